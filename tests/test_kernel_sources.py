"""Rules that the kernel sources keep and no output shows: checked on the text, without a GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "dsv4_attn_b200" / "csrc"
# launched as an ordinary kernel, after everything before it in the stream
ORDINARY = {"decode_simt_kernel"}


def block_end(text, at):
    """Index behind the brace that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced braces")


def kernels():
    found = {}
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__[^{;]*?(\w+)\((?:const )?[\w ]*Args\b[^{;]*\{", text):
            body = text[m.end() - 1:block_end(text, m.end() - 1)]
            # a lambda runs where it is called, not where it stands
            while (lam := re.search(r"auto \w+ = \[[^\]]*\][^{;]*\{", body)) is not None:
                body = body[:lam.start()] + body[block_end(body, lam.end() - 1):]
            found[m.group(1)] = body
    return found


KERNELS = kernels()


def test_every_kernel_is_found():
    launched = set(re.findall(r"\b(\w+_kernel)\b(?!\.cuh)", (CSRC / "api.cu").read_text()))
    assert launched <= set(KERNELS) and len(KERNELS) >= 10


@pytest.mark.parametrize("name", sorted(set(KERNELS) - ORDINARY))
def test_nothing_is_read_before_the_wait_on_the_previous_kernel(name):
    """Every kernel is launched while the one before it in the stream may still run: it waits, unconditionally, before it reads memory."""
    body = KERNELS[name]
    wait = re.search(r"[;{}]\s*ptx::pdl_wait\(\);", body)
    assert wait is not None, "no unconditional wait"
    early = re.search(r"ptx::(ld|ldg|tma_load|tma_gather|bulk_load)\w*\(|plan_row_lengths\(", body[:wait.start()])
    assert early is None, f"{name} reads before its wait: {body[early.start():early.start() + 60]}"


# What may outlive a call: facts about the device or the process, and the frequencies of the theta last used.
KEPT = {"fn", "known", "done", "done_topk", "done_pair", "per_device", "dummy", "known_theta", "known_freq"}
SWITCHES = {"g_dbg", "g_wait_ns", "g_drop_tile", "g_trace", "t_last_error"}


def test_nothing_is_kept_by_an_address_between_calls():
    """State of the host side is what the list says: no tensor map, workspace or check is remembered for a buffer seen before."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "api.cu").read_text())
    inside = set()
    for m in re.finditer(r"\bstatic (?!constexpr)(?:thread_local )?(?:std::atomic<[^>]+>|\w+) ([^;({]+)(?=[;{])", text):
        inside |= {re.match(r"\w+", part.strip()).group(0) for part in m.group(1).split(",")}
    assert inside == KEPT, inside ^ KEPT
    outside = set(re.findall(r"^(?:std::atomic<[^\n]+>|thread_local [^\n=]*?) ?(\w+)(?:\{| =)", text, flags=re.M))
    assert outside == SWITCHES, outside ^ SWITCHES
