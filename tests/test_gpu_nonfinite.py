"""Queries that are NaN or infinite spoil their own head rows and nothing else: not the other heads of the request, not the
requests before and after it (with fewer than 128 heads the unused MMA rows of a request hold the queries of the next), not
the waits of the kernel.  Lengths at which one or both halves of a tile are full, so that a thread's 32 logits are all NaN.
Run with `-m gpu` on a B200."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import dsv4_oracle as orc  # noqa: E402
from tests import gpu_util as gu  # noqa: E402

B, BAD = 3, 1


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dsv4_attn_b200 as d
    return d


def decode(lib, source, H, n, route):
    """(q on the device, call(q) -> (out, lse or None), the oracle's out and lse for the unspoilt queries)"""
    st = lib.new_status("cuda")
    splits = 2 if route == "split" else 1
    if source == "csa":
        case = orc.make_csa_case(seed=1100 + n, B=B, s_q=1, H=H, n_entries=n + 9, topk=n)
        case.indices[0, 0, 5] = -1                      # a gap among the first 64 slots: one half of that tile is not full
        want = orc.csa_sparse_decode(case.q, case.pool, case.block_table, case.indices, case.sm_scale)
        d = gu.csa_to_dev(case)
        plan = lib.plan_csa(B, 1, H, n) if route == "plan" else None
        call = lambda q: lib.csa_sparse_decode(**dict(d, q=q), num_splits=None if plan else splits, plan=plan, status=st)
        q = d["q"]
    elif source == "hca":
        case = orc.make_hca_case(seed=1200 + n, B=B, s_q=1, H=H, kv_len=n - 20, win_len=20, with_sink=True)
        want = orc.hca_dense_decode(case.q, case.pool, case.block_table, case.kv_len, case.win, case.win_len, case.sm_scale, sink=case.sink)
        d = gu.hca_to_dev(case)
        plan = lib.plan_hca(B, 1, H, d["kv_len"], d["win_len"]) if route == "plan" else None
        call = lambda q: lib.hca_dense_decode(**dict(d, q=q), num_splits=None if plan else splits, plan=plan, status=st)
        q = d["q"]
    else:
        case = orc.make_ref_layout_case(seed=1300 + n, B=B, H=H, M_cur=n - 20, swa_len=20)
        q, sink = gu.dev(case.Q, torch.bfloat16), gu.dev(case.sink)
        want = orc.hca_decode_ref_layout(case.Q, case.Kc, case.Kc_s, case.Kc_rope, case.Kswa, case.Kswa_s, case.Kswa_rope, case.sink, case.sm_scale)
        if source == "planes":
            planes = [gu.dev(case.Kc), gu.dev(case.Kc_s), gu.dev(case.Kc_rope, torch.bfloat16), gu.dev(case.Kswa), gu.dev(case.Kswa_s),
                      gu.dev(case.Kswa_rope, torch.bfloat16)]
            call = lambda q: (lib.hca_decode_fwd(q, *planes, sink, case.sm_scale, M_cur=n - 20, swa_len=20), None)
        else:
            rng = np.random.default_rng(n)
            kv, bt = orc.pack_ref_pages(case.Kc, case.Kc_s, case.Kc_rope, 64, rng)
            sw, sbt = orc.pack_ref_pages(case.Kswa, case.Kswa_s, case.Kswa_rope, 64, rng)
            t = [gu.dev(kv), gu.dev(bt), torch.full((B,), n - 20, dtype=torch.int32, device="cuda"), gu.dev(sw), gu.dev(sbt),
                 torch.full((B,), 20, dtype=torch.int32, device="cuda")]
            call = lambda q: lib.hca_packed_decode(q, *t, case.sm_scale, page_size=64, attn_sink=sink, num_splits=splits, status=st)
    return q, call, want, st


ROUTES = [("csa", "static"), ("csa", "split"), ("csa", "plan"), ("hca", "static"), ("hca", "split"), ("hca", "plan"), ("planes", "static"),
          ("packed", "static"), ("packed", "split")]


@pytest.mark.parametrize("source,route", ROUTES)
@pytest.mark.parametrize("H", [16, 128])
@pytest.mark.parametrize("n", [62, 128])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_nonfinite_queries_spoil_their_own_rows_only(lib, source, route, H, n, value):
    q, call, (want, want_lse), st = decode(lib, source, H, n, route)
    for heads in ([3], list(range(H))):                 # one head of a request, all of them
        spoilt = q.clone()
        spoilt.view(B, H, -1)[BAD, heads] = value
        out, lse = call(spoilt)
        torch.cuda.synchronize()
        assert st.cpu().tolist() == [0, 0, 0, 0]
        keep = np.ones((B, H), bool)
        keep[BAD, heads] = False
        what = f"{source} {route} H={H} n={n} {value} heads={len(heads)}"
        gu.check_out(gu.out_to_f32(out).reshape(B, H, -1)[keep], want.reshape(B, H, -1)[keep], what)
        if lse is not None:
            gu.check_lse(lse.cpu().numpy().reshape(B, H)[keep], want_lse.reshape(B, H)[keep], what)
        # the spoilt rows say so, in splits and pieces as well (-inf would read as an empty row)
        assert np.isnan(gu.out_to_f32(out).reshape(B, H, -1)[~keep]).all(), what
        assert lse is None or np.isnan(lse.cpu().numpy().reshape(B, H)[~keep]).all(), what
