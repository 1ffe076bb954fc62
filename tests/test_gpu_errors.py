"""GPU tests of the two error paths of the decode kernel, both driven from the host: (1) a bounded wait
that runs out (the loaders are told to withhold one tile's hand-over, the wait limit is set to a fraction
of a millisecond): the kernel must return, name the wait in `status`, and leave the device usable;
(2) indices, lengths and block-table values that point outside the cache: such entries are left out of
the softmax, never read, and reported with status code 7.  Nothing here faults or hangs the GPU."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import dsv4_oracle as orc  # noqa: E402
from tests import gpu_util as gu  # noqa: E402


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dsv4_attn_b200 as d
    return d


@pytest.mark.parametrize("with_plan", [False, True])
def test_bounded_wait_runs_out_and_kernel_returns(lib, with_plan):
    case = orc.make_hca_case(seed=61, B=2, s_q=1, H=128, kv_len=[300, 200], win_len=[128, 64])
    args = gu.hca_to_dev(case)
    plan = lib.plan_hca(2, 1, 128, args["kv_len"], args["win_len"]) if with_plan else None
    st = lib.new_status("cuda")
    # 200 us; one tile of every block is never handed over (with a plan the two short rows are cut over all
    # SMs, a tile or two per block: the first one is withheld)
    lib.LIB.dsv4_debug_set_wait(200_000, 0 if with_plan else 1)
    try:
        lib.hca_dense_decode(status=st, plan=plan, num_splits=None if with_plan else 1, **args)
        torch.cuda.synchronize()                    # returns: no trap, no fault, no hang
    finally:
        lib.LIB.dsv4_debug_set_wait(0, -1)
    code, block, role, tile = st.cpu().tolist()
    assert code in (1, 2, 3, 4, 5, 8), f"expected a wait code, got {code}"
    assert role in (0, 1, 2, 3, 4) and tile >= -1
    # the next launch is an ordinary one
    st.zero_()
    out, lse = lib.hca_dense_decode(status=st, plan=plan, num_splits=None if with_plan else 1, **args)
    torch.cuda.synchronize()
    assert st.cpu().tolist() == [0, 0, 0, 0]
    want_out, want_lse = orc.hca_dense_decode(case.q, case.pool, case.block_table, case.kv_len, case.win, case.win_len, case.sm_scale)
    gu.check_out(gu.out_to_f32(out), want_out, "after a timed-out launch")
    gu.check_lse(lse.cpu().numpy(), want_lse, "after a timed-out launch")


@pytest.mark.parametrize("source", ["csa", "hca", "planes", "packed"])
@pytest.mark.parametrize("tile", [0, 5, 12])
def test_bounded_wait_at_the_start_middle_and_end_of_a_row(lib, source, tile):
    """The first, a middle and the last tile of rows of 13 withheld: copies and MMAs are on their way, or the fetch warps have
    already finished, when the waits run out.  The launch returns and the next one is right."""
    n, W, H = 740, 64, 64
    st = lib.new_status("cuda")
    if source == "csa":
        case = orc.make_csa_case(seed=64, B=2, s_q=1, H=H, n_entries=n + W, topk=n + W)
        d = gu.csa_to_dev(case)
        want = orc.csa_sparse_decode(case.q, case.pool, case.block_table, case.indices, case.sm_scale)
        call = lambda: lib.csa_sparse_decode(status=st, num_splits=1, **d)
    elif source == "hca":
        case = orc.make_hca_case(seed=65, B=2, s_q=1, H=H, kv_len=n, win_len=W)
        d = gu.hca_to_dev(case)
        want = orc.hca_dense_decode(case.q, case.pool, case.block_table, case.kv_len, case.win, case.win_len, case.sm_scale)
        call = lambda: lib.hca_dense_decode(status=st, num_splits=1, **d)
    else:
        case = orc.make_ref_layout_case(seed=66, B=2, H=H, M_cur=n, swa_len=W)
        q, sink = gu.dev(case.Q, torch.bfloat16), gu.dev(case.sink)
        want = orc.hca_decode_ref_layout(case.Q, case.Kc, case.Kc_s, case.Kc_rope, case.Kswa, case.Kswa_s, case.Kswa_rope, case.sink, case.sm_scale)
        if source == "planes":
            planes = [gu.dev(case.Kc), gu.dev(case.Kc_s), gu.dev(case.Kc_rope, torch.bfloat16), gu.dev(case.Kswa), gu.dev(case.Kswa_s),
                      gu.dev(case.Kswa_rope, torch.bfloat16)]
            # (no room for partials: one split)
            call = lambda: (lib.LIB.hca_decode_fwd(*(t.data_ptr() for t in (q, *planes, sink, out)), None, None, case.sm_scale, 2, H, 448, 64, n, W,
                                                        torch.cuda.current_stream().cuda_stream), out)[1:] + (None,)
            out = torch.empty(2, H, 512, dtype=torch.bfloat16, device="cuda")
        else:
            rng = np.random.default_rng(7)
            kv, bt = orc.pack_ref_pages(case.Kc, case.Kc_s, case.Kc_rope, 64, rng)
            sw, sbt = orc.pack_ref_pages(case.Kswa, case.Kswa_s, case.Kswa_rope, 64, rng)
            full = lambda v: torch.full((2,), v, dtype=torch.int32, device="cuda")
            t = [gu.dev(kv), gu.dev(bt), full(n), gu.dev(sw), gu.dev(sbt), full(W)]
            call = lambda: lib.hca_packed_decode(q, *t, case.sm_scale, page_size=64, attn_sink=sink, num_splits=1, status=st)
    torch.cuda.synchronize()
    lib.LIB.dsv4_debug_set_wait(200_000, tile)
    try:
        call()
        torch.cuda.synchronize()                    # returns: no trap, no fault, no hang
    finally:
        lib.LIB.dsv4_debug_set_wait(0, -1)
    if source != "planes":
        assert st.cpu().tolist()[0] in (1, 2, 3, 4, 5, 6, 8, 9)
    st.zero_()
    out, lse = call()
    torch.cuda.synchronize()
    assert st.cpu().tolist() == [0, 0, 0, 0]
    gu.check_out(gu.out_to_f32(out), want[0], f"{source} after a timed-out launch")
    if lse is not None:
        gu.check_lse(lse.cpu().numpy(), want[1], f"{source} after a timed-out launch")


def test_csa_out_of_range_indices_and_pages_are_left_out(lib):
    case = orc.make_csa_case(seed=62, B=2, s_q=1, H=64, n_entries=[400, 400], topk=256)
    max_pages = case.block_table.shape[1]
    idx = case.indices.copy()
    idx[0, 0, 5] = max_pages * 64 + 3          # beyond the block table
    idx[0, 0, 9] = 2_000_000_000               # far beyond
    bt = case.block_table.copy()
    bad_page_slot = int(idx[1, 0, 0]) >> 6
    bt[1, bad_page_slot] = case.pool.shape[0] + 7       # a table value outside the pool
    # what remains: the same lists with those entries padded out
    ref_idx = idx.copy()
    ref_idx[0, 0, 5] = -1;  ref_idx[0, 0, 9] = -1
    ref_idx[1, 0][(ref_idx[1, 0] >> 6) == bad_page_slot] = -1
    want_out, want_lse = orc.csa_sparse_decode(case.q, case.pool, case.block_table, ref_idx, case.sm_scale)
    for impl in ("mma", "simt"):
        st = lib.new_status("cuda")
        out, lse = lib.csa_sparse_decode(gu.dev(case.q, torch.bfloat16), gu.dev(case.pool), gu.dev(bt), gu.dev(idx), case.sm_scale,
                                         num_splits=1, status=st, impl=impl)
        torch.cuda.synchronize()
        if impl == "mma":
            assert st.cpu().tolist()[0] == 7
        gu.check_out(gu.out_to_f32(out), want_out, f"bad indices {impl}")
        gu.check_lse(lse.cpu().numpy(), want_lse, f"bad indices {impl}")


def test_hca_lengths_beyond_the_cache_are_left_out(lib):
    case = orc.make_hca_case(seed=63, B=2, s_q=1, H=64, kv_len=[200, 100], win_len=[50, 128])
    max_pages = case.block_table.shape[1]
    kv = case.kv_len.copy();  win = case.win_len.copy()
    kv[0, 0] = max_pages * 64 + 100            # claims more compressed entries than the block table holds
    win[1, 0] = 128 + 40                       # claims more window rows than the window buffer holds
    args = gu.hca_to_dev(case)
    args["kv_len"] = gu.dev(kv);  args["win_len"] = gu.dev(win)
    st = lib.new_status("cuda")
    out, lse = lib.hca_dense_decode(status=st, num_splits=1, **args)
    torch.cuda.synchronize()
    assert st.cpu().tolist()[0] == 7
    got = gu.out_to_f32(out)
    assert np.isfinite(got).all() and np.isfinite(lse.cpu().numpy()).all()
    # request 1: everything readable was attended to - the real 100 + 128 rows
    ref_win = case.win_len.copy()
    want_out, want_lse = orc.hca_dense_decode(case.q[1:], case.pool, case.block_table[1:], case.kv_len[1:], case.win[1:], ref_win[1:],
                                              case.sm_scale)
    gu.check_out(got[1:], want_out, "window length beyond the buffer")
    gu.check_lse(lse.cpu().numpy()[1:], want_lse, "window length beyond the buffer")
