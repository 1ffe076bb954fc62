"""Row lengths at the edges of the decode kernel's tiles (64 entries, dealt four at a time to the two blocks of a pair; 16 rows
per reduction step) against the CPU oracle: every source, the cache / window border inside a group of four, and
cache records that take no part filled with NaN bytes, which must not reach the result.  Run with `-m gpu` on a B200."""
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


@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 31, 32, 33, 36, 63, 64, 65, 97, 128, 129, 200])
def test_row_lengths_at_tile_edges(lib, n):
    H = 128 if n % 2 else 16
    st = lib.new_status("cuda")

    def check(got, want, what):
        torch.cuda.synchronize()
        assert st.cpu().tolist() == [0, 0, 0, 0], what
        gu.check_out(gu.out_to_f32(got[0]), want[0], what)
        gu.check_lse(got[1].cpu().numpy(), want[1], what)

    case = orc.make_csa_case(seed=700 + n, B=2, s_q=1, H=H, n_entries=n + 7, topk=n)
    pool = case.pool.copy()
    for b in range(2):
        chosen = set(case.indices[b, 0].tolist())
        for e in range(case.block_table.shape[1] * 64):
            if e not in chosen:
                pool[case.block_table[b, e >> 6], e & 63] = 0x7F
    want = orc.csa_sparse_decode(case.q, pool, case.block_table, case.indices, case.sm_scale)
    d = dict(gu.csa_to_dev(case), kv_pool=gu.dev(pool))
    check(lib.csa_sparse_decode(**d, num_splits=1, status=st), want, f"csa n={n}")
    check(lib.csa_sparse_decode(**d, num_splits=2, status=st), want, f"csa n={n} split")

    win = min(n // 3, 128)
    case = orc.make_hca_case(seed=800 + n, B=2, s_q=1, H=H, kv_len=[n - win, n], win_len=[win, 1], with_sink=True)
    want = orc.hca_dense_decode(case.q, case.pool, case.block_table, case.kv_len, case.win, case.win_len, case.sm_scale, sink=case.sink)
    check(lib.hca_dense_decode(**gu.hca_to_dev(case), num_splits=1, status=st), want, f"hca n={n}")

    case = orc.make_ref_layout_case(seed=900 + n, B=2, H=H, M_cur=n, swa_len=max(win, 1))
    want = orc.hca_decode_ref_layout(case.Q, case.Kc, case.Kc_s, case.Kc_rope, case.Kswa, case.Kswa_s, case.Kswa_rope, case.sink, case.sm_scale)
    got = lib.hca_decode_fwd(gu.dev(case.Q, torch.bfloat16), gu.dev(case.Kc), gu.dev(case.Kc_s), gu.dev(case.Kc_rope, torch.bfloat16), gu.dev(case.Kswa),
                             gu.dev(case.Kswa_s), gu.dev(case.Kswa_rope, torch.bfloat16), gu.dev(case.sink), case.sm_scale, M_cur=n, swa_len=max(win, 1))
    torch.cuda.synchronize()
    gu.check_out(gu.out_to_f32(got), want[0] if isinstance(want, tuple) else want, f"planes n={n}")


class _PagesInOrder:
    """Stands in for the generator that shuffles pages: page numbers follow one another."""
    def __init__(self, seed):
        self.integers = np.random.default_rng(seed).integers

    def permutation(self, n):
        return np.arange(n)


@pytest.mark.parametrize("page", [16, 32, 64])
@pytest.mark.parametrize("m_cur", [0, 1, 62, 66, 131])
def test_packed_pages_fetched_four_tokens_at_a_time(lib, page, m_cur):
    """A group of four rows is fetched as one box only inside a page: window rows that are not aligned to four cross page borders,
    here also into the page that lies next in memory."""
    case = orc.make_ref_layout_case(seed=1000 + m_cur, B=2, H=16, M_cur=140, swa_len=128)
    kv, bt = orc.pack_ref_pages(case.Kc, case.Kc_s, case.Kc_rope, page, _PagesInOrder(1))
    sw, sbt = orc.pack_ref_pages(case.Kswa, case.Kswa_s, case.Kswa_rope, page, _PagesInOrder(2))
    m, w = np.array([m_cur, m_cur + 1], np.int32), np.array([128, 67], np.int32)
    st = lib.new_status("cuda")
    out, lse = lib.hca_packed_decode(gu.dev(case.Q, torch.bfloat16), gu.dev(kv), gu.dev(bt), gu.dev(m), gu.dev(sw), gu.dev(sbt), gu.dev(w),
                                     case.sm_scale, page_size=page, attn_sink=gu.dev(case.sink), num_splits=1, status=st)
    torch.cuda.synchronize()
    assert st.cpu().tolist() == [0, 0, 0, 0]
    want, want_lse = orc.hca_decode_packed_pages(case.Q, kv, bt, m, sw, sbt, w, case.sink, case.sm_scale, page)
    gu.check_out(gu.out_to_f32(out), want, f"page={page} m_cur={m_cur}")
    gu.check_lse(lse.cpu().numpy(), want_lse, f"page={page} m_cur={m_cur}")
