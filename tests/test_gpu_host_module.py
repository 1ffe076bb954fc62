"""The native module behind the operators (csrc/host.cpp).  Run with `-m gpu` on a B200."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dsv4_attn_b200 as d
    return d


def test_other_python_threads_run_during_a_launch(lib):
    """A launch may have to wait for room in the launch queue: it does not hold the interpreter meanwhile.  PyGILState_Check stands in for the
    library's entry points: it returns 1, a launch error, when its caller holds the interpreter."""
    from dsv4_attn_b200 import api
    real = [C.cast(getattr(lib.LIB, name), C.c_void_p).value for name in api.ENTRY_POINTS]
    check = C.cast(C.pythonapi.PyGILState_Check, C.c_void_p).value
    x = torch.zeros(4, 2, 576, dtype=torch.bfloat16, device="cuda")
    pos = torch.zeros(4, dtype=torch.int32, device="cuda")
    pool = torch.zeros(1, 64, 656, dtype=torch.uint8, device="cuda")
    table = torch.zeros(1, 1, dtype=torch.int32, device="cuda")
    idx = torch.zeros(1, 1, 64, dtype=torch.int32, device="cuda")
    plan = lib.plan_csa(1, 1, 16, 64)
    torch.cuda.synchronize()
    api._host.bind(*(a if name.endswith("plan_splits") else check for name, a in zip(api.ENTRY_POINTS, real)))
    try:
        lib.rope_norm(x, pos)
        lib.csa_sparse_decode(torch.zeros(1, 1, 16, 576, dtype=torch.bfloat16, device="cuda"), pool, table, idx, 0.04)
        lib.kv_quantize_insert(torch.zeros(1, 2, 576, dtype=torch.bfloat16, device="cuda"), pool, table, torch.zeros(1, dtype=torch.int32, device="cuda"))
        lib.hca_compress_fwd(torch.zeros(1, 8, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, 8, 64, dtype=torch.bfloat16, device="cuda"),
                             torch.zeros(4, 64, dtype=torch.bfloat16, device="cuda"), 4)
        assert api._host.plan(plan.kind, 1, 1, 16, 64, 0, 0, *plan.lengths, plan.sched) == 0
    finally:
        api._host.bind(*real)
