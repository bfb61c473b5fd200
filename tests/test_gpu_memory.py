"""Device memory that a call takes from the stream-ordered pool: its high-water
mark against what the call is documented to hold."""

import ctypes

import numpy as np
import pytest
import torch
from scipy import sparse

from oracle.rgf_oracle import get_batches
from quatrex_b200 import _lib
from quatrex_b200.datastructures import DSDBCOO
from quatrex_b200.greens_function_solver import RGF
from quatrex_b200.transport import TransportSolver
from quatrex_b200.workloads import make_device

pytestmark = pytest.mark.gpu

CPLX = 16
KEYS = ("density", "transmission", "current_left")
SLACK = 1 << 20  # status words, small tables and the pool's rounding


def _pool():
    cu = ctypes.CDLL("libcuda.so.1")
    dev = ctypes.c_int()
    assert cu.cuDeviceGet(ctypes.byref(dev), torch.cuda.current_device()) == 0
    pool = ctypes.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), dev) == 0
    return cu, pool


def _peak(call):
    """Bytes of the device's default pool in use at the peak of call(), above
    what was in use before."""
    used, high = 7, 8  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, CU_MEMPOOL_ATTR_USED_MEM_HIGH
    cu, pool = _pool()
    torch.cuda.synchronize()
    v = ctypes.c_uint64(0)
    assert cu.cuMemPoolSetAttribute(pool, high, ctypes.byref(v)) == 0  # resets the mark
    before = ctypes.c_uint64()
    assert cu.cuMemPoolGetAttribute(pool, used, ctypes.byref(before)) == 0
    call()
    torch.cuda.synchronize()
    assert cu.cuMemPoolGetAttribute(pool, high, ctypes.byref(v)) == 0
    return v.value - before.value


@pytest.mark.parametrize("n", [64, 256])
def test_sancho_rubio_holds_nine_matrices(n):
    """Nine work matrices per energy, and for n > 64 the inverse's panel scratch."""
    ne = 40
    d, u, lo = make_device(num_blocks=2, block_size=n, num_energies=ne, seed=5).system_blocks()
    a_ii, a_ij, a_ji = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (d[0], u[0], lo[0]))
    x = torch.empty_like(a_ii)
    lib, ctx = _lib.load(), _lib.context(0)

    def call():
        st = lib.qtx_sancho_rubio(ctx, n, ne, a_ii.data_ptr(), n * n, a_ij.data_ptr(), n * n, a_ji.data_ptr(), n * n,
                                  1e-12, 200, x.data_ptr(), None, 0)
        _lib.check(st, ctx, "sancho_rubio")

    panels = n * 32 * CPLX * ne if n > 64 else 0
    assert _peak(call) <= 9 * n * n * CPLX * ne + panels + SLACK


@pytest.mark.parametrize("pattern", [False, True])
@pytest.mark.parametrize("current", [False, True])
def test_selected_solve_holds_twelve_work_matrices(pattern, current):
    """Three block stacks (two more of couplings with the currents), twelve work
    matrices and the inverse's panel scratch, whether the blocks are stored full
    or as patterns."""
    nb, b, ne = 6, 96, 20
    dev = make_device(num_blocks=nb, block_size=b, num_energies=ne, seed=4)
    d, u, lo = dev.system_blocks()
    a = DSDBCOO.from_blocks(d, u, lo, device="cuda")
    if pattern:
        keep = np.random.default_rng(1).random(len(a.rows)) < 0.5
        keep |= a.rows == a.cols
        a = DSDBCOO(a.data[:, torch.from_numpy(keep).cuda()].contiguous(), a.rows[keep], a.cols[keep], a.block_sizes,
                    a.stack_shape)
    out = [DSDBCOO.zeros_like(a) for _ in range(3)]
    solver = RGF(max_batch_size=ne)
    call = lambda: solver.selected_solve(a, a, a, out=out, return_retarded=True, return_current=current)  # noqa: E731
    call()  # pattern tables of the operands
    mats = 3 * nb + 12 + (2 * (nb - 1) if current else 0)
    assert _peak(call) <= (mats * b * b + b * 32) * CPLX * ne + SLACK


def test_leads_in_turn_where_there_is_no_room_for_both():
    """A batch whose leads would decimate together (b = 256, 74 energies) with
    the device filled up to about 1 GB more than the recursion's own work space:
    both leads need 1.4 GB, one 0.7 GB.  The call goes through, with the result
    of a call that has all the memory."""
    nb, b, ne = 2, 256, 74
    dev = make_device(num_blocks=nb, block_size=b, num_energies=ne, seed=6)
    solver = TransportSolver(dev, max_batch_size=ne)
    want = {k: v.clone() for k, v in solver.solve(dev.energies, keys=KEYS).items()}
    out = solver.allocate_outputs(ne, KEYS)
    lib, ctx = _lib.load(), _lib.context(0)
    _lib.check(lib.qtx_ctx_trim(ctx), ctx, "trim")
    torch.cuda.empty_cache()
    sweep = (3 * nb + 20) * b * b * CPLX * ne
    lead = 9 * b * b * CPLX * ne
    free, _ = torch.cuda.mem_get_info()
    ballast = torch.empty(free - sweep - lead - lead // 2, dtype=torch.uint8, device="cuda")
    try:
        got = solver.solve(dev.energies, out)
        for k in KEYS:
            assert torch.equal(got[k], want[k]), k
    finally:
        del ballast
        _lib.check(lib.qtx_ctx_trim(ctx), ctx, "trim")
        torch.cuda.empty_cache()


@pytest.mark.parametrize("b,ne,ne_call", [(64, 148, 148), (128, 74, 74), (256, 74, 74), (256, 149, 74), (300, 9, 9)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_transport_footprint_covers_the_call(b, ne, ne_call, precision):
    """Both leads together, and (149 energies in batches of 75 and 74) a call
    whose last batch decimates together after a larger one in turn."""
    largest = max(get_batches(ne, ne_call)[0])
    dev = make_device(num_blocks=2, block_size=b, num_energies=ne, seed=8)
    solver = TransportSolver(dev, max_batch_size=ne_call, precision=precision)
    out = solver.allocate_outputs(ne, KEYS)
    prec = _lib.QTX_PREC_MIXED if precision == "mixed" else _lib.QTX_PREC_FP64
    lib = _lib.load()
    assert _peak(lambda: solver.solve(dev.energies, out)) <= lib.qtx_transport_footprint(2, b, largest, prec)


def test_server_takes_the_leads_in_turn_to_fit_the_budget():
    """A budget that holds one lead's decimation beside the sweep but not both:
    the request is accepted, runs within the budget and returns the same bits."""
    nb, b, ne = 2, 256, 40
    dev = make_device(num_blocks=nb, block_size=b, num_energies=ne, seed=9)
    solver = TransportSolver(dev, max_batch_size=ne)
    want = solver.solve(dev.energies, keys=KEYS)
    out = solver.allocate_outputs(ne, KEYS)
    e = torch.from_numpy(dev.energies).cuda()
    p = _lib.TransportProblem(
        num_blocks=nb, block_size=b, num_energies=ne, h_diag=solver.h_diag.data_ptr(),
        h_upper=solver.h_upper.data_ptr(), energies=e.data_ptr(), eta=dev.eta, mu_left=dev.mu_left,
        mu_right=dev.mu_right, kt=dev.kt, sr_tol=dev.sr_tol, sr_max_iterations=dev.sr_max_iter, max_batch_size=ne)
    o = _lib.TransportOutputs(**{k: out[k].data_ptr() for k in KEYS})
    lib = _lib.load()
    both = lib.qtx_transport_footprint(nb, b, ne, _lib.QTX_PREC_FP64)
    budget = both - 9 * b * b * CPLX * ne
    cfg = _lib.ServerConfig(device=torch.cuda.current_device(), slots=1, memory_budget=budget, group_max_block_size=0)
    srv = ctypes.c_void_p()
    assert lib.qtx_server_create(ctypes.byref(cfg), ctypes.byref(srv)) == _lib.QTX_OK
    try:
        def call():
            rid, status, lat = ctypes.c_int64(), ctypes.c_int32(-1), ctypes.c_double()
            assert lib.qtx_server_submit(srv, ctypes.byref(p), ctypes.byref(o), _lib.QTX_PREC_FP64, 0,
                                         ctypes.byref(rid)) == _lib.QTX_OK
            assert lib.qtx_server_wait(srv, rid, 60000, ctypes.byref(status), ctypes.byref(lat), None, 0) == 0
            assert status.value == _lib.QTX_OK

        assert _peak(call) <= budget
    finally:
        assert lib.qtx_server_destroy(srv) == 0
    for k in KEYS:
        assert torch.equal(out[k], want[k]), k


def test_host_stack_larger_than_the_device_memory_left():
    """A host stack of blocks stored as patterns (small rows, so the recursion's
    work space decides how many energies fit), with currents, and 2 GB of free
    device memory: the streamed batches fit, and the results are those of a call
    with all the memory."""
    nb, b, ne = 80, 128, 24
    rng = np.random.default_rng(2)
    n = nb * b
    rows = np.concatenate([np.arange(n), np.arange(n - b), np.arange(b, n)])
    cols = np.concatenate([np.arange(n), np.arange(b, n), np.arange(n - b)])
    values = rng.standard_normal(len(rows)) + 1j * rng.standard_normal(len(rows)) + 8.0 * (rows == cols)
    m = DSDBCOO.from_sparray(sparse.coo_matrix((values, (rows, cols)), shape=(n, n)), [b] * nb, (ne,))
    m.data *= rng.uniform(0.5, 1.5, (ne, 1))
    solver = RGF(max_batch_size=ne)
    call = lambda: solver.selected_solve(m, m, m, return_retarded=True, return_current=True)  # noqa: E731
    want = call()
    lib, ctx = _lib.load(), _lib.context(0)
    _lib.check(lib.qtx_ctx_trim(ctx), ctx, "trim")
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    ballast = torch.empty(free - (2 << 30), dtype=torch.uint8, device="cuda")
    try:
        got = call()
    finally:
        del ballast
        _lib.check(lib.qtx_ctx_trim(ctx), ctx, "trim")
        torch.cuda.empty_cache()
    for q in range(3):
        assert np.array_equal(got[q].data, want[q].data), q
    assert np.array_equal(got[3], want[3])
