"""Kernel-level parity on the GPU: the batched complex GEMM against a torch
complex128 matmul, the batched inverse against NumPy/LAPACK, Sancho-Rubio
against the oracle.  Tolerances: relative Frobenius error 1e-12 for a single
GEMM, 1e-10 for inverses of well-conditioned blocks."""


import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from oracle import rgf_oracle as orc
from quatrex_b200 import _lib
from quatrex_b200.obc import SanchoRubio, contact_self_energies
from quatrex_b200.workloads import make_device

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a = a.cpu().numpy() if isinstance(a, torch.Tensor) else a
    b = b.cpu().numpy() if isinstance(b, torch.Tensor) else b
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def _crand(g, *shape):
    return torch.complex(torch.randn(*shape, generator=g, dtype=torch.float64),
                         torch.randn(*shape, generator=g, dtype=torch.float64)).cuda()


def _zgemm(m, n, k, batch, alpha, a, op_a, b, op_b, beta, c, d, sa=None, sb=None):
    lib = _lib.load()
    ctx = _lib.context(0)
    lda = a.shape[-1]
    ldb = b.shape[-1]
    sa = a.shape[-1] * a.shape[-2] if sa is None else sa
    sb = b.shape[-1] * b.shape[-2] if sb is None else sb
    st = lib.qtx_zgemm(ctx, m, n, k, batch, alpha.real, alpha.imag, a.data_ptr(), lda, sa, op_a, b.data_ptr(), ldb,
                       sb, op_b, beta.real, beta.imag, c.data_ptr() if c is not None else None, n, m * n,
                       d.data_ptr(), n, m * n, 0, torch.cuda.current_stream().cuda_stream)
    _lib.check(st, ctx, "zgemm")
    torch.cuda.synchronize()


@pytest.mark.parametrize("m,n,k", [(64, 64, 64), (1, 1, 1), (2, 4, 2), (37, 53, 71), (128, 96, 200), (256, 256, 256)])
@pytest.mark.parametrize("op_a", [0, 1])
@pytest.mark.parametrize("op_b", [0, 1])
def test_zgemm_matches_torch(m, n, k, op_a, op_b):
    g = torch.Generator().manual_seed(m * 1000 + n * 10 + k)
    batch = 3
    a = _crand(g, batch, *((m, k) if op_a == 0 else (k, m)))
    b = _crand(g, batch, *((k, n) if op_b == 0 else (n, k)))
    c = _crand(g, batch, m, n)
    d = torch.empty(batch, m, n, dtype=torch.complex128, device="cuda")
    alpha, beta = complex(0.7, -0.2), complex(-1.0, 0.5)
    _zgemm(m, n, k, batch, alpha, a, op_a, b, op_b, beta, c, d)
    aa = a if op_a == 0 else a.conj().transpose(-1, -2)
    bb = b if op_b == 0 else b.conj().transpose(-1, -2)
    ref = alpha * (aa @ bb) + beta * c
    assert _rel(d, ref) < 1e-13


@pytest.mark.parametrize("op_a,op_b", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("n,batch", [(63, 296), (64, 296), (97, 148), (128, 148), (161, 296)])
def test_zgemm_result_does_not_depend_on_the_tile(n, batch, op_a, op_b):
    """A single product takes the 32 x 32 tile, a batch that fills whole waves
    of the GPU the 64 x 64 one; both run the same sequence per element, so the
    results agree bit for bit (edges of both tiles, one row or column past
    them included)."""
    g = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.randn(batch, n, n, dtype=torch.complex128, device="cuda", generator=g) for _ in range(2))
    big = torch.empty_like(a)
    _zgemm(n, n, n, batch, 1.0 + 0.5j, a, op_a, b, op_b, 0j, None, big)
    one = torch.empty_like(a[:1])
    for e in (0, batch - 1):
        _zgemm(n, n, n, 1, 1.0 + 0.5j, a[e:e + 1].contiguous(), op_a, b[e:e + 1].contiguous(), op_b, 0j, None, one)
        assert torch.equal(one[0], big[e])
    want = (1.0 + 0.5j) * (a.mH if op_a else a) @ (b.mH if op_b else b)
    # two chains of 2 n products each, rounded once a step
    assert _rel(big, want.cpu().numpy()) < 4 * n * 2.0**-53


def test_zgemm_broadcast_operand():
    g = torch.Generator().manual_seed(5)
    a = _crand(g, 1, 48, 48)
    b = _crand(g, 4, 48, 48)
    d = torch.empty(4, 48, 48, dtype=torch.complex128, device="cuda")
    _zgemm(48, 48, 48, 4, 1.0 + 0j, a, 0, b, 0, 0j, None, d, sa=0)
    assert _rel(d, a @ b) < 1e-13


@pytest.mark.parametrize("n", [1, 2, 3, 4, 8, 16, 24, 31, 48, 64, 96, 100, 128, 129, 161, 200, 250, 255, 256, 257, 300,
                               512])
def test_inverse_matches_lapack(n):
    rng = np.random.default_rng(n)
    batch = 5
    a = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    a += np.sqrt(n) * np.eye(n)  # keep the condition number moderate
    ta = torch.from_numpy(a).cuda()
    x = torch.empty_like(ta)
    lib = _lib.load()
    ctx = _lib.context(0)
    st = lib.qtx_inv(ctx, n, batch, ta.data_ptr(), n * n, x.data_ptr(), n * n, torch.cuda.current_stream().cuda_stream)
    _lib.check(st, ctx, "inv")
    ref = np.linalg.inv(a)
    assert _rel(x, ref) < 1e-10
    # in place
    st = lib.qtx_inv(ctx, n, batch, ta.data_ptr(), n * n, ta.data_ptr(), n * n, torch.cuda.current_stream().cuda_stream)
    _lib.check(st, ctx, "inv")
    assert _rel(ta, ref) < 1e-10

@pytest.mark.parametrize("n,batch", [(32, 3), (33, 3), (63, 2), (65, 3), (160, 2), (192, 160), (256, 20), (384, 2),
                                     (385, 2), (511, 2)])
@pytest.mark.parametrize("in_place", [False, True])
def test_inverse_register_and_panel_shapes(n, batch, in_place):
    """Edges of the register kernels (32 and 64 rows) and of the panel kernels
    (128, 256 and 384 rows; 32- and 16-column panels with a remainder), with
    few and with many matrices per launch."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    a[:, np.arange(n), np.arange(n)] += np.sqrt(n)
    ta = torch.from_numpy(a[:, np.roll(np.arange(n), n // 3)].copy()).cuda()
    want = torch.linalg.inv(ta)
    x = ta.clone() if in_place else torch.empty_like(ta)
    lib = _lib.load()
    ctx = _lib.context(0)
    src = x if in_place else ta
    _lib.check(lib.qtx_inv(ctx, n, batch, src.data_ptr(), n * n, x.data_ptr(), n * n, 0), ctx, "inv")
    torch.cuda.synchronize()
    # elimination with partial pivoting: error of order n u times the condition number
    cond = float(torch.linalg.cond(ta).max())
    assert _rel(x, want.cpu().numpy()) < 4 * n * 2.0**-53 * cond


@pytest.mark.parametrize("n", [16, 32, 64, 128])
def test_inverse_of_tied_pivots(n):
    """Hadamard matrices: in the first steps every candidate of a column has
    the same |Re| + |Im| (ties over all the bits the search compares), and
    rows scaled by 1 + k 2^-50 tie in the high word only; H^-1 = H^T / n."""
    h = np.ones((1, 1))
    while h.shape[0] < n:
        h = np.block([[h, h], [h, -h]])
    scale = 1.0 + np.arange(n) * 2.0**-50
    a = np.stack([h, scale[:, None] * h]).astype(np.complex128)
    ta = torch.from_numpy(a).cuda()
    x = torch.empty_like(ta)
    lib = _lib.load()
    ctx = _lib.context(0)
    _lib.check(lib.qtx_inv(ctx, n, 2, ta.data_ptr(), n * n, x.data_ptr(), n * n, 0), ctx, "inv")
    torch.cuda.synchronize()
    want = np.stack([h.T / n, h.T / (n * scale[None, :])])
    # orthogonal up to scale (condition number 1), growth factor n
    assert _rel(x, want) < 4 * n * 2.0**-53


def _one_launch(check):
    """Run `check` (t is this module) in a process whose inverses take no scratch
    (QTX_INV_SPLIT_BELOW=0, read once per process)."""
    env = dict(os.environ, QTX_INV_SPLIT_BELOW="0")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = f"import sys; sys.path[:0] = ['.', 'tests']; import test_gpu_kernels as t; {check}"
    subprocess.run([sys.executable, "-c", code], check=True, env=env, cwd=root, timeout=300)


def _check_one_launch():
    lib, ctx = _lib.load(), _lib.context(0)
    for n, batch in ((65, 3), (100, 3), (128, 3), (129, 3), (256, 150), (257, 2), (512, 2)):
        rng = np.random.default_rng(n)
        a = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
        a[:, np.arange(n), np.arange(n)] += np.sqrt(n)
        t = torch.from_numpy(a[:, np.roll(np.arange(n), n // 3)].copy()).cuda()
        x = torch.empty_like(t)
        _lib.check(lib.qtx_inv(ctx, n, batch, t.data_ptr(), n * n, x.data_ptr(), n * n, 0), ctx, "inv")
        want = torch.linalg.inv(t)
        err = float(torch.linalg.vector_norm(x - want) / torch.linalg.vector_norm(want))
        assert err < 4 * n * 2.0**-53 * float(torch.linalg.cond(t).max()), (n, err)


def test_one_launch_inverse_without_scratch():
    """The form that takes no scratch: every shape of its panel elimination."""
    _one_launch("t._check_one_launch()")


def _check_non_finite(n):
    """A matrix with a column of NaN (every bit set, the sign included), one
    with a single NaN and one with an infinity between finite ones: the finite
    ones come out as without them, nothing outside the output is written, and
    the NaN ones do not come out finite.  A pivot search that lost a NaN row
    named no row, or a used one, and the permutation then pointed anywhere."""
    lib, ctx = _lib.load(), _lib.context(0)
    rng = np.random.default_rng(n)
    a = rng.standard_normal((5, n, n)) + 1j * rng.standard_normal((5, n, n))
    a[:, np.arange(n), np.arange(n)] += np.sqrt(n)
    a.view(np.uint64)[1, :, 2 * (n // 2):2 * (n // 2) + 2] = 0xFFFFFFFFFFFFFFFF
    a[2, n // 3, 0] = complex(np.nan, 1.0)
    a[3, n - 1, n // 2] = complex(0.0, -np.inf)
    buf = torch.full((7, n, n), 7.0, dtype=torch.complex128, device="cuda")
    x = buf[1:6]
    ta = torch.from_numpy(a).cuda()
    st = lib.qtx_inv(ctx, n, 5, ta.data_ptr(), n * n, x.data_ptr(), n * n, 0)
    assert st in (_lib.QTX_OK, _lib.QTX_E_SINGULAR)
    good = ta[[0, 4]].contiguous()
    want = torch.empty_like(good)
    _lib.check(lib.qtx_inv(ctx, n, 2, good.data_ptr(), n * n, want.data_ptr(), n * n, 0), ctx, "inv")
    assert torch.equal(x[[0, 4]], want)
    assert bool((buf[[0, 6]] == 7.0).all())
    for e in (1, 2):  # (an infinity may have a finite inverse: 1 / inf = 0)
        assert not bool(torch.isfinite(torch.view_as_real(x[e])).all())


@pytest.mark.parametrize("n", [1, 5, 32, 33, 64, 65, 97, 128, 129, 256, 257, 384, 385, 512])
def test_inverse_with_nan_and_inf(n):
    _check_non_finite(n)


def test_one_launch_inverse_with_nan_and_inf():
    _one_launch("[t._check_non_finite(n) for n in (65, 97, 128, 129, 256, 257, 512)]")


@pytest.mark.parametrize("n", [96, 200, 256, 300])
def test_inverse_does_not_depend_on_the_batch(n):
    """The first entries of a 130-matrix batch equal a 5-matrix call bit for
    bit, and both match LAPACK."""
    rng = np.random.default_rng(n + 7)
    a = rng.standard_normal((130, n, n)) + 1j * rng.standard_normal((130, n, n))
    a[:, np.arange(n), np.arange(n)] += np.sqrt(n)
    ta = torch.from_numpy(a).cuda()
    big, small = torch.empty_like(ta), torch.empty_like(ta[:5])
    lib = _lib.load()
    ctx = _lib.context(0)
    _lib.check(lib.qtx_inv(ctx, n, 130, ta.data_ptr(), n * n, big.data_ptr(), n * n, 0), ctx, "inv")
    _lib.check(lib.qtx_inv(ctx, n, 5, ta.data_ptr(), n * n, small.data_ptr(), n * n, 0), ctx, "inv")
    assert torch.equal(small, big[:5])
    assert _rel(small, np.linalg.inv(a[:5])) < 1e-10


_FORM_SIZES = (65, 96, 97, 128, 129, 200, 256, 257, 384, 512)


def _form_inputs(n):
    """A random matrix, one of signs (in the first steps every candidate of a
    column ties) and one with a zero column, i.e. an exact zero pivot."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n))
    a[1] = rng.choice([-1.0, 1.0], (n, n))
    a[2, :, n // 2] = 0
    return torch.from_numpy(a).cuda()


def _form_outputs():
    """Per size: the inverse, the status and the message of the call."""
    lib, ctx = _lib.load(), _lib.context(0)
    out = {}
    for n in _FORM_SIZES:
        t = _form_inputs(n)
        x = torch.empty_like(t)
        st = lib.qtx_inv(ctx, n, 3, t.data_ptr(), n * n, x.data_ptr(), n * n, 0)
        out[n] = (x.cpu(), st, lib.qtx_last_error(ctx).decode())
    return out


def test_one_launch_and_panel_inverses_agree(tmp_path):
    """The form without scratch against the panels: the same zero pivot is
    named, and where the panels are equally wide and eliminated by the same
    steps (97 to 256 rows) the results agree bit for bit.  Elsewhere (16-column
    panels up to 96 rows, the pivot row scaled by its own formula above 256)
    each form has an error of order n u times the condition number."""
    path = str(tmp_path / "one.pt")
    _one_launch(f"t.torch.save(t._form_outputs(), {path!r})")
    one, panels = torch.load(path), _form_outputs()
    for n in _FORM_SIZES:
        (x, st, msg), (y, st_p, msg_p) = one[n], panels[n]
        assert st == st_p == _lib.QTX_E_SINGULAR and msg == msg_p and f"pivot {n // 2 + 1})" in msg
        cond = torch.linalg.cond(_form_inputs(n)[:2]).cpu()
        for e in range(2):
            if 96 < n <= 256:
                assert torch.equal(x[e], y[e]), (n, e)
            else:
                err = torch.linalg.vector_norm(x[e] - y[e]) / torch.linalg.vector_norm(y[e])
                assert err < 2 * 4 * n * 2.0**-53 * cond[e], (n, e)


@pytest.mark.parametrize("n,panels", [(32, 0), (64, 0), (65, 3), (100, 4), (256, 8), (300, 19), (512, 32)])
def test_launch_count_of_an_inverse(n, panels):
    """Every launch counts: one for a register inverse, two per panel and the
    final unscrambling for the others, and the two of the status word."""
    a = torch.eye(n, dtype=torch.complex128, device="cuda").repeat(2, 1, 1)
    x = torch.empty_like(a)
    lib, ctx = _lib.load(), _lib.context(0)
    before = lib.qtx_launch_count(ctx)
    _lib.check(lib.qtx_inv(ctx, n, 2, a.data_ptr(), n * n, x.data_ptr(), n * n, 0), ctx, "inv")
    assert lib.qtx_launch_count(ctx) - before == 2 + (2 * panels + 1 if panels else 1)


@pytest.mark.parametrize("n", [200, 256])
@pytest.mark.parametrize("batch", [5, 130])
def test_inverse_output_sixteen_bytes_off(n, batch):
    """The panel update reads and writes adjacent column pairs in one 32-byte
    access only when the matrices start 32-byte aligned; an output batch that
    starts one complex element (16 bytes) into its buffer takes the 16-byte
    accesses and returns the same bits as an aligned one."""
    rng = np.random.default_rng(n + batch)
    a = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    a[:, np.arange(n), np.arange(n)] += np.sqrt(n)
    ta = torch.from_numpy(a).cuda()
    aligned = torch.empty_like(ta)
    buf = torch.empty(batch * n * n + 1, dtype=torch.complex128, device="cuda")
    off = buf[1:].view(batch, n, n)
    assert off.data_ptr() % 32 == 16
    lib = _lib.load()
    ctx = _lib.context(0)
    _lib.check(lib.qtx_inv(ctx, n, batch, ta.data_ptr(), n * n, aligned.data_ptr(), n * n, 0), ctx, "inv")
    _lib.check(lib.qtx_inv(ctx, n, batch, ta.data_ptr(), n * n, off.data_ptr(), n * n, 0), ctx, "inv")
    assert torch.equal(off, aligned)
    assert _rel(aligned[:3], np.linalg.inv(a[:3])) < 1e-10


def test_inverse_needs_pivoting():
    # zero leading diagonal entries: fails without row interchanges
    a = np.array([[0, 1, 2], [1, 0, 3], [4, 5, 0]], dtype=np.complex128)[None]
    ta = torch.from_numpy(a).cuda()
    x = torch.empty_like(ta)
    lib = _lib.load()
    ctx = _lib.context(0)
    _lib.check(lib.qtx_inv(ctx, 3, 1, ta.data_ptr(), 9, x.data_ptr(), 9, 0), ctx, "inv")
    assert _rel(x, np.linalg.inv(a)) < 1e-14


@pytest.mark.parametrize("n", [64, 200, 256])
def test_inverse_pivoting_large_blocks(n):
    """Row-permuted, well-conditioned blocks with a zero diagonal: every
    column needs a row interchange, across panels."""
    rng = np.random.default_rng(n + 1)
    batch = 6
    base = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    base += 2 * np.sqrt(n) * np.eye(n)
    perm = np.roll(np.arange(n), n // 3 + 1)
    a = np.ascontiguousarray(base[:, perm, :])
    assert np.all(np.abs(np.diagonal(a, axis1=1, axis2=2)) < 2 * np.sqrt(n) - 1e-9)
    ta = torch.from_numpy(a).cuda()
    x = torch.empty_like(ta)
    lib = _lib.load()
    ctx = _lib.context(0)
    _lib.check(lib.qtx_inv(ctx, n, batch, ta.data_ptr(), n * n, x.data_ptr(), n * n, 0), ctx, "inv")
    assert _rel(x, np.linalg.inv(a)) < 1e-12


@pytest.mark.parametrize("n", [4, 200])
def test_inverse_singular_block_flags_its_energy(n):
    """A block with a zero column in the middle of a batch returns
    QTX_E_SINGULAR; the other blocks are still inverted correctly."""
    rng = np.random.default_rng(7)
    a = rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n)) + np.sqrt(n) * np.eye(n)
    a[1, :, n // 2] = 0
    ta = torch.from_numpy(a).cuda()
    x = torch.empty_like(ta)
    lib = _lib.load()
    ctx = _lib.context(0)
    st = lib.qtx_inv(ctx, n, 3, ta.data_ptr(), n * n, x.data_ptr(), n * n, 0)
    assert st == _lib.QTX_E_SINGULAR
    torch.cuda.synchronize()
    xc = x.cpu().numpy()
    for e in (0, 2):
        assert _rel(xc[e], np.linalg.inv(a[e])) < 1e-10


def test_inverse_singular_block_raises():
    a = np.zeros((2, 4, 4), dtype=np.complex128)
    a[0] = np.eye(4)
    ta = torch.from_numpy(a).cuda()
    x = torch.empty_like(ta)
    lib = _lib.load()
    ctx = _lib.context(0)
    st = lib.qtx_inv(ctx, 4, 2, ta.data_ptr(), 16, x.data_ptr(), 16, 0)
    assert st == _lib.QTX_E_SINGULAR
    with pytest.raises(np.linalg.LinAlgError):
        _lib.check(st, ctx, "inv")
    # the context stays usable
    st = lib.qtx_inv(ctx, 4, 1, ta.data_ptr(), 16, x.data_ptr(), 16, 0)
    assert st == _lib.QTX_OK


def test_sancho_rubio_matches_oracle():
    dev = make_device(num_blocks=3, block_size=24, num_energies=9, seed=11)
    d, u, lo = dev.system_blocks()
    x_ref, it_ref = orc.sancho_rubio(d[0], u[0], lo[0], 200, 1e-12)
    sr = SanchoRubio(max_iterations=200, convergence_tol=1e-12)
    x = sr(d[0], u[0], lo[0], "left")
    assert _rel(x, x_ref) < 1e-10
    assert sr.last_iterations.max() == it_ref
    # fixed point of the upstream test criterion
    assert _rel(x, np.linalg.inv(d[0] - lo[0] @ x @ u[0])) < 1e-6
    # broadcast couplings (2-D a_ij / a_ji)
    x2 = sr(d[0], u[0][0], lo[0][0], "left")
    assert _rel(x2, x_ref) < 1e-10


def test_sancho_rubio_not_converged_warns():
    dev = make_device(num_blocks=2, block_size=8, num_energies=3, seed=3)
    d, u, lo = dev.system_blocks()
    with pytest.warns(RuntimeWarning):
        SanchoRubio(max_iterations=1, convergence_tol=1e-12)(d[0], u[0], lo[0], "left")


def test_sancho_rubio_singular_decimation_block():
    """An exactly singular decimation block is reported (QTX_E_SINGULAR ->
    LinAlgError), not passed on as silent NaN; the context stays usable."""
    n, ne = 8, 2
    a_ii = torch.zeros(ne, n, n, dtype=torch.complex128, device="cuda")
    a_ij = torch.eye(n, dtype=torch.complex128, device="cuda").repeat(ne, 1, 1)
    x = torch.empty_like(a_ii)
    lib = _lib.load()
    ctx = _lib.context(0)
    st = lib.qtx_sancho_rubio(ctx, n, ne, a_ii.data_ptr(), n * n, a_ij.data_ptr(), n * n, a_ij.data_ptr(), n * n,
                              1e-12, 3, x.data_ptr(), None, 0)
    assert st == _lib.QTX_E_SINGULAR
    with pytest.raises(np.linalg.LinAlgError):
        SanchoRubio(max_iterations=3, convergence_tol=1e-12)(a_ii, a_ij, a_ij, "left")
    dev = make_device(num_blocks=2, block_size=8, num_energies=2, seed=3)
    d, u, lo = dev.system_blocks()
    x_ok = SanchoRubio(max_iterations=200, convergence_tol=1e-12)(d[0], u[0], lo[0], "left")
    x_ref, _ = orc.sancho_rubio(d[0], u[0], lo[0], 200, 1e-12)
    assert _rel(x_ok, x_ref) < 1e-10


def test_contact_self_energies_match_oracle():
    dev = make_device(num_blocks=3, block_size=16, num_energies=5, seed=2)
    d, u, lo = dev.system_blocks()
    ref = orc.obc_self_energies(d, u, lo, dev.energies, dev.mu_left, dev.mu_right, dev.kt)
    f = orc.fermi_dirac(dev.energies - dev.mu_left, dev.kt)
    sr, sl, sg = contact_self_energies(ref["surface"][0], lo[0], u[0], f)
    assert _rel(sr, ref["retarded"][0]) < 1e-12
    assert _rel(sl, ref["lesser"][0]) < 1e-12
    assert _rel(sg, ref["greater"][0]) < 1e-12


@pytest.mark.parametrize("sizes", [[3, 5, 4, 6], [8] * 12, [1, 2, 1, 3, 2]])
def test_block_sort_index_device_matches_host(sizes):
    """DSDBCOO construction on the device: the same stable block-sorting
    permutation as the host rule (and upstream's compute_block_sort_index),
    per-block counts, and an index outside the matrix refused."""
    from quatrex_b200.datastructures import block_sort_index, block_sort_index_device

    rng = np.random.default_rng(len(sizes))
    n = int(np.sum(sizes))
    # random pattern with entries in every block pair (not only the band), shuffled order
    m = (rng.random((n, n)) < 0.3).astype(np.complex128)
    r, c = np.nonzero(m)
    perm = rng.permutation(len(r))
    r, c = r[perm], c[perm]
    got, counts = block_sort_index_device(r, c, sizes)
    want = block_sort_index(r, c, sizes)
    assert np.array_equal(got.cpu().numpy(), want)
    offs = np.concatenate(([0], np.cumsum(sizes)))
    br = np.searchsorted(offs, r, side="right") - 1
    bc = np.searchsorted(offs, c, side="right") - 1
    ref = np.zeros((len(sizes), len(sizes)), dtype=np.int64)
    np.add.at(ref, (br, bc), 1)
    assert np.array_equal(counts, ref)
    with pytest.raises(ValueError):
        block_sort_index_device(np.array([0, n]), np.array([0, 0]), sizes)


@pytest.mark.parametrize("with_overlap", [False, True])
def test_assemble_system_matches_formula(with_overlap):
    """A(E) = (E + i eta) S - diag(V) - Sigma(E) - H on the data rows."""
    from scipy import sparse

    from quatrex_b200.datastructures import DSDBCOO, assemble_system

    rng = np.random.default_rng(3)
    sizes = np.array([3, 4, 3])
    n = int(sizes.sum())
    band = np.abs(np.subtract.outer(np.arange(n), np.arange(n))) <= 3
    hm = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * band
    hm = hm + hm.conj().T + np.eye(n)
    H = DSDBCOO.from_sparray(sparse.coo_matrix(hm), sizes, (1,))
    S = None
    sm = np.eye(n)
    if with_overlap:
        sm = np.eye(n) + 0.1 * band * rng.standard_normal((n, n))
        S = DSDBCOO(np.asarray(sm[H.rows, H.cols], dtype=np.complex128)[None], H.rows, H.cols, sizes, (1,))
    e = np.array([-0.5, 0.1, 0.7])
    v = rng.standard_normal(n)
    sig = (rng.standard_normal((3, H.rows.size)) + 1j * rng.standard_normal((3, H.rows.size)))
    SG = DSDBCOO(sig, H.rows, H.cols, sizes, (3,))
    A = assemble_system(e, 1e-3, H, overlap=S, potential=v, sigma=SG)
    got = A.data.cpu().numpy()
    for k in range(3):
        full = (e[k] + 1e-3j) * sm - np.diag(v) - hm
        want = full[H.rows, H.cols] - sig[k]
        assert np.allclose(got[k], want, rtol=0, atol=1e-13)


@pytest.mark.skipif(not torch.cuda.is_available() or torch.cuda.device_count() < 2,
                    reason="needs two visible CUDA devices")
def test_two_devices_in_one_process():
    """The large shared-memory opt-in of the GEMM and inverse kernels is a
    per-device attribute: a solve on a second device after the first has used
    the library must still launch (and agree with the oracle)."""
    dev = make_device(num_blocks=3, block_size=64, num_energies=4, seed=7)
    d, u, lo = dev.system_blocks()
    x_ref, _ = orc.sancho_rubio(d[0], u[0], lo[0], 200, 1e-12)
    for k in (0, 1):
        with torch.cuda.device(k):
            x = SanchoRubio(max_iterations=200, convergence_tol=1e-12)(d[0], u[0], lo[0], "left")
            assert _rel(x, x_ref) < 1e-10
