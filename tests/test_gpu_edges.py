"""Sizes and layouts at the edges of the kernels' tiles, slices and dispatch rules,
against the oracle or a 64-bit result."""
import ctypes as C

import numpy as np
import pytest

from tests.gpu_util import from_np_colmajor, rel_fro, to_np_colmajor

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24  # half an ulp of FP32


@pytest.mark.parametrize("n,pad", [(1, 0), (7, 1), (8, 0), (31, 2), (33, 3), (511, 0), (512, 4), (513, 0), (1031, 1)])
def test_generation_rows_and_columns(mxp, orc, torch_cuda, n, pad):
    """8 rows per CTA, 32 columns per warp, 512 per pass; vector and scalar stores."""
    p = mxp.panel_matgen(n, 42, lda=n + pad)
    A = to_np_colmajor(p.A, n, n, n + pad)
    Ao, do, rso, bo = orc.matgen(n, 42)
    assert np.array_equal(A.view(np.uint32), Ao.view(np.uint32))
    for got, want in ((p.d, do), (p.rowsum, rso), (p.rhs, bo)):
        assert np.array_equal(got.cpu().numpy().view(np.uint64), want.view(np.uint64))


@pytest.mark.parametrize("n,pad,shift", [(1, 0, 0), (15, 1, 0), (16, 1, 1), (17, 0, 0), (33, 2, 0), (256, 0, 1),
                                         (512, 0, 0), (513, 2, 1), (1031, 0, 0)])
def test_f64_generation_rows_and_pitches(mxp, orc, torch_cuda, n, pad, shift):
    """8 or 16 rows per CTA by the columns' alignment; nothing past the rows."""
    torch = torch_cuda
    ld = n + pad
    buf = torch.full((n * ld + shift + 2,), -3.0, dtype=torch.float64, device="cuda")
    mxp.matgen_f64(n, 42, A=buf[shift:], lda=ld)
    _, d, _, _ = orc.matgen(n, 42, with_matrix=False)
    got = buf[shift:shift + n * ld].view(n, ld)
    assert np.array_equal(got[:, :n].t().cpu().numpy().view(np.uint64), orc.matgen_f64(n, 42, d).view(np.uint64))
    assert torch.all(got[:, n:] == -3.0) and torch.all(buf[:shift] == -3.0) and torch.all(buf[shift + n * ld:] == -3.0)


def test_generation_of_single_outputs(mxp, orc, torch_cuda):
    """Any output may be skipped (NULL)."""
    torch = torch_cuda
    n = 300
    Ao, do, rso, bo = orc.matgen(n, 9, 1)
    L = mxp.lib()
    out = {k: torch.zeros(n, dtype=torch.float64, device="cuda") for k in ("d", "rowsum", "rhs")}
    A = torch.zeros(n * n, dtype=torch.float32, device="cuda")
    ptr = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    for only in ("A", "d", "rowsum", "rhs"):
        a = {k: (t if k == only else None) for k, t in list(out.items()) + [("A", A)]}
        mxp.check(L.mxp_matgen(n, 9, 1, ptr(a["A"]), n, ptr(a["d"]), ptr(a["rowsum"]), ptr(a["rhs"]), None))
    torch.cuda.synchronize()
    assert np.array_equal(to_np_colmajor(A, n, n, n).view(np.uint32), Ao.view(np.uint32))
    for k, want in (("d", do), ("rowsum", rso), ("rhs", bo)):
        assert np.array_equal(out[k].cpu().numpy().view(np.uint64), want.view(np.uint64))


@pytest.mark.parametrize("n", [1, 255, 256, 257, 5000, 20011])
def test_right_hand_side_alone(mxp, orc, torch_cuda, n):
    """The right-hand side by itself is the one of the whole system."""
    torch = torch_cuda
    rhs = torch.full((n + 1,), -2.0, dtype=torch.float64, device="cuda")
    mxp.check(mxp.lib().mxp_matgen(n, 11, 0, None, n, None, None, rhs.data_ptr(), None))
    _, _, _, want = orc.matgen(n, 11, with_matrix=False)
    assert np.array_equal(rhs[:n].cpu().numpy().view(np.uint64), want.view(np.uint64))
    assert float(rhs[n]) == -2.0


def test_batch_generation_is_the_systems(mxp, orc, torch_cuda):
    sizes = [128, 640, 256, 1152]
    bt = mxp.Batch(sizes, [5, 6, 7, 8])
    bt.matgen()
    torch_cuda.cuda.synchronize()
    for i, n in enumerate(sizes):
        A, d, _, rhs = orc.matgen(n, bt.seeds[i])
        assert np.array_equal(bt.matrix(i).cpu().numpy().view(np.uint32), A.view(np.uint32))
        assert np.array_equal(bt.vec(bt.d, i).cpu().numpy(), d)
        assert np.array_equal(bt.vec(bt.rhs, i).cpu().numpy(), rhs)


@pytest.mark.parametrize("m,n,pad", [(1, 1, 0), (5, 63, 0), (300, 64, 1), (301, 65, 0), (1000, 160, 3), (149 * 4, 512, 0),
                                     (9473, 96, 0), (700, 513, 2), (260, 1100, 0)])
def test_panel_solves_against_64_bits(mxp, orc, torch_cuda, m, n, pad):
    """Slices of 4 .. 64 rows, triangles of one block to several launches.  The
    substitution's error is bounded by ~n eps |X| |T| |T^-1|; the blocks are
    diagonally dominant (|T| |T^-1| < 4), and the terms' errors average out."""
    torch = torch_cuda
    T, _, _, _ = orc.matgen(n, 9)
    if n == 1:
        T[0, 0] = 3.0  # the generator's row sum of a 1 x 1 matrix is empty
    assert orc.lib().orc_getrf_nopiv(n, n, T.ctypes.data, n) == 0
    rng = np.random.default_rng(m + n)
    R = rng.uniform(-0.5, 0.5, (m, n)).astype(np.float32)
    dT = from_np_colmajor(torch, T, ld=n + pad)
    T64 = torch.from_numpy(np.ascontiguousarray(T)).double()
    dR = from_np_colmajor(torch, R, ld=m + pad)
    mxp.trsm_right_upper(m, n, dT, n + pad, dR, m + pad)
    want = torch.linalg.solve_triangular(T64.triu(), torch.from_numpy(R).double(), upper=True, left=False)
    tol = 4 * EPS * max(4.0, np.sqrt(n))
    assert rel_fro(to_np_colmajor(dR, m, n, m + pad), want.numpy()) < tol
    dL = from_np_colmajor(torch, np.ascontiguousarray(R.T), ld=n + pad)
    mxp.trsm_left_lower_unit(n, m, dT, n + pad, dL, n + pad)
    want = torch.linalg.solve_triangular(T64, torch.from_numpy(np.ascontiguousarray(R.T)).double(), upper=False,
                                         unitriangular=True)
    assert rel_fro(to_np_colmajor(dL, n, m, n + pad), want.numpy()) < tol


@pytest.mark.parametrize("m,n,pad", [(9472, 48, 0), (9473, 48, 1), (9473, 49, 0), (18945, 64, 0), (18945, 65, 0),
                                     (28417, 65, 3), (28417, 96, 0), (28417, 97, 0)])
def test_right_solves_of_narrow_triangles(mxp, orc, torch_cuda, m, n, pad):
    """Either side of the line between slices and a thread per row; a triangle of more
    than 64 columns goes there in two steps.  Tolerance as above."""
    test_panel_solves_against_64_bits(mxp, orc, torch_cuda, m, n, pad)


@pytest.mark.parametrize("columns,n,pad", [(32, 16, 1), (33, 16, 0), (32, 17, 0), (9472, 16, 0), (9473, 16, 3),
                                           (9473, 17, 0)])
def test_left_solves_of_narrow_triangles(mxp, orc, torch_cuda, columns, n, pad):
    """The same for the left solve: a warp per column, or slices."""
    test_panel_solves_against_64_bits(mxp, orc, torch_cuda, columns, n, pad)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 65, 96, 127, 130, 191, 321])
@pytest.mark.parametrize("pad", [0, 1])
def test_diagonal_block_edges(mxp, orc, torch_cuda, n, pad):
    """Panels of 16, blocks of 64, strips of 32; 16-byte and scalar addresses."""
    torch = torch_cuda
    A, _, _, _ = orc.matgen(n, 5)
    if n == 1:
        A[0, 0] = 3.0
    dA = from_np_colmajor(torch, A, ld=n + pad)
    XU = torch.full((n * n,), float("nan"), dtype=torch.float32, device="cuda")
    XL = torch.full((n * n,), float("nan"), dtype=torch.float32, device="cuda")
    ws = mxp.Workspace(max(n, 128), n, 0)
    mxp.getrf_nopiv_inv(dA, n, n + pad, XU, XL, n, ws)
    got = to_np_colmajor(dA, n, n, n + pad)
    ref = A.copy(order="F")
    assert orc.lib().orc_getrf_nopiv(n, n, ref.ctypes.data, n) == 0
    assert rel_fro(got, ref) < 1e-6
    LU = got.astype(np.float64)
    U, L = np.triu(LU), np.tril(LU, -1) + np.eye(n)
    xu, xl = (to_np_colmajor(x, n, n, n).astype(np.float64) for x in (XU, XL))
    assert np.array_equal(np.tril(xu, -1), np.zeros((n, n))) and np.array_equal(np.triu(xl, 1), np.zeros((n, n)))
    assert np.abs(xu @ U - np.eye(n)).max() < 1e-5 and np.abs(xl @ L - np.eye(n)).max() < 1e-5


@pytest.mark.parametrize("scale", [2.0 ** 119, 2.0 ** -135])
def test_pivots_outside_the_fast_reciprocal(mxp, orc, torch_cuda, scale):
    """Pivots of 2^126 and above, and subnormal ones (just below 2^-126: their
    reciprocals are still finite), take the slow reciprocal; the factors are
    the oracle's of the same block.  The subnormal block's off-diagonals have
    at most 16 bits, and either side rounds each update to that grid: 2^-10."""
    torch = torch_cuda
    n = 140
    A, _, _, _ = orc.matgen(n, 5)
    A = (A * np.float32(2.0 ** 3) * np.float32(scale)).astype(np.float32, order="F")
    dA = from_np_colmajor(torch, A)
    ws = mxp.Workspace(n, n, 0)
    mxp.getrf_nopiv(dA, n, n, ws)
    got = to_np_colmajor(dA, n, n, n).astype(np.float64)
    ref = A.copy(order="F")
    assert orc.lib().orc_getrf_nopiv(n, n, ref.ctypes.data, n) == 0
    ref = ref.astype(np.float64)
    low = np.tril(np.ones((n, n), bool), -1)
    tol = 1e-6 if scale > 1 else 2.0 ** -10
    assert np.all(np.isfinite(got))
    assert rel_fro(got[low], ref[low]) < tol
    assert rel_fro(got[~low] / scale, ref[~low] / scale) < tol


@pytest.mark.parametrize("n,pad", [(1, 0), (63, 1), (65, 0), (129, 3), (705, 1), (1471, 0)])
def test_chain_solve_ragged(mxp, orc, torch_cuda, n, pad):
    """Triangular solves with a factor made elsewhere: ragged last blocks, any pitch."""
    torch = torch_cuda
    A, _, _, _ = orc.matgen(n, 5)
    if n == 1:
        A[0, 0] = 3.0
    assert orc.lib().orc_getrf_nopiv(n, n, A.ctypes.data, n) == 0
    x = np.random.default_rng(n).standard_normal(n)
    dx = torch.from_numpy(x.copy()).cuda()
    ws = mxp.Workspace(n, min(n, 64), 0)
    mxp.lu_solve(from_np_colmajor(torch, A, ld=n + pad), n, n + pad, dx, ws)
    LU = A.astype(np.float64)
    y = np.linalg.solve(np.tril(LU, -1) + np.eye(n), x)
    want = np.linalg.solve(np.triu(LU), y)
    assert np.max(np.abs(dx.cpu().numpy() - want)) <= 1e-12 * np.max(np.abs(want))


def test_chain_solve_keeps_nan(mxp, orc, torch_cuda):
    """A NaN in the right-hand side, whatever its bits, comes out as NaN and does not
    stall the blocks that wait for it."""
    torch = torch_cuda
    n = 200
    A, _, _, _ = orc.matgen(n, 5)
    assert orc.lib().orc_getrf_nopiv(n, n, A.ctypes.data, n) == 0
    x = np.random.default_rng(1).standard_normal(n)
    x.view(np.uint64)[70] = 0xFFFFFFFFFFFFFFFF
    dx = torch.from_numpy(x.copy()).cuda()
    ws = mxp.Workspace(n, 64, 0)
    mxp.lu_solve(from_np_colmajor(torch, A), n, n, dx, ws)
    assert np.all(np.isnan(dx.cpu().numpy()))  # column 70 of L, then U's back substitution, reach every row


@pytest.mark.parametrize("n,b", [(32, 32), (96, 32), (256, 256), (288, 96), (640, 320)])
def test_stored_inverse_solve_edges(mxp, orc, torch_cuda, n, b):
    """One block, few blocks, block sizes that are no power of two."""
    torch = torch_cuda
    p = mxp.panel_matgen(n, 3)
    ws = mxp.Workspace(n, b, 0)
    mxp.panel_lu(p, b, ws)
    LU = p.A.view(n, n).cpu().numpy().T.astype(np.float64)
    x = np.random.default_rng(n).standard_normal(n)
    dx = torch.from_numpy(x.copy()).cuda()
    mxp.lu_solve(p.A, n, n, dx, ws)
    want = np.linalg.solve(np.triu(LU), np.linalg.solve(np.tril(LU, -1) + np.eye(n), x))
    assert np.max(np.abs(dx.cpu().numpy() - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("n,b,form", [(192, 32, 0), (480, 96, 0), (640, 160, 1), (1280, 128, 0), (2000, 200, 0),
                                      (2304, 256, 1), (3200, 640, 0)])
def test_panel_copies_written_by_the_products(mxp, torch_cuda, n, b, form):
    """The FP16 and BF16X2 copies of the panels from the products' epilogues are the
    casts of the stored panels: the same factors bit for bit (b = 200: not that way)."""
    got = []
    for fused in (1, 0):
        p = mxp.panel_matgen(n, 9)
        ws = mxp.Workspace(n, b, form)
        ws.set_option(mxp.OPT_FP8_FUSED_CAST, fused)
        mxp.panel_lu(p, b, ws)
        got.append(p.A.cpu().numpy())
        ws.close()
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("n,b,chain", [(1024, 128, False), (1152, 128, True), (1920, 128, True), (384, 64, False), (512, 64, True),
                                       (2112, 192, False), (2304, 192, True), (5120, 256, False), (8192, 256, True),
                                       (3200, 320, False), (28160, 320, True), (2048, 512, False)])
def test_which_solve_a_factor_takes(mxp, torch_cuda, n, b, chain):
    """Either side of the line between the stored inverses and the chain: the chain's
    results are the chain's bits; the inverses' differ and agree to rounding."""
    torch = torch_cuda
    p = mxp.panel_matgen(n, 3)
    ws = mxp.Workspace(n, b, 0)
    mxp.panel_lu(p, b, ws)
    x = np.random.default_rng(n).standard_normal(n)
    got = []
    for off in (False, True):
        if off:
            ws.set_option(mxp.OPT_TRSV_INV, 0)
        dx = torch.from_numpy(x.copy()).cuda()
        mxp.lu_solve(p.A, n, n, dx, ws)
        got.append(dx.cpu().numpy())
    assert np.array_equal(got[0], got[1]) == chain
    assert np.max(np.abs(got[0] - got[1])) <= 1e-12 * np.max(np.abs(got[1]))


@pytest.mark.parametrize("m,n,k,ldc", [(129, 257, 4096, 132), (300, 260, 4224, 300), (640, 1000, 128, 643),
                                       (4097, 300, 640, 4097), (127, 33, 256, 128), (257, 300, 2048, 260),
                                       (300, 260, 2176, 301)])
def test_fp8_update_short_and_long_k(mxp, orc, torch_cuda, m, n, k, ldc):
    """Both forms of the FP8 kernel, C with 16-byte and with scalar addresses.  FP32
    accumulation in another order: 1e-5 of the sum of the terms' sizes."""
    torch = torch_cuda
    rng = np.random.default_rng(k)
    L = (rng.standard_normal((m, k)) * 1e-2).astype(np.float32)
    U = (rng.standard_normal((k, n)) * 0.5).astype(np.float32)
    Cm = rng.standard_normal((m, n)).astype(np.float32)
    dC = from_np_colmajor(torch, Cm, ld=ldc)
    Lp, Rp = (torch.zeros(r * k, dtype=torch.uint8, device="cuda") for r in (m, n))
    ls, rs = (torch.zeros(-(-r // 128) * -(-k // 128), dtype=torch.uint8, device="cuda") for r in (m, n))
    ws = mxp.Workspace(max(m, n) + k, k, 2)
    mxp.panel_cast_left(2, m, k, from_np_colmajor(torch, L), m, Lp, k, ls)
    mxp.panel_cast_right(2, n, k, from_np_colmajor(torch, U), k, Rp, k, rs)
    mxp.schur_update(2, m, n, k, Lp, k, Rp, k, dC, ldc, ws, ls, rs)
    got = to_np_colmajor(dC, m, n, ldc)
    want = orc.schur_update(2, Cm, L, U)
    bound = np.abs(L.astype(np.float64)) @ np.abs(U.astype(np.float64))
    err = np.abs(got.astype(np.float64) - want.astype(np.float64))
    assert np.all(err <= 1e-5 * bound + 1e-6 * np.abs(want) + 1e-30)
    pad = dC.view(n, ldc)[:, m:]
    assert torch.count_nonzero(pad) == 0  # nothing past the rows


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("b", [64, 128, 256])
def test_batch_strips_any_alignment(mxp, orc, torch_cuda, b, shift):
    """Vector and scalar paths of the panel strips and of the C staging (matrices at a
    16-byte and at a 4-byte address), one tile to several, whole and half ones:
    factors against the oracle at the form's bar, solutions against 64 bits."""
    torch = torch_cuda
    sizes = [128, 384, 256, 896]
    bt = mxp.Batch(sizes, [21, 22, 23, 24])
    bt.set_config(b, 128, 3)
    total = sum(n * n for n in sizes)
    buf = torch.empty(total + 4, dtype=torch.float32, device="cuda")
    bt.A = buf[shift:shift + total]
    bt.matgen()
    bt.solve()
    for i, (n, r) in enumerate(zip(sizes, bt.results())):
        assert r["converged"] == 1 and r["hpl_harness"] < 16.0 and r["info"] == 0
        A, d, _, rhs = orc.matgen(n, bt.seeds[i])
        if n % b == 0:
            assert orc.panel_lu(A, b, 0) == 0
            assert rel_fro(bt.matrix(i).cpu().numpy(), A) <= 1e-3
        x64 = np.linalg.solve(orc.matgen_f64(n, bt.seeds[i], d), rhs)
        x = bt.vec(bt.x, i).cpu().numpy()
        assert np.max(np.abs(x - x64)) / np.max(np.abs(x64)) < 1e-10
    bt.close()


@pytest.mark.parametrize("b", [64, 256])
def test_batch_strips_are_fp32(mxp, orc, torch_cuda, b):
    """Systems of at most two block steps: the first block row and column see no
    FP16 product, so they are FP32 factors, and the split products must leave
    them as close to 64 bits as substitution does (a few eps of their size)."""
    n = 2 * b
    bt = mxp.Batch([n], [31])
    bt.set_config(b, 128, 3)
    bt.matgen()
    bt.solve()
    got = bt.matrix(0).cpu().numpy().astype(np.float64)
    A, _, _, _ = orc.matgen(n, 31)
    A = A.astype(np.float64)
    for k in range(b):  # 64-bit elimination of the first block's pivots
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k, k + 1:])
    for sl in ((slice(b, n), slice(0, b)), (slice(0, b), slice(b, n))):
        assert rel_fro(got[sl], A[sl]) < 4 * EPS
    bt.close()
