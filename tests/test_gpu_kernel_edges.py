"""Kernels chosen by a rule on sizes, at the edges of their ranges, against the
oracle's arithmetic or the general kernel."""
import numpy as np
import pytest
import torch

import f3r_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return F.Context(0)


@pytest.mark.parametrize("grid,blocks,sigma", [
    ((16, 16, 16), 1, 1), ((16, 16, 16), 7, 1), ((16, 16, 16), 4096, 1),  # one block, ragged blocks, single rows
    ((64, 64, 1), 5, 1), ((32, 32, 16), 1, 1),                            # one and several sweeping warps
    ((64, 32, 32), 1, 1),                                                 # longer than the streamed kernel takes
    ((16, 16, 16), 7, 256)])                                              # blocks not contiguous
def test_block_ilu_solve_is_the_oracles(ctx, grid, blocks, sigma):
    """One outer step over one application of M = U^-1 L^-1 to a residual of
    entries +-1 (its norm, a power of two, and the fp16 input are exact): x is
    the fp16 result times one factor, rounded to fp32."""
    A = F.stencil27(*grid, 1, 0.5).scale()
    n = A.shape[0]
    r, i, v = A.arrays()
    b = np.where(F.random_uniform(3, 0.0, 1.0, n) < 0.5, -1.0, 1.0)
    M = O.Mat.from_csr(r, i, v)
    L, U = O.ilu0_bj(M, blocks)
    h = (b / np.sqrt(n)).astype(np.float16)
    want = O.trsv(U, True, O.trsv(L, False, h, prod_fma=True), prod_fma=True).astype(np.float64)
    S = F.Solver(ctx, A, precond=F.PRECOND_ILU0_BJ, ilu_blocks=blocks, sell_sigma=sigma, m2=1, m3=0, m4=1,
                 static_weight=1.0)
    x = np.zeros(n)
    S.solve(b, x, cond=lambda it, e: it >= 1)
    c = np.dot(x, want) / np.dot(want, want)
    assert c != 0 and np.all(np.abs(x / c - want) <= 4 * 2.0 ** -24 * np.abs(want))


@pytest.mark.parametrize("grid,blocks", [((32, 32, 32), 32768), ((32, 32, 32), 4096), ((24, 25, 27), 300), ((40, 40, 1), 33)])
def test_small_ilu_blocks_cost_what_they_hold(ctx, grid, blocks):
    """blocks of one row and of a few: the device memory of a solver does not
    grow with their number (32,768 rows: the matrix and its vectors take under 32
    MB, both factors at 4 words for each they need 12 MB), and a block solve is the oracle's"""
    A = F.stencil27(*grid, 1, 0.5).scale()
    n = A.shape[0]
    r, i, v = A.arrays()
    b = np.where(F.random_uniform(3, 0.0, 1.0, n) < 0.5, -1.0, 1.0)
    L, U = O.ilu0_bj(O.Mat.from_csr(r, i, v), blocks)
    h = (b / np.sqrt(n)).astype(np.float16)
    kw = dict(precond=F.PRECOND_ILU0_BJ, ilu_blocks=blocks, m2=1, m3=0, m4=1, static_weight=1.0)
    F.Solver(ctx, A, **kw).close()  # kernels loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    S = F.Solver(ctx, A, **kw)
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20
    x = np.zeros(n)
    S.solve(b, x, cond=lambda it, e: it >= 1)
    S.close()
    # b's entries are +-1: h is b over a factor that fp16 rounds, the same for every row
    want = O.trsv(U, True, O.trsv(L, False, h, prod_fma=True), prod_fma=True).astype(np.float64)
    c = np.dot(x, want) / np.dot(want, want)
    ulp = 4 * 2.0 ** -24 if float(h[0] * b[0]) ** 2 * n == 1.0 else 2.0 ** -10
    assert c != 0 and np.all(np.abs(x / c - want) <= ulp * np.abs(want).max())


@pytest.mark.parametrize("kind,grid,kw", [
    ("7pt", (64, 3, 2), dict(aligned=True, height=64)), ("7pt", (67, 5, 3), dict(aligned=True)),  # ragged last slices
    ("7pt", (67, 71, 64), dict(aligned=True, height=64)),  # more than one wave: two rows a lane
    ("7pt", (67, 71, 64), dict(aligned=True)), ("7pt", (67, 71, 64), dict()),
    ("7pt", (67, 71, 64), dict(sigma=256)), ("sdainv", (40, 31, 17), dict(aligned=True)),
    ("27pt", (68, 66, 67), dict()), ("27pt", (70, 68, 66), dict()),  # either side of a wave of rows
    # repeating rows (from half a wave of rows, or a wave): one and three windows, ragged grids, both tile sizes
    ("27pt", (40, 31, 17), dict(aligned=True, height=64)), ("27pt", (54, 53, 53), dict(aligned=True)),
    ("27pt", (200, 3, 261), dict(aligned=True)), ("27pt", (101, 67, 59), dict(aligned=True, height=64)),
    ("27pt", (107, 106, 106), dict(aligned=True)),  # rows off the patterns beside a last wave of tiles that is nearly full
    ("27pt", (81, 81, 81), dict(aligned=True)), ("27pt", (97, 90, 81), dict(aligned=True, height=64)),
    ("27pt", (53, 53, 53), dict(sigma=256)), ("27pt", (54, 53, 53), dict(sigma=256)),  # and of half of one (fp64)
])
def test_products_bitexact_across_the_rules(ctx, kind, grid, kw):
    """the thread-a-row, the repeating-row and the bulk-copy kernels on either
    side of the rules that choose between them: the oracle's sums bit for bit"""
    A = (F.stencil27(*grid, 2, 0.5) if kind == "27pt" else F.diffusion7(*grid, 1.5, 3.0, 1)).scale()
    if kind == "sdainv":
        A = A.sdainv()[1]
    r, i, v = A.arrays()
    n = A.shape[0]
    S = F.Sell(ctx, A, **kw)
    x = np.random.default_rng(1).standard_normal(n)
    for vt, dt, tdt, ov, oy, oacc in ((F.F64, np.float64, torch.float64, O.DT_F64, O.DT_F64, O.DT_F64),
                                      (F.F32, np.float32, torch.float32, O.DT_F32, O.DT_F32, O.DT_F32),
                                      (F.F16, np.float32, torch.float32, O.DT_F16, O.DT_F32, O.DT_F32),
                                      (F.F16, np.float16, torch.float16, O.DT_F16, O.DT_F16, O.DT_F32)):
        xd = x.astype(dt)
        y = torch.zeros(n, dtype=tdt, device="cuda")
        S.operate(torch.from_numpy(xd).cuda(), y, val_t=vt)
        torch.cuda.synchronize()
        want = O.spmv(r, i, v, xd, ov, oy, oacc)
        assert np.array_equal(y.cpu().numpy().view(np.uint8), want.view(np.uint8)), vt
        # vectors that start off a 16-byte boundary
        xo, yo = torch.zeros(n + 1, dtype=tdt, device="cuda")[1:], torch.zeros(n + 1, dtype=tdt, device="cuda")[1:]
        xo.copy_(torch.from_numpy(xd))
        S.operate(xo, yo, val_t=vt)
        torch.cuda.synchronize()
        assert np.array_equal(yo.cpu().numpy().view(np.uint8), want.view(np.uint8)), vt
    S.close()


@pytest.mark.parametrize("height", [32, 64])
@pytest.mark.parametrize("nrows,ncols,offsets", [
    (310007, 310033, tuple(range(27))),                                          # more columns than rows
    (310007, 309006, (-1300, -1299, -1298, -40, -39, -38) + tuple(range(-3, 6))),  # fewer
    (310007, 620013, (0, 1, 2, 5, 6, 7, 155000, 155001, 155002, 310003, 310004, 310005)),  # a window past the rows
])
def test_products_of_rectangular_matrices_with_repeating_rows(ctx, height, nrows, ncols, offsets):
    """bands of constant coefficients whose columns do not end where the rows do: the oracle's sums bit for bit"""
    d = np.array(offsets)
    c = np.arange(nrows)[:, None] + d
    keep = (c >= 0) & (c < ncols)
    r = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    i = c[keep].astype(np.int32)
    v = np.broadcast_to(np.random.default_rng(8).standard_normal(len(d)), c.shape)[keep]
    S = F.Sell(ctx, F.HostMatrix.from_csr(r, i, v, ncols), aligned=True, height=height)
    x = np.random.default_rng(9).standard_normal(ncols)
    for vt, dt, tdt, ov, oy, oacc in ((F.F64, np.float64, torch.float64, O.DT_F64, O.DT_F64, O.DT_F64),
                                      (F.F32, np.float32, torch.float32, O.DT_F32, O.DT_F32, O.DT_F32),
                                      (F.F16, np.float32, torch.float32, O.DT_F16, O.DT_F32, O.DT_F32),
                                      (F.F16, np.float16, torch.float16, O.DT_F16, O.DT_F16, O.DT_F32)):
        xd = x.astype(dt)
        y = torch.zeros(nrows, dtype=tdt, device="cuda")
        S.operate(torch.from_numpy(xd).cuda(), y, val_t=vt)
        torch.cuda.synchronize()
        want = O.spmv(r, i, v, xd, ov, oy, oacc)
        assert np.array_equal(y.cpu().numpy().view(np.uint8), want.view(np.uint8)), vt
    S.close()


@pytest.mark.parametrize("n,lo,hi", [(1, 1, 1), (97, 0, 8), (64, 8, 8), (131, 9, 9), (70, 30, 70), (33, 0, 33)])
def test_csr_tiles_bitexact(ctx, n, lo, hi):
    """groups of 32 rows that fit the short tile, fill it, fit the wide one or
    need several, empty rows and a ragged last group among them"""
    rng = np.random.default_rng(n)
    cnt = np.minimum(rng.integers(lo, hi + 1, n), n)
    r = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    i = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in cnt] or [[]]).astype(np.int32)
    v = rng.standard_normal(len(i))
    S = F.Sell(ctx, F.HostMatrix.from_csr(r, i, v, n), csr=True)
    x = rng.standard_normal(n)
    for vt, dt, tdt, ov in ((F.F64, np.float64, torch.float64, O.DT_F64), (F.F32, np.float32, torch.float32, O.DT_F32),
                            (F.F16, np.float16, torch.float16, O.DT_F16)):
        y = torch.zeros(n, dtype=tdt, device="cuda")
        S.operate(torch.from_numpy(x.astype(dt)).cuda(), y, val_t=vt)
        torch.cuda.synchronize()
        want = O.spmv(r, i, v, x.astype(dt), ov, ov, O.DT_F64 if vt == F.F64 else O.DT_F32)
        assert np.array_equal(y.cpu().numpy().view(np.uint8), want.view(np.uint8)), vt
    S.close()


@pytest.mark.parametrize("n,lo,hi", [(97, 16, 16), (101, 0, 17), (130, 64, 64), (129, 1, 65)])
def test_csr_middle_tiles_bitexact(ctx, n, lo, hi):
    """groups that fill a tile of 512 entries or take several, either side of the rows it is chosen for"""
    rng = np.random.default_rng(hi)
    cnt = rng.integers(lo, hi + 1, n)
    cnt[n // 2] = hi
    r = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    i = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in cnt]).astype(np.int32)
    v = rng.standard_normal(len(i))
    S = F.Sell(ctx, F.HostMatrix.from_csr(r, i, v, n), csr=True)
    x = rng.standard_normal(n)
    for vt, dt, ov in ((F.F64, np.float64, O.DT_F64), (F.F32, np.float32, O.DT_F32), (F.F16, np.float16, O.DT_F16)):
        xd = torch.from_numpy(x.astype(dt)).cuda()
        y = torch.zeros_like(xd)
        S.operate(xd, y, val_t=vt)
        torch.cuda.synchronize()
        want = O.spmv(r, i, v, x.astype(dt), ov, ov, O.DT_F64 if vt == F.F64 else O.DT_F32)
        assert np.array_equal(y.cpu().numpy().view(np.uint8), want.view(np.uint8)), vt
    S.close()


@pytest.mark.parametrize("grid", [(13, 11, 7), (32, 32, 32), (70, 69, 63), (97, 90, 71)])
@pytest.mark.parametrize("m2,m3", [(8, 4), (3, 8), (5, 0)])
def test_single_column_levels_are_the_block_kernels(ctx, grid, m2, m3):
    """the single solve's dots, updates and deferred normalisation against the
    K-column kernels: a column of a two-column block, bit for bit, with one and
    two logical blocks a block, 1 to 8 basis vectors and n % 4 of 0 to 3"""
    A = F.stencil27(*grid, 2, 0.5).scale()
    n = A.shape[0]
    X = np.stack([F.random_uniform(k, -1.0, 1.0, n) for k in (1, 2)])
    B = np.stack([A.spmv(x) for x in X])
    S = F.Solver(ctx, A, rel_tol=1e-10, m2=m2, m3=m3, sell_align=1)
    Y = np.zeros_like(B)
    rb = S.solve_multi(B, Y)
    for k in (0, 1):
        y = np.zeros(n)
        r = S.solve(B[k], y)
        assert r.is_solved and r.res_iter == rb[k].res_iter and np.array_equal(y, Y[k])


@pytest.mark.parametrize("kw", [dict(aligned=True), dict(aligned=True, height=64)])
def test_patterns_and_streamed_kernels_agree_on_non_finite_x(ctx, kw):
    """infinities and NaN in x reach the same rows from the row patterns as from
    the streamed kernel (which x off a 16-byte boundary takes), through padding
    and absent entries too"""
    A = F.stencil27(83, 71, 53, 2, 0.5).scale()
    n = A.shape[0]
    S = F.Sell(ctx, A, **kw)
    x = np.random.default_rng(5).standard_normal(n)
    x[[0, 1, 40, n // 2, n - 1]] = [np.inf, np.nan, -np.inf, np.inf, np.nan]
    for vt, tdt in ((F.F64, torch.float64), (F.F32, torch.float32), (F.F16, torch.float32), (F.F16, torch.float16)):
        xa = torch.from_numpy(x).to(tdt).cuda()
        xo = torch.zeros(n + 1, dtype=tdt, device="cuda")[1:]
        xo.copy_(xa)
        ya, yo = torch.zeros_like(xa), torch.zeros_like(xa)
        S.operate(xa, ya, val_t=vt)
        S.operate(xo, yo, val_t=vt)
        torch.cuda.synchronize()
        assert np.array_equal(ya.cpu().numpy(), yo.cpu().numpy(), equal_nan=True), vt
    S.close()


def _rows(per_sm):
    return per_sm * torch.cuda.get_device_properties(0).multi_processor_count


def test_the_library_reports_the_kernel_that_a_product_takes(ctx):
    """the kernels either side of each rule, and what the patterns cannot take:
    varying coefficients, short rows, too few rows"""
    nz = -(-_rows(1024) // (54 * 53))  # half a wave of rows and up
    A = F.stencil27(54, 53, nz, 2, 0.5).scale()
    n = A.shape[0]
    for kw, want in ((dict(aligned=True), ("patterns",) * 3), (dict(aligned=True, height=64), ("patterns", "patterns", "slices")),
                     (dict(csr=True), ("csr",) * 3), (dict(), ("slices", "rows", "rows")),
                     (dict(aligned=True, sigma=256), ("slices",) * 3)):
        S = F.Sell(ctx, A, **kw)
        got = tuple(S.product(vt)["kernel"] for vt in (F.F64, F.F32, F.F16))
        assert got == want, kw
        S.close()
    r, i, v = A.arrays()
    S = F.Sell(ctx, F.HostMatrix.from_csr(r, i, v * np.random.default_rng(0).uniform(1, 2, len(v)), n), aligned=True)
    p = S.product(F.F16)
    assert p["kernel"] == "slices" and p["matrix_bytes"] >= S.info().nnz_padded * 2
    S.close()
    few = F.Sell(ctx, F.stencil27(54, 53, nz - 1, 2, 0.5).scale(), aligned=True)
    assert few.product(F.F32)["kernel"] == ("patterns" if 54 * 53 * (nz - 1) >= _rows(1024) else "slices")
    few.close()
    S = F.Sell(ctx, F.diffusion7(32, 32, 32, 1.5, 3.0, 1).scale(), aligned=True)
    assert S.product(F.F16, F.F32)["kernel"] == "rows" and S.product(F.F16)["listed_rows"] == 0
    with pytest.raises(F.F3RError):
        S.product(F.F32, F.F16)
    S.close()


@pytest.mark.parametrize("width,dtype,want", [(64, F.F16, "rows"), (200, F.F16, "slices"), (64, F.F32, "rows"),
                                              (200, F.F64, "slices")])
def test_long_packed_rows_are_streamed(ctx, width, dtype, want):
    """100,000 rows: a matrix that stays in L2 is worked a thread a row, one that
    does not is streamed, as every packed matrix of long rows once was"""
    n = 100000
    c = (np.arange(n)[:, None] + np.arange(width) * 3) % n
    c.sort(1)
    v = np.random.default_rng(4).standard_normal(n * width)
    r, i = (np.arange(n + 1) * width).astype(np.int32), c.ravel().astype(np.int32)
    S = F.Sell(ctx, F.HostMatrix.from_csr(r, i, v, n), dtypes=(dtype,))
    assert S.product(dtype)["kernel"] == want
    dt, ov = {F.F64: (np.float64, O.DT_F64), F.F32: (np.float32, O.DT_F32), F.F16: (np.float16, O.DT_F16)}[dtype]
    x = np.random.default_rng(5).standard_normal(n).astype(dt)
    y = torch.from_numpy(np.zeros_like(x)).cuda()
    S.operate(torch.from_numpy(x).cuda(), y, val_t=dtype)
    torch.cuda.synchronize()
    want_y = O.spmv(r, i, v, x, ov, ov, O.DT_F64 if dtype == F.F64 else O.DT_F32)
    assert np.array_equal(y.cpu().numpy().view(np.uint8), want_y.view(np.uint8))
    S.close()


@pytest.mark.parametrize("K", [2, 4, 8, 16])
@pytest.mark.parametrize("variant,kw", [(2, dict(sell_align=1)), (1, dict(sell_align=1, sell_c=64))])
def test_block_solves_from_patterns_are_the_single_solves(ctx, K, variant, kw):
    """K columns from row patterns, rows that are no multiple of a 16-byte unit's
    and a ragged last block: every column its single solve bit for bit"""
    A = F.stencil27(54, 53, -(-_rows(1024) // (54 * 53)), variant, 0.5).scale()
    n = A.shape[0]
    S = F.Solver(ctx, A, rel_tol=1e-10, **kw)
    for vt, xt in ((F.F16, F.F16), (F.F32, F.F32)):
        p = S.product(vt, xt, columns=K)
        assert p["kernel"] == "patterns" and 0 < p["listed_rows"] < n // 2
    B = np.stack([F.random_uniform(k, -1.0, 1.0, n) for k in range(K)])
    Y = np.zeros_like(B)
    rb = S.solve_multi(B, Y)
    for k in range(K):
        y = np.zeros(n)
        r = S.solve(B[k], y)
        assert r.is_solved and r.res_iter == rb[k].res_iter and np.array_equal(y, Y[k]), k
    S.close()


@pytest.mark.parametrize("nx,block", [(257, "patterns"), (258, "slices"), (400, "slices")])
def test_patterns_of_long_grid_lines(ctx, nx, block):
    """lines longer than a pattern's block: the single-column product keeps the
    patterns where the K-column one has too many windows; both bit for bit"""
    ny, nz = 40, -(-_rows(1024) // (nx * 40))
    A = F.stencil27(nx, ny, nz, 2, 0.5).scale()
    r, i, v = A.arrays()
    n = A.shape[0]
    S = F.Solver(ctx, A, rel_tol=1e-10, sell_align=1)
    assert S.product(F.F16)["kernel"] == "patterns" and S.product(F.F16, columns=8)["kernel"] == block
    x = np.random.default_rng(2).standard_normal(n)
    for vt, dt, ov, oacc in ((F.F64, np.float64, O.DT_F64, O.DT_F64), (F.F32, np.float32, O.DT_F32, O.DT_F32),
                             (F.F16, np.float16, O.DT_F16, O.DT_F32)):
        xd = torch.from_numpy(x.astype(dt)).cuda()
        y = torch.zeros_like(xd)
        S.operate(xd, y, val_t=vt)
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), O.spmv(r, i, v, x.astype(dt), ov, ov, oacc)), vt
    B = np.stack([F.random_uniform(k, -1.0, 1.0, n) for k in range(2)])
    Y, y = np.zeros_like(B), np.zeros(n)
    S.solve_multi(B, Y)
    S.solve(B[1], y)
    assert np.array_equal(y, Y[1])
    S.close()


def test_a_matrix_that_leaves_no_room_for_patterns_is_streamed(ctx):
    """the patterns are an extra: with device memory for the matrix and not for
    the lists of the rows off them, the matrix works as it did without"""
    A = F.stencil27(12, 400, 400, 2, 0.5).scale()  # lists of a sixth of the rows
    n = A.shape[0]
    x = torch.from_numpy(np.random.default_rng(6).standard_normal(n)).cuda()
    y, z = torch.zeros_like(x), torch.zeros_like(x)
    F.Sell(ctx, A, aligned=True).close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    S = F.Sell(ctx, A, aligned=True)
    S.operate(x, y)
    ctx.synchronize()
    p, total = S.product(F.F64), free - torch.cuda.mem_get_info()[0]
    assert p["kernel"] == "patterns" and p["listed_rows"] > n // 8
    S.close()
    # value copies of 8, 4 and 2 bytes and one of columns
    lists = p["listed_rows"] * 28 * (8 + 4 + 2 + 4)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (total - lists // 2), dtype=torch.uint8, device="cuda")
    try:
        S = F.Sell(ctx, A, aligned=True)
        assert S.product(F.F64)["kernel"] == "slices"
        S.operate(x, z)
        ctx.synchronize()
        S.close()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert torch.equal(y, z)
