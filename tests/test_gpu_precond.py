"""Preconditioners on the GPU vs the CPU oracle.

ILU(0): factor and applications bit-identical to the reference's sequential
LUFactorisationAlgo (same per-row arithmetic, wavefront-parallel order).
Chebyshev: the power-method bounds use device dot products (fixed tree), so
bounds and applications agree to rounding only (1e-12 relative).
"""
import numpy as np
import pytest

from alien_b200 import abi
from oracle import oracle as O
from tests import problems

pytestmark = pytest.mark.gpu


def rnd(n, seed):
    return np.random.default_rng(seed).uniform(-1, 1, n)


STENCIL_SHAPED = {"poisson16", "diffusion12", "convdiff_10x11x12", "diffusion24", "grid_37x21x5"}


@pytest.mark.parametrize("schedule", ["auto", "wavefront"])
@pytest.mark.parametrize("name", ["poisson16", "diffusion12", "convdiff_10x11x12", "diffusion2d_31x9", "ragged",
                                  "diffusion24", "grid_37x21x5"])
def test_ilu0_factor_and_apply_bit_exact(ctx, name, schedule):
    P = abi.diffusion(37, 21, 5, sigma=1.0, smooth=2.0, seed=9) if name == "grid_37x21x5" else problems.get(name)
    A = ctx.matrix(P.row_ptr, P.cols, P.vals)
    pc = abi.Precond(ctx, A, "ilu0", ilu_schedule=schedule)
    expect = abi.ILU_SCHEDULE["stencil_cluster" if schedule == "auto" and name in STENCIL_SHAPED else "wavefront"]
    assert pc.info.ilu_schedule == expect
    np.testing.assert_array_equal(pc.ilu0_values(), O.ilu0_factor(P.row_ptr, P.cols, P.vals))
    for seed in range(3):  # repeated applications (sweep state must reset itself)
        y = rnd(P.n, seed)
        vy, vx = ctx.vector(y), ctx.vector(P.n)
        pc.apply(vy, vx)
        np.testing.assert_array_equal(vx.download(), O.ilu0_apply(P.row_ptr, P.cols, P.vals, y))
    # in place: x and y the same vector
    y = rnd(P.n, 9)
    v = ctx.vector(y)
    pc.apply(v, v)
    np.testing.assert_array_equal(v.download(), O.ilu0_apply(P.row_ptr, P.cols, P.vals, y))
    info = pc.info
    assert info.ilu_levels_lower >= 1 and info.ilu_levels_upper >= 1
    if name == "poisson16":
        assert info.ilu_levels_lower == 3 * 16 - 2


@pytest.mark.parametrize("schedule", ["stencil", "stencil_cluster"])
def test_ilu0_stencil_schedule_refused_for_other_matrices(ctx, schedule):
    P = problems.get("ragged")
    A = ctx.matrix(P.row_ptr, P.cols, P.vals)
    with pytest.raises(abi.AB2Error) as e:
        abi.Precond(ctx, A, "ilu0", ilu_schedule=schedule)
    assert e.value.code == abi.AB2_ERR_BAD_ARG


def test_ilu0_cluster_schedule_needs_its_buffers_in_shared_memory(ctx):
    """600 planes along z: the cluster walk's buffers exceed shared memory,
    so AUTO takes the single-CTA walk and an explicit request is refused."""
    P = abi.diffusion(20, 18, 600, sigma=1.0, smooth=2.0, seed=3)
    A = ctx.matrix(P.row_ptr, P.cols, P.vals)
    pc = abi.Precond(ctx, A, "ilu0")
    assert pc.info.ilu_schedule == abi.ILU_SCHEDULE["stencil"]
    y = rnd(P.n, 4)
    vy, vx = ctx.vector(y), ctx.vector(P.n)
    pc.apply(vy, vx)
    np.testing.assert_array_equal(vx.download(), O.ilu0_apply(P.row_ptr, P.cols, P.vals, y))
    with pytest.raises(abi.AB2Error) as e:
        abi.Precond(ctx, A, "ilu0", ilu_schedule="stencil_cluster")
    assert e.value.code == abi.AB2_ERR_BAD_ARG


def test_diag_apply(ctx):
    P = problems.get("diffusion12")
    A = ctx.matrix(P.row_ptr, P.cols, P.vals)
    pc = abi.Precond(ctx, A, "diag")
    y = rnd(P.n, 1)
    vy, vx = ctx.vector(y), ctx.vector(P.n)
    pc.apply(vy, vx)
    np.testing.assert_array_equal(vx.download(), O.inv_diag(P.row_ptr, P.cols, P.vals) * y)


@pytest.mark.parametrize("saad,lanczos", [(True, False), (True, True), (False, True)])
@pytest.mark.parametrize("name", ["poisson16", "diffusion24", "convdiff_10x11x12"])
def test_chebyshev_variants_bit_exact(ctx, name, saad, lanczos):
    """Saad's recurrence (ChebyshevPreconditioner<.., true>) and Lanczos bounds,
    against the oracle summing its dots in the device tree."""
    P = problems.get(name)
    A = ctx.matrix(P.row_ptr, P.cols, P.vals)
    pc = abi.Precond(ctx, A, "cheb", poly_factor=0.0, poly_order=3, poly_factor_max_iter=20, cheb_saad=saad,
                     cheb_lanczos=lanczos)
    tb = ctx.info.reduction_max_blocks
    x = rnd(P.n, 5)
    vx, vy = ctx.vector(x), ctx.vector(P.n)
    pc.apply(vx, vy)
    exact = O.cheb_apply(P.row_ptr, P.cols, P.vals, x, 0.0, 3, 20, dot_mode=O.DOT_DEVICE_TREE, tree_blocks=tb,
                         saad=saad, lanczos=lanczos)
    np.testing.assert_array_equal(vy.download(), exact)
    pc.apply(vx, vx)  # in place
    np.testing.assert_array_equal(vx.download(), exact)


@pytest.mark.parametrize("name,factor", [("poisson16", 0.0), ("diffusion12", 0.0), ("poisson16", 0.5),
                                         ("ragged", 0.0)])
def test_chebyshev_bounds_and_apply(ctx, name, factor):
    P = problems.get(name)
    A = ctx.matrix(P.row_ptr, P.cols, P.vals)
    pc = abi.Precond(ctx, A, "cheb", poly_factor=factor, poly_order=3, poly_factor_max_iter=12)
    tb = ctx.info.reduction_max_blocks
    # bit-exact against the oracle summing its dots in the device tree
    a, b = O.cheb_bounds(P.row_ptr, P.cols, P.vals, factor, 12, dot_mode=O.DOT_DEVICE_TREE, tree_blocks=tb)
    assert (pc.info.cheb_alpha, pc.info.cheb_beta) == (a, b)
    # and close to the sequential-dot bounds of the reference's order
    a0, b0 = O.cheb_bounds(P.row_ptr, P.cols, P.vals, factor, 12)
    assert abs(pc.info.cheb_alpha - a0) <= 1e-12 * abs(a0)
    assert abs(pc.info.cheb_beta - b0) <= 1e-12 * abs(b0)
    x = rnd(P.n, 3)
    vx, vy = ctx.vector(x), ctx.vector(P.n)
    pc.apply(vx, vy)
    exact = O.cheb_apply(P.row_ptr, P.cols, P.vals, x, factor, 3, 12, dot_mode=O.DOT_DEVICE_TREE, tree_blocks=tb)
    np.testing.assert_array_equal(vy.download(), exact)
    ref = O.cheb_apply(P.row_ptr, P.cols, P.vals, x, factor, 3, 12)
    np.testing.assert_allclose(vy.download(), ref, rtol=0, atol=1e-11 * np.max(np.abs(ref)))
    pc.apply(vx, vx)  # aliasing input/output
    np.testing.assert_array_equal(vx.download(), exact)


# The stencil sweeps one tile per CTA and in 2 x 2-tile thread-block clusters
# (tiles handing boundary values to their cluster neighbours through
# distributed shared memory), on grids whose tiles fill several clusters,
# partly filled clusters and partial tiles included.  Same bits as the
# sequential sweeps.
@pytest.mark.parametrize("schedule", ["stencil", "stencil_cluster"])
@pytest.mark.parametrize("dims", [(130, 75, 7), (40, 40, 6), (16, 100, 3), (100, 16, 3), (20, 18, 340)])
def test_ilu0_stencil_walks_bit_exact(ctx, schedule, dims):
    P = abi.diffusion(*dims, sigma=1.0, smooth=2.0, seed=5)
    A = ctx.matrix(P.row_ptr, P.cols, P.vals)
    pc = abi.Precond(ctx, A, "ilu0", ilu_schedule=schedule)
    assert pc.info.ilu_schedule == abi.ILU_SCHEDULE[schedule]
    for seed in range(2):
        y = rnd(P.n, 20 + seed)
        vy, vx = ctx.vector(y), ctx.vector(P.n)
        pc.apply(vy, vx)
        np.testing.assert_array_equal(vx.download(), O.ilu0_apply(P.row_ptr, P.cols, P.vals, y))


# The strip walk at the edges of its tiles, strips, rings and lanes (odd sides,
# one line, planes below and above the ring sizes), with right-hand sides that
# leave the fast division's range: zeros, tiny and huge values, denormals,
# infinities and NaN.  Same bits as the sequential sweeps.
@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 2, 41), (16, 8, 24), (17, 9, 23), (15, 24, 11), (33, 31, 37)])
@pytest.mark.parametrize("scale", [1.0, 1e-140, 1e140])
def test_ilu0_strip_walk_division_range(ctx, dims, scale):
    P = abi.diffusion(*dims, sigma=1.0, smooth=2.0, seed=7)
    vals = P.vals * scale
    A = ctx.matrix(P.row_ptr, P.cols, vals)
    pc = abi.Precond(ctx, A, "ilu0")  # (a 2 x 2 x 2 profile is no 7-point grid by its entries alone: wavefronts)
    rng = np.random.default_rng(3)
    n = P.n
    y0 = rng.uniform(-1, 1, n)
    zeros = y0 * (rng.uniform(size=n) < 0.3)
    zeros[::5] = -0.0
    wide = y0 * 10.0 ** rng.uniform(-300, 150, n)
    inf, nan = y0.copy(), y0.copy()
    inf[n // 3] = np.inf
    nan[n // 2] = np.nan
    for y in (y0, zeros, wide, np.zeros(n), inf, nan, y0):
        vy, vx = ctx.vector(y), ctx.vector(n)
        pc.apply(vy, vx)
        with np.errstate(all="ignore"):
            ref = O.ilu0_apply(P.row_ptr, P.cols, vals, y)
        got = vx.download()
        np.testing.assert_array_equal(got, ref)
        np.testing.assert_array_equal(np.signbit(got)[~np.isnan(ref)], np.signbit(ref)[~np.isnan(ref)])


def _csr(n, rows):
    """CSR from {row: {col: value}}."""
    rp, ci, vv = [0], [], []
    for i in range(n):
        for c in sorted(rows[i]):
            ci.append(c)
            vv.append(rows[i][c])
        rp.append(len(ci))
    return np.asarray(rp, np.int32), np.asarray(ci, np.int32), np.asarray(vv)


def _random_rows(n, most, span, seed, dense_levels=False):
    rng = np.random.default_rng(seed)
    rows = []
    for i in range(n):
        r = {i: 4.0 + rng.uniform()}
        # dense_levels: every row hangs on row 0 only
        cols = [0] if dense_levels else rng.integers(max(0, i - span), i + 1, rng.integers(0, most + 1))
        for c in cols:
            if c != i:
                r[int(c)] = -rng.uniform()
        rows.append(r)
    for i in range(n):  # the same on the other side of the diagonal
        for c in list(rows[i]):
            if c < i and len([k for k in rows[c] if k > c]) < most:
                rows[c][i] = -rng.uniform()
    return _csr(n, rows)


# Both sweeps by one CTA (AUTO on small factors of matrices that are no 3-D grid)
# against the sequential sweeps and the sweeps across SMs: narrow and wide
# wavefronts, one to nine entries a side (nine is past what is packed), right-hand
# sides outside the fast division's range, FP64 limits of shared memory.
@pytest.mark.parametrize("kind", ["n1", "two", "eight", "nine", "wide", "grid", "limit", "past_limit", "nodiag"])
def test_ilu0_one_cta_sweeps_bit_exact(ctx, kind):
    if kind == "n1":
        rp, ci, vv = _csr(1, [{0: 3.0}])
    elif kind == "two":
        rp, ci, vv = _random_rows(700, 2, 40, 1)
    elif kind == "eight":
        rp, ci, vv = _random_rows(900, 8, 60, 2)
    elif kind == "nine":
        n = 400
        rows = [{c: (12.0 if c == i else -0.3 - 0.01 * (c % 7)) for c in range(max(0, i - 9), min(n, i + 10))}
                for i in range(n)]
        rp, ci, vv = _csr(n, rows)
    elif kind == "wide":
        rp, ci, vv = _random_rows(3000, 2, 10, 3, dense_levels=True)
    elif kind == "nodiag":
        rp, ci, vv = _csr(40, [{c: (2.0 if c == i else -0.5) for c in (i - 1, i, i + 1)
                                if 0 <= c < 40 and not (i == 20 and c == 20)} for i in range(40)])
    else:
        nx, ny = {"grid": (61, 47), "limit": (165, 169), "past_limit": (170, 170)}[kind]
        P = abi.diffusion(nx, ny, 1, sigma=1.0, smooth=2.0, seed=4)
        rp, ci, vv = P.row_ptr, P.cols, P.vals
    n = rp.size - 1
    A = ctx.matrix(rp, ci, vv)
    auto, across = abi.Precond(ctx, A, "ilu0"), abi.Precond(ctx, A, "ilu0", ilu_schedule="wavefront")
    y0 = rnd(n, 7)
    zeros = np.where(np.arange(n) % 3 == 0, y0, -0.0)
    inf = y0.copy()
    inf[n // 2] = np.inf
    for y in (y0, zeros, y0 * 1e-290, y0 * 1e160, np.zeros(n), inf, y0):
        out = []
        for pc in (auto, across):
            vx = ctx.vector(n)
            pc.apply(ctx.vector(y), vx)
            out.append(vx.download())
        with np.errstate(all="ignore"):
            ref = O.ilu0_apply(rp, ci, vv, y)
        np.testing.assert_array_equal(out[0], ref)
        np.testing.assert_array_equal(out[0], out[1])
    v = ctx.vector(y0)
    auto.apply(v, v)  # in place
    np.testing.assert_array_equal(v.download(), O.ilu0_apply(rp, ci, vv, y0))


@pytest.mark.parametrize("saad", [True, False])
@pytest.mark.parametrize("order", [1, 2, 3, 5])
@pytest.mark.parametrize("name", ["poisson16", "ragged", "convdiff_10x11x12"])
def test_chebyshev_first_and_last_step(ctx, name, order, saad):
    """The start fused into the first step (different vectors) and not (in
    place), and the last step's skipped stores: the oracle's bits in both,
    repeatedly."""
    P = problems.get(name)
    A = ctx.matrix(P.row_ptr, P.cols, P.vals)
    pc = abi.Precond(ctx, A, "cheb", poly_factor=0.0, poly_order=order, poly_factor_max_iter=12, cheb_saad=saad)
    tb = ctx.info.reduction_max_blocks
    for seed in range(2):
        x = rnd(P.n, seed)
        exact = O.cheb_apply(P.row_ptr, P.cols, P.vals, x, 0.0, order, 12, dot_mode=O.DOT_DEVICE_TREE, tree_blocks=tb,
                             saad=saad)
        vx, vy = ctx.vector(x), ctx.vector(P.n)
        pc.apply(vx, vy)
        np.testing.assert_array_equal(vy.download(), exact)
        pc.apply(vx, vx)
        np.testing.assert_array_equal(vx.download(), exact)


@pytest.mark.parametrize("n", [1, 2, 311, 312, 313, 624, 1249, 40000])
def test_chebyshev_start_vector_drawn_on_the_device(ctx, n):
    """The power method's start vector (a default-seeded mt19937) around the
    generator's block sizes: the oracle's bounds, bit for bit."""
    rng = np.random.default_rng(n)
    rp, ci, vals = _csr(n, [{c: (rng.uniform(2.5, 4.0) if c == i else -1.0) for c in (i - 1, i, i + 1) if 0 <= c < n}
                            for i in range(n)])
    A = ctx.matrix(rp, ci, vals)
    pc = abi.Precond(ctx, A, "cheb", poly_factor=0.0, poly_order=3, poly_factor_max_iter=3)
    with np.errstate(all="ignore"):  # (n = 1: D^-1 A is the identity, the shifted method divides 0 by 0)
        bounds = O.cheb_bounds(rp, ci, vals, 0.0, 3, dot_mode=O.DOT_DEVICE_TREE,
                               tree_blocks=ctx.info.reduction_max_blocks)
    np.testing.assert_array_equal([pc.info.cheb_alpha, pc.info.cheb_beta], bounds)


# The start goes into Saad's first step where that pays (bands, or few and narrow
# rows): seen by an application's launches, either side of the limits, with the
# oracle's bits in both forms.
@pytest.mark.parametrize("n,per_row,widest,fused", [(900, 3, 24, True), (900, 3, 25, False), (200000, 7, 7, True),
                                                    (200001, 7, 7, False)])
def test_chebyshev_start_fused_where_it_pays(ctx, n, per_row, widest, fused):
    rows = np.repeat(np.arange(n), per_row)
    cols = (rows + np.tile(np.arange(per_row) - per_row // 2, n)) % n
    if widest > per_row:
        rows = np.concatenate([rows, np.full(widest - per_row, 5)])
        cols = np.concatenate([cols, np.arange(100, 100 + widest - per_row)])
    order = np.lexsort((cols, rows))
    rows, cols = rows[order], cols[order]
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    vals = np.where(rows == cols, np.linspace(widest + 1.0, widest + 2.0, n)[rows], -0.5)
    assert np.bincount(rows).max() == widest and (vals.size <= 1400000) == (n <= 200000)
    A = ctx.matrix(rp, cols.astype(np.int32), vals)
    pc = abi.Precond(ctx, A, "cheb", poly_factor=0.0, poly_order=3, poly_factor_max_iter=4, cheb_saad=True)
    x = rnd(n, 3)
    vx, vy = ctx.vector(x), ctx.vector(n)
    before = ctx.launches
    pc.apply(vx, vy)
    assert ctx.launches - before == (2 if fused else 3)
    exact = O.cheb_apply(rp, cols.astype(np.int32), vals, x, 0.0, 3, 4, dot_mode=O.DOT_DEVICE_TREE,
                         tree_blocks=ctx.info.reduction_max_blocks, saad=True)
    np.testing.assert_array_equal(vy.download(), exact)
    A.close()


def test_chebyshev_start_fused_with_bands(ctx):
    P = abi.diffusion(70, 60, 50, sigma=1.0, smooth=2.0, seed=5)  # 1.45 million entries
    x = rnd(P.n, 3)
    for formats, launches in ((abi.FMT_CSR | abi.FMT_ELL | abi.FMT_STENCIL, 2), (abi.FMT_CSR | abi.FMT_ELL, 3)):
        A = ctx.matrix(P.row_ptr, P.cols, P.vals, formats)
        pc = abi.Precond(ctx, A, "cheb", poly_factor=0.0, poly_order=3, poly_factor_max_iter=4, cheb_saad=True)
        vx, vy = ctx.vector(x), ctx.vector(P.n)
        before = ctx.launches
        pc.apply(vx, vy)
        assert ctx.launches - before == launches
        A.close()


def test_ilu0_cluster_schedule_is_refused_before_any_set_up(ctx):
    """Past the planes it is offered for, the request ends with the grid's shape known:
    nothing is factorised or packed for it."""
    P = abi.diffusion(6, 5, 347, sigma=1.0, smooth=2.0, seed=3)
    A = ctx.matrix(P.row_ptr, P.cols, P.vals, abi.FMT_CSR | abi.FMT_ELL | abi.FMT_STENCIL)
    launches = []
    for schedule in ("stencil", "stencil_cluster"):
        before = ctx.launches
        if schedule == "stencil":
            abi.Precond(ctx, A, "ilu0", ilu_schedule=schedule)
        else:
            with pytest.raises(abi.AB2Error) as e:
                abi.Precond(ctx, A, "ilu0", ilu_schedule=schedule)
            assert e.value.code == abi.AB2_ERR_BAD_ARG
        launches.append(ctx.launches - before)
    assert launches[0] - launches[1] >= 7  # extract, fill, factor, pack, both sweeps' coefficients, hand-over words
    A.close()


# Exact zeros in the sweeps: point sources, empty regions, all of it, of both signs,
# and zeros over pivots outside the fast division's range, down to the sign bit.
@pytest.mark.parametrize("dims", [(33, 18, 21), (40, 31, 1)])
@pytest.mark.parametrize("scale", [1.0, 1e-140])
def test_ilu0_zero_dividends(ctx, dims, scale):
    P = abi.diffusion(*dims, sigma=1.0, smooth=2.0, seed=7)
    vals = P.vals * scale
    A = ctx.matrix(P.row_ptr, P.cols, vals)
    pc = abi.Precond(ctx, A, "ilu0")
    vz = ctx.vector(P.n)
    point = np.zeros(P.n)
    point[P.n // 2] = 1.0
    last = np.zeros(P.n)
    last[-1] = -3.0
    half = rnd(P.n, 5)
    half[P.n // 3:] = -0.0
    for y in (point, last, -last, half, np.zeros(P.n), np.full(P.n, -0.0), np.where(np.arange(P.n) % 2 == 0, 0.0, -0.0)):
        pc.apply(ctx.vector(y), vz)
        np.testing.assert_array_equal(vz.download().view(np.int64),
                                      O.ilu0_apply(P.row_ptr, P.cols, vals, y).view(np.int64))
    A.close()


def _layers(layers, per_layer, entries, seed):
    """Rows in layers, each hanging on `entries` rows of the layer before it and as
    many of the one after it (fewer in the outer layers): one wavefront a layer."""
    rng = np.random.default_rng(seed)
    n = layers * per_layer
    rows, cols = [np.arange(n)], [np.arange(n)]
    for step in (-1, 1):
        r = np.repeat(np.arange(n).reshape(layers, per_layer)[(1 if step < 0 else 0):(None if step < 0 else -1)], entries)
        first = np.stack([rng.choice(per_layer, entries, replace=False) for _ in range(r.size // entries)]).ravel()
        rows.append(r)
        cols.append((r // per_layer + step) * per_layer + first)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((cols, rows))
    rows, cols = rows[order], cols[order]
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    vals = np.where(rows == cols, 2.0 * entries + 1.0, -rng.uniform(0.1, 1.0, rows.size))
    return rp, cols.astype(np.int32), vals


# The one-CTA sweeps told from the sweeps across SMs by an application's launches
# (one, two): wavefronts of more rows than the CTA's warps take at a time (its WIDE
# builds) with 2, 4 and 8 entries a side, and a vector that fits shared memory to the
# byte (28 x 970: 225,280) or misses it by eight (159 x 175).
@pytest.mark.parametrize("kind,launches", [("wide2", 1), ("wide4", 1), ("wide8", 1), ("wide9", 2), ("wide3_odd", 1),
                                           ("fits", 1), ("misses", 2)])
def test_ilu0_one_cta_sweeps_run_where_they_should(ctx, kind, launches):
    if kind.startswith("wide"):
        rp, ci, vv = _layers(20, 1300 if kind != "wide3_odd" else 513, int(kind[4]), seed=int(kind[4]))
    else:
        P = abi.diffusion(*((28, 970) if kind == "fits" else (159, 175)), 1, sigma=1.0, smooth=2.0, seed=4)
        rp, ci, vv = P.row_ptr, P.cols, P.vals
    n = rp.size - 1
    A = ctx.matrix(rp, ci, vv, abi.FMT_CSR | abi.FMT_ELL | abi.FMT_F32)
    pc = abi.Precond(ctx, A, "ilu0")
    np.testing.assert_array_equal(pc.ilu0_values(), O.ilu0_factor(rp, ci, vv))
    vz = ctx.vector(n)
    y0 = rnd(n, 11)
    for y in (y0, np.where(np.arange(n) % 3 == 0, y0, -0.0), y0 * 1e-290, y0):
        vy = ctx.vector(y)
        before = ctx.launches
        pc.apply(vy, vz)
        assert ctx.launches - before == launches
        np.testing.assert_array_equal(vz.download(), O.ilu0_apply(rp, ci, vv, y))
    # the same in FP32, inside the mixed solver
    kw = dict(solver="bicgs", precond="ilu0", tol=1e-10, max_outer=10, inner_tol=1e-4, inner_max_iter=500)
    M = abi.Mixed(ctx, A, **kw)
    x = ctx.vector(n)
    st = M.solve(ctx.vector(y0), x)
    o = O.mixed_solve(rp, ci, vv, y0, dot_mode=O.DOT_DEVICE_TREE, tree_blocks=ctx.info.reduction_max_blocks, **kw)
    assert (st.outer_iterations, st.inner_iterations) == (o.outer_iterations, o.inner_iterations)
    np.testing.assert_array_equal(x.download(), o.x)
    M.close()
    A.close()
