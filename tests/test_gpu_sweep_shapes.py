"""The BILU0 factorisation (a warp per row) and the ring-fed block sweeps at the shapes where they can go wrong: rows longer
than the factorisation keeps on chip, levels of one row and levels wider than a
step, a step's remainder, rows with long overflow lists, systems at and beyond what one SM's shared memory holds, and
batches of uneven systems. The factors of every precision, FP64 and mixed sweeps against the oracle bit for bit; the all-FP32 sweeps bit for bit those of
the fixed-thread-count kernels (the same arithmetic in the same order) and within float rounding of the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(n, pairs, seed):
    """A structurally symmetric, diagonally dominant 3 x 3 block system with the given off-diagonal pairs."""
    from ressim_gb300.bsr import BSR
    rng = np.random.default_rng(seed)
    pairs = np.asarray(sorted(set(map(tuple, pairs))), dtype=np.int64).reshape(-1, 2)
    rows = np.concatenate([np.arange(n), pairs[:, 0], pairs[:, 1]])
    cols = np.concatenate([np.arange(n), pairs[:, 1], pairs[:, 0]])
    order = np.lexsort((cols, rows))
    rows, cols = rows[order], cols[order]
    val = 0.2 * rng.standard_normal((rows.size, 3, 3))
    deg = np.bincount(rows, minlength=n)
    val[rows == cols] += (2.0 + deg)[:, None, None] * np.eye(3)
    return BSR(n, 3, np.concatenate([[0], np.cumsum(deg)]).astype(np.int32), cols.astype(np.int32), val.reshape(-1))


def box(nx, ny, nz):
    i = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    return [p for a, b in ((i[:, :, :-1], i[:, :, 1:]), (i[:, :-1], i[:, 1:]), (i[:-1], i[1:])) for p in zip(a.ravel(), b.ravel())]


SHAPES = {
    "one_row": (1, []),
    "chain": (301, [(k, k + 1) for k in range(300)]),                      # 301 levels of one row
    "diagonal": (1003, []),                                                # one level: several steps and a remainder
    "star": (400, [(0, k) for k in range(1, 400)]),                        # an overflow list of 396 entries
    "arrow": (200, [(k, 199) for k in range(199)]),                        # the same in the forward sweep
    "two_colours": (1200, [(k, 600 + (7 * k + j) % 600) for k in range(600) for j in range(5)]),   # every row overflows
    "clique": (130, [(k, k + 1) for k in range(129)] + [(a, b) for a in range(20, 67) for b in range(a + 1, 67)]),   # rows of 47+ blocks
    "box": (9 * 7 * 5, box(9, 7, 5)),
    "slab": (70 * 61 * 2, box(70, 61, 2)),
    "box_13k": (33 * 40 * 10, box(33, 40, 10)),                            # FP32: the vector fills most of the SM
    "box_20k": (40 * 50 * 10, box(40, 50, 10)),                            # no vector fits
}


@pytest.mark.parametrize("name", SHAPES)
def test_sweeps_match_the_oracle(name, oracle):
    from ressim_gb300.solver import DeviceSolver
    n, pairs = SHAPES[name]
    A = system(n, pairs, seed=len(name))
    r = np.random.default_rng(1).standard_normal(3 * n)
    lu, _ = oracle.bilu0_factor(A)
    luf, _ = oracle.bilu0_factor_lean(A)
    f32, _ = oracle.bilu0_factor_f32(A)
    z = {}
    for precision, threads in (("fp64", 0), ("mixed", 0), ("mixed_f32", 0), ("mixed_f32", 256)):
        with DeviceSolver(precond="bilu0", precision=precision, sweep="cta", cpr2_threads=threads) as d:
            d.set_matrix(A)
            d.setup()
            z[precision, threads] = d.precond_apply(r)
            if not threads:                                                # the factorisation, a warp per row
                assert np.array_equal(d.factors(A.nnzb), {"fp64": lu, "mixed": luf, "mixed_f32": f32}[precision])
            if not threads:
                x, res = d.solve(r, tol=1e-8, maxit=100)                   # the input fused with the Krylov updates
                assert res.converged
    assert np.array_equal(z["fp64", 0], oracle.bilu0_apply(A, lu, r))
    assert np.array_equal(z["mixed", 0], oracle.bilu0_apply_fd(A, luf, r))
    assert np.array_equal(z["mixed_f32", 0], z["mixed_f32", 256])
    ref = oracle.bilu0_apply_ff(A, f32, r)
    assert np.linalg.norm(z["mixed_f32", 0] - ref) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("precision", ["fp64", "mixed_f32"])
def test_batch_of_uneven_systems(precision):
    """A batch gives every system the result it has alone, whatever its place in the concatenated arrays (the input's
    16-byte alignment differs from system to system)."""
    from ressim_gb300.solver import DeviceSolver
    mats = [system(n, pairs, seed=3) for n, pairs in (SHAPES[k] for k in ("chain", "one_row", "box", "two_colours", "star"))]
    r = np.random.default_rng(2).standard_normal(sum(3 * A.n for A in mats))
    alone, off = [], 0
    for A in mats:
        with DeviceSolver(precond="bilu0", precision=precision) as d:
            d.set_matrix(A)
            d.setup()
            alone.append(d.precond_apply(r[off:off + 3 * A.n]))
        off += 3 * A.n
    with DeviceSolver(precond="bilu0", precision=precision) as d:
        d.set_batch(mats)
        d.setup()
        assert np.array_equal(d.precond_apply(r), np.concatenate(alone))


@pytest.mark.parametrize("precision", ["mixed", "mixed_f32"])
@pytest.mark.parametrize("form", [1, 2, 3])
def test_multicolour_slabs_match_the_block_kernel(precision, form):
    """The large colours' rows in slabs of 32 (a remainder, colours that do not start on a slab, a batch; rows longer than a
    slab's: cliques of 20 rows, which hold one row of each large colour) give the pre- and post-smoothing of the one-block
    application, which reads the rows where they lie: bit for bit."""
    from ressim_gb300.solver import DeviceSolver
    cliques = [(a, b) for g in range(3) for a in range(100 + 999 * g, 120 + 999 * g) for b in range(a + 1, 120 + 999 * g)]
    mats = [system(61 * 45 * 2 + k, box(61, 45, 2) + cliques + [(61 * 45 * 2 - 1, 61 * 45 * 2)] * k, seed=5 + k) for k in (0, 1)]
    r = np.random.default_rng(4).standard_normal(sum(3 * A.n for A in mats))
    z = []
    for opt in (dict(sweep="cta"), dict(sweep="split", vcycle_form=form)):
        with DeviceSolver(precond="cpr", precision=precision, **opt) as d:
            d.set_batch(mats)
            d.setup()
            z.append(d.precond_apply(r))
    assert np.isfinite(z[0]).all() and np.array_equal(z[0], z[1])


@pytest.mark.parametrize("name", ["star", "arrow", "clique", "two_colours", "long_rows", "slab"])
def test_grid_sweeps_long_rows(name, oracle):
    """The grid-wide sweeps at rows around the length from which a whole warp takes a row, and of one and several rounds of 32
    entries, alone, side by side and dependent on each other within a claim: FP64 and mixed bit for bit the oracle's (and the
    solve, whose input is fused, converges)."""
    from ressim_gb300.solver import DeviceSolver
    long_rows = [(k, 200 + j) for k in range(60) for j in range(5 + k)] + [(k, k + 1) for k in range(60)] + [(a, b) for a in range(300, 340) for b in range(a + 1, 340)]
    n, pairs = SHAPES.get(name, (345, long_rows))
    A = system(n, pairs, seed=9)
    r = np.random.default_rng(7).standard_normal(3 * n)
    ref = {"fp64": lambda: oracle.bilu0_apply(A, oracle.bilu0_factor(A)[0], r), "mixed": lambda: oracle.bilu0_apply_fd(A, oracle.bilu0_factor_lean(A)[0], r)}
    for precision in ("fp64", "mixed", "mixed_f32"):
        with DeviceSolver(precond="bilu0", precision=precision, sweep="grid") as d:
            d.set_matrix(A)
            d.setup()
            z = d.precond_apply(r)
            x, res = d.solve(r, tol=1e-8, maxit=100)
            assert res.converged
        if precision in ref:
            assert np.array_equal(z, ref[precision]())


@pytest.mark.parametrize("form", [1, 3])
@pytest.mark.parametrize("size", [31, 65, 150])
def test_small_colours_match_the_block_kernel(size, form):
    """Cliques whose rows take one, two and three rounds of the small colours' pass (64 entries a round), one system after
    another in a batch and over two applications: bit for bit the one-block application's."""
    from ressim_gb300.solver import DeviceSolver
    clique = [(a, b) for a in range(50, 50 + size) for b in range(a + 1, 50 + size)]
    mats = [system(31 * 22 * 2 + k, box(31, 22, 2) + clique + [(31 * 22 * 2 - 1, 31 * 22 * 2)] * k, seed=11 + k) for k in (0, 1)]
    r = np.random.default_rng(8).standard_normal(sum(3 * A.n for A in mats))
    z = []
    for opt in (dict(sweep="cta"), dict(sweep="split", vcycle_form=form)):
        with DeviceSolver(precond="cpr", precision="mixed_f32", **opt) as d:
            d.set_batch(mats)
            d.setup()
            z.append(d.precond_apply(r))
            assert np.array_equal(d.precond_apply(r), z[-1])
    assert np.isfinite(z[0]).all() and np.array_equal(z[0], z[1])


def test_ring_steps_keep_their_records_until_every_lane_has_read_them(oracle):
    """A step's bytes in the ring are given back only when all lanes of a warp have read theirs: steps whose warps are partly
    filled and mix rows with and without overflow entries, many more steps than the ring holds, more systems than SMs, applied
    again and again -- the oracle's bits every time (FP32: the fixed-thread-count kernel's)."""
    from ressim_gb300.solver import DeviceSolver
    mats = []
    for k in range(170):
        m = 90 + k % 7                                                     # a band with long rows here and there: levels of a few rows
        pairs = [(i, i + d) for i in range(m) for d in (1, 9, 10) if i + d < m] + [(i, i + 5 + j) for i in range(k % 3, m, 11) for j in range(9) if i + 5 + j < m]
        mats.append(system(m, pairs, seed=k))
    r = np.random.default_rng(12).standard_normal(sum(3 * A.n for A in mats))
    off = np.concatenate([[0], np.cumsum([3 * A.n for A in mats])])
    z = {}
    for precision, threads in (("fp64", 0), ("mixed_f32", 0), ("mixed_f32", 256)):
        with DeviceSolver(precond="bilu0", precision=precision, sweep="cta", cpr2_threads=threads) as d:
            d.set_batch(mats)
            d.setup()
            z[precision, threads] = d.precond_apply(r)
            for _ in range(20 if not threads else 0):
                assert np.array_equal(d.precond_apply(r), z[precision, threads])
    for s, A in enumerate(mats):
        b = r[off[s]:off[s + 1]]
        assert np.array_equal(z["fp64", 0][off[s]:off[s + 1]], oracle.bilu0_apply(A, oracle.bilu0_factor(A)[0], b))
    assert np.array_equal(z["mixed_f32", 0], z["mixed_f32", 256])


@pytest.mark.parametrize("n", [1880, 1925, 1960, 2000, 2047, 2048, 2049, 2200, 2295, 2340])
def test_shared_memory_around_the_default_limit(n, oracle):
    """Systems whose vectors need just under 48 KB of dynamic shared memory, beside the kernels' static part: the one-block
    sweeps (24 n and 12 n bytes), the split form's stage with its staging buffers, the coarse V-cycle's vectors."""
    from ressim_gb300.solver import DeviceSolver
    for m, precision in ((n, "fp64"), (2 * n, "mixed_f32"), (n, "mixed_f32")):
        nx = 40
        pairs = [(i, i + 1) for i in range(m - 1) if (i + 1) % nx] + [(i, i + nx) for i in range(m - nx)]
        A = system(m, pairs, seed=6)
        r = np.random.default_rng(6).standard_normal(3 * m)
        z = []
        for opt in (dict(precond="bilu0", sweep="cta", cpr2_threads=256), dict(precond="bilu0", sweep="cta")):   # (the latter: the ring)
            with DeviceSolver(precision=precision, **opt) as d:
                d.set_matrix(A)
                d.setup()
                z.append(d.precond_apply(r))
        assert np.array_equal(z[0], z[1])
        z = []
        for opt in [dict(sweep="cta"), dict(sweep="auto")] + [dict(sweep="split", autotune=False, vcycle_form=3, cpr2_threads=t) for t in (128, 256, 512)]:
            with DeviceSolver(precond="cpr", precision=precision, **opt) as d:
                d.set_matrix(A)
                d.setup()
                z.append(d.precond_apply(r))
        assert np.isfinite(z[0]).all() and all(np.array_equal(z[0], v) for v in z[1:])


@pytest.mark.parametrize("cells", [9900, 10300, 10600, 10900, 11200, 11500])
def test_coarse_levels_around_the_default_limit(cells):
    """The same for the levels below the finest of one system, kept in shared memory by the split form (24 bytes a row)."""
    from ressim_gb300.solver import DeviceSolver
    ny = cells // 100
    A = system(20 * ny * 5, box(20, ny, 5), seed=8)
    r = np.random.default_rng(8).standard_normal(3 * A.n)
    z = []
    for form in (3, 2):
        with DeviceSolver(precond="cpr", vcycle_form=form) as d:
            d.set_matrix(A)
            d.setup()
            z.append(d.precond_apply(r))
            assert 1700 < d.amg_level_sizes()[0][1:].sum() < 2300
    assert np.isfinite(z[0]).all() and np.array_equal(z[0], z[1])


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_f32"])
def test_levels_in_flight_do_not_change_results(precision):
    """Persistent grids from one block on (sweep_inflight) give the factors and the application of the full one, bit for bit."""
    from ressim_gb300.solver import DeviceSolver
    A = system(33 * 40 * 3, box(33, 40, 3), seed=9)
    r = np.random.default_rng(9).standard_normal(3 * A.n)
    out = []
    for inflight in (0, 1, 2, 8):
        with DeviceSolver(precond="cpr", precision=precision, sweep="grid", sweep_inflight=inflight) as d:
            d.set_matrix(A)
            d.setup()
            out.append((d.factors(A.nnzb), d.precond_apply(r)))
    for f, z in out[1:]:
        assert np.array_equal(f, out[0][0]) and np.array_equal(z, out[0][1])


@pytest.mark.parametrize("precond", ["bilu0", "cpr"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_large_batches_of_fp64_vectors(precision, precond, oracle):
    """FP64 vectors of more than 2,000 rows go through the ring in large batches and over the whole GPU in small ones: the
    same bits, and the oracle's."""
    from ressim_gb300.solver import DeviceSolver
    kinds = [system(2600 + k, box(20, 13, 10) + [(2599, 2600)] * (k > 0), seed=k) for k in (0, 1)]
    r = np.random.default_rng(3).standard_normal(3 * 150 * 2601)
    z = {}
    # (a CPR application with the sweeps of one block per system: sweep="grid" forms the second stage's input in another order)
    for copies, sweep, threads in ((150, "auto", 0), (150, "grid", 0) if precond == "bilu0" else (150, "split", 256), (3, "auto", 0)):
        mats = [kinds[k % 2] for k in range(copies)]
        N = sum(3 * A.n for A in mats)
        with DeviceSolver(precond=precond, precision=precision, sweep=sweep, cpr2_threads=threads) as d:
            d.set_batch(mats)
            d.setup()
            if precond == "cpr" and sweep == "auto":
                assert ("bilu0=ring" if copies == 150 else "bilu0=grid") in d.tuning()
            z[copies, sweep == "auto"] = d.precond_apply(r[:N])
    z = {(150, "auto"): z[150, True], (150, "other"): z[150, False], (3, "auto"): z[3, True]}
    N3 = z[3, "auto"].size
    assert np.array_equal(z[150, "auto"], z[150, "other"]) and np.array_equal(z[150, "auto"][:N3], z[3, "auto"])
    if precond == "bilu0":
        A = kinds[0]
        f, _ = (oracle.bilu0_factor if precision == "fp64" else oracle.bilu0_factor_lean)(A)
        ref = (oracle.bilu0_apply if precision == "fp64" else oracle.bilu0_apply_fd)(A, f, r[:3 * A.n])
        assert np.array_equal(z[150, "auto"][:3 * A.n], ref)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_f32"])
def test_factors_of_wide_levels(precision, oracle):
    """Batches whose levels are wide enough for a thread per row, with a singular pivot block in one kind of system and a claim
    that ends in the middle: the oracle's factors bit for bit, and its count of regularised blocks."""
    from ressim_gb300.solver import DeviceSolver
    kinds = [system(100 + k, box(5, 5, 4) + [(99, 100)] * k, seed=k) for k in (0, 1)] + [system(100, box(5, 5, 4), seed=7)]
    v = kinds[2].val.reshape(-1, 9)
    v[0] = 0.0                                                             # block (0, 0): nothing is eliminated from it
    copies = 1303
    mats = [kinds[k % 3] for k in range(copies)]
    with DeviceSolver(precond="bilu0", precision=precision) as d:
        d.set_batch(mats)
        d.setup()
        f = d.factors(sum(A.nnzb for A in mats))
        reg = d.stats().regularised_blocks
    ref = [{"fp64": oracle.bilu0_factor, "mixed": oracle.bilu0_factor_lean, "mixed_f32": oracle.bilu0_factor_f32}[precision](A) for A in kinds]
    assert reg == sum(ref[k % 3][1] for k in range(copies)) >= copies // 3
    assert np.array_equal(f, np.concatenate([ref[k % 3][0].reshape(-1) for k in range(copies)]).reshape(f.shape))


@pytest.mark.parametrize("n", [1, 85, 86, 207530, 207531, 300001])
def test_product_on_the_callers_vectors(n):
    """The permutations into and out of level space at one word a thread, at the line where the grid no longer covers the vector
    in one round (207,531 rows on 152 SMs) and beyond it with a remainder: a diagonal system's product, exact."""
    from ressim_gb300.solver import DeviceSolver
    from ressim_gb300.bsr import BSR
    rng = np.random.default_rng(n)
    val = np.zeros((n, 3, 3))
    val[:, np.arange(3), np.arange(3)] = rng.standard_normal((n, 3))
    order = rng.permutation(n)                                             # couplings that reverse the row order within levels
    x = rng.standard_normal((n, 3))
    pairs = [] if n < 1000 else [(int(min(a, b)), int(max(a, b))) for a, b in zip(order[:500], order[500:1000]) if a != b]
    rows = np.concatenate([np.arange(n), [p[0] for p in pairs], [p[1] for p in pairs]]).astype(np.int64)
    cols = np.concatenate([np.arange(n), [p[1] for p in pairs], [p[0] for p in pairs]]).astype(np.int64)
    o = np.lexsort((cols, rows))
    v = np.concatenate([val, np.zeros((2 * len(pairs), 3, 3))])[o]
    A = BSR(n, 3, np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32), cols[o].astype(np.int32), v.reshape(-1))
    with DeviceSolver(precond="bilu0") as d:
        d.set_matrix(A)
        y = d.spmv(x.reshape(-1))
    assert np.array_equal(y, (val[:, np.arange(3), np.arange(3)] * x).reshape(-1))
