"""The dense LU of the coarsest level (one cluster of blocks, or one block, per system; columns on chip or in global memory) at
its edges: fewer rows than blocks, the line between the two memories (424 / 425 rows in FP64), the largest dense level, batches
beyond one cluster per system, small matrices in large batches, and elimination with interchanges and ties. The pressure
matrix of these systems is chosen entry by entry (blocks are multiples of the identity), against the oracle's CPR
application; the bound is that of the other CPR tests (the back substitution sums in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain_system(m, seed):
    """m rows of which a chain of min(m, 60) spread over the numbering is coupled, the others stand alone (coarsening stalls
    on them): diagonals 1 to 3 against off-diagonals up to 3 of opposite signs, so that the LU interchanges rows and meets
    ties, while ILU(0), which does not interchange, stays stable (every pivot is at least the diagonal)."""
    from ressim_gb300.bsr import BSR
    rng = np.random.default_rng([seed, m])
    ch = np.sort(rng.choice(m, min(m, 60), replace=False))
    up, lo = rng.integers(1, 4, ch.size - 1).astype(float), -rng.integers(1, 4, ch.size - 1).astype(float)
    rows = np.concatenate([np.arange(m), ch[:-1], ch[1:]])
    cols = np.concatenate([np.arange(m), ch[1:], ch[:-1]])
    val = np.concatenate([rng.integers(1, 4, m).astype(float), up, lo])
    order = np.lexsort((cols, rows))
    rows, cols, val = rows[order], cols[order], val[order]
    return BSR(m, 3, np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int32), cols.astype(np.int32),
               (val[:, None, None] * np.eye(3)).reshape(-1))


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_f32"])
@pytest.mark.parametrize("m,copies", [(1, 1), (5, 1), (9, 1), (60, 1), (225, 1), (424, 1), (425, 1), (620, 1), (800, 1), (60, 200), (130, 40), (225, 40),
                                      (425, 40), (300, 150)])
def test_coarse_lu_against_the_oracle(m, copies, precision, oracle):
    from ressim_gb300.solver import DeviceSolver
    kinds = [chain_system(m, seed) for seed in range(min(copies, 3))]
    mats = [kinds[k % len(kinds)] for k in range(copies)]
    r = np.random.default_rng(m).standard_normal((copies, 3 * m))
    with DeviceSolver(precond="cpr", precision=precision) as d:
        d.set_batch(mats)
        d.setup()
        rows, _, dense = d.amg_level_sizes()
        assert list(rows) == [copies * m] and dense == copies * m * m       # one level, dense
        z = d.precond_apply(r.reshape(-1)).reshape(copies, -1)
    bound = 1e-10 if precision == "fp64" else 1e-3
    for k in {0, 1 % copies, 2 % copies, copies - 1}:
        ref = oracle.prec_apply(mats[k], r[k], prec=1)
        assert np.linalg.norm(z[k] - ref) <= bound * np.linalg.norm(ref)
