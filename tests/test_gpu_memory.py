"""Device memory that runs out, and what a set-up reserves: a handle whose budget ends anywhere between its first array and its
last returns RSG_ENOMEM, and again when the call is repeated, never a solve on part of its arrays; a solve that
escalates to FP64 sweep vectors allocates nothing."""
import numpy as np
import pytest

from test_gpu_sweep_shapes import box, system

pytestmark = pytest.mark.gpu

ENOMEM, ESTATE = -3, -4


def code(call):
    from ressim_gb300._lib import RsgError
    try:
        call()
        return 0
    except RsgError as e:
        return e.code


FORMS = [dict(precond="bilu0", precision="fp64"), dict(precond="bilu0", precision="mixed"), dict(precond="bilu0", precision="mixed_f32"),
         dict(precond="cpr", precision="fp64"), dict(precond="cpr", precision="mixed_f32"), dict(precond="cpr", precision="mixed_f32", sweep="split"),
         dict(precond="cpr", precision="mixed_f32", sweep="cta"), dict(precond="cpr", precision="mixed", sweep="grid"),
         dict(precond="cpr", precision="mixed_f32", krylov="gmres", restart=10), dict(precond="cpr_device", precision="fp64")]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(str(v) for v in f.values()))
def test_budget_that_runs_out(form):
    from ressim_gb300.solver import DeviceSolver
    A = system(27 * 17 * 5, box(27, 17, 5), seed=2)                        # 2,295 rows: FP32 on the ring, FP64 vectors grid-wide
    b = np.random.default_rng(3).standard_normal(3 * A.n)
    with DeviceSolver(**form) as d:
        d.set_matrix(A)
        plan = d.stats().device_bytes
        d.setup()
        ready = d.stats().device_bytes
        ref = d.solve(b, 1e-8, 60)[0]
        full = d.stats().device_bytes
    assert plan < ready <= full
    budgets = sorted({*np.linspace(plan, ready, 40).astype(int).tolist(), *np.linspace(ready, full, 8).astype(int).tolist(), ready - 1, full - 1, full})
    seen = set()
    for budget in budgets:
        with DeviceSolver(**form, mem_budget=budget) as d:
            d.set_matrix(A)
            for _ in range(2):
                rc = code(d.setup)
                seen.add(rc)
                if rc:
                    assert rc == ENOMEM
                    assert code(lambda: d.solve(b, 1e-8, 60)) == ESTATE
            if rc == 0:
                rcs = [code(lambda: d.solve(b, 1e-8, 60)) for _ in range(2)]
                assert rcs in ([0, 0], [ENOMEM, ENOMEM])
                assert budget < full or rcs == [0, 0]
                if not rcs[0]:
                    assert np.array_equal(d.solve(b, 1e-8, 60)[0], ref)
    assert seen == {0, ENOMEM}


@pytest.mark.parametrize("precond", ["bilu0", "cpr"])
@pytest.mark.parametrize("sweep", ["auto", "grid", "split", "cta"])
@pytest.mark.parametrize("shape", [(9, 7, 5), (27, 17, 5), (33, 40, 10)])
def test_escalation_takes_no_memory(precond, sweep, shape):
    """Systems below and beyond the length to which FP64 vectors run on the ring, cut off after two iterations: the second
    attempt with FP64 sweep vectors runs within what the set-up held."""
    from ressim_gb300.solver import DeviceSolver
    if precond == "bilu0" and sweep == "split":
        pytest.skip("a form of CPR")
    nx, ny, nz = shape
    A = system(nx * ny * nz, box(nx, ny, nz), seed=4)
    b = np.random.default_rng(5).standard_normal(3 * A.n)
    opt = dict(precond=precond, precision="mixed_f32", sweep=sweep)
    with DeviceSolver(**opt) as d:
        d.set_matrix(A)
        d.setup()
        held = d.stats().device_bytes
    with DeviceSolver(**opt, mem_budget=held) as d:
        d.set_matrix(A)
        d.setup()
        for _ in range(2):
            d.setup()
            before = d.stats().device_bytes                                # (at most `held`: shapes tuned before are not tuned again)
            x, res = d.solve(b, tol=1e-13, maxit=2)
            assert not res.converged and d.stats().escalated_systems == 1 and np.isfinite(x).all()
            assert d.stats().device_bytes == before <= held


# what a handle held after a solve before the sweeps by value words, the ring and the slabs: a budget that was just enough
# for it still is (system, preconditioner, precision, sweep, Krylov method, bytes)
BUDGETS = [("box315", "bilu0", "fp64", "auto", "bicgstab", 729168), ("box315", "bilu0", "mixed_f32", "auto", "bicgstab", 728952),
           ("box315", "cpr", "fp64", "auto", "bicgstab", 2578728), ("box315", "cpr", "mixed_f32", "auto", "bicgstab", 2578444),
           ("box13k", "bilu0", "fp64", "auto", "bicgstab", 32368308), ("box13k", "bilu0", "fp64", "auto", "gmres", 39339124),
           ("box13k", "bilu0", "fp64", "grid", "bicgstab", 25609876), ("box13k", "bilu0", "mixed_f32", "auto", "bicgstab", 32643108),
           ("box13k", "bilu0", "mixed_f32", "auto", "gmres", 39613924), ("box13k", "bilu0", "mixed_f32", "grid", "bicgstab", 29263876),
           ("box13k", "cpr", "fp64", "auto", "bicgstab", 47553864), ("box13k", "cpr", "fp64", "auto", "gmres", 54524680),
           ("box13k", "cpr", "fp64", "grid", "bicgstab", 40795432), ("box13k", "cpr", "fp64", "split", "bicgstab", 47553864),
           ("box13k", "cpr", "mixed_f32", "auto", "bicgstab", 48073480), ("box13k", "cpr", "mixed_f32", "auto", "gmres", 55044296),
           ("box13k", "cpr", "mixed_f32", "grid", "bicgstab", 44694248), ("box13k", "cpr", "mixed_f32", "split", "bicgstab", 48073480),
           ("box13k", "cpr_device", "fp64", "auto", "bicgstab", 35943664), ("box13k", "cpr_device", "fp64", "auto", "gmres", 42914480),
           ("box13k", "cpr_device", "mixed_f32", "auto", "bicgstab", 36188480), ("box13k", "cpr_device", "mixed_f32", "auto", "gmres", 43159296),
           ("box2295c", "cpr", "fp64", "auto", "bicgstab", 11848668), ("box2295c", "cpr", "fp64", "grid", "bicgstab", 10427460),
           ("box2295c", "cpr", "mixed_f32", "auto", "bicgstab", 11907448), ("box2295c", "cpr", "mixed_f32", "grid", "bicgstab", 11196844)]
CLIQUE = [(a, b) for a in range(50, 110) for b in range(a + 1, 110)]


@pytest.mark.parametrize("case", BUDGETS, ids=lambda c: "-".join(c[:5]))
def test_budgets_that_were_enough(case):
    from ressim_gb300.solver import DeviceSolver
    name, precond, precision, sweep, krylov, budget = case
    n, pairs = {"box315": (315, box(9, 7, 5)), "box13k": (13200, box(33, 40, 10)), "box2295c": (2295, box(27, 17, 5) + CLIQUE)}[name]
    A = system(n, pairs, seed=1)
    with DeviceSolver(precond=precond, precision=precision, sweep=sweep, krylov=krylov, restart=10, mem_budget=budget) as d:
        d.set_matrix(A)
        d.setup()
        d.solve(np.ones(3 * n), 1e-6, 2)
        assert d.stats().device_bytes <= budget
