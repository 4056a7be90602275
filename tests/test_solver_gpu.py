"""The fused device solver against the reference's solve_iceflow (golden
vectors made from the reference source) and against the oracle."""

import numpy as np
import pytest
import torch

from igm_b200 import _lib as L
from igm_b200.solver import DeviceAdamSolver
from oracle import iceflow_oracle as O
from tests.gpu_util import dev, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,nsolve", [("f64", 3), ("f32", 2)])
def test_solver_sequence_matches_reference(golden, case, nsolve):
    """Three solves on one optimizer: iteration counts (early stopping), the
    global Adam step counter, the COST history and U, V after each solve."""
    g = golden(f"solver_{case}")
    f64 = case == "f64"
    dt = torch.float64 if f64 else torch.float32
    thk, usurf, A, c = (dev(g[k], dt) for k in ["thk", "usurf", "arrhenius", "slidingco"])
    nz = g["s0_U"].shape[0]
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).to(dt))[1].numpy()
    solver = DeviceAdamSolver(lr=1.0)
    U = torch.zeros((nz,) + tuple(thk.shape), dtype=dt, device="cuda")
    V = torch.zeros_like(U)
    for s in range(nsolve):
        U, V, costs = solver.solve(U, V, thk, usurf, A, c, float(g["dx"]), dz, nbitmax=int(g["nbitmax"]))
        ref_costs = g[f"s{s}_costs"]
        assert len(costs) == len(ref_costs), (len(costs), len(ref_costs))
        assert solver.iterations == int(g[f"s{s}_iterations_after"])
        # FP32: the trajectory's sensitivity (see test_fp32_solver_error_against_fp64)
        np.testing.assert_allclose(costs, ref_costs, rtol=1e-9 if f64 else 1e-4,
                                   atol=(1e-9 if f64 else 1e-4) * np.abs(ref_costs).max())
        e = max(rel_l2(U.cpu().numpy(), g[f"s{s}_U"]), rel_l2(V.cpu().numpy(), g[f"s{s}_V"]))
        assert e < (1e-9 if f64 else 1e-2), e


def _oracle_solve(st, nz, dt, n):
    f = [torch.as_tensor(st[k]).to(dt) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).to(dt))[1]
    Z = torch.zeros((nz,) + tuple(f[0].shape), dtype=dt)
    U, V, c = O.solve_iceflow(Z, Z, *f, 100.0, dz, O.KerasLegacyAdam(lr=1.0), nbitmax=n, early_stopping=False)
    return np.concatenate([U.double().numpy().ravel(), V.double().numpy().ravel()]), c


def _device_solve(st, nz, dt, n):
    f = [dev(st[k], dt) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).to(dt))[1].numpy()
    Z = torch.zeros((nz,) + tuple(f[0].shape), dtype=dt, device="cuda")
    U, V, c = DeviceAdamSolver().solve(Z, Z, *f, 100.0, dz, nbitmax=n, early_stopping=False)
    return np.concatenate([U.double().cpu().numpy().ravel(), V.double().cpu().numpy().ravel()]), c


@pytest.mark.parametrize("n", [1, 10, 30])
def test_fp64_solver_matches_fp64_oracle(n):
    st = O.valley_glacier(40, 36, 100.0, seed=2)
    ref, cref = _oracle_solve(st, 10, torch.float64, n)
    got, c = _device_solve(st, 10, torch.float64, n)
    assert rel_l2(got, ref) < 1e-8, rel_l2(got, ref)
    np.testing.assert_allclose(c, cref, rtol=1e-10)


def test_fp64_solver_100_iterations_within_sensitivity():
    """After 100 iterations a 1e-15 relative perturbation of the inputs moves
    the FP64 oracle solution by ~3e-4 (the trajectory amplifies round-off), so
    the device FP64 solve is bounded by that sensitivity."""
    st = O.valley_glacier(40, 36, 100.0, seed=2)
    ref, cref = _oracle_solve(st, 10, torch.float64, 100)
    rng = np.random.default_rng(0)
    pert = {k: (v * (1 + 1e-15 * rng.standard_normal(v.shape))) if k in ("thk", "usurf", "arrhenius", "slidingco") else v
            for k, v in {k: np.asarray(st[k], np.float64) for k in ("thk", "usurf", "arrhenius", "slidingco")}.items()}
    refp, cpert = _oracle_solve(pert, 10, torch.float64, 100)
    sens = rel_l2(refp, ref)
    got, c = _device_solve(st, 10, torch.float64, 100)
    e = rel_l2(got, ref)
    print(f"device FP64 vs oracle FP64 after 100 iterations: {e:.3e}; oracle sensitivity to 1e-15 input noise: {sens:.3e}")
    assert e <= 10 * sens + 1e-9, (e, sens)
    spread = max(abs(cpert[-1] - cref[-1]), 1e-9 * abs(cref[-1]))
    print(f"final COST: device {c[-1]:.6f}, oracle {cref[-1]:.6f}, perturbed oracle {cpert[-1]:.6f}")
    assert abs(c[-1] - cref[-1]) <= 10 * spread + 1e-3 * abs(cref[-1])


@pytest.mark.parametrize("n", [1, 10, 100])
def test_fp32_solver_error_against_fp64(n):
    """Adam at lr = 1 amplifies rounding (a 1e-7 relative perturbation of the
    inputs moves the FP64 solution by ~3e-3 after 100 iterations), so the FP32
    result is judged against the FP64 oracle relative to the reference
    algorithm's own FP32 error: |U32 - U64| <= 3 |U32_oracle - U64_oracle| + 1e-6."""
    st = O.valley_glacier(40, 36, 100.0, seed=2)
    ref64, c64 = _oracle_solve(st, 10, torch.float64, n)
    ref32, _ = _oracle_solve(st, 10, torch.float32, n)
    got, c = _device_solve(st, 10, torch.float32, n)
    e_dev, e_ref = rel_l2(got, ref64), rel_l2(ref32, ref64)
    print(f"n={n}: device FP32 vs FP64 {e_dev:.3e}; reference algorithm FP32 vs FP64 {e_ref:.3e}")
    assert e_dev <= 3 * e_ref + 1e-6, (e_dev, e_ref)
    _, c32 = _oracle_solve(st, 10, torch.float32, n)
    assert abs(c[-1] - c64[-1]) <= 3 * abs(c32[-1] - c64[-1]) + 1e-5 * abs(c64[-1])


def test_nan_input_stops_with_status():
    st = O.valley_glacier(20, 20, 100.0, seed=1)
    st["thk"][5, 5] = np.nan
    dz = O.compute_zeta_dzeta(O.compute_levels(5, 4.0))[1].numpy()
    Z = torch.zeros((5, 20, 20), device="cuda")
    with pytest.raises(L.IgmError) as ei:
        DeviceAdamSolver().solve(Z, Z, *[dev(st[k]) for k in ["thk", "usurf", "arrhenius", "slidingco"]], 100.0, dz,
                                 nbitmax=20)
    assert ei.value.status == 3


def test_max_iter_caps_and_no_early_stop():
    st = O.valley_glacier(20, 24, 100.0, seed=1)
    dz = O.compute_zeta_dzeta(O.compute_levels(5, 4.0))[1].numpy()
    Z = torch.zeros((5, 20, 24), device="cuda")
    s = DeviceAdamSolver()
    _, _, c = s.solve(Z, Z, *[dev(st[k]) for k in ["thk", "usurf", "arrhenius", "slidingco"]], 100.0, dz,
                      nbitmax=7, early_stopping=False)
    assert len(c) == 7 and s.iterations == 7


def test_fp32_solver_matches_fp32_oracle_to_1e5():
    """FP32 against the FP32 restatement of the reference solver on the same
    inputs, relative L2 of the velocities <= 1e-5, after one iteration -- the
    number of iterations at which that bound is well posed: Adam at lr 1
    moves each velocity by about +-1 per iteration with the sign of its
    gradient, so a rounding difference that flips a near-zero gradient moves
    that node by a full step.  Measured on the oracle alone (this glacier,
    relative L2 of the solution after a 1e-7 relative perturbation of the
    inputs): 3.8e-6 after 1 iteration, 8.6e-5 after 3 and 4.4e-4 after 10;
    beyond one iteration parity is held by
    test_fp32_solver_error_against_fp64 against that sensitivity."""
    st = O.valley_glacier(40, 36, 100.0, seed=2)
    ref, cref = _oracle_solve(st, 10, torch.float32, 1)
    got, c = _device_solve(st, 10, torch.float32, 1)
    e = rel_l2(got, ref)
    print(f"one iteration: device FP32 vs oracle FP32 {e:.3e}")
    assert e <= 1e-5, e
    np.testing.assert_allclose(c, cref, rtol=1e-5)


@pytest.mark.parametrize("n", [0, 1, 2, 5])
@pytest.mark.parametrize("offset", [0, 1])
def test_start_is_read_in_place(n, offset):
    """A solve reads its start where it lies (copied when it is not 16-byte
    aligned) and leaves it unchanged, whatever the number of iterations'
    parity; without ice the gradient and the step are zero.  Against the
    solve in single iterations' entry point from copies and zeroed moments."""
    import ctypes as C
    from igm_b200.kernels import fields_struct, workspace
    st = O.valley_glacier(40, 36, 100.0, seed=4, varying_coeffs=True)
    f = [dev(st[k], torch.float32) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    nz = 6
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0))[1].numpy()
    rng = np.random.default_rng(3)
    base = torch.as_tensor(rng.normal(20, 10, (2, nz * 40 * 36 + 1)).astype(np.float32)).cuda()
    U, V = (base[i, offset:offset + nz * 40 * 36].view(nz, 40, 36) for i in range(2))
    U *= f[0] > 0
    V *= f[0] > 0
    keep = base.clone()
    s = DeviceAdamSolver()
    s.iterations = 3
    Ur, Vr, costs = s.solve(U, V, *f, 100.0, dz, nbitmax=n, early_stopping=False)
    assert torch.equal(base, keep) and len(costs) == n and s.iterations == 3 + n
    g, ph, fs = L.make_grid(1, nz, 40, 36, 100.0, dz), L.make_physics(), fields_struct(*f)
    W = [U.clone(), V.clone(), torch.empty_like(U), torch.empty_like(V)] + [torch.zeros_like(U) for _ in range(4)]
    ctl = torch.zeros(C.sizeof(L.SolverCtl), dtype=torch.uint8, device="cuda")
    cs = torch.zeros(max(n, 1), dtype=torch.float64, device="cuda")
    es = L.EarlyStop()
    wp, wn = workspace("cuda").get(g, U.device)
    lib, stream = L.lib(), L.stream_ptr()
    L.check(lib.igm_solver_begin(L.ptr(ctl), 3, stream))
    L.check(lib.igm_solver_iterate(0, C.byref(g), C.byref(ph), C.byref(fs), *[L.ptr(w) for w in W], C.byref(s.adam),
                                   C.byref(es), n, max(n, 1), L.ptr(ctl), L.ptr(cs), wp, wn, stream))
    ice = f[0] > 0
    for got, ref in zip((Ur, Vr), W[2 * (n % 2):2 * (n % 2) + 2]):
        assert torch.equal(got, torch.where(ice, ref, torch.zeros_like(ref)))
    np.testing.assert_array_equal(costs, cs.cpu().numpy()[:n])


def test_zero_epsilon_without_a_gradient_is_not_a_number():
    """Adam's step 0 / (sqrt(0) + 0) of a node whose gradient is zero: with
    epsilon 0 the solve stops, as the division gives it."""
    st = O.valley_glacier(40, 36, 100.0, seed=4)
    dz = O.compute_zeta_dzeta(O.compute_levels(5, 4.0))[1].numpy()
    Z = torch.zeros((5, 40, 36), device="cuda")
    f = [dev(st[k]) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    assert not bool((f[0] > 0).all())
    with pytest.raises(L.IgmError) as ei:
        DeviceAdamSolver(epsilon=0.0).solve(Z, Z, *f, 100.0, dz, nbitmax=5)
    assert ei.value.status == 3


def test_lazily_negated_start():
    """A start whose memory holds the opposite sign (a negated view) is copied."""
    st = O.valley_glacier(40, 36, 100.0, seed=4)
    dz = O.compute_zeta_dzeta(O.compute_levels(5, 4.0))[1].numpy()
    f = [dev(st[k]) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    U = torch.randn(5, 40, 36, device="cuda") * 10
    got, ref = (DeviceAdamSolver().solve(s, s, *f, 100.0, dz, nbitmax=2) for s in (torch._neg_view(U), -U))
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
