"""Energy and hand-written adjoint kernels (through the C ABI) against the
golden vectors of the reference source and against the oracle.

Tolerances: FP64 kernels to 1e-11 relative; FP32 energy terms to 1e-5
relative; FP32 gradients to 1e-5 relative L2 over the field."""

import numpy as np
import pytest
import torch

from igm_b200 import kernels as K
from oracle import iceflow_oracle as O
from tests.gpu_util import dev, rel_l2

pytestmark = pytest.mark.gpu

CASES = ["small_f64", "small_f32", "nz2_f64", "mid_f32", "mid_f64", "nz16_f64"]


def run(g, grad=True, scale=None):
    f64 = g["U"].dtype == np.float64
    dt = torch.float64 if f64 else torch.float32
    args = [dev(g[k], dt) for k in ["U", "V", "thk", "usurf", "arrhenius", "slidingco"]]
    ns = (g["thk"].shape[0] - 1) * (g["thk"].shape[1] - 1)
    terms, dU, dV = K.energy(*args, float(g["dx"]), g["dzeta"], grad=grad, grad_scale=1.0 / ns if scale is None else scale)
    return terms.cpu().numpy(), dU, dV, ns


@pytest.mark.parametrize("case", CASES)
def test_energy_terms_match_reference(golden, case):
    g = golden(f"energy_{case}")
    terms, _, _, ns = run(g, grad=False)
    tol = 1e-11 if g["U"].dtype == np.float64 else 1e-5
    means = terms / ns
    np.testing.assert_allclose(means, g["means"], rtol=tol, atol=tol * np.abs(g["means"]).max())
    np.testing.assert_allclose(means.sum(), float(g["cost"]), rtol=tol)


@pytest.mark.parametrize("case", CASES)
def test_adjoint_matches_reference_autodiff(golden, case):
    g = golden(f"energy_{case}")
    terms, dU, dV, ns = run(g, grad=True)
    f64 = g["U"].dtype == np.float64
    tol = 1e-11 if f64 else 1e-5
    assert rel_l2(dU.cpu().numpy(), g["gradU"]) < tol
    assert rel_l2(dV.cpu().numpy(), g["gradV"]) < tol
    np.testing.assert_allclose(terms / ns, g["means"], rtol=tol, atol=tol * np.abs(g["means"]).max())


def test_adjoint_central_differences():
    """Central finite differences of the FP64 energy at random nodes
    (eps = 1e-3 m/a) against the FP64 adjoint."""
    st = O.valley_glacier(48, 40, 100.0, seed=3, varying_coeffs=True)
    nz = 10
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).double())[1].numpy()
    rng = np.random.default_rng(0)
    U = rng.normal(20, 15, (nz, 48, 40))
    V = rng.normal(-5, 15, (nz, 48, 40))
    f = [dev(st[k], torch.float64) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    Ud, Vd = dev(U, torch.float64), dev(V, torch.float64)
    _, dU, dV = K.energy(Ud, Vd, *f, 100.0, dz, grad=True, grad_scale=1.0)
    dU, dV = dU.cpu().numpy(), dV.cpu().numpy()
    eps = 1e-3
    errs = []
    for _ in range(200):
        k, j, i = rng.integers(0, nz), rng.integers(0, 48), rng.integers(0, 40)
        which = rng.integers(0, 2)
        base = (Ud if which == 0 else Vd)
        orig = float(base[k, j, i])
        base[k, j, i] = orig + eps
        ep = K.energy(Ud, Vd, *f, 100.0, dz)[0].sum().item()
        base[k, j, i] = orig - eps
        em = K.energy(Ud, Vd, *f, 100.0, dz)[0].sum().item()
        base[k, j, i] = orig
        fd = (ep - em) / (2 * eps)
        ad = (dU if which == 0 else dV)[k, j, i]
        errs.append(abs(fd - ad) / max(abs(ad), 1e-3))
    assert np.median(errs) < 1e-6 and np.max(errs) < 1e-3, (np.median(errs), np.max(errs))


@pytest.mark.parametrize("shape", [(2, 7, 5), (3, 33, 65), (1, 9, 12), (5, 40, 17), (10, 100, 100), (16, 23, 31)])
def test_odd_shapes_against_oracle(shape):
    nz, ny, nx = shape
    rng = np.random.default_rng(nz * 1000 + ny)
    st = O.valley_glacier(ny, nx, 100.0, seed=ny, varying_coeffs=True)
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).double())[1] if nz > 1 else torch.ones(1, dtype=torch.float64)
    U = rng.normal(30, 20, (nz, ny, nx))
    V = rng.normal(0, 20, (nz, ny, nx))
    fl = {k: torch.as_tensor(st[k]).double() for k in ["thk", "usurf", "arrhenius", "slidingco"]}
    cost, means, gU, gV = O.energy_and_grad(torch.as_tensor(U), torch.as_tensor(V), fl["thk"], fl["usurf"],
                                            fl["arrhenius"], fl["slidingco"], 100.0, dz)
    ns = (ny - 1) * (nx - 1)
    terms, dU, dV = K.energy(dev(U, torch.float64), dev(V, torch.float64), *[dev(fl[k]) for k in fl], 100.0,
                             dz.numpy(), grad=True, grad_scale=1.0 / ns)
    np.testing.assert_allclose(terms.cpu().numpy() / ns, torch.stack(means).numpy(), rtol=1e-11, atol=1e-9)
    assert rel_l2(dU.cpu().numpy(), gU.numpy()) < 1e-11
    assert rel_l2(dV.cpu().numpy(), gV.numpy()) < 1e-11
    # FP32 kernel against the FP64 oracle: the FP32 error is stated by this bound
    terms32, dU32, dV32 = K.energy(dev(U, torch.float32), dev(V, torch.float32),
                                   *[dev(fl[k], torch.float32) for k in fl], 100.0, dz.numpy(), grad=True,
                                   grad_scale=1.0 / ns)
    np.testing.assert_allclose(terms32.cpu().numpy() / ns, torch.stack(means).numpy(), rtol=1e-5,
                               atol=1e-5 * float(cost.abs()))
    assert rel_l2(dU32.cpu().numpy(), gU.numpy()) < 2e-5
    assert rel_l2(dV32.cpu().numpy(), gV.numpy()) < 2e-5


def test_batched_equals_separate():
    rng = np.random.default_rng(5)
    nz, ny, nx, B = 4, 21, 26, 3
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0))[1].numpy()
    sts = [O.valley_glacier(ny, nx, 100.0, seed=s, varying_coeffs=True) for s in range(B)]
    U = rng.normal(30, 20, (B, nz, ny, nx)).astype(np.float32)
    V = rng.normal(0, 20, (B, nz, ny, nx)).astype(np.float32)
    F = {k: np.stack([s[k] for s in sts]) for k in ["thk", "usurf", "arrhenius", "slidingco"]}
    tb, dUb, dVb = K.energy(dev(U), dev(V), *[dev(F[k]) for k in F], 100.0, dz, grad=True)
    tot = np.zeros(3)
    for b in range(B):
        t, dU, dV = K.energy(dev(U[b]), dev(V[b]), *[dev(F[k][b]) for k in F], 100.0, dz, grad=True)
        tot += t.cpu().numpy()
        np.testing.assert_array_equal(dU.cpu().numpy(), dUb[b].cpu().numpy())
    np.testing.assert_allclose(tb.cpu().numpy(), tot, rtol=1e-12)


def test_energy_reduction_is_deterministic():
    st = O.valley_glacier(300, 257, 50.0, seed=1, varying_coeffs=True)
    rng = np.random.default_rng(1)
    U = dev(rng.normal(30, 20, (10, 300, 257)).astype(np.float32))
    V = dev(rng.normal(0, 20, (10, 300, 257)).astype(np.float32))
    f = [dev(st[k]) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    dz = O.compute_zeta_dzeta(O.compute_levels(10, 4.0))[1].numpy()
    a = [K.energy(U, V, *f, 50.0, dz, grad=True) for _ in range(3)]
    for t, dU, dV in a[1:]:
        assert torch.equal(t, a[0][0]) and torch.equal(dU, a[0][1]) and torch.equal(dV, a[0][2])


@pytest.mark.parametrize("n,m,fnge", [(2.5, 2.0, False), (3.0, 3.0, True), (4.0, 1.5, True)])
def test_other_physics_against_oracle(n, m, fnge):
    """Glen and Weertman exponents other than 3 and the forced-negative
    gravitational energy take the kernel's general path (generic powers,
    per-layer gravity clamp); FP64 against the FP64 oracle."""
    nz, ny, nx = 6, 37, 45
    rng = np.random.default_rng(int(n * 10 + m))
    st = O.valley_glacier(ny, nx, 100.0, seed=7, varying_coeffs=True)
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).double())[1]
    U = rng.normal(30, 20, (nz, ny, nx))
    V = rng.normal(0, 20, (nz, ny, nx))
    fl = {k: torch.as_tensor(st[k]).double() for k in ["thk", "usurf", "arrhenius", "slidingco"]}
    ph = O.Physics(exp_glen=n, exp_weertman=m, force_negative_gravitational_energy=fnge)
    cost, means, gU, gV = O.energy_and_grad(torch.as_tensor(U), torch.as_tensor(V), fl["thk"], fl["usurf"],
                                            fl["arrhenius"], fl["slidingco"], 100.0, dz, ph)
    ns = (ny - 1) * (nx - 1)
    phys = dict(exp_glen=n, exp_weertman=m, force_negative_gravitational_energy=fnge)
    terms, dU, dV = K.energy(dev(U, torch.float64), dev(V, torch.float64), *[dev(fl[k]) for k in fl], 100.0,
                             dz.numpy(), phys, grad=True, grad_scale=1.0 / ns)
    np.testing.assert_allclose(terms.cpu().numpy() / ns, torch.stack(means).numpy(), rtol=1e-10,
                               atol=1e-10 * float(cost.abs()))
    assert rel_l2(dU.cpu().numpy(), gU.numpy()) < 1e-10
    assert rel_l2(dV.cpu().numpy(), gV.numpy()) < 1e-10


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("ice_rows,value", [((0, 0), 0.0), ((20, 21), 0.0), ((16, 48), 1e12), ((16, 48), float("nan")),
                                            ((16, 48), float("inf"))])
def test_bare_ground(dtype, ice_rows, value):
    """Cells without ice skip their layers: none, one or a third of the rows
    under ice, moving ground everywhere (sliding acts without ice too), and one
    off-ice node (row 60, level 2) with a value whose products overflow or are
    not finite, which must not be skipped.  Against autograd of the oracle in
    FP64; tolerances as above (2e-5 for the FP32 gradient against FP64)."""
    ny, nx, nz = 70, 66, 5
    st = O.valley_glacier(ny, nx, 100.0, seed=5, varying_coeffs=True)
    rng = np.random.default_rng(6)
    thk = np.zeros((ny, nx))
    thk[ice_rows[0]:ice_rows[1]] = rng.uniform(50, 150, (ice_rows[1] - ice_rows[0], nx))
    U, V = rng.normal(20, 10, (nz, ny, nx)), rng.normal(0, 10, (nz, ny, nx))
    if value:
        U[2, 60, 33] = value
    np_dt = np.float32 if dtype == torch.float32 else np.float64
    f64 = [np.asarray(a, np_dt).astype(np.float64) for a in (thk, st["topg"] + thk, st["arrhenius"], st["slidingco"])]
    U, V = U.astype(np_dt), V.astype(np_dt)
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).double())[1]
    ns = (ny - 1) * (nx - 1)
    terms, dU, dV = K.energy(dev(U, dtype), dev(V, dtype), *[dev(a, dtype) for a in f64], 100.0, dz.numpy(), grad=True,
                             grad_scale=1.0 / ns)
    terms2, _, _ = K.energy(dev(U, dtype), dev(V, dtype), *[dev(a, dtype) for a in f64], 100.0, dz.numpy())
    assert np.array_equal(terms.cpu().numpy(), terms2.cpu().numpy(), equal_nan=True)
    if not np.isfinite(value):
        assert not bool(torch.isfinite(terms.sum())) and not bool(torch.isfinite(dU).all())
        ok = torch.ones((ny, nx), dtype=torch.bool)
        ok[58:63, 31:36] = False
        assert bool(torch.isfinite(dU.cpu()[:, ok]).all())
        return
    cost, means, gU, gV = O.energy_and_grad(torch.as_tensor(U).double(), torch.as_tensor(V).double(),
                                            *[torch.as_tensor(a) for a in f64], 100.0, dz)
    tol = 1e-11 if dtype == torch.float64 else 2e-5
    np.testing.assert_allclose(terms.cpu().numpy() / ns, [float(m) for m in means], rtol=tol,
                               atol=tol * max(abs(float(m)) for m in means))
    assert rel_l2(dU.cpu().numpy(), gU.numpy()) < tol
    assert rel_l2(dV.cpu().numpy(), gV.numpy()) < tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("gout", [1.0, -0.37, 0.0])
def test_backward_scale_on_the_device(dtype, gout):
    """The autograd backward, whose scale is divided on the device, against
    the gradient with the same scale given by the host: the same bits."""
    from igm_b200.energy import iceflow_energy
    ny, nx, nz = 33, 41, 4
    st = O.valley_glacier(ny, nx, 100.0, seed=7, varying_coeffs=True)
    rng = np.random.default_rng(8)
    f = [dev(st[k], dtype) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).double())[1].numpy()
    U, V = (dev(rng.normal(5, 9, (nz, ny, nx)), dtype).requires_grad_(True) for _ in range(2))
    g = torch.tensor(gout, dtype=dtype, device="cuda")
    dU, dV = torch.autograd.grad(iceflow_energy(U, V, *f, 100.0, dz), [U, V], grad_outputs=g)
    _, rU, rV = K.energy(U.detach(), V.detach(), *f, 100.0, dz, grad=True, grad_scale=float(g) / ((ny - 1) * (nx - 1)))
    assert torch.equal(dU, rU) and torch.equal(dV, rV)


def test_a_thread_without_a_context():
    """The energy from a thread that has made no CUDA runtime call of its own
    (autograd's backward thread, with buffers from the caching allocator)."""
    import threading
    st = O.valley_glacier(33, 40, 100.0, seed=9)
    f = [dev(st[k], torch.float32) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    dz = O.compute_zeta_dzeta(O.compute_levels(4, 4.0))[1].numpy()
    U = torch.ones((4, 33, 40), device="cuda")
    ref = K.energy(U, U, *f, 100.0, dz, grad=True)
    keep = [torch.empty_like(U) for _ in range(4)]
    del keep  # freed blocks that the thread's allocations reuse
    got = []
    t = threading.Thread(target=lambda: got.append(K.energy(U, U, *f, 100.0, dz, grad=True, terms_out=torch.empty_like(ref[0]))))
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert len(got) == 1 and all(torch.equal(a, b) for a, b in zip(got[0], ref))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(1, 3, 2, 5), (2, 2, 16, 31), (1, 4, 17, 33), (1, 5, 31, 62), (3, 3, 15, 7), (1, 2, 40, 97),
                                   (2, 1, 33, 66), (1, 3, 47, 35)])
def test_16_byte_copies_against_element_copies(dtype, shape):
    """Widths whose rows do not start on 16-byte boundaries: the 16-byte copies
    of aligned arrays against the element copies that arrays off that alignment
    take, bit for bit: energy, gradient and three solver
    iterations, NaN around the arrays."""
    import ctypes as C
    B, nz, ny, nx = shape
    rng = np.random.default_rng(ny * nx)
    dz = O.compute_zeta_dzeta(O.compute_levels(max(nz, 2), 4.0).double())[1].numpy()[:max(nz - 1, 1)]
    thk = rng.uniform(0, 200, (B, ny, nx)) * (rng.random((B, ny, nx)) < 0.6)
    data = [rng.normal(20, 10, (B, nz, ny, nx)), rng.normal(0, 10, (B, nz, ny, nx)), thk, thk + rng.uniform(2000, 2100, thk.shape),
            rng.uniform(20, 150, thk.shape), rng.uniform(0.01, 0.1, thk.shape)]

    def place(a, off):  # the array's values `off` elements past a 16-byte boundary, NaN before and after
        buf = torch.full((a.size + 64,), float("nan"), dtype=dtype, device="cuda")
        v = buf[16 + off:16 + off + a.size]
        v.copy_(torch.as_tensor(a.reshape(-1)))
        return v.view(a.shape)

    got = []
    for off in (0, 1):
        U, V, *f = (place(a, off) for a in data)
        terms, dU, dV = K.energy(U, V, *f, 100.0, dz, grad=True, grad_scale=1e-3)
        terms2, _, _ = K.energy(U, V, *f, 100.0, dz)
        g, ph, fs = K.L.make_grid(B, nz, ny, nx, 100.0, dz), K.L.make_physics(), K.fields_struct(*f)
        W = [place(np.zeros(data[0].shape), off) for _ in range(8)]
        ctl = torch.zeros(C.sizeof(K.L.SolverCtl), dtype=torch.uint8, device="cuda")
        cs = torch.zeros(3, dtype=torch.float64, device="cuda")
        ad, es = K.L.Adam(), K.L.EarlyStop()
        ad.lr, ad.beta_1, ad.beta_2, ad.epsilon = 1.0, 0.9, 0.999, 1e-7
        wp, wn = K.workspace(U.device).get(g, U.device)
        K.L.check(K.L.lib().igm_solver_solve(K.L.dtype_code(dtype), C.byref(g), C.byref(ph), C.byref(fs), K.L.ptr(U), K.L.ptr(V),
                                             *[K.L.ptr(w) for w in W], C.byref(ad), C.byref(es), 0, 3, ctl.data_ptr(),
                                             cs.data_ptr(), wp, wn, K.L.stream_ptr()))
        torch.cuda.synchronize()
        assert int(K.L.SolverCtl.from_buffer_copy(ctl.cpu().numpy().tobytes()).iter) == 3
        got.append([terms, terms2, dU, dV, cs, *[w.clone() for w in W]])
    assert all(bool(torch.isfinite(t).all()) for t in got[0])
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("nx", [64, 66])
@pytest.mark.parametrize("what,value,level", [("U", float("nan"), 0), ("V", float("inf"), 0), ("U", 1e25, 0), ("U", float("nan"), 2),
                                              ("V", float("inf"), 4), ("arrhenius", float("nan"), 0), ("arrhenius", 0.0, 0),
                                              ("usurf", float("nan"), 0), ("usurf", float("inf"), 0),
                                              ("scale", float("nan"), 0), ("scale", float("inf"), 0), ("dzeta", float("nan"), 2)])
def test_bare_ground_hides_nothing(dtype, nx, what, value, level):
    """A value that is not finite far off the ice (row 60; ice in rows 16 ..
    47) shows in the same energy terms and at the same nodes of the gradient as
    with a trace of ice (1e-30 m) on the bare ground, where no layer is skipped."""
    ny, nz = 70, 5
    st = O.valley_glacier(ny, nx, 100.0, seed=5, varying_coeffs=True)
    rng = np.random.default_rng(6)
    ice = np.zeros((ny, nx))
    ice[16:48] = rng.uniform(50, 150, (32, nx))
    f = {"U": rng.normal(20, 10, (nz, ny, nx)), "V": rng.normal(0, 10, (nz, ny, nx)), "usurf": st["topg"] + ice,
         "arrhenius": np.array(st["arrhenius"], np.float64), "slidingco": st["slidingco"]}
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0).double())[1].numpy()
    scale = 1e-3
    if what == "scale":
        scale = value
    elif what == "dzeta":
        dz[level] = value
    else:
        f[what][(level, 60, 33) if what in "UV" else (60, 33)] = value
    got = []
    for thk in (ice, np.where(ice > 0, ice, 1e-30)):
        args = [dev(a, dtype) for a in (f["U"], f["V"], thk, f["usurf"], f["arrhenius"], f["slidingco"])]
        terms, dU, dV = K.energy(*args, 100.0, dz, grad=True, grad_scale=scale)
        only, _, _ = K.energy(*args, 100.0, dz)
        got.append([torch.isfinite(t).cpu() for t in (terms, only, dU, dV)])
    for i, (a, b) in enumerate(zip(*got)):
        assert torch.equal(a, b), (i, (a != b).nonzero()[:8].tolist())


def test_backward_of_a_lazily_negated_gradient():
    """The incoming gradient of an imaginary part of a conjugate is a view whose
    memory holds the opposite sign."""
    from igm_b200.energy import iceflow_energy
    ny, nx, nz = 17, 20, 3
    st = O.valley_glacier(ny, nx, 100.0, seed=7, varying_coeffs=True)
    rng = np.random.default_rng(8)
    f = [dev(st[k], torch.float32) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0))[1].numpy()
    U, V = (dev(rng.normal(5, 9, (nz, ny, nx)), torch.float32).requires_grad_(True) for _ in range(2))
    g = torch.complex(torch.zeros((), device="cuda"), torch.full((), 0.5, device="cuda")).conj().imag
    assert g.is_neg() and float(g) == -0.5
    got = torch.autograd.grad(iceflow_energy(U, V, *f, 100.0, dz), [U, V], grad_outputs=g)
    ref = torch.autograd.grad(iceflow_energy(U, V, *f, 100.0, dz), [U, V], grad_outputs=g.resolve_neg())
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


def test_two_streams_share_no_workspace():
    """Energies and gradients differentiated on two streams at once, without a
    wait between them, against one after another; then one more on each, whose
    scratch they must have left clean."""
    from igm_b200.energy import iceflow_energy
    streams = [torch.cuda.Stream() for _ in range(2)]
    sets, ref = [], []
    for s, n in enumerate((190, 230)):
        st = O.valley_glacier(n, n, 100.0, seed=s, varying_coeffs=True)
        rng = np.random.default_rng(s)
        f = [dev(st[k], torch.float32) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
        dz = O.compute_zeta_dzeta(O.compute_levels(6, 4.0))[1].numpy()
        U, V = (dev(rng.normal(5, 9, (6, n, n)), torch.float32).requires_grad_(True) for _ in range(2))
        sets.append((U, V, *f, 100.0, dz))
        c = iceflow_energy(*sets[s])
        ref.append((c.detach(), *torch.autograd.grad(c, [U, V])))
    with torch.cuda.stream(streams[0]):
        a = K.workspace(torch.device("cuda", 0))
    with torch.cuda.stream(streams[1]):
        b = K.workspace(torch.device("cuda", 0))
    assert a is not b and a is K.workspace(torch.device("cuda", 0), streams[0].cuda_stream)
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(25):
        for s, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                c = iceflow_energy(*sets[s])
                got[s].append((c.detach(), *torch.autograd.grad(c, sets[s][:2])))
    torch.cuda.synchronize()
    for s in range(2):
        for g in got[s]:
            assert all(torch.equal(x, y) for x, y in zip(g, ref[s]))
        with torch.cuda.stream(streams[s]):
            assert torch.equal(iceflow_energy(*sets[s]).detach(), ref[s][0])
    assert all(int(w.buf[:256].sum()) == 0 for w in (a, b))  # tickets and error word


def test_workspaces_are_bounded():
    dev0 = torch.device("cuda", 0)
    made = [K.workspace(dev0, -1 - i) for i in range(K.MAX_WORKSPACES + 3)]  # keys of no stream: nothing is launched
    assert len(K._WS) == K.MAX_WORKSPACES and K.workspace(dev0, -1) is not made[0]
    for i in range(K.MAX_WORKSPACES + 3):
        K._WS.pop((dev0, -1 - i), None)


def test_captured_energies():
    """Two graphs of an energy and its gradient, captured after a warm-up on
    another stream, replayed in turn with other inputs before any eager call on
    the capture's stream."""
    ny, nx, nz = 90, 100, 5
    st = O.valley_glacier(ny, nx, 100.0, seed=3, varying_coeffs=True)
    f = [dev(st[k], torch.float32) for k in ["thk", "usurf", "arrhenius", "slidingco"]]
    dz = O.compute_zeta_dzeta(O.compute_levels(nz, 4.0))[1].numpy()
    U, V = (torch.zeros((nz, ny, nx), device="cuda") for _ in range(2))
    K.energy(U, V, *f, 100.0, dz, grad=True)
    graphs, outs = [], []
    for _ in range(2):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            outs.append(K.energy(U, V, *f, 100.0, dz, grad=True))
    rng = np.random.default_rng(4)
    for g, out in list(zip(graphs, outs))[::-1] * 2:
        U.copy_(torch.as_tensor(rng.normal(20, 10, U.shape)))
        V.copy_(torch.as_tensor(rng.normal(0, 10, U.shape)))
        g.replay()
        ref = K.energy(U, V, *f, 100.0, dz, grad=True)
        assert all(torch.equal(a, b) for a, b in zip(out, ref))
