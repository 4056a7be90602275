"""The plain solver on the device (igm/processes/iceflow/solve/solve.py:11-119).

One fused kernel per iteration (energy + adjoint + Keras-legacy Adam +
FP64 reduction + EarlyStopping); the whole solve is enqueued without host
synchronisation and the host reads the 64-byte control block once at the end.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _lib as L
from .kernels import fields_struct, workspace


class DeviceAdamSolver:
    """Minimises the Blatter-Pattyn energy over (U, V) with Adam.

    ``iterations`` mirrors Keras' ``optimizer.iterations``: it is global to the
    solver object and carries over between solves (the bias correction uses
    it), while the moment slots start from zero at every solve, as the
    reference's fresh ``tf.Variable(U)`` get fresh slots (solve.py:27-28)."""

    def __init__(self, lr=1.0, beta_1=0.9, beta_2=0.999, epsilon=1e-7):
        self.adam = L.Adam()
        self.adam.lr, self.adam.beta_1, self.adam.beta_2, self.adam.epsilon = lr, beta_1, beta_2, epsilon
        self.iterations = 0
        self.last_costs = np.zeros(0)
        self.last_status = 0

    def solve(self, U, V, thk, usurf, arrhenius, slidingco, dx, dzeta, nbitmax=100, phys=None,
              relative_min_delta=0.0002, patience=10, early_stopping=True, mask=True):
        """Returns (U, V, costs) with U, V [Nz, Ny, Nx] (or [B, Nz, Ny, Nx])
        masked to zero where thk == 0 (solve.py:116-117) when ``mask``."""
        batched = U.dim() == 4
        U4 = U if batched else U[None]
        V4 = V if batched else V[None]
        f2 = [t if batched else t[None] for t in (thk, usurf, arrhenius, slidingco)]
        B, nz, ny, nx = U4.shape
        dev = U.device
        g = L.make_grid(B, nz, ny, nx, dx, dzeta)
        ph = phys if isinstance(phys, L.Physics) else L.make_physics(phys)
        # the start is read where it lies (iteration 0 reads it, later ones the two working pairs)
        # unless a copy is needed for its layout, its alignment or a negation that is still to be done
        U4, V4 = (t if t.is_contiguous() and t.data_ptr() % 16 == 0 and not t.is_neg() else t.clone() for t in (U4, V4))
        U0, V0, U1, V1, mU, mV, vU, vV = (torch.empty_like(U4) for _ in range(8))
        # control block and costs in one buffer: one copy to the host
        nctl = (C.sizeof(L.SolverCtl) + 63) // 64 * 64
        rec = torch.empty(nctl + 8 * max(int(nbitmax), 1), dtype=torch.uint8, device=dev)
        ctl, costs = rec.data_ptr(), rec.data_ptr() + nctl
        es = L.EarlyStop()
        es.relative_min_delta, es.patience, es.enabled = float(relative_min_delta), int(patience), int(bool(early_stopping))
        f = fields_struct(*f2)  # (refuses tensors that are not on the device)
        st = L.stream_ptr()
        ws = workspace(dev, st)  # held until the solve has ended
        wp, wn = ws.get(g, dev)
        lib = L.lib()
        if nbitmax > 0:
            rc = lib.igm_solver_solve(L.dtype_code(U.dtype), C.byref(g), C.byref(ph), C.byref(f), L.ptr(U4), L.ptr(V4),
                                      L.ptr(U0), L.ptr(V0), L.ptr(U1), L.ptr(V1), L.ptr(mU), L.ptr(mV), L.ptr(vU),
                                      L.ptr(vV), C.byref(self.adam), C.byref(es), int(self.iterations), int(nbitmax),
                                      ctl, costs, wp, wn, st)
            L.check(rc, "igm_solver_solve")
        else:
            L.check(lib.igm_solver_begin(ctl, int(self.iterations), st), "igm_solver_begin")
            U0, V0 = U4.clone(), V4.clone()
        host = rec.cpu().numpy()
        hc = L.SolverCtl.from_buffer_copy(host[:nctl].tobytes())
        n = int(hc.iter)
        self.iterations += n
        self.last_status = int(hc.status)
        self.last_costs = host[nctl:nctl + 8 * n].view(np.float64).copy()
        if hc.status != 0:
            raise L.IgmError(hc.status, f"solver stopped at iteration {n}: non-finite energy")
        Ur, Vr = (U0, V0) if n % 2 == 0 else (U1, V1)
        if mask:
            w = (C.c_double * nz)(*([0.0] * nz))
            rc = lib.igm_velocity_reduce(L.dtype_code(U.dtype), B, nz, ny, nx, L.ptr(Ur), L.ptr(Vr), L.ptr(f2[0]), 1, w,
                                         None, None, None, None, None, None, None, st)
            L.check(rc, "igm_velocity_reduce(mask)")
        if not batched:
            Ur, Vr = Ur[0], Vr[0]
        return Ur, Vr, self.last_costs
