"""smb_simple process (igm/processes/smb_simple/smb_simple.py:10-50):
ELA mass balance from a [time, gradabl, gradacc, ela, maxacc] table."""

from __future__ import annotations

from bisect import bisect_right
from math import isfinite

import numpy as np

from .. import kernels as K
from .. import state as S


def _interp1d(xs, ys, x):
    """interp1d_tf (igm/utils/math/interp1d_tf.py): piecewise linear, constant
    outside the table."""
    x = np.clip(float(x), float(np.min(xs)), float(np.max(xs)))
    return np.float32(np.interp(x, np.asarray(xs, np.float64), np.asarray(ys, np.float64)))


def _interp_row(table, x):
    """The columns 1 .. of ``table`` (float32 [rows, columns], column 0 the
    times) at time x, as _interp1d gives them: its arithmetic in Python floats
    for a short table of finite, increasing times, which costs a tenth of the
    array calls (16 us a column of a 40 us time step)."""
    if table.shape[0] <= 64:
        rows = table.tolist()
        t = [r[0] for r in rows]
        if all(a < b for a, b in zip(t, t[1:])) and all(map(isfinite, t)) and isfinite(x):
            if x <= t[0] or len(t) == 1:
                return [np.float32(v) for v in rows[0][1:]]
            if x >= t[-1]:
                return [np.float32(v) for v in rows[-1][1:]]
            j = bisect_right(t, x) - 1
            a, b = rows[j], rows[j + 1]
            if all(map(isfinite, a)) and all(map(isfinite, b)):
                dt, dx = b[0] - a[0], x - a[0]
                return [np.float32((v1 - v0) / dt * dx + v0) for v0, v1 in zip(a[1:], b[1:])]
    return [_interp1d(table[:, 0], table[:, k], x) for k in range(1, table.shape[1])]


def initialize(cfg, state):
    c = cfg.processes.smb_simple
    if len(c.array) == 0:
        state.smbpar = np.loadtxt(c.file, skiprows=1, dtype=np.float32)
    else:
        state.smbpar = np.array(c.array[1:]).astype(np.float32)
    state.smbpar = np.atleast_2d(state.smbpar)
    state.tlast_mb = -np.inf


def update(cfg, state):
    with S.update_scope(state):  # host-resident state: the results go back in one batch at the end
        _update(cfg, state)


def _update(cfg, state):
    c = cfg.processes.smb_simple
    t = float(state.t)
    if (t - float(state.tlast_mb)) >= c.update_freq:
        if hasattr(state, "logger"):
            state.logger.info("Construct mass balance at time : " + str(t))
        p = state.smbpar
        gradabl, gradacc, ela, maxacc = _interp_row(p[:, :5], t)
        usurf = S.get(state, "usurf")
        icemask = S.get(state, "icemask") if hasattr(state, "icemask") else None
        smb = K.smb_simple(usurf, gradabl, gradacc, ela, maxacc, icemask=icemask)
        S.put(state, "smb", smb)
        state.tlast_mb = t


def finalize(cfg, state):
    pass
