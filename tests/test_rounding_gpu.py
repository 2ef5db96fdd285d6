"""The step's branch-free quotients, reciprocals and square roots (div_rn, div_by, rcp_rn, sqrt_rn,
intpl1d_grid) against numpy's FP32, bit for bit: the tabulated physics at every node of the energy
grids and the floats beside it, between the nodes, at the ends of the tables and outside them."""
import os
import re

import numpy as np
import pytest

from moquimc_gb300 import build

pytestmark = pytest.mark.gpu

f = np.float32


def _table(name):
    text = open(os.path.join(build.CSRC, "mqi_tables.h")).read()
    body = re.search(name + r"\[[^\]]*\]\s*=\s*\{([^}]*)\}", text).group(1)
    return np.array([float.fromhex(x.strip().rstrip("f")) for x in body.split(",") if x.strip()], np.float32)


def _energies(where):
    nodes = np.concatenate([f(0.1) + np.arange(601, dtype=f) * f(0.5), np.arange(1, 602, dtype=f) * f(0.5)])
    if where == "nodes":
        e = [nodes]
        for to in (f(0), f(np.inf)):
            x = nodes
            for _ in range(3):
                x = np.nextafter(x, to)
                e.append(x)
        return np.unique(np.concatenate(e))
    if where == "between":
        return np.random.default_rng(3).uniform(0.1, 300.0, 200_001).astype(f)
    return np.array([1e-3, 0.05, 0.0999, 0.3, 0.4999, 299.6, 299.7, 300.0, 300.1, 1e3, 1e5], f)


def _lookup(tab, e, e_min, e_max, below):
    i0 = np.clip(((e - f(e_min)) / f(0.5)).astype(np.int64), 0, 599)
    i1 = np.minimum(i0 + 1, 599)
    x0 = f(e_min) + i0.astype(f) * f(0.5)
    x1 = x0 + f(0.5)
    v = tab[i0] + (e - x0) * (tab[i1] - tab[i0]) / (x1 - x0)
    return np.where((e >= f(e_min)) & (e <= f(e_max)), v, below)


@pytest.mark.parametrize("where", ["nodes", "between", "outside"])
def test_step_quotients_are_correctly_rounded(gpu_ctx_factory, where):
    e = _energies(where)
    got = gpu_ctx_factory().eval_physics(e)
    mp, me = f(938.272046), f(0.510998928)
    et = e + mp
    gamma = et / mp
    g2 = gamma * gamma
    r = f(1) / g2
    res = (1.0 - r.astype(np.float64) * g2.astype(np.float64)).astype(f)     # one FMA: exact in FP64, rounded once
    beta = (f(1) - r) - res * r
    ratio = me / mp
    te = f(2) * me * beta * g2 / (f(1) + f(2) * gamma * ratio + ratio * ratio)
    dedx = _table("mqi_tab_dedx")
    want = [_lookup(_table("mqi_tab_cs_p_ion"), e, 0.1, 299.6, f(0)), _lookup(_table("mqi_tab_cs_pp_e"), e, 0.5, 300.0, f(0)),
            _lookup(_table("mqi_tab_cs_po_e"), e, 0.5, 300.0, f(0)), _lookup(_table("mqi_tab_cs_po_i"), e, 0.5, 300.0, f(0)),
            -_lookup(dedx, e, 0.1, 299.6, np.where(e < f(0.1), dedx[0], f(0))), beta, te, np.sqrt(et * et - mp * mp)]
    for k, w in enumerate(want):
        assert w.dtype == np.float32
        np.testing.assert_array_equal(got[:, k], w)
