"""The FP64 step by fast convolution (sbe_conv.cu) at the edges of its size
classes (2..64, 65..128, 129..256, 257..512, 513..1024; odd sizes among them),
against the CPU oracle.

Tolerance 1e-12, derived: a transform of M <= 2048 points carries a rounding
error of about 2^-53 * 3 log2 M ~ 4e-15 of the largest sum; n <= 4 steps of 4
stages with h V / hbar < 1 add at most 16 of them (6e-14), and the oracle's own
sequential sums of Nk <= 1024 terms 2^-53 * 1024 ~ 1e-13 of theirs.
"""

import dataclasses

import numpy as np
import pytest
import torch
from helpers import HBAR, relerr

from oracle import oracle as orc
from pulsesuite_b200 import _lib, abi, device
from pulsesuite_b200 import grid as pgrid
from pulsesuite_b200.batch import WireBatch

pytestmark = pytest.mark.gpu

TOL = 1e-12
EDGES = [2, 3, 37, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024]


def any_grid(nk, kind):
    """A grid of any size: the synthetic wire's spacing law for kind "k0";
    distinct, decaying Veh, Vee, Vhh for kind "distinct"."""
    g = pgrid.wire_grid(64)
    dk = 6.0 / g.radius / max(nk, 16)
    kr = dk * (np.arange(nk) - (nk - 1) / 2.0)
    g = dataclasses.replace(g, nk=nk, dk=dk, kr=kr, L=np.pi / dk)
    q = np.maximum(np.arange(nk), 0.5) * dk * g.radius
    v = g.vprefactor * np.stack([np.exp(-0.3 * q), 1.2 * np.exp(-0.4 * q) / (1 + q),
                                 0.7 / (1 + q * q)])
    if kind != "distinct":
        v[:] = v[0]
    chi = [orc.chi1d_table(getattr(g, f"q{c}"), getattr(g, f"alpha{c}"), g.delta0,
                           getattr(g, f"m{c}"), g.chi_scale) for c in "eh"]
    return g, pgrid.table_block(g, *v, *chi)


def case(nks, kind, screened, seed=0):
    rng = np.random.default_rng(seed)
    gb = [any_grid(nk, kind) for nk in nks]
    grids, blocks = [g for g, _ in gb], [b for _, b in gb]
    tables, tabdata = pgrid.pack_tables(grids, blocks, screened=screened)
    w = np.zeros(len(nks), dtype=abi.WIRE_DTYPE)
    w["table"] = np.arange(len(nks))
    w["npulse"] = rng.integers(0, 3, len(nks))
    w["gap"] = rng.uniform(-1, 1, len(nks)) * 5e-21
    w["gamma"] = 1e13
    w["mscale"] = 4e-29
    w["pscale"] = 1.0
    w["amp"] = rng.uniform(1e7, 1e8, (len(nks), 2))
    w["t0"] = rng.uniform(0, 4e-15, (len(nks), 2))
    w["fwhm"] = 20e-15
    w["phase"] = rng.uniform(0, 6, (len(nks), 2))
    y = []
    for nk in nks:
        n = 0.4 * np.exp(-np.linspace(-2, 2, nk) ** 2) * rng.uniform(0.2, 1)
        p = np.sqrt(n * (1 - n)) * np.exp(1j * rng.uniform(0, 6, nk))
        y.append(np.stack([p.real, p.imag, n, 0.9 * n], 1))
    return grids, tables, tabdata, w, np.concatenate(y)


def batch(grids, tables, tabdata, w, y, screened, p_cap):
    b = WireBatch(grids, w, screened=screened, p_cap=p_cap, tables=tables,
                  tabdata=torch.as_tensor(tabdata, device="cuda"))
    b.set_state(y, y)
    return b


def oracle_wires(w, tables, p_cap):
    ww = w.copy()
    nks = tables["nk"][ww["table"]].astype(np.int64)
    ww["off"] = np.cumsum(nks) - nks
    ww["p_off"] = np.arange(len(ww)) * p_cap
    return ww


def compare(b, y, yo, nks):
    o = 0
    for nk in nks:
        a, r = y[o:o + nk], yo[o:o + nk]
        assert relerr(a[:, :2], r[:, :2]) < TOL and relerr(a[:, 2:], r[:, 2:]) < TOL, nk
        o += nk


@pytest.mark.parametrize("kind,screened", [("k0", False), ("k0", True), ("distinct", False),
                                           ("distinct", True)])
def test_rk4_at_class_edges(cuda, kind, screened):
    n, dt = 4, 1e-15
    grids, tables, tabdata, w, y0 = case(EDGES, kind, screened)
    b = batch(grids, tables, tabdata, w, y0, screened, n)
    b.rk4(n, dt)
    ww, yo = oracle_wires(w, tables, n), y0.reshape(-1).copy()
    Po = orc.rk4(tables, tabdata, ww, yo, n, dt, HBAR, p_stride=1, p_cap=n)
    assert (b.wires()["status"] == 0).all() and (b.wires()["steps"] == n).all()
    compare(b, b.state(), yo.reshape(-1, 4), EDGES)
    for i in range(len(EDGES)):
        assert relerr(b.records(i), Po.reshape(-1, n)[i]) < TOL, EDGES[i]


@pytest.mark.parametrize("kind,screened", [("k0", False), ("distinct", True)])
def test_leapfrog_at_class_edges(cuda, kind, screened):
    n, dt = 4, 2e-17
    grids, tables, tabdata, w, y0 = case(EDGES, kind, screened, seed=1)
    b = batch(grids, tables, tabdata, w, y0, screened, n)
    f = np.random.default_rng(2).uniform(-1e8, 1e8, (len(EDGES), 2 * n))
    b.leapfrog(torch.as_tensor(f, device="cuda"), n, dt)
    ww = oracle_wires(w, tables, n)
    y1, y2 = y0.reshape(-1).copy(), y0.reshape(-1).copy()
    orc.leapfrog(tables, tabdata, ww, y1, y2, f, n, dt, HBAR, p_stride=1, p_cap=n)
    compare(b, b.state(), y2.reshape(-1, 4), EDGES)
    compare(b, b.y1.cpu().numpy(), y1.reshape(-1, 4), EDGES)


@pytest.mark.parametrize("kind,screened", [("k0", True), ("distinct", False)])
def test_rhs_both_sides_of_the_direct_kernel(cuda, kind, screened):
    """One call over sizes of the direct kernel (<= 256) and of the transforms."""
    grids, tables, tabdata, w, y0 = case(EDGES, kind, screened, seed=3)
    b = batch(grids, tables, tabdata, w, y0, screened, 1)
    dy = b.rhs().cpu().numpy()
    ref = orc.rhs(tables, tabdata, oracle_wires(w, tables, 1), y0.reshape(-1), HBAR)
    assert (b.wires()["status"] == 0).all()
    compare(b, dy, ref.reshape(-1, 4), EDGES)


def test_mixed_launch_and_one_class(cuda):
    """One launch over every class gives each wire the bits of its own class's
    launch; a wire outside the class of a PSB_TAB_ONE_CLASS launch is refused."""
    n, dt = 3, 1e-15
    grids, tables, tabdata, w, y0 = case(EDGES, "k0", False, seed=4)
    b = batch(grids, tables, tabdata, w, y0, False, n)
    b.rk4(n, dt)
    c = batch(grids, tables, tabdata, w, y0, False, n)

    def launch(flags, nkmax):
        _lib.call("psb_rk4_f64", *c._common(), None, 0, device.ptr(c.y), c.n_state, nkmax, flags,
                  n, dt, device.ptr(c.P), c.P.shape[0], 1, c.p_cap, abi.as_ptr(c.model),
                  device.stream_ptr())

    launch(abi.PSB_TAB_SHARED_V, 1024)
    assert torch.equal(b.y, c.y) and torch.equal(b.P, c.P)
    launch(abi.PSB_TAB_SHARED_V | abi.PSB_TAB_ONE_CLASS, 1024)
    other = np.array(EDGES) <= 512
    assert (c.wires()["status"][other] == abi.PSB_ERR_SIZE).all()
    assert (c.wires()["status"][~other] == 0).all()
