"""Batched quantum-wire SBE engine: many wires of uneven k grids resident on
one GPU, advanced by the fused sm_100a step kernels.

    b = WireBatch(grids, wires, screened=False)
    P = b.rk4(nsteps, dt, p_stride=1)      # P(t) records, device tensor
    y = b.state()                           # (n_state, 4) float64 on the host

``wires`` is a numpy array of ``abi.WIRE_DTYPE``; ``table`` indexes
``grids``.  The batch assigns the state (``off``) and P(t) (``p_off``)
ranges.  Buffers are torch tensors on the current device; the step entry
points allocate nothing.
"""

import numpy as np
import torch
from scipy.constants import hbar

from . import _lib, abi, coulomb, device


def wire_cost(nk):
    """Time of one wire and stage in a full group of the per-wire split kernel,
    relative (2.2, 2.3, 2.9, 4.6, 10.7 us at Nk 64, 128, 256, 512, 1024)."""
    return 2.0 + 2.6e-3 * nk + 6.0e-6 * nk * nk


def wire_group(n, wmax, sms):
    """Wires per group of the per-wire split kernel for n wires of one grid on
    its share of the SMs: the fewest waves of CTAs times a CTA's time, which
    grows as w + 1 (Nk 512: one wire 8.8 us a stage, ten 50).  Against the
    largest group that a full wave of CTAs leaves, 8 steps of screened wires:
    1600 at Nk 512 3.37 -> 2.12 ms (2 waves of 6, not 2 of 10 with a second of
    12 CTAs), 16384 20.1 -> 19.2, 1024 of Nk 64..512 1.61 -> 1.11 (15 grids
    on ten SMs each, not one wire per CTA)."""
    sms = max(1, int(round(sms)))

    def time(w):
        return -(-(-(-n // w)) // sms) * (w + 1)

    return min(range(1, wmax + 1), key=lambda w: (time(w), -w))


def groups_of(table, wires, wg):
    """Split-form groups (SPLIT_GROUP_DTYPE) of wg of the given wires each, all
    of one table; the last holds what is left.  Unused slots are -1."""
    g = np.zeros(-(-len(wires) // wg), dtype=abi.SPLIT_GROUP_DTYPE)
    g["table"] = table
    g["nw"] = wg
    g["nw"][-1] = len(wires) - (len(g) - 1) * wg
    slots = np.full(len(g) * wg, -1, dtype=np.int64)
    slots[:len(wires)] = wires
    g["wire"] = -1
    g["wire"][:, :wg] = slots.reshape(len(g), wg)
    return g


# Wires times right-hand sides of a call up to which the size classes of an FP64
# step go out in one library call, chained on the caller's stream, and above
# which each has a side stream.  The fork and join cost the host 20 (two classes)
# to 60 us (five); the library's launches cover every class for all wires, and
# the CTAs without a wire cost up to 20 % of a leapfrog step of 20480 wires.  us
# per call, side streams / chained: one leapfrog step of 192 wires of Nk 64, 128,
# 256 52 / 18, of 1536 53 / 25; one RK4 step of 192 46 / 21, four 46 / 54; one
# leapfrog step of 2560 wires of Nk 64 .. 1024 94 / 105.
CHAIN_STAGES = 2048


class WireBatch:
    """``form`` selects the step kernel: "plain" (FP64 throughout,
    psb_rk4_f64) or "split" (exchange sums on the int8 tensor cores as exact
    products of base-254 digits, FP64 right-hand side and state:
    psb_rk4_split for unscreened grids with one shared Coulomb matrix,
    psb_rk4_split_wire for screened grids or distinct Veh, Vee, Vhh)."""

    def __init__(self, grids, wires, screened=False, excitons=True, p_cap=0, tables=None,
                 tabdata=None, form="plain", split_w=None, tune=True):
        device.require_cuda()
        if form not in ("plain", "split"):
            raise ValueError("form must be 'plain' or 'split'")
        self.form = form
        # split form: wires per CTA group by grid size, {nk: 4, 8 or 16}; grids
        # not listed use the built-in rule (see _setup_split)
        self.split_w = dict(split_w or {})
        self.tune = bool(tune)
        self.grids = list(grids)
        self.screened = bool(screened)
        if tables is None:
            tables, tabdata = coulomb.grid_tables(self.grids, screened=screened,
                                                  excitons=excitons)
        self.h_tables = np.ascontiguousarray(tables)
        self.tabdata = tabdata
        self.nkmax = int(self.h_tables["nk"].max())
        w = np.array(wires, dtype=abi.WIRE_DTYPE, copy=True)
        nks = self.h_tables["nk"][w["table"]].astype(np.int64)
        offs = np.zeros(len(w), dtype=np.int64)
        if len(w):
            offs[1:] = np.cumsum(nks)[:-1]
        w["off"] = offs
        self.p_cap = int(p_cap)
        w["p_off"] = np.arange(len(w), dtype=np.int64) * self.p_cap
        self.nks = nks
        self.n_state = int(nks.sum())
        self.nw = len(w)
        self.h_wires = w
        self.d_tables = device.to_device(self.h_tables)
        self.d_wires = device.to_device(w)
        self.y = torch.zeros((self.n_state, 4), dtype=torch.float64, device="cuda")
        self.y1 = None
        self.P = torch.zeros((max(1, self.nw * self.p_cap), 2), dtype=torch.float64,
                             device="cuda")
        # Launch classes by grid size: the widths of the FP64 step kernel (a
        # CTA's threads, registers and shared memory follow from its class).
        # Several classes run concurrently on side streams, the largest grids
        # first: alone, a small class leaves most of the GPU idle.
        self.classes = []
        order = np.argsort(-nks, kind="stable").astype(np.int32)
        for lo, hi in ((512, abi.PSB_MAX_NK), (256, 512), (128, 256), (64, 128), (0, 64)):
            sel = order[(nks[order] > lo) & (nks[order] <= hi)]
            if sel.size == 0:
                continue
            tabs = np.unique(w["table"][sel])
            tf = self.h_tables["flags"][tabs]
            flags = abi.PSB_TAB_ONE_CLASS
            if (tf & abi.PSB_TAB_SCREENED).any():
                flags |= abi.PSB_TAB_SCREENED
            if (tf & abi.PSB_TAB_SHARED_V).all():
                flags |= abi.PSB_TAB_SHARED_V
            self.classes.append((torch.as_tensor(sel, device="cuda"), int(nks[sel].max()), flags))
        most = len(self.classes)  # launches of one call: leapfrog's, rk4's
        if form == "split":
            self._setup_split()
            most = max(most, len(self.split_launches) + len(self.wire_launches))
        self.side_streams = self._streams(most) if most > 1 else []
        self.tab_flags = 0
        if (self.h_tables["flags"] & abi.PSB_TAB_SCREENED).any():
            self.tab_flags |= abi.PSB_TAB_SCREENED
        if (self.h_tables["flags"] & abi.PSB_TAB_SHARED_V).all():
            self.tab_flags |= abi.PSB_TAB_SHARED_V
        self.model = abi.model_array(hbar)

    def _setup_split(self):
        """Wire groups (one CTA each) and the workspace of the split form.

        Unscreened grids with Veh == Vee == Vhh use psb_rk4_split: a group
        holds up to W in {4, 8, 16} wires of one grid sharing one Coulomb
        matrix.  W is chosen per grid by the autotuner (tune.SplitTuner:
        measured per-CTA cost of each W on this device, times the waves of
        CTAs the grid's wire count needs); with ``tune=False`` by a rule
        (W = 8 once a grid has enough wires for roughly two waves of CTAs,
        else 4); ``split_w`` overrides both per grid.  Groups are launched in
        classes of (W, state resident in shared memory or not) so that a
        large grid does not push the small ones out of the resident layout.

        Screened grids and grids with distinct Veh, Vee, Vhh use
        psb_rk4_split_wire (one matrix per wire, the wires of a group
        contracted one after another): W by ``wire_group``, each grid on the
        share of the SMs that its wires' work has in the batch
        (``split_w`` overrides it, 1 .. psb_split_wire_max_group).

        All classes run concurrently on side streams, the one with the
        largest grid first."""
        f = self.h_tables["flags"]
        if ((f & abi.PSB_TAB_EXCITONS) == 0).any():
            raise _lib.PsbError("split form needs tables with excitons (the exchange sums)")
        lib = _lib.load()
        maxnk = {wg: int(lib.psb_split_max_nk(wg)) for wg in (4, 8, 16)}
        resnk = {wg: int(lib.psb_split_max_nk_resident(wg)) for wg in (4, 8, 16)}
        nks = self.h_tables["nk"].astype(np.int64)
        counts = np.bincount(self.h_wires["table"], minlength=len(nks))
        sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
        target = float(np.sum(counts * nks.astype(np.float64) ** 2)) / (2.0 * sms)
        # the per-wire kernel's work in this batch, by which its grids share the SMs
        per_wire_t = [(f[t] & abi.PSB_TAB_SCREENED) or not (f[t] & abi.PSB_TAB_SHARED_V)
                      for t in range(len(nks))]
        wire_work = sum(wire_cost(int(nks[t])) * int(counts[t]) for t in range(len(nks))
                        if per_wire_t[t]) or 1.0
        classes = {}
        wclasses = {}
        for t in np.argsort(-nks, kind="stable"):
            nk = int(nks[t])
            if counts[t] == 0:
                continue
            ws = np.nonzero(self.h_wires["table"] == t)[0]
            tflags = int(f[t]) & (abi.PSB_TAB_EXCITONS | abi.PSB_TAB_SCREENED |
                                  abi.PSB_TAB_SHARED_V)
            per_wire = (tflags & abi.PSB_TAB_SCREENED) or not (tflags & abi.PSB_TAB_SHARED_V)
            if per_wire:
                wmax = int(lib.psb_split_wire_max_group(nk, tflags))
                if wmax < 1:
                    raise _lib.PsbError(f"split form: nk {nk} exceeds the supported maximum "
                                        "for screened or distinct Coulomb matrices")
                wg = wire_group(len(ws), wmax, sms * wire_cost(nk) * len(ws) / wire_work)
                if nk in self.split_w:
                    wg = int(self.split_w[nk])
                    if not 1 <= wg <= wmax:
                        raise ValueError(f"split_w[{nk}] must be 1..{wmax} for these tables")
                key = (wg, tflags)
                target_classes = wclasses
            else:
                wg = 4
                if self.tune:
                    from .tune import shared_tuner

                    wg = shared_tuner().best_width(nk, int(counts[t]))
                elif nk <= maxnk[8] and 8 * nk * nk <= max(target, 4 * nk * nk):
                    wg = 8
                if nk in self.split_w:
                    wg = int(self.split_w[nk])
                    if wg not in (4, 8, 16):
                        raise ValueError("split_w values must be 4, 8 or 16")
                if nk > maxnk[wg]:
                    raise _lib.PsbError(f"split form: nk {nk} exceeds the supported maximum")
                key = (wg, nk <= resnk[wg])
                target_classes = classes
            target_classes.setdefault(key, []).append(groups_of(t, ws, wg))
        self.split_launches = []
        for key in classes:
            ga = np.concatenate(classes[key])
            nkmax = int(nks[ga["table"]].max())
            self.split_launches.append((key[0], device.to_device(ga), len(ga), nkmax))
        # the class with the largest grid first: its CTAs run longest
        self.split_launches.sort(key=lambda l: -l[3])
        # per-wire classes: (W, groups, count, nkmax, table flags)
        self.wire_launches = []
        for key in wclasses:
            ga = np.concatenate(wclasses[key])
            nkmax = int(nks[ga["table"]].max())
            self.wire_launches.append((key[0], device.to_device(ga), len(ga), nkmax, key[1]))
        self.wire_launches.sort(key=lambda l: -l[3])
        self.ws = torch.zeros(int(lib.psb_split_ws_bytes(self.n_state)), dtype=torch.uint8,
                              device="cuda")

    @staticmethod
    def _streams(n):
        """One stream per class, priorities by grid size (the largest grid's
        CTAs run longest, so the CTA scheduler serves them first)."""
        least, greatest = torch.cuda.Stream.priority_range()
        return [torch.cuda.Stream(priority=min(least, greatest + r)) for r in range(n)]

    def _concurrent(self, calls, stream):
        """Run ``calls`` (one per class, each taking its stream) concurrently
        on the side streams, ordered after the work queued on ``stream``
        (default: the current stream) and before what follows on it; a single
        call runs on that stream itself."""
        main = stream if stream is not None else torch.cuda.current_stream()
        if len(calls) == 1:
            calls[0](main)
            return
        if len(calls) > len(self.side_streams):
            raise _lib.PsbError(f"{len(calls)} launches on {len(self.side_streams)} side streams")
        fork = torch.cuda.Event()
        fork.record(main)
        for c, s in zip(calls, self.side_streams):
            s.wait_event(fork)
            c(s)
            join = torch.cuda.Event()
            join.record(s)
            main.wait_event(join)

    # -- state --------------------------------------------------------------
    def set_state(self, y, y1=None):
        self.y.copy_(torch.as_tensor(np.asarray(y, dtype=np.float64).reshape(self.n_state, 4)))
        if y1 is not None:
            if self.y1 is None:
                self.y1 = torch.zeros_like(self.y)
            self.y1.copy_(torch.as_tensor(np.asarray(y1, dtype=np.float64).reshape(-1, 4)))

    def state(self):
        return self.y.cpu().numpy()

    def wires(self):
        """Current wire descriptors (t, steps, status) from the device."""
        return device.to_host_struct(self.d_wires, abi.WIRE_DTYPE)

    def wire_slice(self, i):
        o = int(self.h_wires["off"][i])
        return slice(o, o + int(self.nks[i]))

    def records(self, i):
        """P(t) records of wire i as complex numpy."""
        P = self.P[i * self.p_cap:(i + 1) * self.p_cap].cpu().numpy()
        return P[:, 0] + 1j * P[:, 1]

    def _common(self):
        return (device.ptr(self.d_tables), len(self.h_tables), device.ptr(self.tabdata),
                self.tabdata.numel(), device.ptr(self.d_wires), self.nw)

    # -- entry points -----------------------------------------------------------
    @property
    def launches_per_call(self):
        """Kernel launches of an rk4 call (one per size class; a short FP64
        call over several, CHAIN_STAGES, covers every class up to the largest)."""
        if self.form == "split":
            return len(self.split_launches) + len(self.wire_launches)
        return len(self.classes)

    def rhs(self, stream=None):
        dy = torch.empty_like(self.y)
        flags = self.tab_flags | (abi.PSB_TAB_ONE_CLASS if len(self.classes) == 1 else 0)
        _lib.call("psb_rhs_f64", *self._common(), device.ptr(self.y), device.ptr(dy),
                  self.n_state, self.nkmax, flags, abi.as_ptr(self.model),
                  device.stream_ptr(stream))
        return dy

    def rk4(self, nsteps, dt, p_stride=1, stream=None):
        tail = (int(nsteps), float(dt), device.ptr(self.P), self.P.shape[0], int(p_stride),
                self.p_cap, abi.as_ptr(self.model))
        calls = []
        if self.form == "split":
            ws = (device.ptr(self.y), self.n_state, device.ptr(self.ws), self.ws.numel())
            for wg, groups, ng, nkmax in self.split_launches:
                calls.append(lambda s, a=(device.ptr(groups), ng, wg, nkmax): _lib.call(
                    "psb_rk4_split", *self._common(), *a, *ws, *tail, device.stream_ptr(s)))
            for wg, groups, ng, nkmax, tflags in self.wire_launches:
                calls.append(lambda s, a=(device.ptr(groups), ng, wg, nkmax, tflags): _lib.call(
                    "psb_rk4_split_wire", *self._common(), *a, *ws, *tail, device.stream_ptr(s)))
        else:
            for order, n, nkmax, flags in self._fp64_launches(4 * int(nsteps)):
                calls.append(lambda s, a=(device.ptr(order), n), b=(nkmax, flags): _lib.call(
                    "psb_rk4_f64", *self._common(), *a, device.ptr(self.y), self.n_state, *b,
                    *tail, device.stream_ptr(s)))
        self._concurrent(calls, stream)

    def _fp64_launches(self, stages):
        """(order, n_order, nkmax, tab_flags) of the library calls of an FP64
        step of ``stages`` right-hand sides: one per size class, or one for all
        (see CHAIN_STAGES)."""
        if len(self.classes) > 1 and self.nw * stages <= CHAIN_STAGES:
            return [(None, 0, self.nkmax, self.tab_flags)]
        return [(order, order.numel(), nkmax, flags) for order, nkmax, flags in self.classes]

    def capture(self, nsteps, dt, p_stride=1):
        """A CUDA graph of one ``rk4(nsteps, dt, p_stride)`` call (every size
        class's launch, the split form's side streams and their joins), to
        replay with ``graph.replay()`` on the current stream: one host call
        per step instead of one launch per class plus the stream
        synchronisation.  The graph reads and writes this batch's own state,
        wire descriptors and P(t) buffers, so a caller changes the data
        between replays (``set_state``, the wire descriptors), not the
        shapes.  One eager call first sets the kernels' attributes outside
        the capture (it advances the batch like any rk4 call)."""
        import torch

        self.rk4(nsteps, dt, p_stride=p_stride)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            self.rk4(nsteps, dt, p_stride=p_stride)
        torch.cuda.synchronize()
        return g

    def leapfrog(self, field, nsteps, dt, p_stride=1, stream=None):
        """field: device float64 tensor (nw, 2*n_samples) of sampled E(t_n)."""
        if self.y1 is None:
            self.y1 = self.y.clone()
        assert field.is_cuda and field.dtype == torch.float64 and field.dim() == 2
        calls = [lambda s, a=(device.ptr(order), n), b=(nkmax, flags): _lib.call(
            "psb_leapfrog_f64", *self._common(), *a, device.ptr(self.y1), device.ptr(self.y),
            self.n_state, *b, device.ptr(field), field.shape[1], field.numel(), int(nsteps),
            float(dt), device.ptr(self.P), self.P.shape[0], int(p_stride), self.p_cap,
            abi.as_ptr(self.model), device.stream_ptr(s))
            for order, n, nkmax, flags in self._fp64_launches(int(nsteps))]
        self._concurrent(calls, stream)
