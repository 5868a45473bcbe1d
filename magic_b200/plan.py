"""Plan: one horizontal resolution (l_max, minc) resident on one GPU.

A Plan owns the FP64 Legendre tables (built on the device by
``mt_plan_create``) and exposes the transforms and nonlinear-term builders
on torch CUDA tensors.  Shapes, dtypes and conventions are those of the
reference's ``magic_torch.sht`` (spectral (lm_max,) / (lm_max, B) complex128,
grids (n_theta, n_phi) / (B, n_theta, n_phi) float64 with interleaved N/S
theta rows).  Every call enqueues on the current torch CUDA stream and does not
synchronise the host.
"""

import collections
import ctypes as C

import numpy as np
import torch

from . import _lib
from ._lib import MagicError, check, check_writes, plain, raise_device_status

_CD = torch.complex128
_RD = torch.float64


def _ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else C.c_void_p(0)


class _StatusWatch:
    """Non-blocking check of the split kernels' device status.  After each call
    the status word of its workspace (first int, written by a bounded tensor-pipe
    wait that ran out) is copied on the same stream into a pinned host slot, and
    an event marks when it has landed; poll() raises MagicError for the first
    landed non-zero code.  Nothing is recorded while the stream is being captured
    into a CUDA graph (the caller reads the word after replays instead)."""

    SLOTS = 4096

    def __init__(self):
        self.host = torch.zeros(self.SLOTS, dtype=torch.int32).pin_memory()
        self.pending = collections.deque()
        self.next = 0

    def record(self, work, what):
        if torch.cuda.is_current_stream_capturing():
            return
        self.poll()
        if len(self.pending) >= self.SLOTS:
            self.poll(block=True)
        stream = torch.cuda.current_stream(work.device)
        slot = self.next
        self.next = (self.next + 1) % self.SLOTS
        self.host[slot:slot + 1].copy_(work[:4].view(torch.int32), non_blocking=True)
        ev = torch.cuda.Event()
        ev.record(stream)
        self.pending.append((slot, ev, what))

    def poll(self, block=False):
        while self.pending:
            slot, ev, what = self.pending[0]
            if block:
                ev.synchronize()
            elif not ev.query():
                return
            self.pending.popleft()
            code = int(self.host[slot])
            if code:
                self.pending.clear()
                raise_device_status(code, what)


class Plan:
    """Tables and entry points for one (l_max, minc) grid on one CUDA device.

    Split-precision plans watch the device status of every call (see
    ``poll_status``): a bounded wait on the tensor pipe that ran out is raised
    as MagicError by the next call on the plan, or by ``poll_status``."""

    def __init__(self, l_max, minc=1, precision="fp64", device=None, n_theta_max=0,
                 n_phi_max=0):
        if not torch.cuda.is_available():
            raise RuntimeError("magic_b200 needs a CUDA device (B200); no CPU fallback")
        dev = torch.device(device if device is not None else "cuda")
        if dev.type != "cuda":
            raise ValueError("magic_b200 plans live on CUDA devices")
        self.device = dev if dev.index is not None else torch.device(
            "cuda", torch.cuda.current_device())
        prec = {"fp64": _lib.MT_PREC_FP64, "split": _lib.MT_PREC_SPLIT,
                "ozaki": _lib.MT_PREC_OZAKI}[precision]
        self.precision = precision
        L = _lib.lib()
        desc = _lib.GridDesc(int(l_max), int(minc), int(n_theta_max), int(n_phi_max), prec)
        h = C.c_void_p()
        with torch.cuda.device(self.device):
            check(L.mt_plan_create(C.byref(desc), C.byref(h)))
        self._h = h
        self._sizes = {}
        info = _lib.PlanInfo()
        check(L.mt_plan_get_info(h, C.byref(info)))
        self.l_max = info.l_max
        self.minc = info.minc
        self.n_theta_max = info.n_theta_max
        self.n_phi_max = info.n_phi_max
        self.n_m_max = info.n_m_max
        self.lm_max = info.lm_max
        self.nhs = info.nhs
        ls, l_of, m_of = [], [], []
        pos = 0
        for m in range(0, self.l_max + 1, self.minc):
            ls.append(pos)
            for l in range(m, self.l_max + 1):
                l_of.append(l)
                m_of.append(m)
            pos += self.l_max - m + 1
        self.lStart = np.array(ls)
        self.lm2l = np.array(l_of)
        self.lm2m = np.array(m_of)
        lf = torch.tensor(self.lm2l, dtype=_RD, device=self.device)
        self.dLh = lf * (lf + 1.0)
        self.dPhi = 1j * torch.tensor(self.lm2m, dtype=_RD, device=self.device).to(_CD)
        th = torch.empty(self.n_theta_max, dtype=_RD, device=self.device)
        check(L.mt_plan_copy_tables(h, _ptr(th), None, None, None, self._stream()))
        gi = torch.zeros(self.n_theta_max, dtype=torch.long)
        gi[0::2] = torch.arange(self.nhs)
        gi[1::2] = torch.arange(self.n_theta_max - 1, self.nhs - 1, -1)
        self.grid_idx = gi.to(self.device)
        sin_g = torch.sin(th[self.grid_idx])
        self.O_sin_theta_E2_grid = 1.0 / sin_g ** 2
        self._status = _StatusWatch() if precision != "fp64" else None

    # ------------------------------------------------------ device status
    def poll_status(self, block=False):
        """Raise MagicError if a split-precision call on this plan recorded a
        device-side timeout.  block=False only looks at calls that have already
        finished; block=True waits for every call made so far."""
        if self._status is not None:
            self._status.poll(block)

    def device_status(self, work):
        """Status word of the call that last used ``work`` (synchronises the
        current stream): 0, or the code of the bounded wait that ran out."""
        code = C.c_int(0)
        check(_lib.lib().mt_device_status(_ptr(work), C.byref(code), self._stream()))
        return code.value

    def _watch(self, work, what, fused=False):
        """Record the status word of a call that cleared it: every call of a split
        plan; on digit-split (ozaki) plans only the fused stage (their transforms
        run the FP64 kernels, which leave the word alone)."""
        if self._status is not None and (fused or self.precision == "split"):
            self._status.record(work, what)

    def __del__(self):
        h = getattr(self, "_h", None)
        if h is not None and h.value:
            try:
                _lib.lib().mt_plan_destroy(h)
            except Exception:
                pass
            self._h = None

    # ------------------------------------------------------------ helpers
    # A transform of a small grid takes less time on the device than its call on the
    # host (l_max 16: 10 us against 21): the handle of the current stream instead of a
    # torch.cuda.Stream, addresses as plain integers, and results allocated in the
    # shape that is returned instead of a view of a larger one.
    def _stream(self):
        return _lib.stream_handle(self.device)

    def _work(self, nbytes):
        return torch.empty(max(int(nbytes), 16), dtype=torch.uint8, device=self.device)

    def _scratch(self, B, nf):
        """Workspace of a transform of nf fields of B columns (its size is the plan's)."""
        size = self._sizes.get((B, nf))
        if size is None:
            if len(self._sizes) >= 256:
                self._sizes.clear()
            size = _lib.lib().mt_transform_workspace(self._h, B, nf)
            self._sizes[B, nf] = size
        return self._work(size)

    def _spec(self, x, name):
        """(tensor, columns, row stride, whether 1-D) of a spectral argument."""
        if not isinstance(x, torch.Tensor) or x.device != self.device:
            raise ValueError(f"{name}: expected a tensor on {self.device}")
        n = x.dim()
        if not 1 <= n <= 2 or x.size(0) != self.lm_max:
            raise ValueError(f"{name}: expected shape (lm_max={self.lm_max},[B])")
        if x.dtype != _CD:
            x = x.to(_CD)
        if x.is_conj():
            x = x.resolve_conj()
        if n == 1:
            if x.stride(0) < 1:
                x = x.contiguous()
            return x, 1, x.stride(0), True
        if x.stride(1) != 1 or x.stride(0) < x.size(1):
            x = x.contiguous()
        return x, x.size(1), x.stride(0), False

    def _grid(self, x, name):
        """(tensor, grids, whether 2-D) of a grid argument."""
        if not isinstance(x, torch.Tensor) or x.device != self.device:
            raise ValueError(f"{name}: expected a tensor on {self.device}")
        n = x.dim()
        if not 2 <= n <= 3 or x.size(-2) != self.n_theta_max or x.size(-1) != self.n_phi_max:
            raise ValueError(f"{name}: expected shape ([B,] {self.n_theta_max}, {self.n_phi_max})")
        if x.dtype != _RD:
            x = x.to(_RD)
        if x.is_neg():
            x = x.resolve_neg()
        return x.contiguous(), x.size(0) if n == 3 else 1, n == 2

    def _new_grid(self, B, one):
        shape = (self.n_theta_max, self.n_phi_max)
        return torch.empty(shape if one else (B, *shape), dtype=_RD, device=self.device)

    def _new_spec(self, B, one):
        return torch.empty(self.lm_max if one else (self.lm_max, B), dtype=_CD,
                           device=self.device)

    def tables(self):
        """FP64 tables built on the device: theta_ord, gauss, Plm, dPlm (reference layout)."""
        nt, lm, nhs = self.n_theta_max, self.lm_max, self.nhs
        out = dict(theta_ord=torch.empty(nt, dtype=_RD, device=self.device),
                   gauss=torch.empty(nt, dtype=_RD, device=self.device),
                   Plm=torch.empty(lm, nhs, dtype=_RD, device=self.device),
                   dPlm=torch.empty(lm, nhs, dtype=_RD, device=self.device))
        check(_lib.lib().mt_plan_copy_tables(self._h, _ptr(out["theta_ord"]), _ptr(out["gauss"]),
                                             _ptr(out["Plm"]), _ptr(out["dPlm"]), self._stream()))
        return out

    # -------------------------------------------------------- transforms
    def scal_to_spat(self, Slm, lcut=None):
        X, B, ld, one = self._spec(Slm, "Slm")
        out = self._new_grid(B, one)
        L = _lib.lib()
        ws = self._scratch(B, 1)
        check(L.mt_scal_to_spat(self._h, X.data_ptr(), ld, B, out.data_ptr(), ws.data_ptr(),
                                ws.numel(), self._stream()))
        self._watch(ws, "scal_to_spat")
        return out

    def scal_to_SH(self, sc, lcut=None):
        g, B, one = self._grid(sc, "sc")
        out = self._new_spec(B, one)
        L = _lib.lib()
        ws = self._scratch(B, 1)
        check(L.mt_scal_to_SH(self._h, g.data_ptr(), B, out.data_ptr(), B, ws.data_ptr(),
                              ws.numel(), self._stream()))
        self._watch(ws, "scal_to_SH")
        return out

    def torpol_to_spat(self, Qlm, Slm, Tlm, lcut=None):
        Q, B, ld, one = self._spec(Qlm, "Qlm")
        S, bS, ldS, _ = self._spec(Slm, "Slm")
        T, bT, ldT, _ = self._spec(Tlm, "Tlm")
        if not (B == bS == bT):
            raise ValueError("Qlm, Slm, Tlm must have the same shape")
        if not (ld == ldS == ldT):
            Q, S, T = Q.contiguous(), S.contiguous(), T.contiguous()
            ld = Q.stride(0)
        outs = tuple(self._new_grid(B, one) for _ in range(3))
        L = _lib.lib()
        ws = self._scratch(B, 3)
        check(L.mt_torpol_to_spat(self._h, Q.data_ptr(), S.data_ptr(), T.data_ptr(), ld, B,
                                  *[o.data_ptr() for o in outs], ws.data_ptr(), ws.numel(),
                                  self._stream()))
        self._watch(ws, "torpol_to_spat")
        return outs

    def spat_to_sphertor(self, vt, vp, lcut=None):
        gt, B, one = self._grid(vt, "vt")
        gp, Bp, _ = self._grid(vp, "vp")
        if B != Bp:
            raise ValueError("vt and vp must have the same shape")
        S, T = self._new_spec(B, one), self._new_spec(B, one)
        L = _lib.lib()
        ws = self._scratch(B, 2)
        check(L.mt_spat_to_sphertor(self._h, gt.data_ptr(), gp.data_ptr(), B, S.data_ptr(),
                                    T.data_ptr(), B, ws.data_ptr(), ws.numel(), self._stream()))
        self._watch(ws, "spat_to_sphertor")
        return S, T

    def _grad(self, Slm, scale_dlh):
        X, B, ld, one = self._spec(Slm, "Slm")
        gt, gp = self._new_grid(B, one), self._new_grid(B, one)
        L = _lib.lib()
        ws = self._scratch(B, 2)
        check(L.mt_scal_to_grad_spat(self._h, X.data_ptr(), ld, B, int(scale_dlh),
                                     gt.data_ptr(), gp.data_ptr(), ws.data_ptr(), ws.numel(),
                                     self._stream()))
        self._watch(ws, "scal_to_grad_spat")
        return gt, gp

    def scal_to_grad_spat(self, Slm, lcut=None):
        return self._grad(Slm, False)

    def pol_to_grad_spat(self, Slm, lcut=None):
        return self._grad(Slm, True)

    # ------------------------------------------------- grid-space products
    def _grids(self, arrs, n_r, name):
        out = []
        for i, a in enumerate(arrs):
            if a.shape != (n_r, self.n_theta_max, self.n_phi_max) or a.device != self.device:
                raise ValueError(f"{name}[{i}]: expected ({n_r}, {self.n_theta_max}, "
                                 f"{self.n_phi_max}) on {self.device}")
            out.append(plain(a.to(_RD)).contiguous())
        return out

    def _prof(self, x, n_r):
        # as kernels read it (a time step's profiles): nothing to convert
        if isinstance(x, torch.Tensor) and x.dtype == _RD and x.device == self.device and \
                x.dim() == 1 and x.size(0) == n_r and x.is_contiguous() and not x.is_neg():
            return x
        t = torch.as_tensor(x, dtype=_RD, device=self.device).reshape(-1)
        if t.numel() == 1 and n_r > 1:
            t = t.expand(n_r)
        return plain(t).contiguous()

    def get_nl(self, grids, or2, or4, LFfac):
        """get_nl products (magic_torch/get_nl.py:30-87); grids: 14 (n_r, nt, np)."""
        n_r = grids[0].shape[0]
        ins = self._grids(grids, n_r, "get_nl")
        outs = [torch.empty_like(ins[0]) for _ in range(12)]
        or2 = self._prof(or2, n_r)
        or4 = self._prof(or4, n_r)
        pin = (C.c_void_p * 14)(*[t.data_ptr() for t in ins])
        pout = (C.c_void_p * 12)(*[t.data_ptr() for t in outs])
        check(_lib.lib().mt_get_nl(self._h, n_r, pin, pout, _ptr(or2), _ptr(or4), float(LFfac),
                                   self._stream()))
        return tuple(outs)

    def get_nl_anel(self, grids, prof, LFfac, ViscHeatFac, OhmLossFac, l_mag=True):
        """get_nl_anel products (magic_torch/get_nl_anel.py:41-136); 19 grids in, 13 out.

        ``prof``: dict of radial profiles r, or1, or2, or4, beta, orho1, otemp1, visc,
        lambda_ over the grid levels.
        """
        n_r = grids[0].shape[0]
        ins = self._grids(grids, n_r, "get_nl_anel")
        outs = [torch.empty_like(ins[0]) for _ in range(13)]
        keep = {k: self._prof(prof[k], n_r) for k in
                ("r", "or1", "or2", "or4", "beta", "orho1", "otemp1", "visc", "lambda_")}
        p = _lib.AnelParams(*[k.data_ptr() for k in keep.values()], float(LFfac),
                            float(ViscHeatFac), float(OhmLossFac), int(bool(l_mag)))
        pin = (C.c_void_p * 19)(*[t.data_ptr() for t in ins])
        pout = (C.c_void_p * 13)(*[t.data_ptr() for t in outs])
        check(_lib.lib().mt_get_nl_anel(self._h, n_r, pin, pout, C.byref(p), self._stream()))
        return tuple(outs)

    def courant(self, vr, vt, vp, br, bt, bp, prof, courfac, alffac, LFfac, opm, damp=True):
        """Per-level (dtrkc, dthkc) (magic_torch/courant.py:80-127)."""
        n_r = vr.shape[0]
        mag = br is not None
        g = self._grids([vr, vt, vp] + ([br, bt, bp] if mag else []), n_r, "courant")
        keep = {k: self._prof(prof[k], n_r) for k in
                ("or2", "or4", "orho1", "orho2", "delxr2", "delxh2")}
        mode = (1 if damp else 2) if mag else 0
        p = _lib.CourantParams(*[k.data_ptr() for k in keep.values()], float(courfac),
                               float(alffac), float(LFfac), float(opm), mode)
        dtr = torch.empty(n_r, dtype=_RD, device=self.device)
        dth = torch.empty_like(dtr)
        L = _lib.lib()
        ws = self._work(L.mt_courant_workspace(self._h, n_r))
        bptr = [_ptr(x) for x in g[3:6]] if mag else [C.c_void_p(0)] * 3
        check(L.mt_courant(self._h, n_r, _ptr(g[0]), _ptr(g[1]), _ptr(g[2]), *bptr, C.byref(p),
                           _ptr(dtr), _ptr(dth), _ptr(ws), ws.numel(), self._stream()))
        return dtr, dth

    # --------------------------------------------------- fused stage
    def nl_bouss_workspace(self, n_r, l_mag=True, l_chem=False):
        return _lib.lib().mt_nl_bouss_workspace(self._h, int(n_r), int(l_mag), int(l_chem))

    def nl_bouss(self, fields, prof, LFfac, courfac, alffac, opm, l_mag=True, l_chem=False,
                 damp=True, out=None, work=None, parts=0, LFfac_r=None):
        """Fused Boussinesq nonlinear stage (magic_torch/step_time.py:931-1213, steps 1-3 + CFL).

        ``fields``: dict of spectral (lm_max, n_r) complex128 arrays w, dw, ddw, z, dz, s
        (+ b, db, ddb, aj, dj if l_mag, xi if l_chem).  ``prof``: or2, or4, orho1, orho2,
        delxr2, delxh2 over the n_r levels.  Returns (outputs dict, dtrkc, dthkc); outputs
        are (lm_max, n_r) with boundary columns zero.  LFfac_r: optional per-level
        Lorentz factor replacing LFfac (levels of several runs in one call).
        """
        w = fields["w"]
        n_r = w.shape[1]
        names = ["w", "dw", "ddw", "z", "dz", "s"] + (["b", "db", "ddb", "aj", "dj"] if l_mag
                                                       else []) + (["xi"] if l_chem else [])
        ins = {}
        for k in names:
            x = fields[k]
            if x.shape != (self.lm_max, n_r) or x.dtype != _CD or x.device != self.device:
                raise ValueError(f"fields[{k}]: expected ({self.lm_max}, {n_r}) complex128")
            ins[k] = plain(x).contiguous()
        onames = ["Advr", "Advt", "Advp", "VSr", "VSt"] + (["VxBr", "VxBt", "VxBp"] if l_mag
                                                           else []) + \
            (["VXir", "VXit"] if l_chem else [])
        if out is None:
            out = {k: torch.zeros(self.lm_max, n_r, dtype=_CD, device=self.device) for k in onames}
        keep = {k: self._prof(prof[k], n_r) for k in
                ("or2", "or4", "orho1", "orho2", "delxr2", "delxh2")}
        bi = _lib.BoussIn(*[ins[k].data_ptr() if k in ins else None for k in
                            ("w", "dw", "ddw", "z", "dz", "s", "b", "db", "ddb", "aj", "dj",
                             "xi")], n_r)
        bo = _lib.BoussOut(*[out[k].data_ptr() if k in out else None for k in
                             ("Advr", "Advt", "Advp", "VSr", "VSt", "VxBr", "VxBt", "VxBp",
                              "VXir", "VXit")], out["Advr"].stride(0))
        lf_r = None
        if LFfac_r is not None:
            lf_r = self._prof(LFfac_r, n_r)
            if lf_r.numel() != n_r:
                raise ValueError(f"LFfac_r: expected {n_r} per-level values")
        bp = _lib.BoussParams(*[k.data_ptr() for k in keep.values()], float(LFfac),
                              float(courfac), float(alffac), float(opm), int(l_mag),
                              int(l_chem), (1 if damp else 2) if l_mag else 0, int(parts),
                              lf_r.data_ptr() if lf_r is not None else None)
        dtr = torch.empty(n_r, dtype=_RD, device=self.device)
        dth = torch.empty_like(dtr)
        L = _lib.lib()
        need = L.mt_nl_bouss_workspace(self._h, n_r, int(l_mag), int(l_chem))
        if work is None or work.numel() < need:
            work = self._work(need)
        check_writes([out[k] for k in onames if k in out], L.mt_nl_bouss, self._h, n_r,
                     C.byref(bi), C.byref(bo), C.byref(bp), _ptr(dtr), _ptr(dth), _ptr(work),
                     work.numel(), self._stream())
        self._watch(work, "nl_bouss", fused=True)
        return out, dtr, dth

    def get_td(self, ins, prof, CorFac, D1, l_double_curl=False, l_heat=True, l_mag=True,
               l_chem=False, l_anel=False, out=None):
        """Explicit time-derivative terms of one step (magic_torch/step_time.py:1139-1176):
        get_dwdt or get_dwdt_double_curl, get_dzdt, get_dpdt, get_dsdt, get_dxidt and
        get_dbdt (magic_torch/get_td.py:58-308) completed by finish_exp_pol, _entropy,
        _comp and _mag (update_wp.py:371-385, update_s.py:191-210, update_xi.py:183-202,
        update_b.py:514-528), in one launch.

        ``ins``: dict of (lm_max, n_r) complex128 arrays Advr, Advt, Advp, w, dw, z (plus
        ddw, dz for the double-curl form; VSr, VSt if l_heat; VxBr, VxBt, VxBp if l_mag;
        VXir, VXit if l_chem; optionally heat, the anelastic stage's spectral heating,
        added to the entropy term).  ``prof``: r, or1, or2, or4, orho1, beta over n_r.
        ``D1``: the first-derivative RadialOp.  Returns a dict dwdt, dzdt (+ dpdt without
        the double-curl form, dsdt, dxidt, dbdt, djdt as enabled)."""
        n_r = ins["w"].shape[1]
        need = ["Advr", "Advt", "Advp", "w", "dw", "z"]
        need += ["ddw", "dz"] if l_double_curl else []
        need += ["VSr", "VSt"] if l_heat else []
        need += ["VxBr", "VxBt", "VxBp"] if l_mag else []
        need += ["VXir", "VXit"] if l_chem else []
        need += ["heat"] if l_heat and ins.get("heat") is not None else []
        src = {}
        for k in need:
            x = ins[k]
            if x.shape != (self.lm_max, n_r) or x.dtype != _CD or x.device != self.device:
                raise ValueError(f"ins[{k}]: expected ({self.lm_max}, {n_r}) complex128")
            src[k] = plain(x).contiguous()
        onames = ["dwdt", "dzdt"] + ([] if l_double_curl else ["dpdt"]) + \
            (["dsdt"] if l_heat else []) + (["dxidt"] if l_chem else []) + \
            (["dbdt", "djdt"] if l_mag else [])
        if out is None:
            out = {k: torch.empty(self.lm_max, n_r, dtype=_CD, device=self.device)
                   for k in onames}
        keep = {k: self._prof(prof[k], n_r) for k in ("r", "or1", "or2", "or4", "orho1", "beta")}
        ti = _lib.TdIn(*[src[k].data_ptr() if k in src else None for k in
                         ("Advr", "Advt", "Advp", "VSr", "VSt", "VxBr", "VxBt", "VxBp", "VXir",
                          "VXit", "w", "dw", "ddw", "z", "dz")], n_r,
                        src["heat"].data_ptr() if "heat" in src else None)
        to = _lib.TdOut(*[out[k].data_ptr() if k in out else None for k in
                          ("dwdt", "dzdt", "dpdt", "dsdt", "dxidt", "dbdt", "djdt")],
                        out["dwdt"].stride(0))
        tp = _lib.TdParams(*[keep[k].data_ptr() for k in ("r", "or1", "or2", "or4", "orho1",
                                                          "beta")],
                           float(CorFac), int(l_double_curl), int(l_heat), int(l_mag),
                           int(l_chem), int(l_anel))
        check_writes([out[k] for k in onames if k in out], _lib.lib().mt_get_td, self._h, n_r,
                     C.byref(ti), C.byref(to), C.byref(tp), D1._h if D1 is not None else None,
                     self._stream())
        return out

    def nl_anel_workspace(self, n_r, l_mag=True, l_chem=False):
        L = _lib.lib()
        size = L.mt_nl_anel_f64_workspace if self.precision == "fp64" else L.mt_nl_anel_workspace
        return size(self._h, int(n_r), int(l_mag), int(l_chem))

    def nl_anel(self, fields, prof, LFfac, ViscHeatFac, OhmLossFac, courfac, alffac, opm,
                l_mag=True, l_chem=False, damp=True, out=None, work=None):
        """Anelastic nonlinear stage (magic_torch/step_time.py:1215-1475: transforms,
        get_nl_anel with viscous and Ohmic heating, forward transforms, CFL), fused: the
        tcgen05 pack/GEMM and FP32 phi kernels on split-precision plans, the int8
        digit-plane GEMMs and an FP64 phi kernel on digit-split (ozaki) plans, the FP64
        contractions and the same phi kernel on FP64 plans.

        ``fields``: dict of spectral (lm_max, n_r) complex128 arrays w, dw, ddw, z, dz, s
        (+ b, db, ddb, aj, dj if l_mag, xi if l_chem).  ``prof``: r, or1, or2, or4, beta,
        orho1, orho2, otemp1, visc, lambda_, delxr2, delxh2 over the n_r levels.  Returns
        (outputs dict Advr Advt Advp VSr VSt [VxBr VxBt VxBp] [VXir VXit] heat, dtrkc,
        dthkc); outputs are (lm_max, n_r) with boundary columns zero.
        """
        w = fields["w"]
        n_r = w.shape[1]
        L = _lib.lib()
        names = ["w", "dw", "ddw", "z", "dz", "s"] + (["b", "db", "ddb", "aj", "dj"] if l_mag
                                                       else []) + (["xi"] if l_chem else [])
        ins = {}
        for k in names:
            x = fields[k]
            if x.shape != (self.lm_max, n_r) or x.dtype != _CD or x.device != self.device:
                raise ValueError(f"fields[{k}]: expected ({self.lm_max}, {n_r}) complex128")
            ins[k] = plain(x).contiguous()
        need = self.nl_anel_workspace(n_r, l_mag, l_chem) if n_r >= 3 else 0
        if need == 0:
            raise MagicError("nl_anel needs n_r >= 3")
        onames = ["Advr", "Advt", "Advp", "VSr", "VSt"] + (["VxBr", "VxBt", "VxBp"] if l_mag
                                                           else []) + \
            (["VXir", "VXit"] if l_chem else []) + ["heat"]
        if out is None:
            out = {k: torch.zeros(self.lm_max, n_r, dtype=_CD, device=self.device) for k in onames}
        # FP64 plans take outputs of any layout and type: what the kernels cannot write
        # (complex128 rows of unit stride, one row stride for all) goes through a copy
        given = out
        if self.precision == "fp64":
            o0 = out[onames[0]]
            fits = all(x.shape == (self.lm_max, n_r) and x.dtype == _CD
                       and x.device == self.device and x.stride(1) == 1
                       and x.stride(0) == o0.stride(0) >= n_r
                       for x in (out[k] for k in onames))
            if not fits:
                out = {k: torch.empty(self.lm_max, n_r, dtype=_CD, device=self.device)
                       for k in onames}
            if work is not None and (work.device != self.device or not work.is_contiguous()
                                     or work.dtype != torch.uint8 or work.data_ptr() % 16):
                work = None
        pnames = ("r", "or1", "or2", "or4", "beta", "orho1", "orho2", "otemp1", "visc",
                  "lambda_", "delxr2", "delxh2")
        keep = {k: self._prof(prof[k], n_r) for k in pnames}
        ai = _lib.AnelIn(*[ins[k].data_ptr() if k in ins else None for k in
                           ("w", "dw", "ddw", "z", "dz", "s", "xi", "b", "db", "ddb", "aj",
                            "dj")], n_r)
        ao = _lib.AnelOut(*[out[k].data_ptr() if k in out else None for k in
                            ("Advr", "Advt", "Advp", "VSr", "VSt", "VxBr", "VxBt", "VxBp",
                             "VXir", "VXit", "heat")], out["Advr"].stride(0))
        ap = _lib.AnelStageParams(*[keep[k].data_ptr() for k in pnames], float(LFfac),
                                  float(ViscHeatFac), float(OhmLossFac), float(courfac),
                                  float(alffac), float(opm), int(l_mag), int(l_chem),
                                  (1 if damp else 2) if l_mag else 0)
        dtr = torch.empty(n_r, dtype=_RD, device=self.device)
        dth = torch.empty_like(dtr)
        if work is None or work.numel() < need:
            work = self._work(need)
        run = L.mt_nl_anel_f64 if self.precision == "fp64" else L.mt_nl_anel
        check_writes([out[k] for k in onames if k in out], run, self._h, n_r, C.byref(ai),
                     C.byref(ao), C.byref(ap), _ptr(dtr), _ptr(dth), _ptr(work), work.numel(),
                     self._stream())
        self._watch(work, "nl_anel", fused=True)
        if out is not given:
            for k in onames:
                given[k][:, 0] = 0.0
                given[k][:, -1] = 0.0
                given[k][:, 1:n_r - 1] = out[k][:, 1:-1]
        return given, dtr, dth
