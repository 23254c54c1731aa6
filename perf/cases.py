"""The workloads this framework's speed is measured on.

Each case is one call of a public entry point with the sizes, data and
options of real use: the transmission of a molecular junction or nanowire
over an energy grid (from a single energy, as a host code's own energy loop
calls it, to a few hundred points in one launch), transmission with the
density of states, several terminals with projections, the elastic-dephasing
SCBA, the contour density matrix, the mixed-precision form, and the three
device-pointer primitives a host code's own sweep calls.

Broadenings are 1 meV for devices in eV, tolerances the entry points'
defaults (SGFACC = 1e-9).  Devices come from libnegf_b200.generators with the seed, the
energies lie inside the leads' bands, on a uniform grid with a random offset.
"""
from __future__ import annotations

import ctypes
import math
import weakref

import numpy as np
import torch

from libnegf_b200 import density as D
from libnegf_b200 import generators as G
from libnegf_b200 import native

ETA = 1e-3
DOS_DELTA = 1e-3
DEC_ITERS = 13        # decimation iterations of a typical point at this eta


def listed():
    return [
        # one energy of the small tight-binding device: a host code that keeps its own energy loop
        dict(name="t_one_energy", kind="T", n=32, nbl=20, s=False, pts=1),
        # the same device over its whole energy grid
        dict(name="t_small_grid", kind="T", n=32, nbl=20, s=False, pts=512),
        # molecular junction, odd layer size, a grid that fills a third of the GPU
        dict(name="t_junction", kind="T", n=97, nbl=24, s=False, pts=48),
        # wide non-orthogonal wire, a handful of energies (adaptive refinement of a grid)
        dict(name="t_wide_wire", kind="T", n=384, nbl=6, s=True, pts=12),
        # non-orthogonal nanowire, two transverse k-points, T and DOS: the ordinary production launch
        dict(name="dos_nanowire", kind="DOS", n=256, nbl=12, s=True, pts=320, kpts=2),
        # three terminals on layers of uneven size, transmissions of all pairs and LDOS sets
        dict(name="terminals_uneven", kind="pairs", n=112, nbl=9, pts=40),
        # elastic dephasing, self-consistent, with currents and layer densities
        dict(name="scba_dephasing", kind="scba", n=64, nbl=12, pts=32, niter=8),
        # equilibrium density matrix on the complex contour (one SCF step of a host code)
        dict(name="rho_contour", kind="rho", n=128, nbl=10, np1=20, np2=12, poles=3),
        # wide layers in the mixed-precision form
        dict(name="t_mixed", kind="mixed", n=256, nbl=10, s=True, pts=64),
        # the block product, inverse and decimation a host code's own sweep calls on device pointers
        dict(name="zgemm_blocks", kind="zgemm", n=300, batch=6, dagger=2),
        dict(name="zinv_blocks", kind="zinv", n=200, batch=8),
        dict(name="decimation_leads", kind="dec", n=144, batch=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["T small", "T small", "T mid", "T wide", "DOS", "pairs", "scba", "rho", "mixed", "zgemm",
                       "zinv", "dec"])
    if kind == "T small":
        return dict(kind="T", n=rng.randint(8, 32), nbl=rng.randint(4, 24), s=rng.random() < 0.3,
                    pts=_log(rng, 1, 512))
    if kind == "T mid":
        return dict(kind="T", n=_log(rng, 33, 160), nbl=rng.randint(3, 24), s=rng.random() < 0.5,
                    pts=_log(rng, 1, 96))
    if kind == "T wide":
        return dict(kind="T", n=_log(rng, 161, 384), nbl=rng.randint(2, 6), s=rng.random() < 0.5,
                    pts=_log(rng, 1, 12))
    if kind == "DOS":
        n = _log(rng, 24, 256)
        return dict(kind="DOS", n=n, nbl=rng.randint(3, 12), s=rng.random() < 0.7, pts=_log(rng, 8, 320),
                    kpts=rng.randint(1, 2))
    if kind == "pairs":
        return dict(kind="pairs", n=_log(rng, 24, 112), nbl=rng.randint(4, 9), pts=_log(rng, 4, 40))
    if kind == "scba":
        return dict(kind="scba", n=_log(rng, 16, 64), nbl=rng.randint(4, 12), pts=_log(rng, 4, 32),
                    niter=rng.randint(3, 8))
    if kind == "rho":
        return dict(kind="rho", n=_log(rng, 24, 128), nbl=rng.randint(3, 10), np1=rng.randint(8, 20),
                    np2=rng.randint(6, 12), poles=rng.randint(1, 3))
    if kind == "mixed":
        return dict(kind="mixed", n=_log(rng, 64, 256), nbl=rng.randint(3, 10), s=rng.random() < 0.5,
                    pts=_log(rng, 8, 64))
    if kind == "zgemm":
        return dict(kind="zgemm", n=_log(rng, 20, 400), batch=_log(rng, 1, 64), dagger=rng.randint(0, 2))
    if kind == "zinv":
        return dict(kind="zinv", n=_log(rng, 20, 384), batch=_log(rng, 1, 64))
    return dict(kind="dec", n=_log(rng, 20, 200), batch=_log(rng, 1, 32))


# ---------------------------------------------------------------- inputs
_contexts = {}


def _context(**options):
    """One context per option set for the whole program, as a host code keeps it."""
    key = tuple(sorted(options.items()))
    if key not in _contexts:
        _contexts[key] = native.Context(0, **options)
    return _contexts[key]


class _State:
    """Uploaded devices (released with the state) and the call to make."""

    def __init__(self):
        self.call = None

    def own(self, ctx, did):
        weakref.finalize(self, ctx.release, did)
        return did


def _pl_sizes(case, rng):
    n = case["n"]
    return [n] + [int(rng.integers(max(2, n // 2), n + 1)) for _ in range(case["nbl"] - 2)] + [max(2, (4 * n) // 5)]


def _devices(case, seed):
    """The host description(s) of a case's device."""
    k = case["kind"]
    rng = np.random.default_rng(seed)
    if k == "pairs":
        nbl = case["nbl"]
        return [G.uneven(_pl_sizes(case, rng), seed=seed, cblk=[1, (nbl + 1) // 2, nbl])]
    if k in ("scba", "rho"):
        return [G.transport_c0(nbl=case["nbl"], n=case["n"], seed=seed)]
    if case["s"]:
        dens = min(1.0, max(0.1, 6.0 / case["n"]))
        return G.transport_c1_kpoints([0.4 + 0.9 * i for i in range(case.get("kpts", 1))], nbl=case["nbl"],
                                      n=case["n"], seed=seed, density=dens)
    return [G.transport_c0(nbl=case["nbl"], n=case["n"], seed=seed + 1000 * i) for i in range(case.get("kpts", 1))]


def _points(case, seed):
    """Energies (and the device index of each) of a case."""
    rng = np.random.default_rng(seed + 77)
    nk, pts = case.get("kpts", 1), case["pts"]
    per = -(-pts // nk)
    lo, hi = -1.5, 1.5
    h = (hi - lo) / per
    E = np.concatenate([lo + h * (np.arange(per) + rng.uniform(0.1, 0.9)) for _ in range(nk)])[:pts]
    return np.ascontiguousarray(E), np.repeat(np.arange(nk), per)[:pts].astype(np.int32)


def _ldos_sets(dev):
    half = dev.norb // 2
    return [list(range(1, half + 1)), list(range(half + 1, dev.norb + 1)), list(range(1, dev.norb + 1, 3))]


PAIRS = [(1, 2), (1, 3), (2, 3)]


def _frm(E):
    f = lambda mu: 1.0 / (np.exp((E - mu) / 0.05) + 1.0)
    return np.stack([f(0.3), f(-0.3)], axis=1)


def _contour(case):
    return D.contour_points(-4.0, 0.0, 0.025, 10.0, case["np1"], case["np2"], case["poles"])


def _blocks(case, seed, count):
    """Seeded complex Gaussian blocks on the GPU, column major per block."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["batch"], case["n"], case["n"])
    return [torch.complex(torch.randn(shape, dtype=torch.float64, device="cuda", generator=g),
                          torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)) for _ in range(count)]


def _lead_blocks(case, seed):
    """Ao, Bo, Co of the leads of `batch` energies of one wide lead, column major."""
    n, dev = case["n"], G.transport_c0(nbl=2, n=case["n"], seed=seed)
    h00, h01 = (torch.from_numpy(x[1]).cuda() for x in (dev.lead_h00, dev.lead_h01))
    E, _ = _points(dict(pts=case["batch"]), seed)
    z = torch.from_numpy(E).cuda().to(torch.complex128)[:, None, None] + 1j * ETA
    eye = torch.eye(n, dtype=torch.complex128, device="cuda")
    cm = lambda a: a.transpose(1, 2).contiguous()     # column major per block
    Ao = z * eye - h00
    Bo = (-h01).expand(case["batch"], n, n)
    Co = (-h01.conj().T).expand(case["batch"], n, n)
    return cm(Ao), cm(Bo), cm(Co)


def prepare(case, seed):
    k, st = case["kind"], _State()
    L = native.load()
    stream = torch.cuda.current_stream().cuda_stream if torch.cuda.is_available() else 0
    sp = ctypes.c_void_p(stream)
    if k == "zgemm":
        n, b = case["n"], case["batch"]
        A, B = _blocks(case, seed, 2)
        C = torch.zeros_like(A)
        one = (ctypes.c_double * 2)(1.0, 0.0)
        zero = (ctypes.c_double * 2)(0.0, 0.0)
        dp = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))
        args = (b, n, n, n, one, dp(A), 2 * n * n, dp(B), 2 * n * n, zero, dp(C), 2 * n * n, case["dagger"], sp)
        st.keep = (A, B, C, one, zero)

        def call():
            _ok(L.negf_b200_zgemm_batched(*args))
            return C
    elif k == "zinv":
        n, b = case["n"], case["batch"]
        (A,) = _blocks(case, seed, 1)
        A += 3.0 * math.sqrt(n) * torch.eye(n, dtype=A.dtype, device=A.device)
        X = torch.zeros_like(A)
        info = torch.zeros(b, dtype=torch.int32, device="cuda")
        work = torch.empty(int(L.negf_b200_zinv_work_bytes(b, n)), dtype=torch.uint8, device="cuda")
        dp = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))
        args = (b, n, dp(A), dp(X), ctypes.cast(info.data_ptr(), ctypes.POINTER(ctypes.c_int32)),
                ctypes.c_void_p(work.data_ptr()), sp)
        st.keep = (A, X, info, work)

        def call():
            _ok(L.negf_b200_zinv_batched(*args))
            return X, info
    elif k == "dec":
        n, b = case["n"], case["batch"]
        Ao, Bo, Co = _lead_blocks(case, seed)
        Go = torch.zeros_like(Ao)
        nc = torch.zeros(b, dtype=torch.int32, device="cuda")
        work = torch.empty(int(L.negf_b200_decimation_work_bytes(b, n)), dtype=torch.uint8, device="cuda")
        dp = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))
        args = (b, n, dp(Ao), dp(Bo), dp(Co), dp(Go), ctypes.cast(nc.data_ptr(), ctypes.POINTER(ctypes.c_int32)),
                1e-9, 300, ctypes.c_void_p(work.data_ptr()), sp)
        st.keep = (Ao, Bo, Co, Go, nc, work)

        def call():
            _ok(L.negf_b200_decimation_batched(*args))
            return Go, nc
    else:
        options = {}
        if k == "mixed":
            options = dict(precision=8)
        if k == "scba":
            options = dict(scba_niter=case["niter"])
        ctx = _context(**options)
        devs = _devices(case, seed)
        ids = np.array([st.own(ctx, ctx.upload(d)) for d in devs], dtype=np.int32)
        did = int(ids[0])
        if k == "rho":
            z, w = _contour(case)

            def call():
                (d, u, l), (dc, cd), nc, status = ctx.density(did, z, w)
                return d, u, l, dc, cd, nc, status
        else:
            E, which = _points(case, seed)
            if k == "pairs":
                ctx.set_dos_proj(did, _ldos_sets(devs[0]))
                call = lambda: ctx.transmissions(did, E, PAIRS, eta=ETA, ldos=True, dos_delta=DOS_DELTA)
            elif k == "scba":
                frm, cpl = _frm(E), np.full(devs[0].norb, 0.05)

                def call():
                    r = ctx.meir_wingreen(did, E, frm, coupling=cpl, eta=ETA)
                    return [r[q] for q in ("curr", "layer_curr", "layer_dens", "scba_iter", "ncyc", "status")]
            elif k == "DOS":
                pid = ids[which]
                call = lambda: ctx.transmission_dos(pid, E, eta=ETA, dos_delta=DOS_DELTA)
            else:
                call = lambda: ctx.transmission(did, E, eta=ETA)
    st.call = call
    return st


def _ok(rc):
    if rc != 0:
        raise RuntimeError("status %d" % rc)


def run(state):
    return state.call()


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    k, n = case["kind"], case["n"]
    unit = 8.0 * n ** 3                       # one complex block product or inverse
    blk = 16.0 * n * n
    if k == "zgemm":
        return dict(bytes=3 * blk * case["batch"], flops=unit * case["batch"])
    if k == "zinv":
        return dict(bytes=2 * blk * case["batch"], flops=unit * case["batch"])
    if k == "dec":
        return dict(bytes=4 * blk * case["batch"], flops=(7 * DEC_ITERS + 1) * unit * case["batch"])
    nbl = case["nbl"]
    pts = case["np1"] + case["np2"] + case["poles"] if k == "rho" else case["pts"]
    per_layer = {"T": 3, "mixed": 3, "DOS": 7, "pairs": 7, "scba": 18, "rho": 9}[k]
    if k == "scba":
        per_layer *= case["niter"]
    ncont = 3 if k == "pairs" else 2
    if k == "pairs":
        unit *= 0.45                          # layers of half to the full size
        blk *= 0.6
    units = nbl * per_layer + ncont * (7 * DEC_ITERS + 3) + 2
    ns = 2 if case.get("s") else 1
    blocks = case.get("kpts", 1) * ns * (3 * nbl + 2 * ncont + ncont)
    out = 8.0 * pts * (1 + (nbl * n if k in ("DOS", "pairs") else 0)) + (3 * blk * nbl if k == "rho" else 0)
    return dict(bytes=blocks * blk + out, flops=units * unit * pts)


# ---------------------------------------------------------------- the same outputs in plain 64-bit torch
def _t(x):
    x = torch.from_numpy(np.ascontiguousarray(x, dtype=np.complex128))
    return x.cuda() if torch.cuda.is_available() else x


def _dag(a):
    return a.conj().transpose(-1, -2)


def _spec(a):
    return 1j * (a - _dag(a))


def _tr(a):
    return a.diagonal(dim1=-2, dim2=-1).sum(-1)


def _decimate(A, B, C, tol=1e-9):
    As, ok = A.clone(), 0
    for _ in range(300):
        g = torch.linalg.inv(A)
        x = g @ C
        C1 = C @ x
        ok = ok + 1 if float(C1.abs().max()) <= tol else 0
        if ok > 1:
            break
        s = B @ x
        y = g @ B
        As = As - s
        A = A - s - C @ y
        B, C = B @ y, C1
    return torch.linalg.inv(As)


def _contact(dev, c, z):
    """(surface GF, Tlc, Tcl, self-energy) of contact c at the energies z (npts)."""
    z = z[:, None, None]
    L = dev.lead_h00[c].shape[0]
    eye = torch.eye(L, dtype=torch.complex128, device=z.device)
    s00 = eye if dev.lead_s00 is None else _t(dev.lead_s00[c])
    s01 = torch.zeros_like(eye) if dev.lead_s01 is None else _t(dev.lead_s01[c])
    h00, h01, hmc = _t(dev.lead_h00[c]), _t(dev.lead_h01[c]), _t(dev.hmc[c])
    smc = torch.zeros_like(hmc) if dev.smc is None else _t(dev.smc[c])
    gs = _decimate(z * s00 - h00, z * s01 - h01, _dag(z.conj() * s01 - h01))
    tlc, tcl = z * smc - hmc, _dag(z.conj() * smc - hmc)
    return gs, tlc, tcl, tlc @ gs @ tcl


def _esh(dev, z, sig):
    z = z[:, None, None]
    i = lambda m: torch.eye(m, dtype=torch.complex128, device=z.device)
    no_s = dev.s_diag is None
    d = [z * (i(h.shape[0]) if no_s else _t(dev.s_diag[q])) - _t(h) for q, h in enumerate(dev.h_diag)]
    u = [z * (0.0 if no_s else _t(dev.s_upper[q])) - _t(h) for q, h in enumerate(dev.h_upper)]
    l = [z * (0.0 if no_s else _t(dev.s_lower[q])) - _t(h) for q, h in enumerate(dev.h_lower)]
    for c, cb in enumerate(dev.cblk):
        d[cb - 1] = d[cb - 1] - sig[c]
    return d, u, l


def _diag_green(d, u, l, every):
    """Gr(1,1) (or every diagonal block) by the recursive sweeps."""
    nbl = len(d)
    g = [None] * nbl
    g[-1] = torch.linalg.inv(d[-1])
    for q in range(nbl - 2, -1, -1):
        g[q] = torch.linalg.inv(d[q] - u[q] @ g[q + 1] @ l[q])
    G = [g[0]]
    for q in range(1, nbl if every else 1):
        G.append(g[q] + g[q] @ l[q - 1] @ G[-1] @ u[q - 1] @ g[q])
    return G


def _dense(dev, z, sig):
    d, u, l = _esh(dev, z, sig)
    off = np.concatenate([[0], np.cumsum(dev.pl_size)])
    M = torch.zeros((z.shape[0], off[-1], off[-1]), dtype=torch.complex128, device=z.device)
    sl = [slice(int(off[q]), int(off[q + 1])) for q in range(dev.nbl)]
    for q in range(dev.nbl):
        M[:, sl[q], sl[q]] = d[q]
        if q + 1 < dev.nbl:
            M[:, sl[q], sl[q + 1]] = u[q]
            M[:, sl[q + 1], sl[q]] = l[q]
    return M, sl


def _np(a):
    return a.cpu().numpy()


def _exact_t(devs, E, which, want_dos):
    T = np.zeros(E.size)
    dos = np.zeros((E.size, devs[0].norb))
    for k, dev in enumerate(devs):
        at = np.nonzero(which == k)[0]
        for q in range(0, at.size, 64):
            sel = at[q:q + 64]
            e = _t(E[sel])
            sig = [_contact(dev, c, e + 1j * ETA)[3] for c in range(2)]
            d, u, l = _esh(dev, e + (1j * DOS_DELTA if want_dos else 0.0), sig)
            Gd = _diag_green(d, u, l, want_dos)
            gam, g = _spec(sig[0]), Gd[0]
            T[sel] = _np((_tr(gam @ _spec(g)) - _tr(gam @ g @ gam @ _dag(g))).real.abs())
            if want_dos:
                dos[sel] = _np(torch.cat([-x.diagonal(dim1=-2, dim2=-1).imag / math.pi for x in Gd], dim=1))
    return T, dos


def _exact_pairs(dev, E):
    e = _t(E)
    sig = [_contact(dev, c, e + 1j * ETA)[3] for c in range(dev.ncont)]
    M, sl = _dense(dev, e + 1j * DOS_DELTA, sig)
    Gr = torch.linalg.inv(M)
    T = []
    for ni, nf in PAIRS:
        a, b = (ni, nf) if dev.cblk[ni - 1] < dev.cblk[nf - 1] else (nf, ni)
        g = Gr[:, sl[dev.cblk[b - 1] - 1], sl[dev.cblk[a - 1] - 1]]
        T.append(_tr(_spec(sig[b - 1]) @ g @ _spec(sig[a - 1]) @ _dag(g)).real.abs())
    dos = -Gr.diagonal(dim1=-2, dim2=-1).imag / math.pi
    led = [dos[:, torch.tensor(s, device=dos.device) - 1].sum(1) for s in _ldos_sets(dev)]
    return _np(torch.stack(T, 1)), _np(torch.stack(led, 1))


def _exact_scba(dev, E, frm, cpl, niter, tol=1e-7):
    e, f, c2 = _t(E), _t(frm), _t(cpl * cpl)
    sig = [_contact(dev, c, e + 1j * ETA)[3] for c in range(2)]
    M, sl = _dense(dev, e, sig)
    blk = [sl[cb - 1] for cb in dev.cblk]
    gam = [_spec(s) for s in sig]
    npts, norb = M.shape[0], M.shape[1]
    sr = torch.zeros((npts, norb), dtype=torch.complex128, device=M.device)
    sn, old = torch.zeros_like(sr), None
    done = torch.zeros(npts, dtype=torch.bool, device=M.device)
    Gr = Gn = None
    for it in range(niter + 1):
        g = torch.linalg.inv(M - torch.diag_embed(sr))
        s = torch.diag_embed(sn)
        for c in range(2):
            s[:, blk[c], blk[c]] += f[:, c, None, None] * gam[c]
        gn = g @ s @ _dag(g)
        Gr = g if Gr is None else torch.where(done[:, None, None], Gr, g)
        Gn = gn if Gn is None else torch.where(done[:, None, None], Gn, gn)
        new = Gn.diagonal(dim1=-2, dim2=-1)
        if old is not None:
            done = done | ((new - old).abs().max(1).values < tol)
        old, sr, sn = new.clone(), c2 * Gr.diagonal(dim1=-2, dim2=-1), c2 * new
        if bool(done.all()):
            break
    curr = [-(_tr(gam[c] @ Gn[:, blk[c], blk[c]]) - f[:, c] * _tr(gam[c] @ _spec(Gr[:, blk[c], blk[c]]))).real
            for c in range(2)]
    lc = [-(_tr(M[:, sl[q], sl[q + 1]] @ Gn[:, sl[q + 1], sl[q]])
            - _tr(Gn[:, sl[q], sl[q + 1]] @ M[:, sl[q + 1], sl[q]])).imag for q in range(dev.nbl - 1)]
    ld = [_tr(Gn[:, s, s]).real for s in sl]
    return [_np(torch.stack(x, 1)) for x in (curr, lc, ld)]


def _exact_rho(dev, z, w):
    zt, wt = _t(z), _t(w)[:, None, None]
    cont = [_contact(dev, c, zt) for c in range(2)]
    M, sl = _dense(dev, zt, [x[3] for x in cont])
    Gr = torch.linalg.inv(M)
    R = _spec((wt * Gr).sum(0))
    d = [_np(R[s, s]) for s in sl]
    u = [_np(R[sl[q], sl[q + 1]]) for q in range(dev.nbl - 1)]
    l = [_np(R[sl[q + 1], sl[q]]) for q in range(dev.nbl - 1)]
    dc, cd = [], []
    for c, (gs, tlc, tcl, _) in enumerate(cont):
        on = _t(dev.hmc[c] != 0).real
        g = Gr[:, sl[dev.cblk[c] - 1], sl[dev.cblk[c] - 1]]
        lc = (wt * -(g @ tlc @ gs)).sum(0) * on
        cl = (wt * -(gs @ tcl @ g)).sum(0) * on.T
        dc.append(_np(1j * (lc - _dag(cl))))
        cd.append(_np(1j * (cl - _dag(lc))))
    return d, u, l, dc, cd


def exact(case, seed):
    k = case["kind"]
    if k == "zgemm":
        A, B = (x.transpose(1, 2) for x in _blocks(case, seed, 2))
        A = _dag(A) if case["dagger"] == 1 else A
        B = _dag(B) if case["dagger"] == 2 else B
        return (A @ B).transpose(1, 2).contiguous()
    if k == "zinv":
        (A,) = _blocks(case, seed, 1)
        A += 3.0 * math.sqrt(case["n"]) * torch.eye(case["n"], dtype=A.dtype, device=A.device)
        return torch.linalg.inv(A), None
    if k == "dec":
        Ao, Bo, Co = (x.transpose(1, 2) for x in _lead_blocks(case, seed))
        return _decimate(Ao, Bo, Co).transpose(1, 2).contiguous(), None
    devs = _devices(case, seed)
    if k == "rho":
        return (*_exact_rho(devs[0], *_contour(case)), None, None)
    E, which = _points(case, seed)
    if k == "pairs":
        return (*_exact_pairs(devs[0], E), None, None)
    if k == "scba":
        return [*_exact_scba(devs[0], E, _frm(E), np.full(devs[0].norb, 0.05), case["niter"]), None, None, None]
    T, dos = _exact_t(devs, E, which, k == "DOS")
    return (T, dos, None, None) if k == "DOS" else (T, None, None)
