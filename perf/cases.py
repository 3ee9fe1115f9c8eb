"""What is measured: calls of the electron-phonon stage as a user's program makes them.

Every case is one system (crystal cell, k-grid, spheres, bands, KB projectors),
made by letzelphc_gb300.synth with wavefunctions, dV_scf and eigenvectors drawn
from the seed, held by one LelphGPU context, and one public entry point:

  call = "unfold_run"  prepare() on the resident wavefunctions, then run_device()
                       on every (q, k) pair: the stage after a wavefunction update
         "run"         run_device() on every (q, k) pair of a prepared context
         "elphq"       compute_elphq(): the reference's per-q stage, host dV in,
                       host matrix elements out
         "star"        compute_elphq_star(): the same with the q-star expansion
         "dmats"       dmats(): representation matrices of some symmetries at every k
         "ingest"      set_q_dvscf_qe(): a q-point loaded from QE's file layout

exact() restates the path with torch in 64 bits (G-space order: FFT of dV psi_k
per mode and band, contraction over the k+q sphere, KB term), with the truncated
pi that the path's conventions prescribe.
"""
import dataclasses
import math

import numpy as np
import torch

from letzelphc_gb300 import synth
from letzelphc_gb300.elph import LelphGPU, OUT_C64, OUT_C128

PI = synth.ELPH_PI


def _case(name, call, kind, a, fft, k, nq, bands, npw, precision, spin="none", timerev=False, lmax=1, nsym=0):
    c = dict(call=call, kind=kind, a=a, fft="x".join(map(str, fft)), k="x".join(map(str, k)), nq=nq, bands=bands,
             npw_lo=npw[0], npw_hi=npw[1], precision=precision, spin=spin, timerev=timerev, lmax=lmax, nsym=nsym)
    if name:
        c["name"] = name
    return c


def listed():
    l12 = ("l12", 7.1, (48, 48, 48))
    return [
        # smallest call: one q of a 2-atom crystal, 64 k-points, 8 bands, in the default (FP64) precision --
        # a convergence test on a small cell, where launches and host work count
        _case("small_q_fp64", "elphq", "diamond", 10.26, (24, 24, 24), (4, 4, 4), 1, 8, (400, 400), "fp64"),
        # the same call in the mixed form
        _case("small_q_mixed", "elphq", "diamond", 10.26, (24, 24, 24), (4, 4, 4), 1, 8, (400, 400), "mixed"),
        # the production batch of the benchmark's cell: 8 q x 512 k, 12 modes, 32 bands, from the resident
        # plane-wave coefficients to complex64 matrix elements on the device
        _case("l12_batch_mixed", "unfold_run", *l12, (8, 8, 8), 8, 32, (2500, 2500), "mixed"),
        # one q of the same cell the way the reference's driver calls its stage: host dV in, host complex128 out
        _case("l12_q_host_mixed", "elphq", *l12, (8, 8, 8), 1, 32, (2500, 2500), "mixed"),
        # 2-D slab with vacuum, hexagonal cell, ragged spheres (npw differs from k to k), long z axis
        _case("slab_batch_mixed", "run", "hex2d", 6.0, (36, 36, 216), (12, 12, 1), 4, 40, (1800, 2600), "mixed"),
        # spinors with spin-orbit coupling, nmag = 4, d projectors, 64 bands: the widest real-space tile
        _case("soc_batch_mixed", "run", "rocksalt8", 8.0, (60, 60, 60), (4, 4, 4), 1, 64, (5000, 5000), "mixed",
              spin="soc", lmax=2),
        # a 16-atom cell with 200 bands (beyond the real-space tile): the G-space route
        _case("wide_batch_mixed", "run", "sc16", 10.0, (96, 96, 96), (2, 2, 2), 1, 200, (12000, 12000), "mixed"),
        # the FP64 form, which results are validated with
        _case("l12_batch_fp64", "unfold_run", *l12, (4, 4, 4), 1, 32, (2500, 2500), "fp64"),
        # collinear spins, time reversal, an odd band count, small ragged spheres
        _case("lsda_odd_mixed", "unfold_run", "zincblende", 10.2, (30, 30, 32), (6, 6, 6), 3, 13, (350, 700), "mixed",
              spin="lsda", timerev=True),
        # representation matrices of 8 symmetries at 512 k: what the driver writes before the q loop
        _case("dmats_mixed", "dmats", *l12, (8, 8, 8), 0, 32, (2500, 2500), "mixed", nsym=8),
        # an irreducible q expanded over its star of 12, Dmats made on the way
        _case("star_mixed", "star", *l12, (4, 4, 4), 1, 32, (2500, 2500), "mixed"),
        # a q-point read from a QE dvscf file: pattern basis to modes, (z, y, x) to (x, y, z)
        _case("ingest_qe", "ingest", *l12, (4, 4, 4), 1, 32, (2500, 2500), "mixed"),
    ]


_LATTICE = {"diamond": (10.26, 2, "3"), "zincblende": (10.2, 2, "3"), "l12": (7.1, 4, "3"),
            "hex2d": (6.0, 3, "2"), "rocksalt8": (8.0, 8, "3")}


def _friendly(n, even):
    while True:
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1 and n % even == 0:
            return n
        n += 1


def _box(kind, a, npw):
    """A QE-like FFT box for spheres of npw plane waves: about 4.2 times the sphere's radius on each axis."""
    A = synth._structure(kind, a)[0]
    gc = math.sqrt(synth._ecut_for(npw, np.linalg.inv(A).T, 0))
    return tuple(_friendly(int(4.2 * np.linalg.norm(A[:, i]) * gc) + 3, 2 if i == 1 else 4) for i in range(3))


def draw(rng):
    call = rng.choice(["unfold_run", "run", "run", "elphq", "dmats", "star", "ingest"])
    kind = rng.choice(["diamond", "zincblende", "l12", "hex2d", "rocksalt8"])
    a, natom, dim = _LATTICE[kind]
    npw = int(math.exp(rng.uniform(math.log(250), math.log(2800))))
    ragged = rng.random() < 0.5
    lo, hi = (int(0.75 * npw), npw) if ragged else (npw, npw)
    n = rng.choice([2, 3, 4, 5, 6])
    k = (n, n, 1) if dim == "2" else (n, n, n)
    bands = int(math.exp(rng.uniform(math.log(3), math.log(64.99))))
    spin = rng.choice(["none", "none", "none", "lsda", "soc"])
    precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
    if call == "star":
        bands = min(bands, 56)  # the star rotation holds four band x band matrices in shared memory
    nq = 1 if call in ("elphq", "star", "ingest") else 0 if call == "dmats" else rng.choice([1, 2, 3])
    fft = _box(kind, a, hi)
    # no drawn case above a share of the largest listed one
    npairs = max(1, nq) * int(np.prod(k))
    ns = 2 if spin == "soc" else 1
    cost = npairs * 3 * natom * bands * max(8, bands) * (2 if spin == "lsda" else ns * ns) * npw
    cap = 2.0e11 if precision == "mixed" else 6.0e9
    if cost > cap:
        bands = max(3, int(bands * math.sqrt(cap / cost)))
    return _case(None, call, kind, a, fft, k, nq, bands, (lo, hi), precision, spin=spin,
                 timerev=kind == "zincblende" and rng.random() < 0.5, lmax=rng.choice([1, 1, 2]),
                 nsym=rng.choice([1, 2, 4]) if call == "dmats" else 0)


# ------------------------------------------------------------------ inputs

_geometry = {}


def _ints(text):
    return tuple(int(v) for v in text.split("x"))


def _structure_of(case):
    """Cell, symmetries, k-points, spheres and form factors: the same for every seed."""
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "call", "nq", "bands", "precision", "nsym")))
    if key not in _geometry:
        o = dict(kind=case["kind"], a=case["a"], fft=_ints(case["fft"]), kgrid=_ints(case["k"]), qpts=[], nbnds=1,
                 npw=(case["npw_lo"], case["npw_hi"]) if case["npw_lo"] < case["npw_hi"] else case["npw_lo"],
                 ls=tuple(range(case["lmax"] + 1)), seed=1000, timerev=case["timerev"])
        if case["spin"] == "soc":
            o.update(nspinor=2, nmag=4, soc=True)
        if case["spin"] == "lsda":
            o.update(nspin=2, nmag=2)
        if len(_geometry) > 32:
            _geometry.clear()
        _geometry[key] = synth.make_system("case", o)
    return _geometry[key]


def _qpoints(case):
    """The first nq irreducible points of the k-grid after Gamma (Gamma too when there are several)."""
    s = _structure_of(case)
    q = synth.reduce_grid(_ints(case["k"]), s.sym_R, s.alat)
    n = case["nq"]
    if n == 1 and len(q) > 1:
        return q[-1:] if case["call"] != "star" else q[len(q) // 2:len(q) // 2 + 1]
    return q[:n]


def _cplx(gen, *shape):
    return torch.complex(torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64),
                         torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64))


def _system(case, seed):
    """The system with the seed's wavefunctions (orthonormal), eigenvectors (unitary) and dV_scf (smooth, unit rms)."""
    s = _structure_of(case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))
    nb, nm = case["bands"], s.nmodes
    wfc = []
    for m in s.miller:
        c = _cplx(gen, s.nspin, s.nspinor * len(m), nb)
        q = torch.linalg.qr(c)[0].transpose(1, 2).contiguous()
        wfc.append(q.reshape(s.nspin, nb, s.nspinor, len(m)).cpu().numpy())
    N = s.fft_dims
    f = [torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64) for n in N]
    Mi = torch.stack(torch.meshgrid(*f, indexing="ij"), -1)
    G2 = ((Mi @ torch.tensor(np.linalg.inv(s.alat), device="cuda")) ** 2).sum(-1)
    gcut = math.sqrt(synth._ecut_for(float(np.mean([len(m) for m in s.miller])), np.linalg.inv(s.alat).T, 0))
    gauss = torch.exp(-G2 / (2.0 * (0.3 * gcut) ** 2))
    qs = _qpoints(case)
    eig, dv = [], []
    for _ in qs:
        v = torch.fft.ifftn(_cplx(gen, nm, s.nmag, *N) * gauss, dim=(2, 3, 4))
        v /= (v.abs() ** 2).mean().sqrt()
        dv.append(v.cpu().numpy())
        eig.append(torch.linalg.qr(_cplx(gen, nm, nm))[0].cpu().numpy())
        del v
    torch.cuda.empty_cache()
    return dataclasses.replace(s, nbnds=nb, wfc=wfc, qpts=qs, eigVec=eig, dVscf=dv)


def _patterns(s, seed):
    """QE's displacement patterns (unitary) of a file."""
    rng = np.random.default_rng(int(seed) % (1 << 62))
    z = rng.standard_normal((s.nmodes, s.nmodes)) + 1j * rng.standard_normal((s.nmodes, s.nmodes))
    return np.linalg.qr(z)[0]


def _star_symmetries(s, q):
    """First symmetry that produces each member of the star of q, the identity first."""
    qc = np.linalg.inv(s.alat).T @ q
    seen, syms = np.zeros((0, 3)), []
    for i, R in enumerate(s.sym_R):
        sq = s.alat.T @ (R @ qc)
        if synth.find_kidx_in_list(seen, sq) < 0:
            seen = np.vstack([seen, sq])
            syms.append(i)
    return syms


def prepare(case, seed):
    s = _system(case, seed)
    ctx = LelphGPU(s, case["precision"])
    st = {"call": case["call"], "s": s, "ctx": ctx}
    if case["call"] in ("run", "unfold_run"):
        for i, q in enumerate(s.qpts):
            ctx.set_q(i, q, s.eigVec[i], s.dVscf[i])
        ctx.prepare()
        st["qslots"] = np.repeat(np.arange(len(s.qpts), dtype=np.int32), s.nk_bz)
        st["kbz"] = np.tile(np.arange(s.nk_bz, dtype=np.int32), len(s.qpts))
        st["out"] = OUT_C64 if case["precision"] == "mixed" else OUT_C128
        st["g"] = torch.empty((len(st["kbz"]), s.nmodes, s.nspin, s.nbnds, s.nbnds), device="cuda",
                              dtype=torch.complex64 if case["precision"] == "mixed" else torch.complex128)
    elif case["call"] == "star":
        st["syms"] = _star_symmetries(s, s.qpts[0])
        st["out"] = OUT_C64 if case["precision"] == "mixed" else OUT_C128
        ctx.prepare()
    elif case["call"] == "elphq":
        ctx.prepare()
    elif case["call"] == "ingest":
        st["pats"] = _patterns(s, seed)
        st["raw"] = np.ascontiguousarray(np.transpose(s.dVscf[0], (0, 1, 4, 3, 2)))
    elif case["call"] == "dmats":
        n = min(case["nsym"], len(s.sym_R))
        pick = np.linspace(0, len(s.sym_R) - 1, n).astype(int)
        st["ops"] = (s.sym_R[pick], s.sym_tau[pick], s.sym_trev[pick])
    return st


def run(st):
    s, ctx, call = st["s"], st["ctx"], st["call"]
    if call == "unfold_run":
        ctx.prepare()
    if call in ("run", "unfold_run"):
        ctx.run_device(st["qslots"], st["kbz"], st["g"].data_ptr(), out=st["out"])
        return st["g"]
    if call == "elphq":
        return ctx.compute_elphq(s.qpts[0], s.eigVec[0], s.dVscf[0])
    if call == "star":
        return ctx.compute_elphq_star(s.qpts[0], s.eigVec[0], s.dVscf[0], st["syms"], out=st["out"])
    if call == "dmats":
        return ctx.dmats(*st["ops"])
    return ctx.set_q_dvscf_qe(0, s.qpts[0], s.eigVec[0], st["pats"], st["raw"], want_dv=True)


# ------------------------------------------------------------------ floors

def work(case):
    """Inputs read once, outputs written once.  Flops of a (q, k) pair: the product dV psi_k on the 8 npw
    differences G' - G of its spheres for every (mode, band of k), and the cheaper of transforming it (5 M log2 M)
    and contracting over the k+q sphere, and contracting it on those M points directly."""
    s = _structure_of(case)
    nb, nm, ns = case["bands"], s.nmodes, s.nspinor
    npw = 0.5 * (case["npw_lo"] + case["npw_hi"])
    N = float(np.prod(s.fft_dims))
    mixed = case["precision"] == "mixed"
    wfc = 16.0 * s.nk_ibz * s.nspin * nb * ns * npw
    dv = 16.0 * nm * s.nmag * N
    nq = len(_qpoints(case)) if case["nq"] else 0
    if case["call"] == "ingest":
        return {"bytes": 2 * dv, "flops": 8.0 * nm * nm * s.nmag * N}
    if case["call"] == "dmats":
        n = float(min(case["nsym"], len(s.sym_R)) * s.nk_bz * s.nspin)
        return {"bytes": wfc + 16.0 * n * nb * nb, "flops": 8.0 * n * nb * nb * ns * npw}
    M = 8.0 * npw
    rows = float(nm * nb * ns * s.nspin)
    pair = rows * (8.0 * ns * M + min(5.0 * M * math.log2(M) + 8.0 * nb * npw, 8.0 * nb * M))
    pairs = nq * s.nk_bz
    out = (8.0 if mixed and case["call"] != "elphq" else 16.0) * nm * s.nspin * nb * nb * pairs
    flops = pair * pairs
    nbytes = out + nq * dv + wfc
    if case["call"] == "star":
        m = len(_star_symmetries(s, _qpoints(case)[0])) - 1
        flops += m * s.nk_bz * s.nspin * (8.0 * nb * nb * ns * npw + 16.0 * nm * nb ** 3)
        nbytes += m * out
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ 64-bit restatement

def _t(x):
    return torch.as_tensor(np.asarray(x), device="cuda")


def _su2(R, trev):
    """Spinor rotation of a (possibly improper) operation, -i sigma_y after it for time reversal."""
    s = (R / np.linalg.det(R)).reshape(9)
    if abs(s[6] + 1) < 1e-5:
        al, be, de = 0.0, PI / 2.0, math.atan2(s[1], s[2])
    elif abs(s[6] - 1) < 1e-5:
        al, be, de = 0.0, -PI / 2.0, math.atan2(-s[1], -s[2])
    else:
        be = -math.asin(s[6])
        al = math.atan2(s[3] / math.cos(be), s[0] / math.cos(be))
        de = math.atan2(s[7] / math.cos(be), s[8] / math.cos(be))
    px, py, pz = np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.diag([1, -1])
    one = np.eye(2)
    u = ((math.cos(al / 2) * one - 1j * math.sin(al / 2) * pz) @ (math.cos(be / 2) * one - 1j * math.sin(be / 2) * py)
         @ (math.cos(de / 2) * one - 1j * math.sin(de / 2) * px))
    return np.array([[0, -1], [1, 0]]) @ u if trev else u


def _spin(u, w):
    return w if w.shape[-2] == 1 else torch.einsum("ab,...bp->...ap", _t(u), w)


def _crys(s, tau):
    return s.blat.T @ tau / (2 * PI)


def _unfold(s, k):
    """Miller indices, coefficients (spin, band, spinor, npw) and S(k+G) of full-BZ point k."""
    ik, sym = (int(v) for v in s.kmap[k])
    R, tr = s.sym_R[sym], bool(s.sym_trev[sym])
    W = np.rint(s.alat.T @ R @ np.linalg.inv(s.alat).T).astype(np.int64)
    n = s.miller[ik].astype(np.int64) @ W.T
    kc = s.alat.T @ (R @ s.kibz[ik])
    ph = np.exp(-2j * PI * ((n + kc) @ _crys(s, s.sym_tau[sym])))
    c = _spin(_su2(R, tr), _t(s.wfc[ik])) * _t(ph)
    return n, (c.conj().resolve_conj() if tr else c), (s.gvec[ik] + s.kibz[ik]) @ R.T


def _ylm(l, m, v):
    """Real spherical harmonics of the rows of v, without the Condon-Shortley sign; 0 (l > 0) at the origin."""
    r = np.sqrt((v * v).sum(1))
    zero = r < 1e-6
    x = v[:, 2] / np.where(zero, 1.0, r)
    a = abs(m)
    p = np.ones(len(v))
    for i in range(1, a + 1):
        p = p * (2 * i - 1) * np.sqrt(np.maximum(0.0, 1 - x * x))
    lo, hi = np.zeros(len(v)), p
    for i in range(a + 1, l + 1):
        lo, hi = hi, ((2 * i - 1) * x * hi - (i + a - 1) * lo) / (i - a)
    phi = np.arctan2(v[:, 1], v[:, 0])
    ang = 1.0 if m == 0 else math.sqrt(2) * (np.cos(a * phi) if m > 0 else np.sin(a * phi))
    y = hi * ang * math.sqrt(math.factorial(l - a) * (2 * l + 1) / (4 * PI * math.factorial(l + a)))
    return np.where(zero, 0.0 if l else 1.0 / math.sqrt(4 * PI), y)


def _channels(s, it):
    return [(i, int(round(s.PP_table[i, it, 0] - 1))) for i in range(s.nltimesj)]


def _projections(s, k, c, K):
    """Per atom: sum_G beta_x(G) conj(c(G)), (projector, x, spin, band, spinor), x = 0 the projector, 1..3 times K_x."""
    ik = int(s.kmap[k][0])
    out = []
    for ia in range(s.natom):
        it = int(s.atom_type[ia])
        ph = np.exp(-2j * PI * (K @ s.atom_pos[ia]))
        b = []
        for i, l in _channels(s, it):
            for m in range(-l, l + 1):
                b0 = s.Fk[ik][i, it] * ph * _ylm(l, m, K)
                b.append(np.stack([b0] + [b0 * K[:, x] * s.Fsign[i, it] for x in range(3)]))
        out.append(torch.einsum("jxp,...p->jx...", _t(np.array(b)), c.conj()))
    return out


def _nonlocal(s, Pk, Pq, eig):
    """KB term (mode, spin, band of k, band of k+q)."""
    buf = []
    for ia in range(s.natom):
        it = int(s.atom_type[ia])
        n = Pk[ia].shape[0]
        f = np.zeros((n, n, s.nspinor, s.nspinor), complex)
        at = 0
        for i, l in _channels(s, it):
            w = 2 * l + 1
            fc = None if s.fCoeff is None else s.fCoeff[s.ntype * i + it]
            j = int(round(s.PP_table[i, it, 1]))
            fac = (j + 1.0) / (4.0 * l + 2.0) if j != 0 and not s.is_soc_present else 1.0
            blk = np.einsum("ij,st->ijst", np.eye(w), np.eye(s.nspinor)) * fac if fc is None else fc
            f[at:at + w, at:at + w] = blk
            at += w
        z = torch.einsum("ijst,jxamt->ixams", _t(f), Pk[ia].conj())
        buf.append(torch.einsum("ixans,iams->xamn", Pq[ia][:, 1:], z[:, 0])
                   - torch.einsum("ians,ixams->xamn", Pq[ia][:, 0], z[:, 1:]))
    return -2j * PI * synth.ELPH_E2 * torch.einsum("vj,jsmn->vsmn", _t(eig), torch.cat(buf))


def _kplus(s, q):
    d = s.kbz_crys[None] - (s.kbz_crys + q)[:, None]
    return [int(v) for v in np.argmin((np.abs(d - np.rint(d))).sum(-1), 1)]


def _elphq(s, iq):
    """g (k, mode, spin, band of k, band of k+q) of q-point iq."""
    q, eig, dv = s.qpts[iq], s.eigVec[iq], _t(s.dVscf[iq])
    N, nN = s.fft_dims, int(np.prod(s.fft_dims))
    nb, ns = s.nbnds, s.nspinor
    kq = _kplus(s, q)
    un, pr = {}, {}

    def get(k):
        if k not in un:
            if len(un) > 256:
                un.clear()
                pr.clear()
            un[k] = _unfold(s, k)
            pr[k] = _projections(s, k, un[k][1], un[k][2])
        return un[k], pr[k]
    g = torch.empty((s.nk_bz, s.nmodes, s.nspin, nb, nb), dtype=torch.complex128, device="cuda")
    step = max(1, int(2.0e8 // (nb * ns * nN)))
    for k in range(s.nk_bz):
        (n1, c1, K1), P1 = get(k)
        (n2, c2, K2), P2 = get(kq[k])
        ulm = np.rint(s.alat.T @ (_sk(s, kq[k]) - _sk(s, k)) - q).astype(np.int64)
        box = torch.zeros((s.nspin, nb, ns, nN), dtype=torch.complex128, device="cuda")
        box[..., _t(np.ravel_multi_index(tuple((n1 % N).T), N))] = c1
        psi = torch.fft.ifftn(box.reshape(s.nspin, nb, ns, *N), dim=(3, 4, 5), norm="forward")
        at = _t(np.ravel_multi_index(tuple(((n2 + ulm) % N).T), N))
        bs = nb if step > 1 else max(1, int(2.0e8 // (ns * nN)))
        for v in range(0, s.nmodes, step):
            for sp in range(s.nspin):
                for b in range(0, nb, bs):
                    p = psi[sp, b:b + bs]
                    d = dv[v:v + step]
                    if ns == 2 and s.nmag == 4:
                        d = d.reshape(d.shape[0], 2, 2, *N)
                        pd = torch.einsum("vstxyz,btxyz->vbsxyz", d, p)
                    else:
                        pd = d[:, None, sp:sp + 1] * p[None]
                    f = torch.fft.fftn(pd, dim=(3, 4, 5), norm="forward").reshape(d.shape[0], p.shape[0], ns, nN)
                    g[k, v:v + step, sp, b:b + bs] = torch.einsum("vmsp,nsp->vmn", f[..., at], c2[sp].conj())
                    del pd, f
        g[k] += _nonlocal(s, P1, P2, eig)
    return g


def _sk(s, k):
    return s.sym_R[s.kmap[k][1]] @ s.kibz[s.kmap[k][0]]


def _kcart(s):
    return s.kbz_crys @ s.blat.T / (2 * PI)


def _dmat(s, R, tau, trev, k):
    """<psi_{Rk, b}| U(R) |psi_{k, a}>, (spin, b, a)."""
    kR = _kplus_one(s, s.alat.T @ (R @ _kcart(s)[k]))
    n1, c1, _ = _unfold(s, k)
    n2, c2, _ = _unfold(s, kR)
    W = np.rint(s.alat.T @ R @ np.linalg.inv(s.alat).T).astype(np.int64)
    # U(R) on the unfolded state: rotate, translate, conjugate for time reversal (k -> -k is inside R)
    n = n1 @ W.T
    kc = s.alat.T @ (R @ _sk(s, k))
    a = _spin(_su2(R, trev), c1) * _t(np.exp(-2j * PI * ((n + kc) @ _crys(s, tau))))
    a = a.conj() if trev else a
    ulm = np.rint(s.alat.T @ (_sk(s, kR) - R @ _sk(s, k))).astype(np.int64)
    N = s.fft_dims
    pos = torch.full((int(np.prod(N)),), -1, dtype=torch.long, device="cuda")
    pos[_t(np.ravel_multi_index(tuple((n % N).T), N))] = torch.arange(len(n), device="cuda")
    to = pos[_t(np.ravel_multi_index(tuple(((n2 + ulm) % N).T), N))]
    b = c2[..., to >= 0]
    return torch.einsum("sbtp,satp->sba", b.conj(), a[..., to[to >= 0]])


def _kplus_one(s, k):
    d = s.kbz_crys - k
    return int(np.argmin(np.abs(d - np.rint(d)).sum(-1)))


def exact(case, seed):
    if case.get("name") == "l12_batch_mixed":
        return None  # 4096 pairs of 384 transforms of 48^3 in FP64: over 20 s
    s = _system(case, seed)
    call = case["call"]
    if call == "ingest":
        M = _t(s.eigVec[0]) @ _t(_patterns(s, seed)).conj().T
        return torch.einsum("vp,p...->v...", M, _t(s.dVscf[0]))
    if call == "dmats":
        n = min(case["nsym"], len(s.sym_R))
        pick = np.linspace(0, len(s.sym_R) - 1, n).astype(int)
        return torch.stack([_dmat(s, s.sym_R[i], s.sym_tau[i], bool(s.sym_trev[i]), k) for i in pick
                            for k in range(s.nk_bz)])
    if call in ("run", "unfold_run"):
        return torch.cat([_elphq(s, i) for i in range(len(s.qpts))])
    g = _elphq(s, 0)
    if call == "elphq":
        return g
    q, kc = s.qpts[0], _kcart(s)
    kq = _kplus(s, q)
    syms = _star_symmetries(s, q)
    out = torch.empty((len(syms), *g.shape), dtype=g.dtype, device="cuda")
    out[0] = g
    for i, S in enumerate(syms[1:], 1):
        R, tau, tr = s.sym_R[S], s.sym_tau[S], bool(s.sym_trev[S])
        D = torch.stack([_dmat(s, R, tau, tr, k) for k in range(s.nk_bz)])
        for k in range(s.nk_bz):
            # D[k+q] and conj(D[k]) on the two band indices, the element conjugated for time reversal
            gk = g[k].conj() if tr else g[k]
            r = torch.einsum("sma,vsab,snb->vsmn", D[k].conj(), gk, D[kq[k]])
            out[i, _kplus_one(s, s.alat.T @ (R @ kc[k]))] = r
    return out
