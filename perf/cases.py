"""Timed cases of the walker-step library: what a run of this framework spends its time on.

A run is a loop of propagation steps with a re-orthonormalisation every 5 and an energy measurement
every 10; the cases are those three, over the trial wavefunctions, Hamiltonian factorisations and
precisions that a user chooses between:

  step         one phaseless step of a single-determinant trial (Propagator.Propagate)
  nomsd_step   the same with a trial of several Slater determinants (NOMSDMulti)
  phmsd_step   the same with a particle-hole expansion (PHMSD)
  thc_step     the same over the tensor-hypercontraction Hamiltonian
  energy       the mixed-estimator energy of a single-determinant trial (NOMSD.Energy)
  phmsd_energy the same for a particle-hole expansion (PHMSDWavefunction.Energy)
  orthogonalize  det_ops.orthogonalize

Sizes are those of this repository's benchmark (M=200, 50+50 electrons, 1600 Cholesky vectors,
1024 walkers; PHMSD: M=120, 30+30, 960, 4096 determinants, 512 walkers), its small test system
(M=32), its molecules (BH: M=19, 78 vectors, 34 determinants; N2: M=28, 134 vectors, 50
determinants; 1536 walkers each) and generic odd ones between.

Systems are synthetic as in safire_b200/synth.py (one-body part plus decaying real symmetric
Cholesky vectors, trial = lowest eigenvectors).  The walkers are the trial plus complex noise, as
a few steps leave them; the weights are around 1; the fields are uniforms in a device buffer.
A step overwrites its walkers, so each pass first puts the walker buffer back (one device copy).
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

CLOSED, COLLINEAR = 1, 2
C128, F64 = torch.complex128, torch.float64
WEIGHT, PHASE, PSEUDO_ELOC, OVLP, THETA, NPROP = 0, 1, 2, 6, 10, 11
VBIAS_BOUND, ORDER = 50.0, 6


def _case(kind, name=None, **kw):
    d = dict(kind=kind, M=32, nup=8, ndn=8, Nc=128, W=64, collinear=False, mixed=False, dt=0.005)
    d.update(kw)
    if name:
        d["name"] = name
    return d


def listed():
    return [
        # the smallest call: a test-sized system in complex128, bound by launches
        _case("step", "step_small_c128", M=32, nup=8, ndn=8, Nc=128, W=64, dt=0.01),
        # a molecule (BH) with 34 determinants, open-shell walkers, a production population
        _case("nomsd_step", "nomsd_step_bh_c128", M=19, nup=3, ndn=3, Nc=78, W=1536, ndet=34,
              collinear=True, dt=0.01),
        # a molecule (N2) with a particle-hole expansion
        _case("phmsd_step", "phmsd_step_n2_c128", M=28, nup=7, ndn=7, Nc=134, W=1536, ndet=50,
              nocc=5, nvirt=8, collinear=True, dt=0.01),
        # the benchmark's step in mixed precision: nine tenths of a production run's calls
        _case("step", "step_mixed", M=200, nup=50, ndn=50, Nc=1600, W=1024, mixed=True),
        # sizes that do not take the FP16 split (M = 4 mod 8) and leave ragged tiles and waves
        _case("step", "step_mixed_ragged", M=108, nup=27, ndn=27, Nc=516, W=300, mixed=True),
        # the benchmark's step in complex128, the drop-in precision
        _case("step", "step_c128", M=200, nup=50, ndn=50, Nc=1600, W=1024),
        # complex128, open shell, odd in every size
        _case("step", "step_odd_c128", M=101, nup=23, ndn=21, Nc=403, W=257, collinear=True),
        # the benchmark's energy measurement in mixed precision
        _case("energy", "energy_mixed", M=200, nup=50, ndn=50, Nc=1600, W=1024, mixed=True),
        # an energy measurement in complex128 at an odd medium size
        _case("energy", "energy_odd_c128", M=130, nup=33, ndn=33, Nc=777, W=300),
        # the benchmark's particle-hole energy measurement, the longest single call
        _case("phmsd_energy", "phmsd_energy_mixed", M=120, nup=30, ndn=30, Nc=960, W=512,
              ndet=4096, nocc=20, nvirt=40, collinear=True, mixed=True),
        # tensor hypercontraction: Nc is the number of field components, nu the points
        _case("thc_step", "thc_step_c128", M=100, nup=25, ndn=25, Nc=350, nu=500, W=256),
        # re-orthonormalisation of the benchmark's walkers
        _case("orthogonalize", "orthogonalize", M=200, nup=50, ndn=0, Nc=1, W=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "nomsd_step", "phmsd_step", "energy", "energy",
                       "phmsd_energy", "thc_step", "orthogonalize"])
    dt = rng.choice([0.005, 0.01])
    if kind == "nomsd_step":
        M = _log(rng, 8, 32)
        nup = rng.randint(2, max(2, M // 4))
        col = rng.random() < 0.5
        return _case(kind, M=M, nup=nup, ndn=rng.randint(1, nup) if col else nup,
                     Nc=rng.randint(3 * M, 5 * M), W=_log(rng, 32, 1536), ndet=_log(rng, 2, 40),
                     collinear=col, dt=dt)
    if kind == "phmsd_step":
        M = _log(rng, 20, 48)
        nup = rng.randint(4, M // 4)
        return _case(kind, M=M, nup=nup, ndn=rng.randint(4, nup), Nc=rng.randint(3 * M, 6 * M),
                     W=_log(rng, 32, 1024), ndet=_log(rng, 16, 128), nocc=4,
                     nvirt=rng.randint(5, 8), collinear=True, dt=dt)
    if kind == "phmsd_energy":
        M = _log(rng, 24, 120)
        nup = rng.randint(5, M // 4)
        nvirt = rng.randint(6, min(40, M - nup))
        return _case(kind, M=M, nup=nup, ndn=rng.randint(5, nup), Nc=8 * rng.randint(M // 2, M),
                     W=_log(rng, 16, 256), ndet=_log(rng, 32, 2048), nocc=min(20, nup - 1),
                     nvirt=nvirt, collinear=True, mixed=rng.random() < 0.5, dt=dt)
    if kind == "thc_step":
        M = _log(rng, 20, 100)
        nup = rng.randint(3, M // 4)
        return _case(kind, M=M, nup=nup, ndn=nup, Nc=rng.randint(2 * M, 4 * M),
                     nu=rng.randint(3 * M, 5 * M), W=_log(rng, 32, 256), dt=dt)
    if kind == "orthogonalize":
        M = _log(rng, 16, 220)
        return _case(kind, M=M, nup=rng.randint(2, min(64, M // 2)), ndn=0, Nc=1,
                     W=_log(rng, 32, 1024), dt=dt)
    M = _log(rng, 16, 200)
    nup = rng.randint(2, max(2, M // 4))
    W = _log(rng, 32, 1024)
    if rng.random() < 0.5:  # mixed precision: closed shell, multiples of 4
        M = M // 4 * 4
        return _case(kind, M=M, nup=nup, ndn=nup, Nc=4 * rng.randint(M, 2 * M), W=W, mixed=True,
                     dt=dt)
    if kind == "energy":
        W = min(W, 400)
    col = rng.random() < 0.4
    return _case(kind, M=M, nup=nup, ndn=rng.randint(1, nup) if col else nup,
                 Nc=rng.randint(3 * M, 8 * M), W=W, collinear=col, dt=dt)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _sym(a):
    return 0.5 * (a + a.transpose(0, 1))


def _inputs(case, seed):
    """Everything that the seed decides, as torch CUDA tensors (PHMSD trials on the host)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    M, Nc, W = case["M"], case["Nc"], case["W"]

    def randn(*s):
        return torch.randn(s, generator=g, device="cuda", dtype=F64)

    def crandn(*s):
        return torch.complex(randn(*s), randn(*s))

    x = SimpleNamespace(case=case, M=M, Nc=Nc, W=W, dt=case["dt"], g=g)
    x.wt = COLLINEAR if case["collinear"] else CLOSED
    x.nel = [case["nup"]] + ([case["ndn"]] if case["collinear"] else [])
    if case["kind"] == "orthogonalize":
        x.S = [torch.eye(M, x.nel[0], device="cuda", dtype=F64) + 0.3 / math.sqrt(M)
               * crandn(W, M, x.nel[0])]
        return x
    x.h1 = torch.diag(-2.0 + 4.0 * torch.arange(M, device="cuda", dtype=F64) / M)
    x.h1 = x.h1 + 0.1 * _sym(randn(M, M))
    decay = torch.exp(torch.arange(Nc, device="cuda", dtype=F64) * (-8.0 / max(Nc, 200)))
    if case["kind"] == "thc_step":
        nu = case["nu"]
        x.X = randn(M, nu) / math.sqrt(M)
        x.Luv = 0.5 * decay * randn(nu, Nc) / math.sqrt(nu)
        x.L = None
    else:
        x.L = _sym(randn(M, M, Nc)) * (0.5 / math.sqrt(M)) * decay
    _, orb = torch.linalg.eigh(x.h1)
    x.orb = orb
    x.PsiT = [[orb[:, :n].t().contiguous() for n in x.nel]]  # [determinant][spin] [N][M], real
    x.ci = torch.ones(1, dtype=C128, device="cuda")
    if case["kind"] == "nomsd_step":
        # rotated copies of the lowest determinant, coefficients falling off
        for _ in range(1, case["ndet"]):
            x.PsiT.append([torch.linalg.qr(orb[:, :n] + 0.5 / math.sqrt(M) * randn(M, n))[0]
                           .t().contiguous() for n in x.nel])
        d = torch.arange(case["ndet"], device="cuda", dtype=F64)
        x.ci = 0.2 * crandn(case["ndet"]) * torch.exp(-0.2 * d)
        x.ci[0] = 1.0
    if case["kind"].startswith("phmsd"):
        from safire_b200.synth import make_phmsd_trial
        x.trial = make_phmsd_trial(M, case["nup"], case["ndn"], orb.cpu().numpy(),
                                   nocc=case["nocc"], nvirt=case["nvirt"], ndet=case["ndet"],
                                   seed=int(seed))
        # the reference determinant leads with a positive coefficient, as the files have it
        x.trial.coef[0] = 2.0
        x.trial.coef /= np.linalg.norm(x.trial.coef)
    x.S = [x.PsiT[0][s].t() + 0.3 / math.sqrt(M) * crandn(W, M, n) for s, n in enumerate(x.nel)]
    x.weight = 0.5 + torch.rand(W, generator=g, device="cuda", dtype=F64)
    x.u = torch.rand(W, Nc, generator=g, device="cuda", dtype=F64)
    return x


def _likn(x):
    if x.L is None:
        x.L = torch.einsum("iu,ku,un->ikn", x.X, x.X, x.Luv)
    return x.L


def _log_overlap(x, PsiT, S):
    """log det(PsiT_s S_s) summed over the spins (doubled for closed shells), [W]."""
    tot = torch.zeros(S[0].shape[0], dtype=C128, device="cuda")
    for P, A in zip(PsiT, S):
        sign, logabs = torch.linalg.slogdet(torch.matmul(P.to(C128), A))
        tot = torch.complex(tot.real + logabs, tot.imag + torch.angle(sign))
        tot = torch.complex(tot.real, torch.remainder(tot.imag + math.pi, 2 * math.pi) - math.pi)
    return 2 * tot if x.wt == CLOSED else tot


def _explicit_trial(x):
    """PHMSD: the determinants one by one, and their coefficients in sum_k c_k <D_k|S>."""
    t = x.trial
    orbmat = [torch.from_numpy(np.ascontiguousarray(o.real)).cuda() for o in t.orbmat]
    occ = []
    for s in (0, 1):
        rows = [np.array(t.refc[s])]
        for n in sorted(t.exc[s]):
            for e in t.exc[s][n]:
                o = np.array(t.refc[s])
                o[e[:n]] = e[n:]
                rows.append(o)
        occ.append(rows)
    dets = [[orbmat[0][torch.from_numpy(occ[0][a]).long().cuda()],
             orbmat[1][torch.from_numpy(occ[1][b]).long().cuda()]]
            for a, b in zip(t.det_up, t.det_dn)]
    return dets, torch.from_numpy(np.ascontiguousarray(t.coef)).cuda(), orbmat, occ


def _multi_overlap(x, dets, coef, S):
    """log sum_d coef_d exp(log <D_d|S>) and the per-determinant logs [ndet][W]."""
    ov = torch.stack([_log_overlap(x, P, S) for P in dets])
    z = ov + torch.log(coef)[:, None]
    m = torch.gather(z, 0, z.real.argmax(0, keepdim=True))
    return (m + torch.log(torch.exp(z - m).sum(0)))[0], ov


def _total_overlap(x):
    if x.case["kind"] == "nomsd_step":
        return _multi_overlap(x, x.PsiT, x.ci.conj(), x.S)[0]
    if x.case["kind"] == "phmsd_step":
        dets, coef, _, _ = _explicit_trial(x)
        return _multi_overlap(x, dets, coef, x.S)[0]
    return _log_overlap(x, x.PsiT[0], x.S)


def _density(P, A):
    """Compact density matrices [W][N][M] of the walkers A with the determinant P [N][M]."""
    T = torch.matmul(P.to(C128), A)
    return torch.linalg.solve(T.transpose(1, 2), A.transpose(1, 2))


def _energies(x, G):
    """(E1, EXX, EJ) [W][3] from the compact density matrices G[s] of the first determinant."""
    scl = 2.0 if x.wt == CLOSED else 1.0
    W = G[0].shape[0]
    L = _likn(x)
    E = torch.zeros(W, 3, dtype=C128, device="cuda")
    K = torch.zeros(W, x.Nc, dtype=C128, device="cuda")
    for s, Gs in enumerate(G):
        P, N = x.PsiT[0][s], x.nel[s]
        E[:, 0] += scl * (Gs * (P @ x.h1)).sum((1, 2))
        step = max(1, int(2e8 / (W * N * N)))
        for n0 in range(0, x.Nc, step):
            Ln = L[:, :, n0:n0 + step]
            nc = Ln.shape[2]
            Lnak = torch.einsum("ai,ikn->kna", P, Ln).reshape(x.M, nc * N)
            T = torch.complex(torch.matmul(Gs.real, Lnak), torch.matmul(Gs.imag, Lnak))
            T = T.reshape(W, N, nc, N)
            E[:, 1] -= 0.5 * scl * (T * T.transpose(1, 3)).sum((1, 2, 3))
            K[:, n0:n0 + nc] += torch.einsum("wana->wn", T)
    E[:, 2] = 0.5 * scl * scl * (K * K).sum(1)
    return E


def _trial_energy(x):
    """Local energy of the first determinant at itself: the run's first Eshift."""
    S = [P.t().to(C128)[None] for P in x.PsiT[0]]
    return float(_energies(x, [_density(P, A) for P, A in zip(x.PsiT[0], S)]).sum().real)


# ---------------------------------------------------------------------------------------------
# the framework's side
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    from safire_b200 import afqmc as A
    from safire_b200 import capi
    x = _inputs(case, seed)
    st = SimpleNamespace(case=case, kind=case["kind"], A=A)
    if st.kind == "orthogonalize":
        st.start = x.S[0].contiguous()
        st.S = torch.empty_like(st.start)
        st.logdet = torch.zeros(x.W, dtype=C128, device="cuda")
        torch.cuda.synchronize()
        return st
    st.prec = A.PREC_MIXED if case["mixed"] else A.PREC_FP64
    h1 = x.h1.cpu().numpy()[None].astype(np.complex128)
    PsiT = [[p.cpu().numpy().astype(np.complex128) for p in d] for d in x.PsiT]
    ndn = case["ndn"]
    if st.kind == "thc_step":
        st.ham = A.HamiltonianOperations.thc(x.wt, x.M, case["nup"], ndn, x.X.cpu().numpy(),
                                             x.Luv.cpu().numpy(), h1, 0.0, PsiT[0])
    else:
        L = x.L.cpu().numpy()[None]
        if st.kind != "phmsd_energy":
            st.ham = A.HamiltonianOperations(x.wt, x.M, case["nup"], ndn, L, h1, 0.0, PsiT[0])
    st.wset = A.WalkerSet(x.wt, x.M, case["nup"], ndn, x.W)
    for s, S in enumerate(x.S):
        st.wset.SlaterMatrices(s).copy_(S)
    props = st.wset.properties()
    props[:, WEIGHT] = x.weight.to(C128)
    props[:, PHASE] = 1.0
    if st.kind == "energy":
        st.wfn = A.NOMSD(st.ham)
        torch.cuda.synchronize()
        return st
    if st.kind.startswith("phmsd"):
        st.ph = A.PHMSD(x.trial)
        st.ph.set_hamiltonian(L, h1, 0.0)
        st.wfn = A.PHMSDWavefunction(st.ph)
    if st.kind == "phmsd_energy":
        torch.cuda.synchronize()
        return st
    st.prop = A.Propagator(st.ham, A.default_params(dt=case["dt"], precision=st.prec), x.W)
    if case["mixed"]:
        # the Taylor variant that the autotuner keeps: FP16 split where the sizes allow it
        if st.ham.set_split_format(capi.SPLIT_AUTO):
            st.ham.set_taylor_fused(4)
    if st.kind == "nomsd_step":
        st.hams = [st.ham] + [A.HamiltonianOperations(x.wt, x.M, case["nup"], ndn, L, h1, 0.0, P)
                              for P in PsiT[1:]]
        st.multi = A.NOMSDMulti(st.hams, x.ci.cpu().numpy())
        st.prop.set_trial(st.multi)
    if st.kind == "phmsd_step":
        st.prop.set_trial(st.ph)
    st.Eshift = _trial_energy(x)
    props[:, PSEUDO_ELOC] = st.Eshift
    props[:, OVLP] = _total_overlap(x)
    st.start = st.wset.buffer.clone()
    st.u = x.u
    st.out = ([st.wset.SlaterMatrices(s) for s in range(len(x.nel))]
              + [props[:, p] for p in (WEIGHT, PHASE, PSEUDO_ELOC, OVLP)])
    for t in st.out:
        t.walker_set = st.wset  # the library owns the memory: it lives as long as the views
    torch.cuda.synchronize()
    return st


def run(st):
    if st.kind == "orthogonalize":
        st.S.copy_(st.start)
        st.logdet.zero_()
        st.A.det_ops.orthogonalize(st.S, st.logdet)
        return [st.S, st.logdet]
    if st.kind in ("energy", "phmsd_energy"):
        return list(st.wfn.Energy(st.wset, set_properties=False, precision=st.prec))
    st.wset.buffer.copy_(st.start)
    st.prop.Propagate(st.wset, st.Eshift, st.u)
    return st.out


# ---------------------------------------------------------------------------------------------
# the work that cannot be avoided
# ---------------------------------------------------------------------------------------------
def work(case):
    M, Nc, W = case["M"], case["Nc"], case["W"]
    nel = [case["nup"]] + ([case["ndn"]] if case["collinear"] else [])
    kind = case["kind"]
    ntot = sum(nel)
    walkers = 16.0 * W * (M * ntot + NPROP)
    if kind == "orthogonalize":
        # Gram matrix and application of the triangular factor, complex, half of each
        return {"bytes": 2 * walkers, "flops": 8.0 * W * M * nel[0] * nel[0]}
    tensor = 8.0 * M * (M + 1) / 2 * Nc  # the symmetric Cholesky vectors
    overlap = sum(4.0 * M * n * n + 8.0 / 3 * n ** 3 for n in nel)
    green = overlap + sum(16.0 / 3 * n ** 3 + 8.0 * n * n * M for n in nel)
    if kind == "energy":
        exchange = sum(4.0 * n * n * M * Nc + 8.0 * n * n * Nc for n in nel)
        return {"bytes": walkers + 8.0 * Nc * ntot * M + 64.0 * W,
                "flops": W * (green + exchange)}
    if kind == "phmsd_energy":
        # per spin and Cholesky vector: the half-rotated rows, the tables over (electron,
        # virtual), and for an average excitation of two holes n^3 + 2 n^2 complex products
        fl = 0.0
        for n in nel:
            nact, nv, nh = max(nel) + case["nvirt"], case["nvirt"], case["nocc"]
            fl += 4.0 * n * M * nact + 8.0 * (n * nv * n + nh * nv * n) + 8.0 * 16 * case["ndet"] / 2
        return {"bytes": walkers + 8.0 * M * Nc * 2 * (max(nel) + case["nvirt"]) + 64.0 * W,
                "flops": W * Nc * fl}
    prop = sum((2 * 4.0 + ORDER * 8.0) * M * M * n for n in nel)
    vhs = 4.0 * M * (M + 1) / 2 * Nc
    vbias = sum(4.0 * M * n * Nc for n in nel)
    ndet = 1
    if kind in ("nomsd_step", "phmsd_step"):
        vbias = 4.0 * M * (M + 1) / 2 * Nc * len(nel)
    if kind == "nomsd_step":
        ndet = case["ndet"]
    if kind == "thc_step":
        nu = case["nu"]
        tensor = 8.0 * (nu * Nc + M * nu)
        vbias = 4.0 * nel[0] * M * nu + 4.0 * nel[0] * nu + 4.0 * nu * Nc
        vhs = 4.0 * nu * Nc + 4.0 * M * (M + 1) / 2 * nu
    return {"bytes": 2 * walkers + tensor + 8.0 * W * Nc,
            "flops": W * (prop + vhs + vbias + ndet * (green + overlap))}


def tolerance(case):
    # about four times the largest relative error against exact() over the listed sizes and some
    # seventy drawn ones (phmsd_energy in mixed precision at the listed size: against complex128)
    if case["kind"] == "orthogonalize":
        return {"rel": 1e-14}
    if case["kind"] in ("energy", "phmsd_energy"):
        return {"rel": 6e-6} if case["mixed"] else {"rel": 1e-13}
    # a step: the weight moves by the log overlap's error, the pseudo energy by that over dt
    return {"rel": 4e-4} if case["mixed"] else {"rel": 1e-12}


# ---------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------
def _probit(p):
    """The inverse normal CDF by the published rational approximation that the fields use."""
    a = [-3.969683028665376e+01, 2.209460984245205e+02, -2.759285104469687e+02,
         1.383577518672690e+02, -3.066479806614716e+01, 2.506628277459239e+00]
    b = [-5.447609879822406e+01, 1.615858368580409e+02, -1.556989798598866e+02,
         6.680131188771972e+01, -1.328068155288572e+01, 1.0]
    c = [-7.784894002430293e-03, -3.223964580411365e-01, -2.400758277161838e+00,
         -2.549732539343734e+00, 4.374664141464968e+00, 2.938163982698783e+00]
    d = [7.784695709041462e-03, 3.224671290700398e-01, 2.445134137142996e+00,
         3.754408661907416e+00, 1.0]

    def poly(k, x):
        r = torch.zeros_like(x)
        for v in k:
            r = r * x + v
        return r

    tail = torch.minimum(p, 1 - p)
    q = torch.sqrt(-2 * torch.log(torch.clamp(tail, min=1e-300)))
    lo = poly(c, q) / poly(d, q)
    q = p - 0.5
    mid = poly(a, q * q) * q / poly(b, q * q)
    return torch.where(p < 0.02425, lo, torch.where(p > 0.97575, -lo, mid))


def _clamp(z):
    m = z.abs()
    return torch.where(m > VBIAS_BOUND, z * (VBIAS_BOUND / torch.clamp(m, min=1e-300)), z)


def _cmm(a, b):
    """complex @ real"""
    return torch.complex(torch.matmul(a.real, b), torch.matmul(a.imag, b))


def _vbias_single(x, P, S):
    a = math.sqrt(x.dt) * (2.0 if x.wt == CLOSED else 1.0)
    L = _likn(x)
    v = 0
    for Ps, A in zip(P, S):
        Lnak = torch.einsum("ai,ikn->akn", Ps, L).reshape(-1, x.Nc)
        v = v + a * _cmm(_density(Ps, A).reshape(A.shape[0], -1), Lnak)
    return v


def _vbias_multi(x, dets, coef, S):
    a = math.sqrt(x.dt) * (2.0 if x.wt == CLOSED else 1.0)
    tot, ov = _multi_overlap(x, dets, coef, S)
    wd = coef[:, None] * torch.exp(ov - tot)
    G = [torch.zeros(x.W, x.M, x.M, dtype=C128, device="cuda") for _ in S]
    for k, P in enumerate(dets):
        for s, A in enumerate(S):
            G[s] += wd[k][:, None, None] * torch.matmul(P[s].t().to(C128), _density(P[s], A))
    return sum(a * _cmm(g.reshape(x.W, -1), _likn(x).reshape(-1, x.Nc)) for g in G)


def _step_exact(x):
    Eshift = _trial_energy(x)
    old = _total_overlap(x)
    kind, dt, L = x.case["kind"], x.dt, _likn(x)
    phi = [P.t().to(C128)[None] for P in x.PsiT[0]]
    vMF = _vbias_single(x, x.PsiT[0], phi)[0].real
    v0 = -0.5 * L.reshape(x.M, -1) @ L.reshape(x.M, -1).t()
    Lf = L.reshape(-1, x.Nc).t()
    H1 = dt * (x.h1 + v0) + math.sqrt(dt) * (vMF @ Lf).reshape(x.M, x.M)
    e, U = torch.linalg.eigh(-0.5 * _sym(H1))
    P1 = (U * torch.exp(e)) @ U.t()
    P1 = torch.where(P1.abs() > 1e-8, P1, torch.zeros_like(P1)).to(C128)
    dets = coef = None
    if kind == "nomsd_step":
        dets, coef = x.PsiT, x.ci.conj()
    elif kind == "phmsd_step":
        dets, coef, _, _ = _explicit_trial(x)
    vb = _vbias_single(x, x.PsiT[0], x.S) if dets is None else _vbias_multi(x, dets, coef, x.S)
    vdiff = 1j * (_clamp(vb) - _clamp(vMF.to(C128)))
    X = _probit(x.u) + vdiff
    hw = (-vdiff * (X - 0.5 * vdiff)).sum(1)
    mf = -0.5 * (vMF * vMF).sum() + 1j * (X * vMF).sum(1)
    V = math.sqrt(dt) * _cmm(X, Lf).reshape(x.W, x.M, x.M)
    x.S = [torch.matmul(P1, S) for S in x.S]
    for s, S in enumerate(x.S):
        T, R = S, S
        for n in range(1, ORDER + 1):
            T = (1j / n) * torch.matmul(V, T)
            R = R + T
        x.S[s] = torch.matmul(P1, R)
    new = _total_overlap(x)
    dth = new.imag - old.imag - mf.imag
    eloc = (mf - hw - (new - old)) / dt
    hi, lo = Eshift + 10.0 * math.sqrt(2 / dt), Eshift - math.sqrt(2 / dt)
    eloc = torch.complex(torch.clamp(eloc.real, lo, hi), eloc.imag)
    f = torch.exp(-dt * (eloc - Eshift))
    weight = x.weight * torch.clamp(torch.cos(dth), min=0.0) * f.abs()
    weight = torch.clamp(weight, max=max(100.0, 0.1 * x.W)).to(C128)
    return x.S + [weight, f / f.abs(), eloc, new]


def _phmsd_energy_exact(x):
    """Every distinct excitation's own terms, then the sum over the determinants."""
    t, L = x.trial, x.L
    dets, coef, orbmat, occ = _explicit_trial(x)
    cost = sum(8.0 * x.W * x.Nc * len(occ[s]) * x.nel[s] ** 3 for s in (0, 1))
    if cost > 1.5e13:
        return None
    ov, e1, ex, K = [], [], [], []
    for s in (0, 1):
        n_u, N = len(occ[s]), x.nel[s]
        o = torch.from_numpy(np.array(occ[s])).long().cuda()
        act = torch.matmul(orbmat[s].to(C128), x.S[s])            # [W][nact][N]
        hrot = torch.matmul((orbmat[s] @ x.h1).to(C128), x.S[s])
        T = act[:, o]                                             # [W][n_u][N][N]
        sign, la = torch.linalg.slogdet(T)
        ov.append(torch.complex(la, torch.angle(sign)))
        Ti = torch.linalg.inv(T)
        e1.append(torch.einsum("wuab,wuba->wu", hrot[:, o], Ti))
        xs = torch.zeros(x.W, n_u, dtype=C128, device="cuda")
        ks = torch.zeros(x.W, n_u, x.Nc, dtype=C128, device="cuda")
        step = max(1, int(1e8 / (n_u * N * N * 4)))
        for n in range(x.Nc):
            B = torch.matmul((orbmat[s] @ L[:, :, n]).to(C128), x.S[s])
            for w in range(0, x.W, step):
                a = torch.matmul(B[w:w + step][:, o], Ti[w:w + step])
                xs[w:w + step] += (a * a.transpose(2, 3)).sum((2, 3))
                ks[w:w + step, :, n] = torch.diagonal(a, dim1=2, dim2=3).sum(-1)
        ex.append(xs)
        K.append(ks)
    iu, idn = (torch.from_numpy(np.array(v)).long().cuda() for v in (t.det_up, t.det_dn))
    z = ov[0][:, iu] + ov[1][:, idn] + torch.log(coef)
    m = torch.gather(z, 1, z.real.argmax(1, keepdim=True))
    f = torch.exp(z - m)
    den = f.sum(1)
    E = torch.zeros(x.W, 3, dtype=C128, device="cuda")
    E[:, 0] = (f * (e1[0][:, iu] + e1[1][:, idn])).sum(1) / den
    E[:, 1] = -0.5 * (f * (ex[0][:, iu] + ex[1][:, idn])).sum(1) / den
    for w in range(x.W):
        k = K[0][w, iu] + K[1][w, idn]
        E[w, 2] = 0.5 * (f[w] * (k * k).sum(1)).sum() / den[w]
    return [E, m[:, 0] + torch.log(den)]


def exact(case, seed):
    x = _inputs(case, seed)
    if case["kind"] == "orthogonalize":
        Q, R = torch.linalg.qr(x.S[0])
        d = torch.diagonal(R, dim1=1, dim2=2)
        return [Q * (d / d.abs())[:, None, :], torch.log(d.abs()).sum(1).to(C128)]
    if case["kind"] == "energy":
        G = [_density(P, A) for P, A in zip(x.PsiT[0], x.S)]
        return [_energies(x, G), _log_overlap(x, x.PsiT[0], x.S)]
    if case["kind"] == "phmsd_energy":
        return _phmsd_energy_exact(x)
    return _step_exact(x)
