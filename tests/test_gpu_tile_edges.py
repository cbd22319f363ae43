"""Sizes at which the kernels change tile, register or thread layout, against numpy or complex128.

The bounds are rounding bounds: eps = 2^-53 times the length of the sums and the condition or
magnitude of the operands, with a factor of a few tens for the constant."""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import rand_c, rel_err, to_dev, to_host

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.mark.parametrize("N", [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 28, 29, 32, 33, 40, 41,
                               50, 57, 63, 64, 65])
@pytest.mark.parametrize("W", [1, 37, 300])
def test_inverse_logdet(cuda, N, W):
    """Inverses and log determinants.  A matrix with a zero first column is singular exactly: its
    inverse is zero, and its log determinant takes the smallest number in the zero pivot's place and
    goes on with the rows and columns that remain."""
    from safire_b200 import afqmc as A
    rs = np.random.default_rng(N)
    a = rand_c(rs, W, N, N)
    a[:, np.arange(N), np.arange(N)] *= 1e-3  # pivoting matters
    d_inv = torch.zeros((W, N, N), dtype=torch.complex128, device=cuda)
    d_log = torch.zeros(W, dtype=torch.complex128, device=cuda)
    A.det_ops.inverse_logdet(to_dev(a), d_inv, d_log)
    inv, log = to_host(d_inv), to_host(d_log)
    for w in range(W):
        cond = np.linalg.cond(a[w])
        assert np.linalg.norm(inv[w] @ a[w] - np.eye(N), 2) < 50 * N * EPS * cond
        sign, la = np.linalg.slogdet(a[w])
        assert abs(log[w].real - la) < 50 * N * EPS * cond
        assert abs(np.exp(1j * log[w].imag) - sign) < 50 * N * EPS * cond
    a[:, :, 0] = 0.0
    d_log.zero_()
    A.det_ops.inverse_logdet(to_dev(a), d_inv, d_log)
    assert np.all(to_host(d_inv) == 0)
    log = to_host(d_log)
    for w in range(W):
        rest = a[w, 1:, 1:]
        cond = np.linalg.cond(rest) if N > 1 else 1.0
        sign, la = np.linalg.slogdet(rest)
        tol = 50 * N * EPS * cond + 1e-12  # the logarithm of the smallest number, -708, has 1e-13
        assert abs(log[w].real - np.log(np.finfo(float).tiny) - la) < tol
        assert abs(np.exp(1j * log[w].imag) - sign) < tol


@pytest.mark.parametrize("M,N", [(9, 1), (8, 8), (30, 9), (40, 31), (64, 32), (70, 50), (80, 64),
                                 (101, 83)])
def test_orthogonalize(cuda, M, N):
    from safire_b200 import afqmc as A
    rs = np.random.default_rng(M)
    W = 5
    S = np.eye(M, N) + rand_c(rs, W, M, N, scale=0.3 / np.sqrt(M))
    d, ld = to_dev(S), torch.zeros(W, dtype=torch.complex128, device=cuda)
    A.det_ops.orthogonalize(d, ld)
    Q, ld = to_host(d), to_host(ld)
    for w in range(W):
        q, r = np.linalg.qr(S[w])
        ph = np.diag(r) / np.abs(np.diag(r))
        tol = 50 * N * EPS * np.linalg.cond(S[w])
        assert np.linalg.norm(Q[w].conj().T @ Q[w] - np.eye(N), 2) < 50 * N * EPS
        assert np.max(np.abs(Q[w] - q * ph)) < tol
        assert abs(ld[w] - np.sum(np.log(np.abs(np.diag(r))))) < tol


@pytest.mark.parametrize("M,N", [(5, 1), (19, 3), (32, 8), (32, 32), (33, 9), (64, 16), (65, 24),
                                 (101, 23), (128, 32), (129, 8), (70, 33)])
@pytest.mark.parametrize("order", [0, 1, 6])
@pytest.mark.parametrize("W", [3, 140])  # N > 16, M > 64: GEMM launches, and one launch for an SM each
def test_propagate(cuda, M, N, order, W):
    from safire_b200 import afqmc as A
    rs = np.random.default_rng(M + N)
    P1 = np.eye(M) + rand_c(rs, M, M, scale=0.1 / np.sqrt(M))
    V = rand_c(rs, W, M, M, scale=0.5 / np.sqrt(M))
    S = rand_c(rs, W, M, N)
    d = torch.zeros((W, M * N + 3), dtype=torch.complex128, device=cuda)  # a longer walker row
    view = d[:, :M * N].unflatten(1, (M, N))
    view.copy_(to_dev(S))
    A.det_ops.Propagate(view, to_dev(P1), to_dev(V), order)
    T = P1 @ S
    R = T.copy()
    for n in range(1, order + 1):
        T = (1j / n) * (V @ T)
        R = R + T
    want = P1 @ R
    assert np.max(np.abs(to_host(view) - want)) < 50 * M * EPS * np.max(np.abs(want))
    assert torch.all(d[:, M * N:] == 0)


def _ham(M, N, Nc, L):
    from safire_b200 import afqmc as A
    _, orb = np.linalg.eigh(np.diag(np.arange(M, dtype=float)) + 0.1)
    return A.HamiltonianOperations(A.CLOSED, M, N, N, L[None], np.eye(M)[None].astype(complex),
                                   0.0, [orb[:, :N].T.astype(complex)])


@pytest.mark.parametrize("W,M,Nc", [(1, 5, 3), (9, 8, 16), (33, 17, 40), (64, 32, 260), (257, 30, 37),
                                    (256, 100, 21), (300, 41, 19)])
def test_vhs_vbias_shapes(cuda, W, M, Nc):
    """vbias and vHS of symmetric vectors (pairs computed once where that pays) and of vectors
    with one bit of one element changed (every pair computed): the other elements are the same
    bit for bit."""
    from safire_b200 import afqmc as A
    rs = np.random.default_rng(W)
    N = max(1, M // 4)
    L = rs.standard_normal((M, M, Nc))
    L = L + L.transpose(1, 0, 2)
    X, G = rand_c(rs, W, Nc), rand_c(rs, W, N * M)
    ham = _ham(M, N, Nc, L)
    V = to_host(ham.vHS(to_dev(X), 0.01))[0].reshape(W, M * M)
    want = 0.1 * (X.real @ L.reshape(M * M, Nc).T + 1j * (X.imag @ L.reshape(M * M, Nc).T))
    scale = 0.1 * np.max(np.abs(X)) * np.max(np.abs(L))
    assert np.max(np.abs(V - want)) < 20 * Nc * EPS * scale
    L2 = L.copy()
    L2[0, 1, 0] = np.nextafter(L2[0, 1, 0], 1e9)
    V2 = to_host(_ham(M, N, Nc, L2).vHS(to_dev(X), 0.01))[0].reshape(W, M * M)
    keep = np.arange(M * M) != 1
    assert np.array_equal(V[:, keep], V2[:, keep])
    Lnak = ham.tensors().Lnak[0].real.reshape(Nc, N * M)
    v = torch.zeros((W, Nc), dtype=torch.complex128, device=cuda)
    ham.vbias(to_dev(G), v, 0.01)
    want = 0.2 * (G.real @ Lnak.T + 1j * (G.imag @ Lnak.T))
    scale = 0.2 * np.max(np.abs(G)) * np.max(np.abs(Lnak))
    assert np.max(np.abs(to_host(v) - want)) < 20 * N * M * EPS * scale


@pytest.mark.parametrize("M,N", [(257, 1), (41, 20), (67, 25), (130, 33)])  # K = N M, 1 to 12 mod 16
@pytest.mark.parametrize("W", [1, 20, 70, 300])
@pytest.mark.parametrize("real", [True, False])
def test_vbias_split_sum(cuda, M, N, W, real):
    """The force bias where its sum over K is split over CTAs (few walkers and vectors), with a ragged
    last K tile and numbers of K tiles that the parts do not divide, for real and complex trials."""
    from safire_b200 import afqmc as A
    Nc = 37
    rs = np.random.default_rng(W + M)
    L = rs.standard_normal((M, M, Nc))
    psi = np.linalg.qr(rand_c(rs, M, N))[0].T
    ham = A.HamiltonianOperations(A.CLOSED, M, N, N, (L + L.transpose(1, 0, 2))[None],
                                  np.eye(M)[None].astype(complex), 0.0,
                                  [psi.real.astype(complex) if real else psi])
    G = rand_c(rs, W, N * M)
    v = torch.zeros((W, Nc), dtype=torch.complex128, device=cuda)
    ham.vbias(to_dev(G), v, 0.01)
    Lnak = ham.tensors().Lnak[0].reshape(Nc, N * M)
    scale = 0.2 * np.max(np.abs(G)) * np.max(np.abs(Lnak))
    assert np.max(np.abs(to_host(v) - 0.2 * G @ Lnak.T)) < 20 * N * M * EPS * scale


@pytest.mark.parametrize("M,N,W,ndet", [(9, 1, 3, 1), (17, 5, 40, 3), (64, 16, 9, 1), (75, 33, 30, 2),
                                       (41, 20, 300, 2)])
def test_real_trial(cuda, M, N, W, ndet):
    """Overlaps and density matrices of a real trial take the products with a real matrix; one
    element with the imaginary part 1e-300, which no sum can feel, takes the complex ones: the
    results are the same bit for bit."""
    from safire_b200 import afqmc as A
    rs = np.random.default_rng(M)
    L = np.zeros((M, M, 2))
    hij = np.eye(M)[None].astype(complex)
    S = to_dev(np.eye(M, N) + rand_c(rs, W, M, N, scale=0.3 / np.sqrt(M)))
    out = []
    psi = [np.linalg.qr(np.eye(M, N) + 0.3 * rs.standard_normal((M, N)) / np.sqrt(M))[0].T.astype(complex)
           for _ in range(ndet)]
    for im in (0.0, 1e-300):
        hams = []
        for P in psi:
            P = P.copy()
            P[0, 0] += 1j * im
            hams.append(A.HamiltonianOperations(A.CLOSED, M, N, N, L[None], hij, 0.0, [P]))
        wset = A.WalkerSet(A.CLOSED, M, N, N, W)
        wset.init_from_trial(hams[0])
        wset.SlaterMatrices(0).copy_(S)
        t = A.NOMSDMulti(hams, np.arange(1.0, ndet + 1).astype(complex)) if ndet > 1 else A.NOMSD(hams[0])
        lo = t.Log_Overlap(wset)
        G, ov = t.MixedDensityMatrix(wset)
        out.append([to_host(x) for x in (lo, G, ov)])
    for a, b in zip(*out):
        assert np.all(np.isfinite(a.view(float))) and np.array_equal(a, b)


@pytest.mark.parametrize("ndet,W", [(2, 1), (31, 5), (32, 3), (33, 9), (70, 4)])
def test_determinant_sums(cuda, ndet, W):
    """Log overlap and density matrix of several determinants at the lanes' remainders, against
    numpy: the sums are weighted means, so eps times their length and the conditions of the
    overlap matrices bounds the error."""
    from safire_b200 import afqmc as A
    M, N = 7, 2
    rs = np.random.default_rng(ndet)
    psi = rs.standard_normal((ndet, N, M))
    S = np.eye(M, N) + rand_c(rs, W, M, N, scale=0.3)
    ci = rs.uniform(0.1, 1.0, ndet)
    L, hij = np.zeros((M, M, 2)), np.eye(M)[None].astype(complex)
    hams = [A.HamiltonianOperations(A.CLOSED, M, N, N, L[None], hij, 0.0, [p.astype(complex)])
            for p in psi]
    wset = A.WalkerSet(A.CLOSED, M, N, N, W)
    wset.init_from_trial(hams[0])
    wset.SlaterMatrices(0).copy_(to_dev(S))
    md = A.NOMSDMulti(hams, ci.astype(complex))
    T = np.einsum("dai,wib->wdab", psi, S)
    f = ci * np.linalg.det(T) ** 2
    cond = np.max(np.linalg.cond(T)) * np.max(np.sum(np.abs(f), 1) / np.abs(np.sum(f, 1)))
    lo = to_host(md.Log_Overlap(wset))
    assert np.max(np.abs(np.exp(lo - np.log(np.sum(f, 1))) - 1)) < 50 * ndet * EPS * cond
    G = to_host(md.MixedDensityMatrix(wset)[0]).reshape(W, M, M)
    Gd = np.einsum("dai,wdba,wkb->wdik", psi, np.linalg.inv(T), S)
    want = np.einsum("wd,wdik->wik", f / np.sum(f, 1, keepdims=True), Gd)
    assert np.max(np.abs(G - want)) < 50 * ndet * EPS * cond * np.max(np.abs(Gd))


@pytest.mark.parametrize("N", [1, 5, 8, 10, 16, 17, 20, 25, 30, 32, 33, 40, 41, 50])
@pytest.mark.parametrize("fmt", [1, 2])  # TF32, FP16 split
def test_exchange_tiles(cuda, N, fmt):
    """The tensor-core exchange at every tile layout, ragged in walkers and vectors, against the
    complex128 energy.  Operands keep 22 bits and the sums run in FP32: 2^-21 per element of the
    rows' magnitude, a few 1e-6 relative of sums that hardly cancel (their diagonal leads)."""
    from safire_b200 import afqmc as A
    M, Nc, W = 104, 56, 29
    rs = np.random.default_rng(N)
    L = 0.1 * rs.standard_normal((M, M, Nc))
    ham = _ham(M, N, Nc, L + L.transpose(1, 0, 2))
    ham.set_split_format(fmt)
    G = to_dev(rand_c(rs, W, N * M, scale=0.05)
               + np.eye(N, M).reshape(-1)[None] * (1 + 0.1 * rs.random((W, 1))))
    E, R = (torch.zeros((W, 3), dtype=torch.complex128, device=cuda) for _ in range(2))
    ham.energy(E, G, precision=A.PREC_MIXED)
    ham.energy(R, G)
    assert ham.device_error_flag() == 0
    E, R = to_host(E), to_host(R)
    for c in (1, 2):
        assert np.max(np.abs(E[:, c] - R[:, c])) < 2e-5 * np.max(np.abs(R[:, c])), c


@pytest.mark.parametrize("nup,ndn,nocc,nvirt,Nc,ndet", [(1, 1, 1, 2, 1, 6), (5, 4, 3, 5, 7, 60),
                                                        (8, 7, 4, 6, 8, 90), (9, 9, 6, 7, 17, 120),
                                                        (13, 11, 8, 9, 18, 200), (30, 30, 20, 40, 15, 300)])
def test_phmsd_energy_index_groups(cuda, nup, ndn, nocc, nvirt, Nc, ndet):
    """The mixed-precision particle-hole energy (groups of eight Cholesky indices, single-precision
    tables) at remainders of the group, of the product tiles and of the lanes, against complex128.
    Sums of a few hundred products at 2^-24, amplified by the excitation blocks' inverses: the
    5e-5 of the comparison with the oracle."""
    from safire_b200 import afqmc as A
    from safire_b200.synth import make_hamiltonian, make_phmsd_trial
    M, W = nup + nvirt + 2, 5
    M += -M % 8  # the tensor-core rows
    h1, Likn = make_hamiltonian(M, Nc, 0.9, seed=M)
    _, C = np.linalg.eigh(h1)
    t = make_phmsd_trial(M, nup, ndn, C, nocc=nocc, nvirt=nvirt, ndet=ndet, seed=M,
                         max_level=min(4, 2 * nocc))
    rs = np.random.default_rng(M + Nc)
    S = [C[None, :, :n] + rand_c(rs, W, M, n, scale=0.2 / np.sqrt(M)) for n in (nup, ndn)]
    wbuf = to_dev(np.concatenate([S[0].reshape(W, -1), S[1].reshape(W, -1), np.zeros((W, 11))], 1))
    ph = A.PHMSD(t)
    ph.set_hamiltonian(Likn[None], h1[None].astype(complex), 0.3)
    out = []
    for prec in (A.PREC_FP64, A.PREC_MIXED):
        ph.set_precision(prec)
        E = torch.zeros((W, 3), dtype=torch.complex128, device=cuda)
        ov = torch.zeros(W, dtype=torch.complex128, device=cuda)
        ph.Energy(wbuf, E, ov)
        out.append(to_host(E))
    scale = np.max(np.abs(out[0]), axis=0)
    assert np.all(np.abs(out[1] - out[0]) < 5e-5 * scale)


@pytest.mark.parametrize("M,N,Nc,W", [(40, 13, 8, 1), (64, 32, 16, 9), (72, 32, 44, 130), (128, 32, 8, 5),
                                      (104, 50, 264, 33), (136, 50, 24, 7), (256, 32, 8, 2),
                                      (168, 50, 16, 3)])
@pytest.mark.parametrize("fmt", [1, 2])  # TF32, FP16 split
def test_mixed_vbias_ranges(cuda, M, N, Nc, W, fmt):
    """The force bias summed over ranges of its K = N M (one, and several) in mixed precision, against
    complex128, at the edges of the blocks that split its rows (2048, 4096 and 8192 values).  Operands
    keep 22 bits, and a range's running sum in FP32 loses up to 2^-23 of itself with each MMA (16
    elements in FP16, 8 in TF32); it is about the size of a result, of which the largest of the
    deviations is taken as eight."""
    from safire_b200 import afqmc as A
    rs = np.random.default_rng(M)
    Nc -= Nc % 8 if fmt == 2 else 0  # the FP16 split takes multiples of 8
    L = rs.standard_normal((M, M, Nc))
    ham = _ham(M, N, Nc, L + L.transpose(1, 0, 2))
    ham.set_split_format(fmt)
    G = to_dev(rand_c(rs, W, N * M))
    v, r = (torch.empty((W, Nc), dtype=torch.complex128, device=cuda) for _ in range(2))
    ham.vbias(G, v, 0.01, precision=A.PREC_MIXED)
    ham.vbias(G, r, 0.01)
    assert ham.device_error_flag() == 0
    v, r = to_host(v), to_host(r)
    step, K = (8, N * M) if fmt == 2 else (4, N * M)
    S = next((c for c in range(16, 1, -1) if K % (c * step) == 0 and K // c >= 512), 1)
    bound = 8 * (2.0 ** -21 + K / S / (2 * step) * 2.0 ** -23)
    assert np.max(np.abs(v - r)) < bound * np.sqrt(np.mean(np.abs(r) ** 2))


@pytest.mark.parametrize("nup,ndn", [(1, 1), (16, 15), (23, 24), (33, 34), (47, 48), (67, 66), (119, 1),
                                     (120, 120)])
def test_energy_block_sums(cuda, nup, ndn):
    """The complex128 energy at the sizes around which a CTA of its block sums takes eight, four, two
    and one Cholesky vectors, up to the 120 electrons whose block fills an SM's shared memory."""
    from oracle import afqmc as O
    from safire_b200 import afqmc as A
    M, Nc, W = max(nup, ndn) + 1, 11, 3
    rs = np.random.default_rng(nup)
    L = rs.standard_normal((M, M, Nc))
    args = (A.COLLINEAR, M, nup, ndn, (L + L.transpose(1, 0, 2))[None],
            np.eye(M)[None].astype(complex), 0.0,
            [np.linalg.qr(rs.standard_normal((M, n)))[0].T.astype(complex) for n in (nup, ndn)])
    G = rand_c(rs, W, (nup + ndn) * M)
    E = torch.zeros((W, 3), dtype=torch.complex128, device=cuda)
    A.HamiltonianOperations(*args).energy(E, to_dev(G))
    # each of the products' sums has M terms, each energy N^2 Nc of their products
    assert rel_err(to_host(E), O.Real3IndexFactorization(*args).energy(G)) < 50 * (M + nup) * EPS
