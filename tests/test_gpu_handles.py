"""What the handles keep between calls follows what they were given: several propagators of one
Hamiltonian, mean fields that change, captured steps beside other calls, host threads."""
import numpy as np
import pytest
import torch

from safire_b200.synth import make_workload
from tests.gpu_helpers import rand_c, rel_err, to_dev, to_host

pytestmark = pytest.mark.gpu
# one mixed-precision step against complex128 (operands of 22 bits, FP32 sums); the propagators of two
# time steps below differ by a percent
TOL_STEP = 1e-5


def _system():
    """M = 48 (both plane formats), its Hamiltonian handle and some field uniforms."""
    from safire_b200 import afqmc as A
    wl = make_workload("cfg1", W=8, M=48, N=6, Nc=40)
    ham = A.HamiltonianOperations(wl.walker_type, wl.M, wl.nup, wl.ndn, wl.Likn, wl.hij, wl.E0,
                                  wl.PsiT)
    u = to_dev(np.random.default_rng(3).random((wl.W, wl.Nc)), torch.float64)
    return wl, ham, u


def _walkers(wl, ham):
    from safire_b200 import afqmc as A
    ws = A.WalkerSet(wl.walker_type, wl.M, wl.nup, wl.ndn, wl.W)
    ws.init_from_trial(ham)
    A.NOMSD(ham).Energy(ws, set_properties=True)
    ws.setProperty(A.capi.PSEUDO_ELOC, sum(ws.getProperty(p) for p in
                                           (A.capi.E1, A.capi.EXX, A.capi.EJ)))
    return ws


def _step(wl, ham, prop, u):
    ws = _walkers(wl, ham)
    prop.Propagate(ws, 0.0, u)
    return to_host(ws.SlaterMatrices(0)).copy()


@pytest.mark.parametrize("mode", [0, 2, 4])  # a launch per product, fused TF32, fused FP16
def test_mixed_step_takes_its_own_propagator(cuda, mode):
    """Mixed steps of propagators that follow one another on a Hamiltonian (another time step after
    the first is gone, whose memory the second is likely to get; two at a time, in turn; another
    mean field) each apply their own exp(-dt H1 / 2), as the complex128 steps do."""
    from safire_b200 import afqmc as A
    wl, ham, u = _system()
    ham.set_taylor_fused(mode)

    def new(dt, precision):
        return A.Propagator(ham, A.default_params(dt=dt, precision=precision), wl.W)

    want = {dt: _step(wl, ham, new(dt, A.PREC_FP64), u) for dt in (0.01, 0.05)}
    assert rel_err(want[0.01], want[0.05]) > 100 * TOL_STEP
    for dt in (0.01, 0.05, 0.01):
        prop = new(dt, A.PREC_MIXED)
        assert rel_err(_step(wl, ham, prop, u), want[dt]) < TOL_STEP, dt
        del prop
    props = {dt: new(dt, A.PREC_MIXED) for dt in want}
    for _ in range(2):
        for dt, prop in props.items():
            assert rel_err(_step(wl, ham, prop, u), want[dt]) < TOL_STEP, dt
    # the mean field moves between the one-body propagator and the fields
    vMF = props[0.05].P1_vMF()[1] + 0.3
    ref = new(0.05, A.PREC_FP64)
    ref.set_trial(None, vMF)
    moved = _step(wl, ham, ref, u)
    assert rel_err(moved, want[0.05]) > 100 * TOL_STEP
    props[0.05].set_trial(None, vMF)
    assert rel_err(_step(wl, ham, props[0.05], u), moved) < TOL_STEP
    assert ham.device_error_flag() == 0


def test_captured_mixed_step_beside_another_propagator(cuda):
    """A captured mixed step keeps its propagator while another one of the Hamiltonian steps."""
    from safire_b200 import afqmc as A
    wl, ham, u = _system()
    ham.set_taylor_fused(4)
    a, b = (A.Propagator(ham, A.default_params(dt=dt, precision=A.PREC_MIXED), wl.W)
            for dt in (0.01, 0.05))
    want = _step(wl, ham, a, u)
    ws, eshift = _walkers(wl, ham), torch.zeros(1, dtype=torch.float64, device=cuda)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.Propagate_dev(ws, eshift, u)
    _step(wl, ham, b, u)
    g.replay()
    assert np.array_equal(to_host(ws.SlaterMatrices(0)), want)


def _phmsd():
    from safire_b200 import afqmc as A
    from safire_b200.synth import make_hamiltonian, make_phmsd_trial
    M, nup, ndn, Nc = 12, 3, 2, 10
    h1, Likn = make_hamiltonian(M, Nc, 0.9, seed=7)
    _, C = np.linalg.eigh(h1)
    t = make_phmsd_trial(M, nup, ndn, C, nocc=2, nvirt=4, ndet=12, seed=3, max_level=2)
    hij = h1[None].astype(complex)
    ph = A.PHMSD(t)
    ph.set_hamiltonian(Likn[None], hij, 0.2)
    return t, C, hij, Likn, ph


def _phmsd_G(ph, C, W, block=0, seed=1):
    M, n = C.shape[0], (3, 2)
    rs = np.random.default_rng(seed)
    S = [C[None, :, :k] + rand_c(rs, W, M, k, scale=0.2 / np.sqrt(M)) for k in n]
    wbuf = to_dev(np.concatenate([x.reshape(W, -1) for x in S], 1))
    G = torch.empty((W, sum(ph.info()[3:5]), M), dtype=torch.complex128, device="cuda")
    ov = torch.empty(W, dtype=torch.complex128, device="cuda")
    return wbuf, G, ov, lambda: ph.MixedDensityMatrix(wbuf, G, ov, block=block)


def test_phmsd_captured_step_beside_larger_calls(cuda):
    """A captured step of 600 walkers with a particle-hole trial, after the density matrix of 1200 on
    the same handle: the buffers of 512 and more walkers are not replaced, so its replays write where
    the capture did, bit for bit what an eager step gives."""
    from safire_b200 import afqmc as A
    t, C, hij, Likn, ph = _phmsd()
    W = 600
    ham = A.HamiltonianOperations(A.COLLINEAR, t.M, t.nup, t.ndn, Likn[None], hij, 0.2,
                                  [t.orbmat[s][t.refc[s]] for s in (0, 1)])
    prop = A.Propagator(ham, A.default_params(dt=0.01), W)
    prop.set_trial(ph)
    u = to_dev(np.random.default_rng(4).random((W, ham.Nc)), torch.float64)
    eshift = torch.zeros(1, dtype=torch.float64, device=cuda)

    def walkers():
        ws = A.WalkerSet(A.COLLINEAR, t.M, t.nup, t.ndn, W)
        ws.init_from_trial(ham)
        return ws
    eager, ws = walkers(), walkers()
    prop.Propagate_dev(eager, eshift, u)
    want = to_host(eager.buffer).copy()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        prop.Propagate_dev(ws, eshift, u)
    _, G, ov, call = _phmsd_G(ph, C, 2 * W)
    call()
    big = to_host(G).copy()
    g.replay()
    assert np.array_equal(to_host(ws.buffer), want)
    call()
    assert np.array_equal(to_host(G), big)


@pytest.mark.parametrize("W", [512, 513, 1300])
def test_phmsd_density_matrix_captured(cuda, W):
    """The density matrix under capture: with the buffers of a smaller call it runs in blocks of what
    they hold, with its own in one, and both give what blocks of 100 give."""
    _, C, _, _, ph = _phmsd()
    _, G, _, call = _phmsd_G(ph, C, W, block=100)
    call()
    want = to_host(G).copy()
    for first in (512, W):
        ph = _phmsd()[-1]
        _phmsd_G(ph, C, first)[-1]()
        _, G, _, call = _phmsd_G(ph, C, W)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call()
        g.replay()
        assert np.array_equal(to_host(G), want), first


def test_failed_call_leaves_no_error(cuda):
    """A call that the runtime refuses (a block sum of 121 electrons passes an SM's shared memory)
    reports it, and neither a later call nor the caller's own runtime finds the error again."""
    from safire_b200 import afqmc as A
    from safire_b200.capi import AfqmcError
    with pytest.raises(AfqmcError):
        _energy_call(122, 121, A.PREC_FP64)()
    assert torch.isfinite(torch.ones(4, device=cuda).exp()).all()
    assert np.all(np.isfinite(to_host(_energy_call(24, 5, A.PREC_FP64)()).view(float)))


def _energy_call(M, N, precision):
    from safire_b200 import afqmc as A
    rs = np.random.default_rng(N)
    L = rs.standard_normal((M, M, 24))
    psi = np.linalg.qr(rs.standard_normal((M, N)))[0].T.astype(complex)
    ham = A.HamiltonianOperations(A.CLOSED, M, N, N, (L + L.transpose(1, 0, 2))[None],
                                  np.eye(M)[None].astype(complex), 0.0, [psi])
    G = to_dev(rand_c(rs, 4, N * M))

    def call():
        E = torch.zeros((4, 3), dtype=torch.complex128, device="cuda")
        ham.energy(E, G, precision=precision)
        return E
    return call


def _det_op_call(name, W, M, N):
    from safire_b200 import afqmc as A
    rs = np.random.default_rng(N)
    S = to_dev(np.eye(M, N) + rand_c(rs, W, M, N, scale=0.3 / np.sqrt(M)))
    if name == "inverse":
        A_ = S[:, :N].contiguous()

        def call():
            inv, ld = torch.empty_like(A_), torch.zeros(W, dtype=torch.complex128, device="cuda")
            A.det_ops.inverse_logdet(A_, inv, ld)
            return inv
    elif name == "orthogonalize":
        def call():
            q, ld = S.clone(), torch.zeros(W, dtype=torch.complex128, device="cuda")
            A.det_ops.orthogonalize(q, ld)
            return q
    else:
        P1 = to_dev(np.eye(M) + rand_c(rs, M, M, scale=0.1 / np.sqrt(M)))
        V = to_dev(rand_c(rs, W, M, M, scale=0.5 / np.sqrt(M)))

        def call():
            q = S.clone()
            A.det_ops.Propagate(q, P1, V)
            return q
    return call


@pytest.mark.parametrize("kind", ["propagate_gemm", "propagate_fused", "inverse", "orthogonalize",
                                  "energy", "energy_mixed"])
def test_host_threads(cuda, kind):
    """Two host threads, each on a stream of its own, whose calls take the same kernels at sizes that
    need different amounts of shared memory: every call succeeds and returns what it returns alone."""
    import threading
    from safire_b200 import afqmc as A
    calls = {"propagate_gemm": lambda: [_det_op_call("propagate", 150, 64, 64),
                                        _det_op_call("propagate", 24, 200, 64)],
             "propagate_fused": lambda: [_det_op_call("propagate", 4, 128, 32),
                                         _det_op_call("propagate", 4, 65, 32)],
             "inverse": lambda: [_det_op_call("inverse", 4, 70, 64), _det_op_call("inverse", 4, 70, 57)],
             "orthogonalize": lambda: [_det_op_call("orthogonalize", 4, 90, 85),
                                       _det_op_call("orthogonalize", 4, 70, 64)],
             "energy": lambda: [_energy_call(104, 100, A.PREC_FP64), _energy_call(104, 60, A.PREC_FP64)],
             "energy_mixed": lambda: [_energy_call(104, 50, A.PREC_MIXED),
                                      _energy_call(104, 33, A.PREC_MIXED)]}[kind]()
    want = [c() for c in calls]
    torch.cuda.synchronize()
    errors, start = [], threading.Barrier(len(calls))

    def run(call, expect):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(150):
                    got = call()
                torch.cuda.current_stream().synchronize()
                if not torch.equal(got, expect):
                    errors.append(f"another result: {(got - expect).abs().max().item():.2e}")
        except Exception as e:  # raised again on the test's own thread
            errors.append(repr(e))

    threads = [threading.Thread(target=run, args=a) for a in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
