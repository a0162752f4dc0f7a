"""GPU: the stage kernels over every state count and slot count they are
instantiated for, where lanes fall outside the tile, sites have no bath or
several, and the ADOs leave a remainder of the grid -- against the oracle
(tolerances of test_gpu_parity.py: 1e-13 of the largest element for one
derivative; a step of the RK4 polynomial adds a few roundings per stage, so
1e-13 of the largest element again)."""
import numpy as np
import pytest

import heom_b200 as hb
import heom_oracle as ho

pytestmark = pytest.mark.gpu

TOL = 1e-13


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def hamiltonian(n, cplx):
    h = ho.synthetic_hamiltonian(n, 40 + n).astype(np.complex128)
    if cplx:
        im = np.triu(np.random.default_rng(n).normal(0.0, 20.0, size=(n, n)), 1)
        h = h + 1j * (im - im.T)
    return h if cplx else h.real


def problem(n, m, depth, cplx, baths_per_state=1):
    if baths_per_state == 1:
        coupling = None
    else:  # bath i on sites i and i + 1, the last site with a single one
        coupling = np.array([[i, (i + 1) % n] for i in range(n)], np.int32)
        coupling[n - 1, 1] = -1
    return ho.build_problem(ho.make_system(hamiltonian(n, cplx), [35.0 + i for i in range(n)],
                                           [50.0 + i for i in range(n)], [0.0] * n, m, 300.0, depth,
                                           coupling=coupling))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n,m,depth,bps", [(n, m, 3 if n * m <= 12 else 2, 1) for n in range(1, 9) for m in (1, 2, 3)] +
                         [(2, 8, 2, 1), (7, 5, 1, 1), (8, 8, 1, 1), (3, 1, 4, 2), (5, 2, 2, 2), (8, 1, 3, 2), (7, 3, 1, 2)])
def test_small_states(n, m, depth, bps, cplx):
    prob = problem(n, m, depth, cplx, min(bps, n))
    y = np.random.default_rng(n * 10 + m).normal(size=prob.state_len)
    dt = 0.5e-15
    ref = ho.derivative(prob, y)
    step = y
    for _ in range(2):
        step = ho.rk4_step(prob, dt, step)
    for scheme in ("product", "horner"):
        with hb.Heom.from_problem(prob, scheme=scheme) as H:
            if scheme == "product":
                bi, bo = H.buffer(), H.buffer()
                bi.write(y)
                H.solve(bi, bo)
                assert rel(bo.read(), ref) <= TOL
                bi.close(), bo.close()
            H.set_state(y)
            H.rk4_steps(dt, 2)
            assert rel(H.get_state(), step) <= TOL


@pytest.mark.parametrize("n,m,depth", [(7, 2, 2), (5, 1, 3), (10, 1, 2)])
def test_flow_buffers_are_the_neighbour_terms(n, m, depth):
    """The plus and the minus terms of an evaluation add up to the derivative without its commutator and
    same term, which are written out here from the tables."""
    prob = problem(n, m, depth, False)
    nodes = prob.graph.nodes
    y = np.random.default_rng(5).normal(size=prob.state_len)
    w = y.view(np.complex128).reshape(nodes, n, n)
    hs = prob.hamiltonian.view(np.complex128).reshape(n, n) / 1.05457148e-34
    same = np.asarray(prob.pf_same).view(np.complex128)
    pair = -(same[:, None] + same[None, :]) * (1.0 - np.eye(n))
    rest = 1j * (w @ hs - hs @ w) + (np.asarray(prob.pf_same_sum).view(np.complex128)[:, None, None] + pair) * w
    ref = ho.derivative(prob, y).view(np.complex128).reshape(nodes, n, n)
    with hb.Heom.from_problem(prob) as H:
        b = [H.buffer() for _ in range(4)]
        b[0].write(y)
        H.set_flow_buffers(b[2], b[3])
        H.solve(b[0], b[1], acc_coeff=1.0)
        above, below = (x.read().view(np.complex128).reshape(nodes, n, n) for x in b[2:])
        H.set_flow_buffers(None, None)
        for x in b:
            x.close()
    assert np.max(np.abs(above + below - (ref - rest))) <= 1e-12 * np.max(np.abs(ref))
    last = np.asarray(prob.graph.tuples).reshape(nodes, -1).sum(axis=1) == depth
    assert np.all(above[last] == 0.0) and np.all(below[0] == 0.0)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n,m,depth,bps", [(n, m, 2, 1) for n in range(9, 17) for m in (1, 2)] +
                         [(9, 3, 2, 1), (10, 5, 1, 1), (16, 3, 1, 1), (11, 1, 2, 2), (12, 2, 1, 2)])
def test_teams(n, m, depth, bps, cplx):
    """9 to 16 states: even and odd counts (threads that own no sector, the padding half), one to eight slots."""
    prob = problem(n, m, depth, cplx, bps)
    y = np.random.default_rng(n * 10 + m).normal(size=prob.state_len)
    step = ho.rk4_step(prob, 0.5e-15, y)
    for scheme in ("product", "horner"):
        with hb.Heom.from_problem(prob, scheme=scheme) as H:
            H.set_state(y)
            H.rk4_steps(0.5e-15, 1)
            got = H.get_state()
            assert rel(got, step) <= TOL
    with hb.Heom.batch([hb.Heom.tables_of(prob)] * 2) as H:  # the fragments of an instance per ADO
        H.set_state(np.concatenate([y, 2.0 * y]))
        H.rk4_steps(0.5e-15, 1)
        both = H.get_state()
    assert rel(both[:y.size], step) <= TOL and rel(both[y.size:], 2.0 * step) <= TOL
