"""Performance cases of the SQD framework, each through its public entry points.

Kinds of case (``case["kind"]``):

* ``product``  one Hamiltonian-vector product ``DeviceOperator.matvec`` -- what an eigensolver or a
  user's own iteration calls over and over; ``form`` is the operator's mode (``free``: matrix-free
  lookups, ``conn``: cached connectivity, the default of ``sqd()``, ``csr``: cached elements);
* ``solve``    ``ground_locg`` on a prepared operator from a seeded random start, to double precision;
* ``sqd``      the whole drop-in call ``sqd(hamiltonian, samples)`` on 0/1 sample rows;
* ``batch``    ``BatchedSQD.matvec``: the products of many independent problems in one call;
* ``setup``    from device samples with duplicates to the first product (``uniquify_device``,
  ``SQDProblem``, ``matvec``), what a user pays once per set of samples;
* ``train``    one optimiser step of the warm-start network (``train_step`` and ``step``);
* ``predict``  the network's outputs on every state of a subspace (``predict``);
* ``circuit``  ``svsim`` of a Pauli-rotation circuit.

Hamiltonians (``case["model"]``): ``random`` (random Pauli sums of locality 1 to 4), ``hubbard``
(Fermi-Hubbard lattices, Jordan-Wigner) and ``electronic`` (random two-body Hamiltonians with the
structure of molecules).  States: ``sector`` draws uniformly from the fixed-particle-number sector;
``near`` draws what a sampler of a low-energy state returns -- configurations with at most one
doubly occupied site (Hubbard) or a few excitations above the lowest orbitals (electronic).
"""
import functools
import math

import numpy as np
import torch

from rqutils_gb300.batch import BatchedSQD
from rqutils_gb300.device import DeviceOperator, DeviceSubspace, DeviceTerms
from rqutils_gb300.ground_locg import ground_locg
from rqutils_gb300.paulis.symplectic import PauliSumXZ
from rqutils_gb300.sqd import SQDProblem, sqd, uniquify_device
from rqutils_gb300.svsim import CircuitXZ, svsim
from rqutils_gb300.warmstart import NPARAMS, WarmStartMLP
from rqutils_gb300 import workloads

DEV = 'cuda'
LATTICES = {8: (4, 2), 9: (3, 3), 12: (4, 3), 16: (4, 4)}


def listed():
    return [
        # a quick product on a few hundred states (notebook-sized problem): latency only
        dict(name='product_small', kind='product', model='random', qubits=12, terms=60, states='sector',
             rows=449, form='free', dtype='complex128'),
        # the repository's 20-qubit benchmark problem: K = 200 terms, 16,384 states, complex128
        dict(name='product_random20', kind='product', model='random', qubits=20, terms=200, states='sector',
             rows=16384, form='free', dtype='complex128'),
        # the headline product: Hubbard 4x4 (32 spin-orbitals), 2^20 sampled states, complex64
        dict(name='product_hubbard', kind='product', model='hubbard', qubits=32, terms=0, states='sector',
             rows=1 << 20, form='free', dtype='complex64'),
        # molecule-shaped Hamiltonian with thousands of X groups and 64-bit keys, matrix-free
        dict(name='product_electronic', kind='product', model='electronic', qubits=36, terms=12000, states='near',
             rows=150001, form='free', dtype='float64'),
        # the cached-connectivity product inside every default solve, on a connected subspace
        dict(name='product_cached', kind='product', model='hubbard', qubits=32, terms=0, states='near',
             rows=1 << 18, form='conn', dtype='float64'),
        # ordinary use of the drop-in: samples of a 20-qubit molecule in, ground state out
        dict(name='sqd_call', kind='sqd', model='electronic', qubits=20, terms=4000, states='near', rows=3001),
        # the eigensolver on the Hubbard subspace of the warm-start study
        dict(name='solve_hubbard', kind='solve', model='hubbard', qubits=32, terms=0, states='near',
             rows=1 << 18, variant='fast', precision='mixed'),
        # many independent problems at once (parameter scans, bootstrap resamples)
        dict(name='batch_product', kind='batch', problems=48, qubits=40, rows=1 << 16, form='free', dtype='complex64'),
        # samples with duplicates, half a million distinct, to an operator with cached connectivity
        dict(name='setup_samples', kind='setup', model='hubbard', qubits=32, terms=0, states='near', rows=600011),
        # a training step of the warm-start network at the batch size of fit()
        dict(name='train_step', kind='train', rows=65536),
        # the network's start vector data on every state of a subspace
        dict(name='predict_states', kind='predict', rows=1 << 18),
        # a state-vector run of a Trotter-like circuit
        dict(name='circuit_20', kind='circuit', qubits=20, gates=120),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _model(rng, rows_hi, near=None):
    model = rng.choice(['random', 'hubbard', 'electronic']) if near is None else rng.choice(['hubbard', 'electronic'])
    if model == 'random':
        n = rng.randint(12, 40)
        rows = _log_int(rng, 300, min(rows_hi, math.comb(n, n // 2) // 2))
        return dict(model=model, qubits=n, terms=_log_int(rng, 50, 2000), states='sector', rows=rows)
    if model == 'hubbard':
        ns = rng.choice([9, 12, 16])
        states = near or rng.choice(['near', 'sector'])
        nu = ns // 2
        most = (math.comb(ns, nu) * (1 + nu * (ns - (ns - nu))) if states == 'near'
                else math.comb(ns, nu) * math.comb(ns, ns - nu)) // 2
        return dict(model=model, qubits=2 * ns, terms=0, states=states, rows=_log_int(rng, 300, min(rows_hi, most)))
    orb = rng.choice([8, 10, 12, 14, 16, 18])
    most = min(rows_hi, 150000, math.comb(orb, orb // 2) ** 2 // 16)
    return dict(model=model, qubits=2 * orb, terms=_log_int(rng, 1000, 12000), states=near or 'near',
                rows=_log_int(rng, 300, most))


def draw(rng):
    kind = rng.choice(['product', 'product', 'product', 'solve', 'sqd', 'batch', 'setup', 'train', 'predict', 'circuit'])
    if kind == 'product':
        m = _model(rng, 1 << 20)
        real = m['model'] != 'random'
        dtype = rng.choice(['float32', 'float64', 'complex64', 'complex128'] if real else ['complex64', 'complex128'])
        return dict(kind=kind, form=rng.choice(['free', 'free', 'conn', 'csr']), dtype=dtype, **m)
    if kind == 'solve':
        m = _model(rng, 1 << 18, 'near')
        m['rows'] = max(m['rows'], 1000)
        return dict(kind=kind, variant=rng.choice(['fast', 'reference']), precision=rng.choice(['fp64', 'mixed']), **m)
    if kind == 'sqd':
        orb = rng.choice([7, 8, 9, 10])
        return dict(kind=kind, model='electronic', qubits=2 * orb, terms=_log_int(rng, 1000, 6000), states='near',
                    rows=_log_int(rng, 200, 4000))
    if kind == 'batch':
        return dict(kind=kind, problems=rng.randint(4, 48), qubits=rng.randint(20, 40), rows=_log_int(rng, 1 << 12, 1 << 16),
                    form=rng.choice(['free', 'conn']), dtype=rng.choice(['complex64', 'complex128']))
    if kind == 'setup':
        return dict(kind=kind, **_model(rng, 600011, 'near'))
    if kind == 'train':
        return dict(kind=kind, rows=128 * _log_int(rng, 4, 512))
    if kind == 'predict':
        return dict(kind=kind, rows=_log_int(rng, 1000, 1 << 18))
    return dict(kind=kind, qubits=rng.randint(8, 20), gates=_log_int(rng, 20, 120))


# ---------------------------------------------------------------------------------------------
# inputs (the Hamiltonian as labels and coefficients, states as sorted int64 on the device)
# ---------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _electronic(orbitals, terms):
    return workloads.chemistry_jw(orbitals, np.random.default_rng(orbitals), keep=terms)


@functools.lru_cache(maxsize=8)
def _electronic_sum(orbitals, terms):
    return PauliSumXZ.from_paulisum(_electronic(orbitals, terms), force_real=True, add_padding=True)


def _labels(case, seed):
    rng = np.random.default_rng(seed)
    if case['model'] == 'random':
        return workloads.random_pauli_masks(rng, case['qubits'], case['terms'])
    if case['model'] == 'hubbard':
        lx, ly = LATTICES[case['qubits'] // 2]
        return workloads.hubbard_jw(lx, ly, 1.0, float(rng.uniform(3., 6.)), True)
    return _electronic(case['qubits'] // 2, case['terms'])


def _pauli_sum(case, seed):
    if case['model'] == 'electronic':  # a program keeps its molecule, the samples change
        return _electronic_sum(case['qubits'] // 2, case['terms'])
    return PauliSumXZ.from_paulisum(_labels(case, seed), force_real=True, add_padding=True)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _fixed_weight(g, n, weight, count):
    """count uniform n-bit words of the given weight."""
    top = torch.rand((count, n), generator=g, device=DEV).argsort(dim=1)[:, :weight]
    return torch.bitwise_left_shift(torch.ones_like(top), top).sum(dim=1)


def _near_words(g, n, weight, count):
    """count n-bit words: the lowest `weight` orbitals filled, then 0 to 4 random excitations."""
    filled = (torch.arange(n, device=DEV) < weight).to(torch.float32)
    depth = torch.rand(count, generator=g, device=DEV).log().div(math.log(0.55)).floor()
    depth = depth.clamp(max=min(4, weight, n - weight))[:, None]
    r = torch.rand((count, n), generator=g, device=DEV)
    rank = [(r + 2. * k).argsort(dim=1).argsort(dim=1) for k in (1. - filled, filled)]
    flip = (rank[0] < depth) | (rank[1] < depth)  # `depth` of the filled ones and of the empty ones
    return ((filled.bool() ^ flip).to(torch.int64) << torch.arange(n, device=DEV)).sum(dim=1)


def _draw_words(case, g, count, seed):
    n = case['qubits']
    half = n // 2
    if case['model'] == 'random':
        return _fixed_weight(g, n, half, count)
    if case['model'] == 'hubbard' and case['states'] == 'near':
        pool = workloads.low_double_occupancy_states(np.random.default_rng(0), _pool_size(half), half)
        idx = torch.randint(0, len(pool), (count,), generator=g, device=DEV)
        return torch.from_numpy(pool.view(np.int64)).to(DEV)[idx]
    w_up = half // 2
    w_dn = half - w_up if case['model'] == 'hubbard' else w_up
    make = _near_words if case['states'] == 'near' else _fixed_weight
    return make(g, half, w_up, count) | (make(g, half, w_dn, count) << half)


@functools.lru_cache(maxsize=4)
def _pool_size(ns):
    up = ns // 2
    return math.comb(ns, up) * (1 + up * up if ns % 2 == 0 else 1 + up * (ns - up - 1) + up)


def _states(case, seed):
    """Sorted distinct states (int64, device), case['rows'] of them where the model has as many."""
    g = _gen(seed)
    have = torch.empty(0, dtype=torch.int64, device=DEV)
    need = case['rows']
    for _ in range(40):
        more = _draw_words(case, g, int(1.2 * (need - have.numel())) + 64, seed)
        have = torch.unique(torch.cat([have, more]))
        if have.numel() >= need:
            break
    if have.numel() > need:
        keep = torch.randperm(have.numel(), generator=g, device=DEV)[:need]
        have = have[keep].sort().values
    return have


def _samples(case, seed):
    """case['rows'] samples (device words, unsorted) of 5/6 as many distinct states."""
    s = _states(dict(case, rows=max(1, case['rows'] * 5 // 6)), seed)
    g = _gen(seed + 2)
    again = s[torch.randint(0, s.numel(), (case['rows'] - s.numel(),), generator=g, device=DEV)]
    words = torch.cat([s, again])
    return words[torch.randperm(words.numel(), generator=g, device=DEV)]


def _vector(rows, dtype, seed):
    dt = getattr(torch, dtype)
    v = torch.randn(rows, dtype=dt, device=DEV, generator=_gen(seed + 1))
    return v / torch.linalg.vector_norm(v)


_LEVELS = {'free': (0, 0), 'conn': (1, 0), 'csr': (1, 2)}


# ---------------------------------------------------------------------------------------------
# batches
# ---------------------------------------------------------------------------------------------
def _batch_parts(case, seed):
    """[(labels, coeffs, n, states)] of the batch: qubits from 16 up, terms and rows log-uniform."""
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(case['problems'] * case['rows'])
    parts = []
    for p in range(case['problems']):
        n = int(sizes.integers(16, case['qubits'] + 1))
        k = int(round(math.exp(sizes.uniform(math.log(100), math.log(1000)))))
        top = min(case['rows'], math.comb(n, n // 2) // 2)
        rows = int(round(math.exp(sizes.uniform(math.log(1 << 10), math.log(top)))))
        labels, coeffs = workloads.random_pauli_masks(rng, n, k)
        s = _states(dict(model='random', qubits=n, states='sector', rows=rows), seed + 7919 * (p + 1))
        parts.append((labels, coeffs, n, s))
    return parts


# ---------------------------------------------------------------------------------------------
# the network and circuits
# ---------------------------------------------------------------------------------------------
def _net_params(seed):
    g = torch.Generator().manual_seed(int(seed))
    p = torch.zeros(NPARAMS)
    o = 0
    for count, scale in ((256 * 64, 1 / 6.), (256, 0.1), (256 * 256, 1 / 16.), (256, 0.1), (512, 1 / 16.), (2, 0.1)):
        p[o:o + count] = torch.randn(count, generator=g) * scale
        o += count
    return p


def _net_features(states, u):
    """(rows, 64) float64 network inputs of states with parameters u (rows,)."""
    f = torch.zeros((states.numel(), 64), dtype=torch.float64, device=DEV)
    f[:, :32] = 2. * ((states[:, None] >> torch.arange(32, device=DEV)) & 1).double() - 1.
    t = (u - 5.) / 3.
    f[:, 32], f[:, 33], f[:, 34] = t, t * t, t * t * t
    return f


def _train_inputs(case, seed):
    rows = case['rows']
    g = _gen(seed)
    s = _fixed_weight(g, 16, 8, rows) | (_fixed_weight(g, 16, 8, rows) << 16)
    u = 2. + 6. * torch.rand(rows, generator=g, device=DEV, dtype=torch.float64)
    x = _net_features(s, u).to(torch.bfloat16)
    tgt = torch.empty((rows, 3), device=DEV)
    tgt[:, 0] = torch.randn(rows, generator=g, device=DEV)
    tgt[:, 1] = torch.where(torch.rand(rows, generator=g, device=DEV) < 0.5, -1., 1.)
    tgt[:, 2] = (torch.randn(rows, generator=g, device=DEV) ** 2).clamp(0.05, 20.)
    return x, tgt


def _circuit(case, seed):
    """Trotter-like layers of rx, rz, rzz, ry and x gates as (x, z, cos, sin) arrays."""
    n, ng = case['qubits'], case['gates']
    rng = np.random.default_rng(seed)
    x, z = np.zeros(ng, np.int64), np.zeros(ng, np.int64)
    ang = rng.uniform(-np.pi, np.pi, ng)
    c, s = np.cos(-ang / 2), np.sin(-ang / 2)
    for k in range(ng):
        q = int(rng.integers(n))
        name = ('rx', 'rx', 'rzz', 'rzz', 'rz', 'ry', 'x')[int(rng.integers(7))]
        if name in ('rx', 'ry', 'x'):
            x[k] = 1 << q
        if name in ('rz', 'ry'):
            z[k] = 1 << q
        if name == 'rzz':
            z[k] = (1 << q) | (1 << ((q + 1) % n))
        if name == 'x':
            c[k], s[k] = 0., -1.
    return x, z, c, s


# ---------------------------------------------------------------------------------------------
# prepare / run / work
# ---------------------------------------------------------------------------------------------
def _operator(case, seed, states):
    sub = DeviceSubspace(states, num_qubits=case['qubits'])
    return DeviceOperator(DeviceTerms(_pauli_sum(case, seed)), sub, mode=case.get('form', 'conn'))


def prepare(case, seed):
    kind = case['kind']
    if kind == 'product':
        s = _states(case, seed)
        return dict(kind=kind, op=_operator(case, seed, s), x=_vector(s.numel(), case['dtype'], seed))
    if kind == 'solve':
        s = _states(case, seed)
        return dict(kind=kind, op=_operator(case, seed, s), x0=_vector(s.numel(), 'float64', seed),
                    variant=case['variant'], precision=case['precision'])
    if kind == 'sqd':
        n = case['qubits']
        words = _samples(case, seed)
        bits = (words[:, None] >> torch.arange(n - 1, -1, -1, device=DEV)) & 1
        return dict(kind=kind, ham=_pauli_sum(case, seed), samples=bits.to(torch.uint8).cpu().numpy())
    if kind == 'batch':
        parts = _batch_parts(case, seed)
        hams = [PauliSumXZ.from_paulisum((a, b), force_real=True, add_padding=True) for a, b, _, _ in parts]
        b = BatchedSQD(hams, [s.cpu().numpy().view(np.uint64) for _, _, _, s in parts],
                       cache_level=_LEVELS[case['form']])
        return dict(kind=kind, b=b, x=_vector(b.D, case['dtype'], seed))
    if kind == 'setup':
        samples = _samples(case, seed)
        return dict(kind=kind, ham=_pauli_sum(case, seed), samples=samples,
                    x=_vector(samples.numel(), 'float64', seed))
    if kind == 'train':
        net = WarmStartMLP(params=_net_params(seed))
        x, tgt = _train_inputs(case, seed)
        return dict(kind=kind, net=net, x=x, xt=x.T.contiguous(), tgt=tgt,
                    out=torch.empty((case['rows'], 2), device=DEV), loss=torch.zeros(1, dtype=torch.float64, device=DEV))
    if kind == 'predict':
        s = _states(dict(model='hubbard', qubits=32, states='sector', rows=case['rows']), seed)
        return dict(kind=kind, net=WarmStartMLP(params=_net_params(seed)), s=s, u=3. + (seed % 97) / 32.)
    x, z, c, sn = _circuit(case, seed)
    return dict(kind=kind, circ=CircuitXZ(x, z, c, sn, case['qubits']), init=_circuit_start(case, seed))


def _circuit_start(case, seed):
    return seed % (1 << case['qubits'])


def run(state):
    kind = state['kind']
    if kind == 'product':
        return state['op'].matvec(state['x'])
    if kind == 'solve':
        # a solve to (nearly) double precision; the default test scales with the vector's length
        e, x, _ = ground_locg(state['op'], state['x0'], maxiter=3000, tol=1e-300, target_rel=1e-12,
                              variant=state['variant'], precision=state['precision'])
        return dict(energy=e, vector=x)
    if kind == 'sqd':
        e, x, basis = sqd(state['ham'], state['samples'])
        return dict(energy=e, vector=x, basis=basis)
    if kind == 'batch':
        return state['b'].matvec(state['x'])
    if kind == 'setup':
        s = uniquify_device(state['samples'])
        p = SQDProblem(state['ham'], s, cache_level=(1, 0))
        return dict(states=s, diagonal=p.op.diag0, product=p.op.matvec(state['x'][:s.numel()]))
    if kind == 'train':
        net = state['net']
        grads = net.train_step(state['x'], state['xt'], state['tgt'], out=state['out'], loss=state['loss'])
        net.step(1e-3)
        return dict(out=state['out'], loss=state['loss'], grads=grads, params=net.params)
    if kind == 'predict':
        return state['net'].predict(state['s'], state['u'])
    return svsim(state['circ'], state['init'])


_SIZE = {'float32': 4, 'float64': 8, 'complex64': 8, 'complex128': 16}


def work(case):
    kind = case['kind']
    if kind == 'product':  # states, x and y once
        b = _SIZE[case['dtype']]
        return dict(bytes=case['rows'] * (8 + 2 * b) + 24 * case['terms'], flops=2 * case['rows'])
    if kind == 'solve':  # the states, the start and the ground state
        return dict(bytes=case['rows'] * 24, flops=2 * case['rows'])
    if kind == 'sqd':
        return dict(bytes=case['rows'] * (2 * case['qubits'] + 8), flops=2 * case['rows'])
    if kind == 'batch':
        rows = case['problems'] * (case['rows'] - 1024) / math.log(case['rows'] / 1024.)
        return dict(bytes=rows * (8 + 2 * _SIZE[case['dtype']]), flops=2 * rows)
    if kind == 'setup':
        return dict(bytes=case['rows'] * 8 * 2, flops=case['rows'])
    if kind == 'train':
        return dict(bytes=case['rows'] * (2 * 128 + 12 + 8) + NPARAMS * 32,
                    flops=case['rows'] * 2 * 3 * (64 * 256 + 256 * 256 + 512))
    if kind == 'predict':
        return dict(bytes=case['rows'] * 16 + NPARAMS * 4, flops=case['rows'] * 2 * (64 * 256 + 256 * 256 + 512))
    n = 1 << case['qubits']
    return dict(bytes=16 * n, flops=6 * n * case['gates'])


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, from the Pauli labels
# ---------------------------------------------------------------------------------------------
def _masks(labels):
    """(x, z, number of Y) of Pauli labels, character 0 = highest qubit."""
    n = len(labels[0])
    ch = np.array(labels, dtype=f'<U{n}').view('<U1').reshape(len(labels), n)
    w = np.left_shift(np.int64(1), np.arange(n - 1, -1, -1, dtype=np.int64))
    x = np.where((ch == 'X') | (ch == 'Y'), w, 0).sum(axis=1)
    z = np.where((ch == 'Z') | (ch == 'Y'), w, 0).sum(axis=1)
    return x, z, (ch == 'Y').sum(axis=1)


def _sign(v):
    """(-1)^popcount(v), float64."""
    for k in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> k)
    return 1. - 2. * (v & 1).double()


def _elements(labels, coeffs, s):
    """(rows, cols, values) of the projected Hamiltonian, group by group of equal X masks."""
    x, z, ny = _masks(labels)
    c = np.asarray(coeffs, dtype=np.complex128) * np.array([1, -1j, -1, 1j])[ny % 4]
    order = np.argsort(x, kind='stable')
    start = np.flatnonzero(np.r_[True, np.diff(x[order]) != 0])
    for a, b in zip(start, np.r_[start[1:], len(order)]):
        t = s ^ int(x[order[a]])
        at = torch.searchsorted(s, t).clamp(max=s.numel() - 1)
        rows = torch.nonzero(s[at] == t).flatten()
        if not rows.numel():
            continue
        sr = s[rows]
        v = torch.zeros(rows.numel(), dtype=torch.complex128, device=s.device)
        for k in order[a:b]:
            v += _sign(sr & int(z[k])) * complex(c[k])
        yield rows, at[rows], v


def _apply(labels, coeffs, s, x):
    y = torch.zeros(s.numel(), dtype=torch.complex128, device=s.device)
    for rows, cols, v in _elements(labels, coeffs, s):
        y[rows] += v * x[cols]
    return y


def _ground(labels, coeffs, s, x0):
    """Ground pair of a real projected Hamiltonian: dense, or Lanczos with full orthogonalisation and
    restarts; the vector's sign as that of its overlap with x0."""
    r, c, v = (torch.cat(p) for p in zip(*_elements(labels, coeffs, s)))
    D = s.numel()
    h = torch.sparse_coo_tensor(torch.stack([r, c]), v.real, (D, D)).coalesce().to_sparse_csr()
    if D <= 2500:
        w, q = torch.linalg.eigh(h.to_dense())
        e, x = w[0], q[:, 0]
    else:
        x = x0 / torch.linalg.vector_norm(x0)
        for _ in range(12):
            q, al, be = [x], [], []
            for k in range(160):
                u = torch.mv(h, q[-1])
                al.append(torch.dot(u, q[-1]))
                basis = torch.stack(q)
                for _ in range(2):
                    u = u - basis.T @ (basis @ u)
                be.append(torch.linalg.vector_norm(u))
                if float(be[-1]) < 1e-13:
                    break
                q.append(u / be[-1])
            m = len(al)
            t = torch.diag(torch.stack(al))
            if m > 1:
                off = torch.stack(be[:m - 1])
                t = t + torch.diag(off, 1) + torch.diag(off, -1)
            w, p = torch.linalg.eigh(t.cpu())
            x = torch.stack(q[:m]).T @ p[:, 0].to(x.device)
            x = x / torch.linalg.vector_norm(x)
            e = torch.dot(x, torch.mv(h, x))
            if float(torch.linalg.vector_norm(torch.mv(h, x) - e * x)) < 1e-13 * max(1., abs(float(e))):
                break
    if float(torch.dot(x, x0)) < 0.:
        x = -x
    return float(e), x


def _gelu(z):
    return 0.5 * z * (1. + torch.tanh(math.sqrt(2. / math.pi) * (z + 0.044715 * z ** 3)))


def _network(p, x):
    w1, b1, w2, b2, w3, b3 = (v.to(x.device) for v in torch.split(p, [256 * 64, 256, 256 * 256, 256, 512, 2]))
    h = _gelu(x @ w1.view(256, 64).T + b1)
    h = _gelu(h @ w2.view(256, 256).T + b2)
    return h @ w3.view(2, 256).T + b3


def exact(case, seed):
    kind = case['kind']
    if kind == 'product':
        s = _states(case, seed)
        x = _vector(s.numel(), case['dtype'], seed).to(torch.complex128)
        y = _apply(*_labels(case, seed), s, x)
        return y if case['dtype'].startswith('complex') else y.real.contiguous()
    if kind == 'solve':
        s = _states(case, seed)
        e, x = _ground(*_labels(case, seed), s, _vector(s.numel(), 'float64', seed))
        return dict(energy=e, vector=x)
    if kind == 'sqd':
        words = torch.unique(_samples(case, seed))
        x0 = torch.zeros(words.numel(), dtype=torch.float64, device=DEV)
        x0[int(torch.argmin(_diagonal(*_labels(case, seed), words)))] = 1.
        e, x = _ground(*_labels(case, seed), words, x0)
        return dict(energy=e, vector=x.cpu().numpy(), basis=None)
    if kind == 'batch':
        parts = _batch_parts(case, seed)
        x = _vector(sum(p[3].numel() for p in parts), case['dtype'], seed).to(torch.complex128)
        xs = torch.split(x, [p[3].numel() for p in parts])
        return torch.cat([_apply(a, b, s, v) for (a, b, _, s), v in zip(parts, xs)])
    if kind == 'setup':
        samples = _samples(case, seed)
        words = torch.unique(samples)
        x = _vector(samples.numel(), 'float64', seed)[:words.numel()]
        return dict(states=None, diagonal=_diagonal(*_labels(case, seed), words),
                    product=_apply(*_labels(case, seed), words, x.to(torch.complex128)).real.contiguous())
    if kind == 'train':
        x, tgt = _train_inputs(case, seed)
        p = _net_params(seed).double().to(DEV).requires_grad_()
        out = _network(p, x.double())
        t = tgt.double()
        loss = (t[:, 2] * ((out[:, 0] - t[:, 0]) ** 2 + torch.nn.functional.softplus(-t[:, 1] * out[:, 1]))).mean()
        loss.backward()
        g = p.grad
        # the first Adam step from zero moments: m / (1 - b1) = g, v / (1 - b2) = g^2
        return dict(out=out.detach(), loss=loss.detach().reshape(1), grads=g, params=p.detach() - 1e-3 * g / (g.abs() + 1e-8))
    if kind == 'predict':
        s = _states(dict(model='hubbard', qubits=32, states='sector', rows=case['rows']), seed)
        u = torch.full((s.numel(),), 3. + (seed % 97) / 32., dtype=torch.float64, device=DEV)
        return _network(_net_params(seed).double(), _net_features(s, u))
    n = 1 << case['qubits']
    i = torch.arange(n, device=DEV)
    psi = torch.zeros(n, dtype=torch.complex128, device=DEV)
    psi[_circuit_start(case, seed)] = 1.
    for x, z, c, s in zip(*_circuit(case, seed)):
        psi = 1j * float(s) * _sign(i & int(z)) * psi[i ^ int(x)] + float(c) * psi
    return psi


def _diagonal(labels, coeffs, s):
    x, z, _ = _masks(labels)
    d = torch.zeros(s.numel(), dtype=torch.float64, device=DEV)
    for k in np.flatnonzero(x == 0):
        d += _sign(s & int(z[k])) * float(coeffs[k])
    return d
