"""The persistent LOBPCG kernel against the CUDA-graph loop of the same iteration, where its layout
changes: one block and many, one to 32 lanes per row, lists that fit in shared memory and not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def built():
    from rqutils_gb300._build import build
    build()


def _operator(name, D, cache_level, real):
    from rqutils_gb300 import workloads
    from rqutils_gb300.paulis.symplectic import PauliSumXZ
    from rqutils_gb300.sqd import SQDProblem
    rng = np.random.default_rng(D)
    if name == 'hubbard':
        labels, coeffs = workloads.hubbard_jw(4, 4, 1.0, 4.0, True)
        S = workloads.low_double_occupancy_states(rng, D)
    else:  # 'dense': most of a small space, long rows
        n = int(np.ceil(np.log2(D)))
        labels, coeffs = workloads.random_pauli_masks(rng, n, 400, locality=(1, n))
        S = np.sort(rng.choice(1 << n, size=D, replace=False)).astype(np.uint64)
        if real:
            labels = [s if s.count('Y') % 2 == 0 else s.replace('Y', 'X') for s in labels]
    ham = PauliSumXZ.from_paulisum((labels, coeffs), force_real=True, add_padding=True)
    return SQDProblem(ham, S, cache_level=cache_level).op


@pytest.mark.parametrize('name,D,cache_level,real', [
    ('dense', 5, (1, 0), True),           # one block, more lanes than rows
    ('dense', 700, (1, 0), False),        # a few blocks, 32 lanes per row
    ('dense', 700, (1, 2), True),
    ('dense', 8192, (1, 0), False),       # 21,000 elements per block: past the shared memory
    ('hubbard', 9001, (1, 0), True),      # several lanes per row
    ('hubbard', 120001, (1, 2), True),    # one lane per row
])
@pytest.mark.parametrize('variant', ['fast', 'reference'])
def test_persistent_kernel_equals_graph_loop(name, D, cache_level, real, variant):
    import torch
    from rqutils_gb300.ground_locg import lobpcg_solve
    op = _operator(name, D, cache_level, real)
    dt = torch.float64 if op.is_real else torch.complex128
    x0 = torch.randn(D, dtype=dt, device='cuda', generator=torch.Generator('cuda').manual_seed(D))
    kw = dict(variant=variant, target_rel=1e-9, tol=1e-300, maxiter=600)
    e1, x1, i1 = lobpcg_solve(op, x0, use_graph=1, **kw)
    e2, x2, i2 = lobpcg_solve(op, x0, use_graph=2, **kw)
    assert i1['converged'] == i2['converged']
    # the same iteration up to the rounding of its reductions, as for the golden cases
    assert abs(i1['niter'] - i2['niter']) <= 1, (i1, i2)
    assert abs(e1 - e2) <= 1e-12 * max(1., abs(e2))
    if i1['converged']:
        assert abs(torch.vdot(x1, x2).item()) > 1 - 1e-10
    r = torch.linalg.vector_norm(op.matvec(x1) - e1 * x1)
    if i1['converged']:
        assert r <= 1.01e-9 * abs(e1)


@pytest.mark.parametrize('variant', ['fast', 'reference'])
def test_threads_with_different_sizes(variant):
    """A thread's large solve and products run after another thread's small ones (the runtime keeps one
    shared-memory limit per kernel for all threads): large, small on a second thread, large again."""
    import threading
    import torch
    from rqutils_gb300.ground_locg import lobpcg_solve
    from rqutils_gb300 import workloads
    from rqutils_gb300.device import DeviceOperator, DeviceSubspace, DeviceTerms
    from rqutils_gb300.paulis.symplectic import PauliSumXZ
    large, small = _operator('dense', 8192, (1, 0), False), _operator('dense', 40, (1, 0), False)
    rng = np.random.default_rng(1)
    many, few = (PauliSumXZ.from_paulisum(workloads.random_pauli_masks(rng, 16, k, locality=(1, 16)), force_real=True,
                                          add_padding=True) for k in (6000, 2500))  # both above 2,048 X groups
    S = np.sort(rng.choice(1 << 16, size=500, replace=False)).astype(np.uint64)
    free = [DeviceOperator(DeviceTerms(h), DeviceSubspace(S, num_qubits=16), mode='free') for h in (many, few)]

    def run(op, free_op):
        dt = torch.float64 if op.is_real else torch.complex128
        x0 = torch.randn(op.D, dtype=dt, device='cuda', generator=torch.Generator('cuda').manual_seed(op.D))
        x = torch.ones(500, dtype=torch.complex128, device='cuda')
        return lobpcg_solve(op, x0, variant=variant, maxiter=20)[0], free_op.matvec(x)

    first = run(large, free[0])
    other = []
    t = threading.Thread(target=lambda: other.append(run(small, free[1])))
    t.start()
    t.join()
    assert other
    again = run(large, free[0])
    assert again[0] == first[0] and torch.equal(again[1], first[1])
