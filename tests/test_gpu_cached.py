"""The tiled cached products (CONN, CSR): the same additions in the same order as the matrix-free
product, so the same bits, at the edges of the tiles (rows per block, products per pass)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def built():
    from rqutils_gb300._build import build
    build()


def _operators(n, K, D, real, seed):
    from rqutils_gb300 import workloads
    from rqutils_gb300.paulis.symplectic import PauliSumXZ
    from rqutils_gb300.sqd import SQDProblem
    rng = np.random.default_rng(seed)
    labels, coeffs = workloads.random_pauli_masks(rng, n, K, locality=(1, n))
    if real:  # an even number of Y per term
        labels = [s if s.count('Y') % 2 == 0 else s.replace('Y', 'X') for s in labels]
    ham = PauliSumXZ.from_paulisum((labels, coeffs), force_real=True, add_padding=True)
    S = np.sort(rng.choice(1 << n, size=D, replace=False)).astype(np.uint64)
    return [SQDProblem(ham, S, cache_level=c).op for c in ((0, 0), (1, 0), (1, 2))]


# D around the tile heights (16 to 256 rows), row lists from empty (sparse subspace) to several
# passes over the product buffer (a 10-qubit space with 900 groups: ~900 elements per row)
@pytest.mark.parametrize('n,K,D', [(1, 2, 1), (3, 5, 7), (10, 1500, 1024), (12, 200, 15), (12, 200, 17),
                                   (14, 300, 4863), (14, 300, 4864), (14, 300, 4865), (30, 60, 5000),
                                   (18, 400, 200001)])
@pytest.mark.parametrize('dtype', ['float32', 'float64', 'complex64', 'complex128'])
def test_cached_products_equal_matrix_free_bits(n, K, D, dtype):
    import torch
    free, conn, csr = _operators(n, K, D, dtype.startswith('float'), 100 * n + D % 97)
    x = torch.randn(D, dtype=getattr(torch, dtype), device='cuda', generator=torch.Generator('cuda').manual_seed(D))
    y = free.matvec(x)
    assert torch.equal(conn.matvec(x), y)
    # cached elements are computed in 64 bits; a 32-bit vector rounds them after their sum
    z = csr.matvec(x)
    if dtype in ('float64', 'complex128'):
        assert torch.equal(z, y)
    else:
        ref = csr.matvec(x.to(torch.float64 if dtype == 'float32' else torch.complex128))
        assert torch.linalg.vector_norm(z - ref) <= 1e-6 * torch.linalg.vector_norm(ref)


@pytest.mark.parametrize('mode', [1, 2])
def test_cached_products_keep_infinities_and_nan(mode):
    """Non-finite entries reach the rows connected to them and no others."""
    import torch
    ops = _operators(12, 80, 700, True, 5)
    x = torch.randn(700, dtype=torch.float64, device='cuda', generator=torch.Generator('cuda').manual_seed(1))
    x[3], x[10] = float('inf'), float('nan')
    y, z = ops[0].matvec(x), ops[mode].matvec(x)
    assert torch.equal(torch.isfinite(y), torch.isfinite(z))
    ok = torch.isfinite(y)
    assert torch.equal(y[ok], z[ok])


def _clustered_states(rng, n, D):
    """D states of two half-filled n / 2-bit blocks, few excitations above the lowest orbitals."""
    half, have = n // 2, np.zeros(0, np.uint64)
    while len(have) < D:
        words = np.zeros(2 * D, np.uint64)
        for block in range(2):
            w = np.full(2 * D, (1 << (half // 2)) - 1, np.uint64)
            for _ in range(3):  # up to three excitations, each with probability 1/2
                a, b = rng.integers(0, half // 2, 2 * D), rng.integers(half // 2, half, 2 * D)
                m = (np.uint64(1) << a.astype(np.uint64)) | (np.uint64(1) << b.astype(np.uint64))
                ok = (rng.random(2 * D) < 0.5) & (((w >> a.astype(np.uint64)) & np.uint64(1)) == 1) & \
                    (((w >> b.astype(np.uint64)) & np.uint64(1)) == 0)
                w = np.where(ok, w ^ m, w)
            words |= w << np.uint64(block * half)
        have = np.unique(np.concatenate([have, words]))
    return np.sort(rng.choice(have, size=D, replace=False))


# one to 32 lanes per row, 32- and 64-bit keys, more hits between two resolutions than the queue
# holds, and (36 qubits) the clustered launch: several passes, the sector test, spread tiles
@pytest.mark.parametrize('n,keep,D', [(20, 3000, 100), (20, 3000, 2500), (28, 4000, 30001), (36, 6000, 60000)])
@pytest.mark.parametrize('dtype', ['float32', 'float64', 'complex64', 'complex128'])
def test_clustered_subspaces(n, keep, D, dtype):
    import torch
    from rqutils_gb300 import workloads
    from rqutils_gb300.device import DeviceOperator, DeviceSubspace, DeviceTerms
    from rqutils_gb300.paulis.symplectic import PauliSumXZ
    rng = np.random.default_rng(n)
    ham = PauliSumXZ.from_paulisum(workloads.chemistry_jw(n // 2, rng, keep=keep), force_real=True,
                                   add_padding=True)
    S = _clustered_states(rng, n, D)
    terms = DeviceTerms(ham)
    x = torch.randn(D, dtype=getattr(torch, dtype), device='cuda', generator=torch.Generator('cuda').manual_seed(D))
    y = DeviceOperator(terms, DeviceSubspace(S, num_qubits=n, line_filter=False), mode='free').matvec(x)
    for masks in (None, (0, 0), ((1 << n // 4) - 1, ((1 << n) - 1) ^ ((1 << n // 4) - 1))):
        sub = DeviceSubspace(S, num_qubits=n, filter_masks=masks)
        assert torch.equal(DeviceOperator(terms, sub, mode='free').matvec(x), y)
    conn = DeviceOperator(terms, sub, mode='conn')
    assert conn.nnz >= 2 * D  # 3 to 40 a row
    assert torch.equal(conn.matvec(x), y)


@pytest.mark.parametrize('first', [True, False])
@pytest.mark.parametrize('D', [1100, 1983, 1984, 1985, 2047, 2048, 2049, 4097])
@pytest.mark.parametrize('dtype', ['float64', 'complex64', 'complex128'])
def test_short_rows_equal_matrix_free_bits(D, first, dtype):
    """Fewer elements than rows, at the edges of a warp's 64 rows and a block's 512: 32 rows of up to 32
    elements (several times 32 for one warp, at either end of the array) among empty ones."""
    import torch
    from rqutils_gb300 import workloads
    from rqutils_gb300.paulis.symplectic import PauliSumXZ
    from rqutils_gb300.sqd import SQDProblem
    rng = np.random.default_rng(D)
    labels, coeffs = workloads.random_pauli_masks(rng, 5, 150, locality=(1, 5))
    if dtype == 'float64':
        labels = [s if s.count('Y') % 2 == 0 else s.replace('Y', 'X') for s in labels]
    labels = ['IZ' + 'I' * 17 + s for s in labels]
    ham = PauliSumXZ.from_paulisum((labels, coeffs), force_real=True, add_padding=True)
    group = np.arange(32) + (0 if first else 1 << 23)
    # spread states differ from each other and from the group above the bits that the terms flip
    spread = (rng.choice(np.arange(1, 1 << 18), size=D - 32, replace=False) << 5) + rng.integers(0, 32, D - 32)
    S = np.sort(np.concatenate([group, spread])).astype(np.uint64)
    free, conn, csr = [SQDProblem(ham, S, cache_level=c).op for c in ((0, 0), (1, 0), (1, 2))]
    assert 32 * 16 < conn.c.nnz < D
    x = torch.randn(D, dtype=getattr(torch, dtype), device='cuda', generator=torch.Generator('cuda').manual_seed(D))
    y = free.matvec(x)
    assert torch.equal(conn.matvec(x), y)
    if dtype != 'complex64':
        assert torch.equal(csr.matvec(x), y)
    else:
        ref = csr.matvec(x.to(torch.complex128))
        assert torch.linalg.vector_norm(csr.matvec(x) - ref) <= 1e-6 * torch.linalg.vector_norm(ref)


def test_binary_search_lists_do_not_read_a_line_filter():
    """The C interface takes a binary-search subspace whose lmap is set: rq_subspace_build leaves it
    unfilled and there are no hash arrays, so the lists come from the states alone."""
    import torch
    from rqutils_gb300 import _lib as L
    from rqutils_gb300 import workloads
    from rqutils_gb300.device import DeviceOperator, DeviceSubspace, DeviceTerms
    from rqutils_gb300.paulis.symplectic import PauliSumXZ
    rng = np.random.default_rng(3)
    ham = PauliSumXZ.from_paulisum(workloads.random_pauli_masks(rng, 12, 80), force_real=True, add_padding=True)
    S = np.sort(rng.choice(1 << 12, size=700, replace=False)).astype(np.uint64)
    terms = DeviceTerms(ham)
    sub = DeviceSubspace(S, num_qubits=12, lookup='bsearch')
    lmap = torch.zeros(1 << 12, dtype=torch.int32, device='cuda')
    sub.c.lmap, sub.c.lbits, sub.c.lwbits, sub.c.lshift = L.ptr(lmap), 9, 8, 2
    for mode in ('conn', 'csr'):
        got = DeviceOperator(terms, sub, mode=mode)
        ref = DeviceOperator(terms, DeviceSubspace(S, num_qubits=12), mode=mode)
        assert ref.nnz > 0
        for a, b in zip(got.connectivity(), ref.connectivity()):
            assert np.array_equal(a, b)
        if mode == 'csr':
            assert torch.equal(got.val, ref.val)


# rows shorter than one element, tiles of average rows, several passes over the product buffer
@pytest.mark.parametrize('n,K,D', [(18, 200, 700), (16, 200, 700), (12, 300, 1500), (10, 1500, 300)])
def test_real_products_are_not_rounded_before_the_sum(n, K, D):
    """Real products: each element's product enters its row's sum exactly.  In 64 bits that is a fused
    multiply-add per element in list order, bit for bit; in 32 bits the error of a row of m elements stays
    within its own rounding plus what compensated sums leave, 2 m (m + 2) 2^-48 of the summed magnitudes
    (a rounded product alone leaves 2^-25 of itself)."""
    import torch
    from fractions import Fraction
    ops = _operators(n, K, D, True, 7 * n)
    x = torch.randn(D, dtype=torch.float64, device='cuda', generator=torch.Generator('cuda').manual_seed(D))
    rowptr, col, _ = ops[2].connectivity()
    val, diag = ops[2].val.cpu().numpy(), ops[2].diag0.cpu().numpy() if ops[2].diag0 is not None else np.zeros(D)
    assert (rowptr[-1] < D) == (n == 18)
    xh = x.cpu().numpy()
    y = np.zeros(D)
    for i in range(D):
        s = Fraction(float(diag[i])) * Fraction(float(xh[i]))
        for e in range(rowptr[i], rowptr[i + 1]):
            s = Fraction(float(s)) + Fraction(float(val[e])) * Fraction(float(xh[col[e]]))
        y[i] = float(s)
    for op in ops:
        assert np.array_equal(op.matvec(x).cpu().numpy(), y)
    x32 = x.float()
    v32, d32, xf = val.astype(np.float32).astype(float), diag.astype(np.float32).astype(float), x32.cpu().numpy().astype(float)
    got = ops[2].matvec(x32).cpu().numpy().astype(float)
    for i in range(D):
        p = np.append(v32[rowptr[i]:rowptr[i + 1]] * xf[col[rowptr[i]:rowptr[i + 1]]], d32[i] * xf[i])
        exact = float(sum(map(Fraction, p)))  # (products of 24-bit factors are exact in 64 bits)
        m = len(p)
        assert abs(got[i] - exact) <= 2. ** -23 * abs(exact) + 2 * m * (m + 2) * 2. ** -48 * np.abs(p).sum(), i


# one row more than the queue's resident rows and fewer, most of a space and all of it; groups around the
# 64 that a lane probes between two resolutions
@pytest.mark.parametrize('D', [155648, 155649, 262144])
@pytest.mark.parametrize('groups', [63, 64, 65, 129])
@pytest.mark.parametrize('dtype', ['float32', 'complex64'])
def test_dense_subspaces_equal_bits(D, groups, dtype):
    """Dense subspaces, whose lanes resolve their own hits, against the product without a line filter."""
    import torch
    from rqutils_gb300.device import DeviceOperator, DeviceSubspace, DeviceTerms
    from rqutils_gb300.paulis.symplectic import PauliSumXZ
    rng = np.random.default_rng(groups)
    masks = rng.choice(np.arange(1, 1 << 18), size=groups, replace=False)
    labels, coeffs = ['I' * 18, 'Z' * 18], [0.3, 0.7]
    for m in masks:
        x = ''.join('X' if m >> (17 - k) & 1 else 'I' for k in range(18))
        z = ''.join('Z' if c == 'I' and rng.random() < 0.5 else c for c in x)
        labels += [x, z] if x != z else [x]
        coeffs += list(rng.normal(size=2 if x != z else 1))
    if dtype == 'complex64':  # an odd number of Y: a term with an imaginary part
        labels = [s.replace('X', 'Y', 1) if k % 3 == 2 else s for k, s in enumerate(labels)]
    ham = PauliSumXZ.from_paulisum((labels, np.array(coeffs)), force_real=True, add_padding=True)
    S = np.sort(rng.choice(1 << 18, size=D, replace=False)).astype(np.uint64)
    terms, sub = DeviceTerms(ham), DeviceSubspace(S, num_qubits=18)
    assert terms.J == groups + 1 and sub.c.lshift <= 7
    x = torch.randn(D, dtype=getattr(torch, dtype), device='cuda', generator=torch.Generator('cuda').manual_seed(D))
    y = DeviceOperator(terms, DeviceSubspace(S, num_qubits=18, line_filter=False), mode='free').matvec(x)
    op = DeviceOperator(terms, sub, mode='free')
    assert torch.equal(op.matvec(x), y)
    op.check_errors()
