"""One two-site split against numpy's SVD at the edges of the Jacobi and QR
kernels: block and panel remainders, row groups of 32, tall and wide theta,
rank below the bonds, and graded spectra, in both forms and both split rules'
exact path.

A split that truncates nothing gives L R = theta.  The bound on the relative
Frobenius error: the QR, the Jacobi and the recovery product are each backward
stable, with errors of at most about N eps of ||theta||; three of them and a
factor of two are 6 N eps, N = max(rows, cols).
"""
import numpy as np
import pytest

import wqc_cuda as W
from wqc_cuda import circuits as C

pytestmark = pytest.mark.gpu


def cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def split(ctx, dl, k, dr, grade, precision, seed):
    """Sites of bonds dl, k, dr through one CZ: (theta, L R, kept bond)."""
    rng = np.random.default_rng(seed)
    chi = max(dl, k, dr, min(2 * dl, 2 * dr, 256))
    d = np.exp(-np.linspace(0.0, grade, k))
    sites = [cplx(rng, 1, 2, dl), cplx(rng, dl, 2, k) * d, d[:, None, None] * cplx(rng, k, 2, dr), cplx(rng, dr, 2, 1)]
    m = W.CudaMps(4, chi, ctx=ctx, precision=precision)
    m.set_split_rule(W.SPLIT_RULE_EXACT)
    for q, t in enumerate(sites):
        m.set_site(q, t)
    m.apply_gates(C.gates_array([C.g2(C.CZ, 1, 2)]))
    theta = (sites[1].reshape(2 * dl, k) @ sites[2].reshape(k, 2 * dr)).reshape(dl, 2, 2, dr)
    theta[:, 1, 1] *= -1
    theta = theta.reshape(2 * dl, 2 * dr)
    left, right = m.site(1), m.site(2)
    kept = int(m.bond_dims()[1])
    m.close()
    return theta, left.reshape(2 * dl, kept) @ right.reshape(kept, 2 * dr), kept


# (dl, k, dr): rows 2 dl, cols 2 dr, rank min(2 dl, 2 dr, 2 k) after the CZ.
SHAPES = [
    (1, 1, 1), (1, 2, 5), (4, 4, 4), (7, 9, 7), (8, 8, 8), (9, 9, 9), (15, 15, 16), (16, 16, 16), (17, 20, 17),
    (31, 40, 31), (32, 32, 32), (33, 33, 33), (47, 50, 47), (48, 60, 49), (64, 64, 64), (65, 70, 65), (96, 100, 96),
    (97, 99, 98), (128, 128, 128),
    (128, 16, 8), (8, 16, 128), (100, 60, 31), (3, 4, 128),   # tall and wide
    (32, 5, 32), (64, 3, 64), (128, 10, 128), (50, 1, 50),    # rank below the bonds
]


@pytest.mark.parametrize("dl,k,dr", SHAPES)
@pytest.mark.parametrize("grade", [0.0, 8.0])
def test_split_keeps_theta(cuda_ctx, dl, k, dr, grade):
    theta, got, kept = split(cuda_ctx, dl, k, dr, grade, W.PRECISION_FP64, dl + k + dr)
    sv = np.linalg.svd(theta, compute_uv=False)
    assert kept == int((sv > 1e-12).sum())
    assert np.linalg.norm(got - theta) <= 6 * max(theta.shape) * np.finfo(float).eps * np.linalg.norm(theta)


# Columns past the cluster Jacobi's 384 rows (staged), groups of QR panels.
@pytest.mark.parametrize("dl,k,dr", [(129, 130, 129), (192, 200, 192), (193, 193, 193), (256, 256, 256),
                                     (256, 30, 100), (256, 20, 256)])
@pytest.mark.parametrize("precision", [W.PRECISION_FP64, W.PRECISION_FP32])
def test_large_split_keeps_the_leading_part(cuda_ctx, dl, k, dr, precision):
    theta, got, kept = split(cuda_ctx, dl, k, dr, 4.0, precision, dl + k + dr)
    u, sv, vh = np.linalg.svd(theta)
    assert kept == min(int((sv > 1e-12).sum()), 256)
    ref = (u[:, :kept] * sv[:kept]) @ vh[:kept]
    # A cut turns an error e of theta into e sigma_kept / gap of the kept part.
    gap = sv[kept - 1] - sv[kept] if kept < len(sv) and sv[kept] > 1e-12 else np.inf
    amplify = 1.0 + (sv[kept - 1] / gap if np.isfinite(gap) else 0.0)
    assert np.linalg.norm(got - ref) <= 6 * max(theta.shape) * np.finfo(float).eps * np.linalg.norm(theta) * amplify


@pytest.mark.parametrize("dl,k,dr", [(4, 4, 4), (9, 9, 9), (33, 33, 33), (65, 20, 64), (128, 128, 128)])
def test_split_keeps_theta_in_the_precision_form(cuda_ctx, dl, k, dr):
    theta, got, kept = split(cuda_ctx, dl, k, dr, 3.0, W.PRECISION_FP32, dl + k + dr)
    sv = np.linalg.svd(theta, compute_uv=False)
    assert kept == int((sv > 1e-12).sum())
    assert np.linalg.norm(got - theta) <= 6 * max(theta.shape) * np.finfo(float).eps * np.linalg.norm(theta)


def test_tasks_of_unlike_shapes_in_one_wave(cuda_ctx):
    """A wave's cluster tasks share a launch, each on its own cluster size; the
    result is that of every split on its own."""
    rng = np.random.default_rng(5)
    bonds = [1, 2, 90, 90, 3, 12, 12, 5, 30, 40, 2, 1]
    n, chi = len(bonds) - 1, 128
    sites = [cplx(rng, bonds[q], 2, bonds[q + 1]) for q in range(n)]

    def state():
        m = W.CudaMps(n, chi, ctx=cuda_ctx)
        m.set_split_rule(W.SPLIT_RULE_EXACT)
        for q, t in enumerate(sites):
            m.set_site(q, t)
        return m

    pairs = [1, 5, 8]  # disjoint; rows and cols 4 x 180, 24 x 10, 60 x 4
    together = state()
    together.apply_gates(C.gates_array([C.g2(C.CNOT, p, p + 1) for p in pairs]))
    for p in pairs:
        alone = state()
        alone.apply_gates(C.gates_array([C.g2(C.CNOT, p, p + 1)]))
        a = np.einsum("asg,gtb->astb", alone.site(p), alone.site(p + 1))
        b = np.einsum("asg,gtb->astb", together.site(p), together.site(p + 1))
        assert np.linalg.norm(a - b) <= 12 * 180 * np.finfo(float).eps * np.linalg.norm(a)
        alone.close()
    together.close()


@pytest.mark.parametrize("dl,k,dr", [(8, 16, 4), (16, 32, 16), (32, 50, 30), (64, 128, 64)])
@pytest.mark.parametrize("multiplicity", [2, 5])
def test_clusters_of_equal_singular_values(cuda_ctx, dl, k, dr, multiplicity):
    """Any small inner product turns a pair of equal columns by a large angle,
    so the iteration may not stop on the size of the inner products alone."""
    rng = np.random.default_rng(k + multiplicity)
    k = min(k, 2 * dl, 2 * dr)
    s = np.repeat(np.exp(-np.arange(-(-k // multiplicity)) / 3.0), multiplicity)[:k]
    u = np.linalg.qr(cplx(rng, 2 * dl, k))[0]
    v = np.linalg.qr(cplx(rng, 2 * dr, k))[0]
    theta = (u * s) @ v.conj().T
    m = W.CudaMps(4, 256, ctx=cuda_ctx)  # launch shapes of the upper bounds, far above the bonds
    m.set_split_rule(W.SPLIT_RULE_EXACT)
    for q, shape in enumerate([(1, 2, 100), (100, 2, 256), (256, 2, 100), (100, 2, 1)]):
        m.set_site(q, cplx(rng, *shape))
    sites = [cplx(rng, 1, 2, dl), (u * np.sqrt(s)).reshape(dl, 2, k), (np.sqrt(s)[:, None] * v.conj().T).reshape(k, 2, dr),
             cplx(rng, dr, 2, 1)]
    for q, t in enumerate(sites):
        m.set_site(q, t)
    m.apply_two_qubit_at_positions(1, 2, np.eye(4), True)
    kept = int(m.bond_dims()[1])
    assert kept == int((s > 1e-12).sum())
    left, right = m.site(1).reshape(2 * dl, kept), m.site(2).reshape(kept, 2 * dr)
    assert np.linalg.norm(left @ right - theta) <= 6 * 2 * max(dl, dr) * np.finfo(float).eps * np.linalg.norm(theta)
    # Both sides are U sqrt(S) and sqrt(S) V^H: their Gram matrices are S.
    for gram in (left.conj().T @ left, right @ right.conj().T):
        assert np.linalg.norm(gram - np.diag(np.diag(gram))) <= 6 * 2 * max(dl, dr) * np.finfo(float).eps * s[0] / s[kept - 1]
    m.close()


@pytest.mark.parametrize("precision", [W.PRECISION_FP64, W.PRECISION_FP32])
def test_wide_register_shares_launches_between_long_and_short_columns(cuda_ctx, precision):
    """64 qubits at chi 128: a saturated wave's 128-column tasks would like
    blocks of 16 columns beside the 256-column tasks' instance, which is compiled
    for 12 warps.  CZs commute, so the bonds stay 2 while their bounds, which
    the launches are shaped by, grow to 128.  Against the oracle: a split of the
    unit state errs by 6 N eps, N = 4, and there are fewer than layers n of them."""
    import oracle as O

    n, chi, layers = 64, 128, 18
    g = [C.g1(C.RY, q, 0.1 + 0.6 * np.sin(q) ** 2) for q in range(n)]
    for k in range(layers):
        g += [C.g2(C.CZ, q, q + 1) for q in range(k % 2, n - 1, 2)]
    gates = C.gates_array(g)
    m = W.CudaMps(n, chi, ctx=cuda_ctx, precision=precision)
    m.apply_gates(gates)
    ref = O.run(n, chi, gates)
    assert m.split_records()["chi"].tolist() == ref.records()["chi"].tolist()
    amp, want = m.amplitude_zero(), ref.amplitude_zero()
    assert abs(amp - want) <= layers * n * 24 * np.finfo(float).eps
    m.close()


@pytest.mark.parametrize("precision", [W.PRECISION_FP64, W.PRECISION_FP32])
def test_short_columns_beside_the_longest(cuda_ctx, precision):
    """Two splits of one wave, 26 columns and 256, and each on its own."""
    rng = np.random.default_rng(9)
    bonds = [1, 2, 13, 20, 13, 2, 4, 128, 128, 128, 4, 2, 1]
    n = len(bonds) - 1
    sites = [cplx(rng, bonds[q], 2, bonds[q + 1]) for q in range(n)]
    pairs = [2, 7]  # 26 x 26 and 256 x 256

    def state(gates):
        m = W.CudaMps(n, 128, ctx=cuda_ctx, precision=precision)
        m.set_split_rule(W.SPLIT_RULE_EXACT)
        for q, t in enumerate(sites):
            m.set_site(q, t)
        m.apply_gates(C.gates_array([C.g2(C.CNOT, p, p + 1) for p in gates]))
        return m

    together = state(pairs)
    for p in pairs:
        alone = state([p])
        a = np.einsum("asg,gtb->astb", alone.site(p), alone.site(p + 1))
        b = np.einsum("asg,gtb->astb", together.site(p), together.site(p + 1))
        assert a.shape == b.shape
        # A random 256 x 256 theta is cut to 128 values; neighbours of the cut
        # lie about sigma_1 / 256 apart, which amplifies each side's 6 N eps.
        assert np.linalg.norm(a - b) <= 12 * 256 * 256 * np.finfo(float).eps * np.linalg.norm(a)
        alone.close()
    together.close()
