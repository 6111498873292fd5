"""Pauli expectations from shared environments against the terms' dense
contraction, around the tile edges and on both sides of the rule that sends
small bonds to the walk over all sites; batches; shot marginals.

Bound: an expectation of a unit state is a chain of products of backward
stable factors of norm at most 1, 2 n contractions of up to 2 chi terms, so
its error is below 4 n chi eps; half a dozen such factors are allowed."""
import numpy as np
import pytest

import wqc_cuda as W
from wqc_cuda import circuits as C

pytestmark = pytest.mark.gpu

PAULI = {"I": np.eye(2), "X": np.array([[0, 1], [1, 0]]), "Y": np.array([[0, -1j], [1j, 0]]), "Z": np.diag([1, -1])}


def sites(n, chi, seed):
    rng = np.random.default_rng(seed)
    b = [min(2 ** min(i, n - i, 20), chi) for i in range(n + 1)]
    out = []
    for q in range(n):
        a = rng.standard_normal((2 * b[q + 1], b[q])) + 1j * rng.standard_normal((2 * b[q + 1], b[q]))
        out.append(np.linalg.qr(a)[0].conj().T.reshape(b[q], 2, b[q + 1]))
    return out


def value(tensors, label):
    n = len(tensors)
    env = np.ones((1, 1), dtype=complex)
    for q, t in enumerate(tensors):
        op = np.einsum("st,atb->asb", PAULI[label[n - 1 - q]], t)
        env = np.tensordot(np.tensordot(env, op, (0, 0)), t.conj(), ((0, 1), (0, 1)))
    return env[0, 0].real


def labels_of(n, seed):
    rng = np.random.default_rng(seed)
    out = ["I" * n, "X" * n, "Z" + "I" * (n - 1), "I" * (n - 1) + "Y"]
    for _ in range(6):
        lo = int(rng.integers(0, n))
        hi = int(rng.integers(lo, n)) + 1
        out.append("I" * lo + "".join(rng.choice(list("IXYZ"), hi - lo)) + "I" * (n - hi))
    return out


@pytest.mark.parametrize("n,chi", [(1, 1), (2, 2), (6, 3), (9, 15), (9, 16), (10, 17), (11, 24), (11, 25), (12, 33),
                                   (13, 48), (14, 64), (15, 127), (18, 200)])
def test_expectation_matches_dense_contraction(cuda_ctx, n, chi):
    tensors = sites(n, chi, 7 * n + chi)
    m = W.CudaMps(n, chi, ctx=cuda_ctx)
    for q, t in enumerate(tensors):
        m.set_site(q, t)
    labels = labels_of(n, n)
    tol = 24 * n * chi * np.finfo(float).eps
    for lab in labels:
        assert abs(m.expectation([lab], [1.0]) - value(tensors, lab)) <= tol
    coeffs = np.arange(1, len(labels) + 1) * (0.5 + 0.25j)
    want = sum(c * value(tensors, lab) for c, lab in zip(coeffs, labels))
    assert abs(m.expectation(labels, coeffs) - want) <= tol * np.abs(coeffs).sum()
    m.close()


@pytest.mark.parametrize("n,chis", [(6, [2, 3, 8]), (12, [40, 33, 7])])
def test_batch_expectation_matches_single_states(cuda_ctx, n, chis):
    gates = [C.gates_array(C.ry_rz_brickwork(n, 9, s)) for s in range(len(chis))]
    labels, coeffs = labels_of(n, 3), np.linspace(0.1, 1.0, 10)
    b = W.CudaBatch([n] * len(chis), chis, ctx=cuda_ctx)
    b.apply_slices(gates)
    got = b.expectations(labels, coeffs)
    for s, chi in enumerate(chis):
        m = W.run(n, chi, gates[s], ctx=cuda_ctx)
        tensors = [m.site(q) for q in range(n)]
        want = sum(c * value(tensors, lab) for c, lab in zip(coeffs, labels))
        # The slices' own splits differ from a single state's by rounding, 1e-10 at most.
        assert abs(got[s] - want) <= 1e-10 * np.abs(coeffs).sum()
        m.close()
    b.close()


@pytest.mark.parametrize("n,chis", [(12, [40, 8, 33, 24, 8]), (10, [3, 32, 16, 20])])
def test_a_slice_has_the_same_expectation_in_any_batch(cuda_ctx, n, chis):
    """Bit for bit: whether a slice's terms walk its sites or share chains is
    decided by its own bonds."""
    gates = [C.gates_array(C.ry_rz_brickwork(n, 9, s)) for s in range(len(chis))]
    labels, coeffs = labels_of(n, 3), np.linspace(0.1, 1.0, 10)

    def values(which):
        b = W.CudaBatch([n] * len(which), [chis[s] for s in which], ctx=cuda_ctx)
        b.apply_slices([gates[s] for s in which])
        out = [complex(x) for x in b.expectations(labels, coeffs)]
        b.close()
        return out

    together = values(range(len(chis)))
    assert together == [values([s])[0] for s in range(len(chis))]
    assert together[::-1] == values(range(len(chis))[::-1])


@pytest.mark.parametrize("n,chi", [(5, 4), (10, 17), (12, 40)])
def test_first_qubit_of_the_shots_follows_its_marginal(cuda_ctx, n, chi):
    tensors = sites(n, chi, n)
    m = W.CudaMps(n, chi, ctx=cuda_ctx)
    for q, t in enumerate(tensors):
        m.set_site(q, t)
    shots = 20000
    draws = m.sample(range(n), shots, 11)
    for q in (0, n // 2, n - 1):
        p1 = 0.5 * (1.0 - value(tensors, "I" * (n - 1 - q) + "Z" + "I" * q))
        ones = int(((draws >> np.uint64(q)) & np.uint64(1)).sum())
        assert abs(ones - shots * p1) <= 6 * np.sqrt(shots * max(p1 * (1 - p1), 1e-3))
    m.close()


@pytest.mark.parametrize("n,chi,cap", [(14, 64, 64), (12, 33, 256)])
@pytest.mark.parametrize("kib", [6000, 3600, 1200, 330])
def test_expectation_makes_do_with_less_memory(cuda_ctx, n, chi, cap, kib):
    """A device without room for the chains: fewer terms at a time (3600 KiB at
    bond 64), then the walk over all sites, at last of one term (256 KiB and the
    labels at bond 64).  No trace of the refused allocations is left."""
    tensors = sites(n, chi, 7 * n + chi)
    labels = labels_of(n, n)
    coeffs = np.linspace(1.0, 2.0, len(labels))
    want = sum(c * value(tensors, lab) for c, lab in zip(coeffs, labels))
    m = W.CudaMps(n, cap, ctx=cuda_ctx)
    for q, t in enumerate(tensors):
        m.set_site(q, t)
    before = W.last_oom()
    m.debug_limit_bytes(kib << 10)
    tol = 24 * n * chi * np.finfo(float).eps * coeffs.sum()
    assert abs(m.expectation(labels, coeffs) - want) <= tol
    assert W.last_oom() == before
    m.debug_limit_bytes(0)
    assert abs(m.expectation(labels, coeffs) - want) <= tol
    m.close()


def test_batch_expectation_makes_do_with_less_memory(cuda_ctx):
    """Slices on both sides of the walking rule, all walking one term at a time."""
    n, chis = 12, [40, 33, 7]
    b = W.CudaBatch([n] * len(chis), chis, ctx=cuda_ctx)
    b.apply_slices([C.gates_array(C.ry_rz_brickwork(n, 9, s)) for s in range(len(chis))])
    labels, coeffs = labels_of(n, 3), np.linspace(0.1, 1.0, 10)
    b.debug_limit_bytes(200 << 10)
    little = b.expectations(labels, coeffs)
    b.debug_limit_bytes(0)
    tol = 24 * n * 40 * np.finfo(float).eps * np.abs(coeffs).sum() * 2  # either value's bound; states of norm near 1
    assert np.abs(little - b.expectations(labels, coeffs)).max() <= tol
    b.close()


def test_a_read_that_finds_no_memory_is_refused_and_the_next_one_works(cuda_ctx):
    n, chi = 14, 64
    m = W.CudaMps(n, chi, ctx=cuda_ctx)
    for q, t in enumerate(sites(n, chi, 1)):
        m.set_site(q, t)
    m.debug_limit_bytes(64 << 10)
    for read in (lambda: m.expectation(["Z" * n], [1.0]), lambda: m.sample(range(n), 10, 1)):
        with pytest.raises(W.WqcCudaError) as e:
            read()
        assert e.value.code == W.ERR_OOM and e.value.required > e.value.available
    m.debug_limit_bytes(0)
    assert np.isfinite(m.expectation(["Z" * n], [1.0])) and len(m.sample(range(n), 10, 1)) == 10
    m.close()


def test_shots_need_room_for_the_bonds_not_for_the_capacity(cuda_ctx):
    """Right environments of bonds up to 32 take 60 KiB and their product's half
    32 KiB; at the capacity of 256 they would take 14 MiB."""
    n = 12
    tensors = sites(n, 32, 5)
    draws = []
    for cap, kib in ((256, 400), (256, 0), (64, 0)):
        m = W.CudaMps(n, cap, ctx=cuda_ctx)
        for q, t in enumerate(tensors):
            m.set_site(q, t)
        m.debug_limit_bytes(kib << 10)
        draws.append(m.sample(range(n), 500, 3).tolist())
        m.close()
    assert draws[0] == draws[1] == draws[2]


def free_bytes():
    import torch

    return torch.cuda.mem_get_info()[0]


def read_state(ctx, n, chi, terms):
    """A loaded state and a Pauli sum on it, with its value."""
    tensors = sites(n, chi, n + chi)
    m = W.CudaMps(n, chi, ctx=ctx)
    for q, t in enumerate(tensors):
        m.set_site(q, t)
    labels = (labels_of(n, n) * (terms // 10 + 1))[:terms]
    coeffs = np.full(terms, 1.0 / terms)
    want = sum(c * value(tensors, lab) for c, lab in zip(coeffs[:10], labels[:10])) * (terms / 10)
    return m, labels, coeffs, want


def test_reads_of_many_states_keep_one_pool(cuda_ctx):
    """What reads keep is bounded for the device, not for each state, and is
    given back with the states or when the free memory is asked for."""
    states = [read_state(cuda_ctx, 16, 128, 400) for _ in range(6)]
    cuda_ctx.device_info()  # nothing idle
    before = free_bytes()
    for m, labels, coeffs, want in states:
        assert abs(m.expectation(labels, coeffs) - want) <= 24 * 16 * 128 * np.finfo(float).eps
        m.sample(range(16), 10, 1)
    assert before - free_bytes() <= 512 << 20
    cuda_ctx.device_info()
    assert before - free_bytes() <= 4 << 20  # the allocator's granularity
    for m, *_ in states:
        m.close()


def test_a_state_that_needs_what_reads_keep_gets_it(cuda_ctx):
    import torch

    cuda_ctx.device_info()
    free0 = free_bytes()
    m, labels, coeffs, want = read_state(cuda_ctx, 16, 128, 400)
    cost = free0 - free_bytes()
    m.expectation(labels, coeffs)
    idle = free0 - cost - free_bytes()
    assert 64 << 20 <= idle <= 512 << 20
    ballast = torch.empty(free_bytes() - cost + idle // 2, dtype=torch.uint8, device="cuda")
    try:
        assert free_bytes() < cost
        other = W.CudaMps(16, 128, ctx=cuda_ctx)
        other.close()
        assert abs(m.expectation(labels, coeffs) - want) <= 24 * 16 * 128 * np.finfo(float).eps
    finally:
        del ballast
        torch.cuda.empty_cache()
    m.close()


def test_reads_of_several_threads_at_once(cuda_ctx):
    """Threads with a state each share the pool, a block to one call at a time."""
    import threading

    shapes = [(12, 40, 30), (14, 64, 50), (13, 33, 10), (12, 90, 20)]
    states = [read_state(cuda_ctx, *s) for s in shapes]
    wrong = []

    def work(k):
        m, labels, coeffs, want = states[k]
        n, chi, _ = shapes[k]
        shots = m.sample(range(n), 50, k).tolist()
        for _ in range(20):
            if abs(m.expectation(labels, coeffs) - want) > 24 * n * chi * np.finfo(float).eps:
                wrong.append(("value", k))
            if m.sample(range(n), 50, k).tolist() != shots:
                wrong.append(("shots", k))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(states))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for m, *_ in states:
        m.close()
