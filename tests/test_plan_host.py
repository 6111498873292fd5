"""The planner's SVD launches against the limits of their kernels, on the CPU.

A wave's cluster Jacobi tasks share a launch, so its threads are those of its
widest blocks and its instance that of its longest columns: the combination
has to fit, not each task by itself.  Brickwork circuits deep enough that every
bond stands at its bound, over the widths where the number of splits of a wave
changes the choice of cluster sizes."""
import ctypes

import numpy as np
import pytest

import wqc_cuda as W
from wqc_cuda import circuits as C

WAVE, KERNEL, TASKS, CLUSTER, THREADS, THREAD_LIMIT, SMEM, SMEM_LIMIT = range(8)


def launches(n, chi, precision, rule, slices=0, max_cluster=16, force=0, layers=None):
    layers = 2 * int(np.ceil(np.log2(chi))) + 2 if layers is None else layers
    gates = C.gates_array([C.g2(C.CZ, q, q + 1) for k in range(layers) for q in range(k % 2, n - 1, 2)])
    out, total = np.zeros((1 << 16, 8), np.int32), ctypes.c_uint32()
    rc = W.lib().wqc_debug_svd_launches(n, chi, slices, precision, rule, 148, max_cluster, force, gates.ctypes.data,
                                        len(gates), out.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), len(out),
                                        ctypes.byref(total))
    assert rc == W.OK and total.value <= len(out)
    return out[: total.value]


def check(rows, what):
    over = rows[(rows[:, THREADS] > rows[:, THREAD_LIMIT]) | (rows[:, SMEM] > rows[:, SMEM_LIMIT]) |
                (rows[:, CLUSTER] < 1)]
    assert len(over) == 0, f"{what}: {len(over)} launches do not fit, the first {over[0].tolist()}"


@pytest.mark.parametrize("precision", [W.PRECISION_FP64, W.PRECISION_FP32, W.PRECISION_TF32X3])
@pytest.mark.parametrize("rule", [W.SPLIT_RULE_REFERENCE, W.SPLIT_RULE_EXACT, -1])
@pytest.mark.parametrize("chi", [16, 48, 64, 96, 100, 128, 192, 256])
def test_every_launch_fits_its_kernel(precision, rule, chi):
    if rule == -1 and precision != W.PRECISION_FP64:
        pytest.skip("the adjoint takes the plain form only")
    for n in [*range(2, 20, 3), *range(20, 132), 160, 200, 255, 256]:
        check(launches(n, chi, precision, rule), f"{n} qubits")


@pytest.mark.parametrize("precision", [W.PRECISION_FP64, W.PRECISION_FP32])
@pytest.mark.parametrize("force", [1, 2, 4, 8, 16])
def test_every_launch_of_a_tuned_context_fits(precision, force):
    for n in (9, 14, 20, 57, 64):
        for chi in (20, 64, 100, 128, 200, 256):
            check(launches(n, chi, precision, W.SPLIT_RULE_EXACT, force=force), f"{n} qubits, chi {chi}")


@pytest.mark.parametrize("precision", [W.PRECISION_FP64, W.PRECISION_FP32])
@pytest.mark.parametrize("slices,max_cluster", [(1, 16), (6, 16), (6, 8), (0, 8)])
def test_every_launch_of_batches_and_smaller_clusters_fits(precision, slices, max_cluster):
    for n in (9, 20, 57, 64):
        for chi in (20, 64, 100, 128, 200, 256):
            check(launches(n, chi, precision, W.SPLIT_RULE_REFERENCE, slices, max_cluster), f"{n} qubits, chi {chi}")


def test_waves_that_already_fitted_keep_one_launch():
    """50 qubits at chi 128, where every combination fits as it is: a saturated
    wave's exact SVDs are one launch, its range finder's and fallbacks one each."""
    rows = launches(50, 128, W.PRECISION_FP64, W.SPLIT_RULE_REFERENCE)
    last = rows[rows[:, WAVE] == rows[:, WAVE].max()]
    assert len(last) == 3 and (last[:, KERNEL] == 0).all()
