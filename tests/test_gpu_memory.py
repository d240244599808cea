"""Calls that meet a full device: they fail with cudaErrorMemoryAllocation and
leave nothing behind, or do without the memory where there is another way.
The full device is a request beyond any device's memory, or the library's
allocation limit."""
import ctypes

import numpy as np
import pytest

from conftest import affine_of

pytestmark = pytest.mark.gpu

OUT_OF_MEMORY = 2  # cudaErrorMemoryAllocation


@pytest.fixture()
def limit(gb):
    yield gb.alloc_limit_set
    gb.alloc_limit_set(0)


def _cudart():
    """The CUDA runtime that libgbprover.so loaded (found in this process's maps)."""
    return ctypes.CDLL(next(ln.split()[-1] for ln in open("/proc/self/maps") if "libcudart.so" in ln))


def _graph_bytes(gb):
    """device memory that captured graphs hold, in use or idle"""
    v = ctypes.c_uint64()
    assert _cudart().cudaDeviceGetGraphMemAttribute(0, 2, ctypes.byref(v)) == 0  # cudaGraphMemAttrReservedMemCurrent
    return v.value


def _demand_too_much(gb, orc):
    """16 polynomials of 2^31 values: 1 TiB"""
    src = gb.Bls12_381FrDeviceVec.upload(orc.fr_random(256, np.random.default_rng(0)))
    with pytest.raises(gb.MsmError) as e:
        gb.fr_device_coeff_to_extended_coset_batch(src, 16, 16, 31)
    assert e.value.code == OUT_OF_MEMORY
    src.free()


def test_a_failed_allocation_does_not_fail_the_next_call(gb, orc):
    v = orc.fr_random(100, np.random.default_rng(1))
    _demand_too_much(gb, orc)
    assert (gb.bls12_381_fr_invert_assign(v) == orc.fr_batch_invert(v)).all()


def test_a_failed_allocation_takes_back_what_graphs_keep(gb, orc):
    rng = np.random.default_rng(2)
    n = 1 << 15
    bases = gb.g1_generator_mul(orc.fr_random(n, rng))
    scal = orc.fr_random(n, rng)
    ctx = gb.Bls12_381G1MsmContext(bases)
    want = affine_of(orc, orc.g1_msm(bases, scal))
    captures = gb.msm_graph_stats()[0]
    for _ in range(3):
        assert (affine_of(orc, ctx.msm(scal)) == want).all()
    assert gb.msm_graph_stats()[0] > captures
    held = _graph_bytes(gb)
    assert held > 0
    _demand_too_much(gb, orc)
    assert _graph_bytes(gb) < held
    assert (affine_of(orc, ctx.msm(scal)) == want).all()
    ctx.close()
