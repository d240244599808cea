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
    launches = gb.msm_graph_stats()[1]
    for _ in range(3):
        assert (affine_of(orc, ctx.msm(scal)) == want).all()
    assert gb.msm_graph_stats()[1] > launches
    held = _graph_bytes(gb)
    assert held > 0
    _demand_too_much(gb, orc)
    assert _graph_bytes(gb) < held
    assert (affine_of(orc, ctx.msm(scal)) == want).all()
    ctx.close()


@pytest.mark.parametrize("kind", ["context", "plain"])
def test_batches_without_room_for_the_affine_rounds(gb, orc, limit, kind):
    """3 x 2^16 points take 170 MB and more for their affine rounds and no other buffer
    of more than 40 MB: with less than that at hand they run without rounds."""
    rng = np.random.default_rng(3)
    n, count = 1 << 16, 3
    bases = gb.g1_generator_mul(orc.fr_random(n, rng))
    scal = orc.fr_random(n * count, rng).reshape(count, n, 4)
    want = [affine_of(orc, orc.g1_msm(bases, scal[i])) for i in range(count)]
    ctx = gb.Bls12_381G1MsmContext(bases)
    gb.msm_graphs_enable(False)
    try:
        for most in (0, 64 << 20, 0):
            limit(most)
            got = ctx.batch(scal) if kind == "context" else gb.bls12_381_g1_msm_batch(bases, scal)
            for i in range(count):
                assert (affine_of(orc, got[i]) == want[i]).all(), (most, i)
    finally:
        gb.msm_graphs_enable(True)
    limit(1 << 20)
    with pytest.raises(gb.MsmError) as e:
        ctx.batch(scal)
    assert e.value.code == OUT_OF_MEMORY
    limit(0)
    assert (affine_of(orc, ctx.batch(scal)[0]) == want[0]).all()
    ctx.close()


@pytest.mark.parametrize("count", [5000, 11500])
def test_batch_in_slices_and_groups(gb, orc, count):
    """5000 MSMs of 1024 points are 123 M digits, more than a slice of the
    affine rounds' list; 11500 are more than one group of a batch as well.  Their
    results come in order."""
    rng = np.random.default_rng(4)
    n = 1024
    bases = gb.g1_generator_mul(orc.fr_random(n, rng))
    dv = gb.fr_random_chacha20(bytes(range(32)), 0, n * count)[0]
    ctx = gb.Bls12_381G1MsmContext(bases)
    got = ctx.device_batch(dv, 0, n, count)
    scal = dv.download().reshape(count, n, 4)
    some = set(range(0, count, 500)) | set(range(4200, 5000, 40)) | {count - 1}
    if count > 10923:  # 2^28 digits
        some |= {10921, 10922, 10923, 10924}
    for i in sorted(some):
        assert (affine_of(orc, got[i]) == affine_of(orc, orc.g1_msm(bases, scal[i]))).all(), i
    ctx.close()
    dv.free()


def test_graph_without_room_for_its_scratch(gb, orc, limit):
    """A captured batch whose launch finds no memory runs launch by launch (and
    without rounds), and is captured again once there is room."""
    rng = np.random.default_rng(5)
    n, count = 1 << 16, 2
    bases = gb.g1_generator_mul(orc.fr_random(n, rng))
    scal = orc.fr_random(n * count, rng).reshape(count, n, 4)
    want = [affine_of(orc, orc.g1_msm(bases, scal[i])) for i in range(count)]
    ctx = gb.Bls12_381G1MsmContext(bases)

    def check():
        got = ctx.batch(scal)
        for i in range(count):
            assert (affine_of(orc, got[i]) == want[i]).all()

    def replayed(calls):
        before = gb.msm_graph_stats()[1]
        for _ in range(calls):
            check()
        return gb.msm_graph_stats()[1] - before

    assert replayed(3) >= 2
    limit(64 << 20)
    assert replayed(2) == 0
    limit(0)
    assert replayed(3) >= 1
    ctx.close()


def test_batches_with_much_scratch_are_not_captured(gb, orc):
    rng = np.random.default_rng(6)
    n, count = 1 << 18, 16
    ctx = gb.Bls12_381G1MsmContext(gb.g1_generator_mul(orc.fr_random(n, rng)))
    dv = gb.fr_random_chacha20(bytes(range(32)), 0, n * count)[0]
    stats = gb.msm_graph_stats()
    first = ctx.device_batch(dv, 0, n, count)
    for _ in range(2):
        assert (affine_of(orc, ctx.device_batch(dv, 0, n, count)) == affine_of(orc, first)).all()
    assert gb.msm_graph_stats() == stats
    for _ in range(3):
        ctx.device_batch(dv, 0, n, 1)
    assert gb.msm_graph_stats()[1] > stats[1]
    ctx.close()
    dv.free()


def test_grand_products_scratch(gb, orc):
    """12 chained sets over 2^18 rows take their result and little beside it."""
    rng = np.random.default_rng(7)
    n, m = 1 << 18, 12
    cols = gb.fr_random_chacha20(bytes(range(32)), 0, n * m)[0]
    perms = gb.fr_random_chacha20(bytes(range(1, 33)), 0, n * m)[0]
    beta, gamma = orc.fr_random(2, rng)
    deltas, blinds = orc.fr_random(m, rng), orc.fr_random(m, rng)
    rt, pool, v = _cudart(), ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0

    def products():
        out = gb.fr_permutation_products_device(cols, perms, n, m, 1, beta, gamma, orc.fr_omega(18), deltas, blinds, 1)
        out.download(1)
        out.free()

    products()
    assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(v)) == 0  # cudaMemPoolAttrUsedMemCurrent
    used = v.value
    assert rt.cudaMemPoolSetAttribute(pool, 8, ctypes.byref(ctypes.c_uint64(0))) == 0  # cudaMemPoolAttrUsedMemHigh
    products()
    assert rt.cudaMemPoolGetAttribute(pool, 8, ctypes.byref(v)) == 0
    assert v.value - used < 32 * n * m * 1.25
    cols.free()
    perms.free()


def _transformed(gb, log_n, count, inverse, most, limit, values):
    dv = gb.Bls12_381FrDeviceVec.upload(values["v"])
    limit(most)
    dv.ntt_zeta_batch(log_n, count, inverse, values["scale"], values["first"], values["one"])
    limit(0)
    out = dv.download()
    dv.free()
    return out


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("log_n,count,most", [(13, 64, 8 << 20),   # no room for the scratch copy (16 MB)
                                              (23, 1, 400 << 20)])  # for the tables (512 MB, copy 256)
def test_transforms_without_room_for_the_staged_passes(gb, orc, limit, log_n, count, most, inverse):
    """They run in place with the common twiddle table, output factors
    included; the first of 64 is checked against the oracle."""
    rng = np.random.default_rng(log_n)
    one, scale, first = orc.fr_const(orc.CONST_ONE), *orc.fr_random(2, rng)
    values = {"v": orc.fr_random(count << log_n, rng), "one": one, "scale": scale, "first": first}
    short = _transformed(gb, log_n, count, inverse, most, limit, values)
    assert (short == _transformed(gb, log_n, count, inverse, 0, limit, values)).all()
    if log_n == 13:
        want = orc.fr_ntt(values["v"][:1 << 13], 13, inverse)
        factors = np.array([orc.fr_mul(scale, f) for f in (one, first, one)])
        want = np.array([orc.fr_mul(w, factors[i % 3]) for i, w in enumerate(want)])
        assert (short[:1 << 13] == want).all()


def test_extension_without_room_for_the_tables(gb, orc, limit):
    """2^21 coefficients to 2^24 values: result and copy 512 MB, tables 1 GB."""
    src = gb.fr_random_chacha20(bytes(range(32)), 0, 1 << 21)[0]
    limit(700 << 20)
    short = gb.fr_device_coeff_to_extended_coset_batch(src, 1 << 21, 1, 24)
    limit(0)
    full = gb.fr_device_coeff_to_extended_coset_batch(src, 1 << 21, 1, 24)
    assert (short.download() == full.download()).all()
    for v in (src, short, full):
        v.free()


def test_ragged_transforms_without_room(gb, orc, limit):
    rng = np.random.default_rng(8)
    logs = [16, 3, 12, 10, 14, 1, 0]
    one, scale, first, second = orc.fr_const(orc.CONST_ONE), *orc.fr_random(3, rng)
    off = np.concatenate([[0], np.cumsum([1 << lg for lg in logs])[:-1]]).astype(np.uint64)
    v = orc.fr_random(sum(1 << lg for lg in logs), rng)
    got = []
    for most in (2 << 20, 0):  # the scratch copy is 2.8 MB
        dv = gb.Bls12_381FrDeviceVec.upload(v)
        limit(most)
        dv.ntt_ragged(off, logs, True, scale, first, second)
        limit(0)
        got.append(dv.download())
        dv.free()
    assert (got[0] == got[1]).all()
    for o, lg in zip(off.astype(int), logs):
        if lg:
            want = orc.fr_ntt(v[o:o + (1 << lg)], lg, True)
            factors = [scale, orc.fr_mul(scale, first), orc.fr_mul(scale, second)]
            for i in (0, 1, (1 << lg) // 2, (1 << lg) - 1):
                assert (got[1][o + i] == orc.fr_mul(want[i], factors[i % 3])).all()


def test_transform_without_room_builds_no_tables(gb, orc, limit):
    """Where the scratch copy (512 MB) has no room, the tables (256 MB), which
    would stay, are not built either."""
    import torch
    log_n, count = 22, 4
    one = orc.fr_const(orc.CONST_ONE)
    dv = gb.fr_random_chacha20(bytes(range(32)), 0, count << log_n)[0]
    dv.download(1)
    free = torch.cuda.mem_get_info()[0]
    limit(400 << 20)
    dv.ntt_zeta_batch(log_n, count, True, one, one, one)
    limit(0)
    dv.download(1)
    assert free - torch.cuda.mem_get_info()[0] < 200 << 20  # the common table is 64 MB
    dv.free()
