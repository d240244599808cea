"""KZG opening helpers on the GPU through the C ABI, bit-exact against the
oracle's eval_polynomial and kate_division (arithmetic.rs:53-116)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ln,count", [(1, 1), (7, 3), (2048, 2), (8193, 1), (1 << 16, 4)])
def test_eval_polys(gb, orc, ln, count):
    rng = np.random.default_rng(ln + count)
    polys = orc.fr_random(ln * count, rng)
    z = orc.fr_random(1, rng)[0]
    dv = gb.Bls12_381FrDeviceVec.upload(polys)
    got = gb.bls12_381_fr_device_eval_polys(dv, ln, count, z)
    for p in range(count):
        assert (got[p] == orc.fr_eval_poly(polys[p * ln:(p + 1) * ln], z)).all()
    dv.free()


def test_eval_polys_shape_errors(gb, orc):
    dv = gb.Bls12_381FrDeviceVec.upload(orc.fr_random(10, np.random.default_rng(0)))
    z = orc.fr_from_ints([3])[0]
    with pytest.raises(gb.MsmError):
        gb.bls12_381_fr_device_eval_polys(dv, 3, 3, z)
    with pytest.raises(gb.MsmError):
        gb.bls12_381_fr_device_eval_polys(dv, 0, 1, z)
    dv.free()


@pytest.mark.parametrize("ln,count,zero", [(2, 1, False), (100, 3, False), (4097, 2, False),
                                           (1 << 17, 1, False), (300, 2, True)])
def test_kate_divide(gb, orc, ln, count, zero):
    rng = np.random.default_rng(ln * 3 + count)
    polys = orc.fr_random(ln * count, rng)
    z = orc.fr_from_ints([0])[0] if zero else orc.fr_random(1, rng)[0]
    dv = gb.Bls12_381FrDeviceVec.upload(polys)
    q = gb.fr_device_kate_divide(dv, ln, count, z)
    got = q.download().reshape(count, ln, 4)
    for p in range(count):
        want = orc.fr_kate_division(polys[p * ln:(p + 1) * ln], z)
        assert (got[p, :ln - 1] == want).all()
        assert (got[p, ln - 1] == 0).all()
    q.free()
    dv.free()


@pytest.mark.parametrize("pre_words,n", [(0, 5000), (6, 4096), (8, 1 << 16), (14, 12345)])
def test_device_random_draw_matches_host(gb, pre_words, n):
    """gb_fr_random_chacha20 gives the values fr_random would draw from the
    same rng state, and the host rng ends at the same word."""
    from gb_prover.rng import ChaCha20Rng, fr_random
    a, b = ChaCha20Rng.from_label("draw"), ChaCha20Rng.from_label("draw")
    a._words(pre_words)
    b._words(pre_words)
    want = fr_random(a, n)
    vec, used = gb.fr_random_chacha20(b.seed, b.word_position(), n)
    b.skip_words(used)
    assert (vec.download() == want).all()
    assert a.word_position() == b.word_position()
    vec.free()


def test_eval_many_matches_single_evaluations(gb, orc):
    """gb_fr_device_eval_many over requests of different vectors, counts and
    points equals one evaluation call per request (itself pinned to the
    oracle in this file)."""
    import numpy as np
    rng = np.random.default_rng(91)
    n = 1 << 12
    vecs = [gb.Bls12_381FrDeviceVec.upload(orc.fr_random(c * n, rng)) for c in (3, 1, 5)]
    pts = orc.fr_random(6, rng)
    reqs = [(vecs[0], 3, pts[0]), (vecs[1], 1, pts[1]), (vecs[2], 5, pts[2]), (vecs[0], 3, pts[3]),
            (vecs[2], 5, pts[4]), (vecs[1], 1, orc.fr_from_ints([0])[0])]
    got = gb.fr_device_eval_many(reqs, n)
    for (v, c, p), g in zip(reqs, got):
        assert (g == gb.bls12_381_fr_device_eval_polys(v, n, c, p)).all()
    want0 = orc.fr_eval_poly(vecs[1].download()[:n], pts[1])
    assert (got[1][0] == want0).all()


@pytest.mark.parametrize("ln,count", [(1, 2), (2, 1), (255, 1), (256, 3), (257, 2), (513, 1), (1 << 14, 1),
                                      ((1 << 14) + 1, 1), (1 << 17, 1), ((1 << 17) + 1, 1), (3 << 16, 1),
                                      ((3 << 16) + 1, 1), (1 << 19, 1), ((1 << 19) + 1, 1), ((1 << 20) + 2049, 1)])
@pytest.mark.parametrize("point", ["random", "zero", "one"])
def test_kate_divide_tile_edges(gb, orc, ln, count, point):
    """Around the block's scan (256), the changes of coefficients a thread (2^14
    and 3 * 2^16 in all) and the carry pass (above 256 tiles of 512 and 2048)."""
    rng = np.random.default_rng(ln + count)
    polys = orc.fr_random(ln * count, rng)
    z = orc.fr_random(1, rng)[0] if point == "random" else orc.fr_from_ints([int(point == "one")])[0]
    dv = gb.Bls12_381FrDeviceVec.upload(polys)
    q = gb.fr_device_kate_divide(dv, ln, count, z)
    got = q.download().reshape(count, ln, 4)
    for p in range(count):
        if ln > 1:
            assert (got[p, :ln - 1] == orc.fr_kate_division(polys[p * ln:(p + 1) * ln], z)).all()
        assert (got[p, ln - 1] == 0).all()
    q.free()
    dv.free()


@pytest.mark.parametrize("ln,requests", [(1, 1), (255, 2), (256, 1), (257, 1), (4096, 3), (4097, 3),
                                         ((1 << 20) + 5, 1), ((1 << 14) + 1, 608), ((1 << 14) - 1, 608)])
def test_eval_many_slice_edges(gb, orc, ln, requests):
    """Around a slice of 4096, with more than one level of slices, and with
    slices of 16384 (many requests)."""
    rng = np.random.default_rng(ln + requests)
    coeffs = orc.fr_random(ln, rng)
    points = orc.fr_random(requests, rng)
    dv = gb.Bls12_381FrDeviceVec.upload(coeffs)
    got = gb.fr_device_eval_many([(dv, 1, z) for z in points], ln)
    for r in range(0, requests, 101):
        assert (got[r][0] == orc.fr_eval_poly(coeffs, points[r])).all()
    dv.free()


@pytest.mark.parametrize("ln,count", [(1, 1), (1, 700), (31, 3), (32, 40), (33, 40), (127, 2), (512, 3), (512, 70000),
                                      (513, 3), (513, 455), (513, 456), (4096, 456), (4097, 304), (4097, 455),
                                      (4097, 1000), (6145, 1000), (8193, 304), (16385, 304), (16384, 303)])
def test_eval_polys_forms(gb, orc, ln, count):
    """Polynomials by a warp and by 256 threads each, with 16, 32 and 64
    coefficients a thread, one slice and several, in one call and at one point."""
    rng = np.random.default_rng(ln + count)
    dv = gb.fr_random_chacha20(bytes(range(32)), 0, ln * count)[0]
    z = orc.fr_random(1, rng)[0]
    got = gb.bls12_381_fr_device_eval_polys(dv, ln, count, z)
    some = sorted({0, count // 2, count - 1} | set(range(0, count, max(1, count // 5))))
    host = dv.download().reshape(count, ln, 4)
    for p in some:
        assert (got[p] == orc.fr_eval_poly(host[p], z)).all(), p
    dv.free()


def test_eval_many_short_at_many_points(gb, orc):
    """A warp a polynomial with the powers made there (many points) and with
    the points' powers given (few points, many polynomials each)."""
    rng = np.random.default_rng(8)
    for ln, requests, count in ((40, 300, 1), (40, 3, 100), (700, 500, 1), (700, 2, 300)):
        coeffs, points = orc.fr_random(ln * count, rng), orc.fr_random(requests, rng)
        dv = gb.Bls12_381FrDeviceVec.upload(coeffs)
        got = gb.fr_device_eval_many([(dv, count, z) for z in points], ln)
        for r in range(0, requests, max(1, requests // 7)):
            for p in range(0, count, max(1, count // 5)):
                assert (got[r][p] == orc.fr_eval_poly(coeffs[p * ln:(p + 1) * ln], points[r])).all(), (r, p)
        dv.free()


def test_kate_divide_by_x_is_a_copy(gb, orc):
    """Point zero: one launch, whatever the length."""
    ln, count = 5000, 3
    polys = orc.fr_random(ln * count, np.random.default_rng(9))
    dv = gb.Bls12_381FrDeviceVec.upload(polys)
    before = gb.launch_counter()
    q = gb.fr_device_kate_divide(dv, ln, count, np.zeros(4, dtype=np.uint64))
    assert gb.launch_counter() == before + 1
    got, polys = q.download().reshape(count, ln, 4), polys.reshape(count, ln, 4)
    assert (got[:, :-1] == polys[:, 1:]).all() and (got[:, -1] == 0).all()
    q.free()
    dv.free()
