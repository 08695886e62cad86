"""The product's per-point geometry (csrc/simplex.cuh), compiled for the host, against the oracle:
per-pixel simplex keys bit-exact, barycentric weights to the last bit or one unit off it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import GOLDEN_CASES, GOLDEN_CASES_F64, ROOT, bits, golden_positions, load_golden


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("shim") / "libsimplex_host.so")
    subprocess.check_call([
        "g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", out,
        "-I", os.path.join(ROOT, "permutohedral_lattice_b200", "csrc"),
        os.path.join(ROOT, "tests", "helpers", "simplex_host_shim.cpp")])
    return ctypes.CDLL(out)


def assert_weights_close(got, want):
    """Bit-exact up to the reference's double rounding: at most one unit in the last place of a weight
    near 1, and rare."""
    diff = np.abs(got.astype(np.float64) - want.astype(np.float64))
    assert diff.max() <= 2.0 ** -23
    assert (diff > 0).mean() <= 1e-4


def run_shim(shim, pos, scale):
    n, pd = pos.shape
    keys = np.zeros((n, pd + 1, pd), np.int16)
    w = np.zeros((n, pd + 1), np.float32)
    fp = ctypes.POINTER(ctypes.c_float)
    rc = shim.simplex_host(pos.ctypes.data_as(fp), scale.ctypes.data_as(fp), n, pd,
                           keys.ctypes.data_as(ctypes.POINTER(ctypes.c_short)), w.ctypes.data_as(fp))
    assert rc == 0
    return keys, w


@pytest.mark.parametrize("case", GOLDEN_CASES)
def test_keys_and_weights_match_golden(case, shim, oracle):
    g = load_golden(case)
    pos = np.ascontiguousarray(golden_positions(g, oracle), np.float32)
    keys, w = run_shim(shim, pos, oracle.scale_factors(pos.shape[1]))
    assert np.array_equal(keys, g["pixel_keys"])
    assert_weights_close(w, g["pixel_weights"])


@pytest.mark.parametrize("pd", [2, 3, 4, 5, 16])
def test_keys_and_weights_match_oracle_random(pd, shim, oracle):
    rng = np.random.default_rng(pd)
    pos = (rng.standard_normal((20000, pd)) * rng.choice([0.1, 1.0, 10.0, 50.0], (20000, 1))
           ).astype(np.float32)
    pos[:100] = np.round(pos[:100])          # exact ties on lattice hyperplanes
    pos[100:200] = 0.0
    keys, w = run_shim(shim, pos, oracle.scale_factors(pd))
    res = oracle.filter(np.ones((len(pos), 1), np.float32), pos)
    assert np.array_equal(keys, res.pixel_keys())
    assert_weights_close(w, res.pix_weight)


def run_shim_f64(shim, pos, scale):
    n, pd = pos.shape
    keys = np.zeros((n, pd + 1, pd), np.int16)
    w = np.zeros((n, pd + 1), np.float64)
    dp = ctypes.POINTER(ctypes.c_double)
    rc = shim.simplex_host_f64(pos.ctypes.data_as(dp), scale.ctypes.data_as(dp), n, pd,
                               keys.ctypes.data_as(ctypes.POINTER(ctypes.c_short)), w.ctypes.data_as(dp))
    assert rc == 0
    return keys, w


@pytest.mark.parametrize("case", GOLDEN_CASES_F64)
def test_double_keys_and_weights_match_golden_bit_for_bit(case, shim, oracle):
    g = load_golden(case)
    pos = np.ascontiguousarray(golden_positions(g, oracle), np.float64)
    keys, w = run_shim_f64(shim, pos, oracle.scale_factors(pos.shape[1], np.float64))
    assert np.array_equal(keys, g["pixel_keys"])
    assert np.array_equal(bits(w), bits(g["pixel_weights"]))


@pytest.mark.parametrize("pd", [2, 3, 4, 5, 16])
def test_double_keys_and_weights_match_oracle_random(pd, shim, oracle):
    rng = np.random.default_rng(100 + pd)
    pos = rng.standard_normal((20000, pd)) * rng.choice([0.1, 1.0, 10.0, 50.0], (20000, 1))
    pos[:100] = np.round(pos[:100])
    pos[100:200] = 0.0
    keys, w = run_shim_f64(shim, pos, oracle.scale_factors(pd, np.float64))
    res = oracle.filter(np.ones((len(pos), 1)), pos, dtype=np.float64)
    assert np.array_equal(keys, res.pixel_keys())
    assert np.array_equal(bits(w), bits(res.pix_weight))


def test_reciprocal_division_is_the_ieee_quotient(shim):
    rng = np.random.default_rng(1)
    fp = ctypes.POINTER(ctypes.c_float)
    shim.small_int_to_float_host.restype = ctypes.c_float
    for c in (0, 1, 2, 511, 1023, 65535, 8388607):
        assert shim.small_int_to_float_host(c) == float(c)
    for b in (80.0, 0.0625, 8.0, 0.125, 16.0, 0.1, 5.0, 3.0, 0.2, 0.7, 1e-3, 123.456, 2.0 ** -20, 3e6):
        a = np.concatenate([np.arange(0, 4096, dtype=np.float32), rng.random(200000, dtype=np.float32),
                            (rng.standard_normal(200000) * 1000).astype(np.float32)])
        out = np.empty_like(a)
        shim.div_by_rcp_host(a.ctypes.data_as(fp), ctypes.c_float(b), len(a), out.ctypes.data_as(fp))
        assert np.array_equal(bits(out), bits(a / np.float32(b))), b


def point_records(shim, pos, scale):
    n, pd = pos.shape
    low16 = np.zeros((n, pd), np.uint16)
    found, settled = np.zeros((n, pd + 1), np.int32), np.zeros((n, pd + 1), np.int32)
    rc = shim.point_records_host(*(ctypes.c_void_p(a.ctypes.data) for a in (pos, scale)), n, pd,
                                 int(pos.dtype == np.float64),
                                 *(ctypes.c_void_p(a.ctypes.data) for a in (low16, found, settled)))
    assert rc == 0
    return low16, found, settled


def keys_by_steps(low16, rank):
    """Keys of every remainder as build_tiles steps from one to the next: a coordinate for every rank, packed in four
    bits (ranks outside 1..16 fall out of the words)."""
    n, pd = low16.shape
    keys = np.zeros((n, pd + 1, pd), np.int64)
    for p in range(n):
        coord = [0] * 17
        for i in range(1, pd):
            if 1 <= rank[p, i] <= 16:
                coord[rank[p, i]] = (coord[rank[p, i]] + i) & 15
        k = low16[p].astype(np.int64)
        keys[p, 0] = k
        for r in range(1, pd + 1):
            k = k + 1
            taken = pd - r + 1
            if taken != rank[p, pd]:
                k[coord[taken]] -= pd + 1
            keys[p, r] = k
    return keys & 0xFFFF


def keys_by_ranks(low16, rank):
    """The same from the ranks, one byte each in four words."""
    n, pd = low16.shape
    keys = np.zeros((n, pd + 1, pd), np.int64)
    for p in range(n):
        words = [sum(int(rank[p, 4 * j + b]) << (8 * b) for b in range(4)) & 0xFFFFFFFF for j in range(pd // 4)]
        for r in range(pd + 1):
            for i in range(pd):
                above = (words[i // 4] + (127 - (pd - r)) * 0x01010101) & 0xFFFFFFFF
                keys[p, r, i] = int(low16[p, i]) + r - (pd + 1) * ((above >> (8 * (i & 3) + 7)) & 1)
    return keys & 0xFFFF


def features_without_a_simplex(dtype):
    """pd = 16: tame points first, then NaN, infinite, huge and (double) merely large features."""
    rng = np.random.default_rng(5)
    pos = rng.standard_normal((60, 16)) * 3.0
    pos[20:30, rng.integers(0, 16, 10)] = np.nan
    pos[30:40, 3] = np.inf
    pos[40:50] *= 1e9
    pos[50:60] *= 1e5 if dtype == np.float64 else 1e30
    return pos.astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_both_ways_to_a_key_agree_whatever_the_features(dtype, shim, oracle):
    pos = features_without_a_simplex(dtype)
    low16, found, settled = point_records(shim, pos, oracle.scale_factors(16, dtype))
    assert np.array_equal(found[:20], settled[:20])                     # real simplices stay as they are
    assert np.array_equal(np.sort(settled, 1), np.tile(np.arange(17), (60, 1)))
    steps, ranks = keys_by_steps(low16, settled), keys_by_ranks(low16, settled)
    assert np.array_equal(steps, ranks)
    # without settling they part: a slot of the tile's hash is then read that nobody wrote
    assert (keys_by_steps(low16, found) != keys_by_ranks(low16, found))[20:].any()


def far_features(pd, n=256):
    """Features beyond the integers of a float: neighbouring floats, whose low 16 bits differ by one."""
    return (1e8 + np.random.default_rng(0).integers(0, 40, (n, pd)) * 8.0).astype(np.float32)


def test_splats_of_two_remainders_can_have_one_key(shim, oracle):
    """Why a tile's splat may only stand for splats of its own remainder."""
    low16, found, _ = point_records(shim, far_features(2), oracle.scale_factors(2))
    remainders = {}
    for point in keys_by_steps(low16, found):
        for r, key in enumerate(point):
            remainders.setdefault(key.tobytes(), set()).add(r)
    assert max(len(rs) for rs in remainders.values()) > 1
