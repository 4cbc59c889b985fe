"""The arithmetic identities the tensor-core kernels rest on, checked on the CPU against the oracle's block decode
(no GPU, no product code): what must hold for the kernels' operand formats to be EXACT.

* Q4_K with integer weights (csrc/grouped_tc.cu): w = d * sc * q - dmin * m (kquant.rs:505-526), so
  W . x = sum_blocks d * [sum (sc * q) * x] - sum_subblocks (dmin * m) * X with X the sub-block sums of x;
  sc * q <= 945 is exact in fp16, and so is 2^-14 sc * q, the fp16 product of a nibble's bits (2^-24 q or 2^-20 q) and 2^10 sc or 2^6 sc;
  -(dmin * m) times a power of two of the row is exact as fp16 hi + lo.
* IQ3_XXS with exact weights: w = d / 4 * (grid magnitude) * sign * (2 s + 1), the product of the last three an integer exact
  in fp16 (csrc/grouped_tc.cu); the magnitude alone exact in bf16 (csrc/iq3_mma.cuh) and a signed byte (csrc/grouped_mma.cu).
* Activations of those kernels: a row times a power of two as two fp16 numbers (csrc/operand_rows.cuh), three for the
  sub-block sums of csrc/grouped_mma.cu, whose activations are four digits in base 256 of a block and, of a wide one, what they leave over;
  its integer sums fit.
* Router operands (csrc/router_tc.cu): an fp32 value is the exact sum of three bf16 numbers (round, round, round).
"""
import os
import re

import numpy as np
import pytest

SEED = 0xD3770B200


def _bf16_rn(x):
    """float32 array -> the nearest bf16 (ties to even), returned as float32."""
    u = np.ascontiguousarray(x, np.float32).view(np.uint32).astype(np.uint64)
    r = ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32)
    return r.view(np.float32)


def _q4k_fields(blocks, n_blocks):
    """d, dmin [nb] float32; sc, m [nb, 8] integers; q [nb, 256] integers, element order of kquant.rs:505-526."""
    b = np.frombuffer(blocks, np.uint8).reshape(n_blocks, 144)
    d = b[:, 0:2].copy().view(np.float16).astype(np.float32).reshape(n_blocks)
    dmin = b[:, 2:4].copy().view(np.float16).astype(np.float32).reshape(n_blocks)
    s = b[:, 4:16].astype(np.int64)
    sc = np.empty((n_blocks, 8), np.int64)
    m = np.empty((n_blocks, 8), np.int64)
    for j in range(8):
        if j < 4:
            sc[:, j] = s[:, j] & 63
            m[:, j] = s[:, j + 4] & 63
        else:
            sc[:, j] = (s[:, j + 4] & 0xF) | ((s[:, j - 4] >> 6) << 4)
            m[:, j] = (s[:, j + 4] >> 4) | ((s[:, j] >> 6) << 4)
    qs = b[:, 16:144].astype(np.int64).reshape(n_blocks, 4, 32)
    q = np.empty((n_blocks, 4, 64), np.int64)
    q[:, :, :32] = qs & 0xF   # low nibbles first, then the high nibbles of the same 32 bytes
    q[:, :, 32:] = qs >> 4
    return d, dmin, sc, m, q.reshape(n_blocks, 256)


def _mins_operand(dmin, m):
    """The A operand of the mins as csrc/grouped_tc.cu forms it for one row: dmin [blocks] fp16, m [blocks, 8] -> (hi, lo) fp16
    and the power of two both carry.  Each step is one fp16 operation."""
    ex = min(30, 39 - int(np.max(dmin.view(np.uint16) & 0x7FFF) >> 10))
    scale = np.float16(2.0 ** (ex - 15))
    dm = dmin * -scale
    prod = dm.astype(np.float64)[:, None] * m
    hi = prod.astype(np.float16)
    return hi, (prod - hi.astype(np.float64)).astype(np.float16), float(scale)  # the fma rounds the exact remainder once


def test_q4k_mins_of_any_size_fit_fp16():
    """Every exponent of the largest dmin of a row, up to fp16's largest number: nothing overflows; the product is exact where the
    scaled dmin is a normal number, and off by 2^-35 of the row's largest min where it is not."""
    rng = np.random.RandomState(4)
    m = np.tile(np.array([0, 1, 2, 31, 32, 61, 62, 63]), (8, 1))
    for top in range(31):
        for _ in range(50):
            bits = ((rng.randint(0, top + 1, 8) << 10) | rng.randint(0, 1024, 8) | (rng.randint(0, 2, 8) << 15)).astype(np.uint16)
            bits[rng.randint(8)] = (top << 10) | 0x3FF
            dmin = bits.view(np.float16)
            with np.errstate(over="raise"):
                hi, lo, scale = _mins_operand(dmin, m)
            assert np.isfinite(hi).all() and np.isfinite(lo).all()
            want = -(dmin.astype(np.float64)[:, None] * m)
            err = np.abs((hi.astype(np.float64) + lo.astype(np.float64)) / scale - want)
            normal = (np.abs(dmin.astype(np.float64)) * scale >= 2.0 ** -14) | (scale >= 1.0)
            assert not err[normal].any()
            assert err.max() <= 2.0 ** -35 * 64 * np.abs(dmin.astype(np.float64)).max()


def test_q4k_integer_weight_decomposition(orc):
    k, n = 1024, 24
    nb = k // 256
    w = orc.synth_blocks(orc.Q4_K, SEED, 901, n * nb)
    x = orc.synth_normal(SEED, 902, 1.0, k)
    want = orc.gemv_scalar(orc.Q4_K, w, k, n, x).astype(np.float64)
    d, dmin, sc, m, q = _q4k_fields(w, n * nb)
    # the field extraction is the format's: rebuilding the weights gives the oracle's dequantised row
    wq = (d[:, None, None] * sc[:, :, None]) * q.reshape(-1, 8, 32) - (dmin[:, None] * m)[:, :, None]
    deq = np.stack([orc.dequant_row(orc.Q4_K, w[r * nb * 144:(r + 1) * nb * 144], k) for r in range(n)])
    assert np.allclose(wq.reshape(n, k), deq, rtol=1e-6, atol=1e-7)
    # (1) sc * q is an integer <= 945: exact in fp16, and one fp16 fma (1024 + q) * sc - 1024 * sc gives it
    iw = sc[:, :, None] * q.reshape(-1, 8, 32)
    assert iw.max() <= 945 and np.array_equal(iw.astype(np.float16).astype(np.int64), iw)
    big = (1024 + q.reshape(-1, 8, 32)).astype(np.float16)      # 0x6400 | q
    assert np.array_equal(big.astype(np.int64), 1024 + q.reshape(-1, 8, 32))
    c = (-1024.0 * sc).astype(np.float16)
    assert np.array_equal(c.astype(np.float64), -1024.0 * sc)   # six bits times 2^10: exact
    fma = (big.astype(np.float64) * sc[:, :, None] + c.astype(np.float64)[:, :, None]).astype(np.float16)  # rounds once
    assert np.array_equal(fma.astype(np.int64), iw)
    # the same times 2^-14, without a constant to add: the bits of a nibble as a number below the normal ones, times a power of two of sc
    for shift in (0, 4):
        bits = (q.reshape(-1, 8, 32) << shift).astype(np.uint16).view(np.float16)
        by = (2.0 ** (10 - shift) * sc).astype(np.float16)
        assert np.array_equal(by.astype(np.float64), 2.0 ** (10 - shift) * sc)
        prod = bits * by[:, :, None]  # fp16 x fp16, rounded once
        assert np.array_equal(prod.astype(np.float64) * 2.0 ** 14, iw) and np.all((prod == 0) | (prod >= 2.0 ** -14))
    # (2) -(dmin * m) times the row's power of two is exact as fp16 hi + lo
    v = -(dmin[:, None].astype(np.float64) * m)
    hi, lo, scale = _mins_operand(dmin.astype(np.float16), m)
    assert np.array_equal((hi.astype(np.float64) + lo.astype(np.float64)) / scale, v)
    # (3) the decomposition: block sums scaled by d, minus the offsets against the sub-block sums of x
    xs = x.astype(np.float64).reshape(nb, 8, 32)
    main = np.einsum("rbsi,bsi->rb", iw.reshape(n, nb, 8, 32).astype(np.float64), xs) * d.reshape(n, nb)
    corr = np.einsum("rbs,bs->r", v.reshape(n, nb, 8), xs.sum(axis=2))
    got = main.sum(axis=1) + corr
    rms = np.sqrt(np.mean(want * want))
    assert np.max(np.abs(got - want)) <= 2e-6 * rms   # the oracle's own fp32 rounding


def test_activation_rows_as_scaled_fp16_parts(orc):
    """Rows scaled by a power of two so that the largest element is in [512, 1024): two fp16 parts carry 22 bits, three all bits of
    the elements above 1/1024 of the largest and 2^-34 of the largest below; the sub-block sums stay inside fp16's range."""
    x = orc.synth_normal(SEED, 903, 37.5, 4096).astype(np.float32)
    x[7] = 3.1e4      # an outlier, as SwiGLU outputs have
    x[11] = 1e-7
    for row in (x, x[1024:2048]):  # with the outlier, and without
        mx = np.max(np.abs(row))
        up = np.uint32((127 + 9 - (int(mx.view(np.uint32) >> 23) - 127)) << 23).view(np.float32)
        xs = row * up
        assert 512 <= np.max(np.abs(xs)) < 1024
        rest, parts = xs.copy(), []
        for _ in range(3):
            parts.append(rest.astype(np.float16))
            rest = rest - parts[-1].astype(np.float32)  # exact
        xs64 = xs.astype(np.float64)
        two = parts[0].astype(np.float64) + parts[1].astype(np.float64)
        assert np.max(np.abs(two - xs64)) <= 2.0 ** -22 * 1024 + 2.0 ** -25
        three = two + parts[2].astype(np.float64)
        large = np.abs(xs64) >= 1.0
        assert large.any() and np.array_equal(three[large], xs64[large])
        assert np.max(np.abs(three - xs64)) <= 2.0 ** -25  # 2^-34 of 512
        assert np.max(np.abs(xs64.reshape(-1, 32).sum(axis=1))) < 65504


def test_iq3xxs_integers_are_exact(orc):
    k = 512
    w = orc.synth_blocks(orc.IQ3_XXS, SEED, 904, k // 256)
    row = orc.dequant_row(orc.IQ3_XXS, w, k).astype(np.float64)
    b = np.frombuffer(w, np.uint8).reshape(-1, 98)
    d = b[:, 0:2].copy().view(np.float16).astype(np.float64).reshape(-1)
    s = (b[:, 66:98].copy().view(np.uint32).reshape(-1, 8) >> 28).astype(np.int64)  # of the word of each 32-element sub-block
    mag = row.reshape(-1, 8, 32) / (d[:, None] * (0.5 + s) * 0.5)[:, :, None]         # grid magnitude x sign
    assert np.allclose(mag, np.round(mag), atol=1e-3)
    mag = np.round(mag)
    assert np.max(np.abs(mag)) <= 62
    assert np.array_equal(_bf16_rn(mag), mag) and np.array_equal(mag.astype(np.float16).astype(np.float64), mag)
    iw = mag * (2 * s + 1)[:, :, None]
    assert np.max(np.abs(iw)) <= 62 * 31 and np.array_equal(iw.astype(np.float16).astype(np.float64), iw)
    assert np.allclose((d / 4)[:, None, None] * iw, row.reshape(-1, 8, 32), rtol=1e-6, atol=0)


def test_three_bf16_parts_carry_an_fp32_exactly(orc):
    x = np.concatenate([orc.synth_normal(SEED, 905, 1.0, 20000), orc.synth_normal(SEED, 906, 0.02, 20000),
                        np.array([0.0, 1.0, -1.0, 3.0e38, 1.17549435e-38, 16777215.0, 1.0 + 2.0 ** -23], np.float32)])
    hi = _bf16_rn(x)
    r1 = (x - hi).astype(np.float32)
    assert np.array_equal(r1.astype(np.float64), x.astype(np.float64) - hi.astype(np.float64))   # exact remainder
    mid = _bf16_rn(r1)
    r2 = (r1 - mid).astype(np.float32)
    assert np.array_equal(r2.astype(np.float64), r1.astype(np.float64) - mid.astype(np.float64))
    lo = _bf16_rn(r2)
    assert np.array_equal(hi.astype(np.float64) + mid.astype(np.float64) + lo.astype(np.float64), x.astype(np.float64))


def _digits(x):
    """Four digits in base 256, -128 .. 127, of a block times the power of two that puts its largest element into [2^30, 2^31), or into half of it
    where four digits do not reach; and what that leaves over, in fifteenths, -7 .. 7."""
    s = 157 - ((int(np.max(np.abs(x)).view(np.uint32)) + 0x10101) >> 23)
    scaled = np.ldexp(x.astype(np.float64), s)
    v = np.rint(scaled).astype(np.int64)
    b = ((v + 0x00808080) ^ 0x00808080).astype(np.int32).view(np.uint32)
    digits = np.stack([(b >> (8 * j)).astype(np.uint8).view(np.int8) for j in range(4)]).astype(np.int64)
    return digits, v, np.clip(np.rint((scaled - v) * 15), -7, 7), s


def _wide(x):
    """Blocks [n, 256] of which fewer than 8 lanes (of eight elements each) have one that is exact as an integer (2^24 or more after the scaling),
    or none of some four lanes, and other lanes are not zero."""
    ex = (np.max(np.abs(x), axis=1).view(np.uint32) + 0x10101) >> 23
    v = np.abs(np.ldexp(x.astype(np.float64), 157 - ex.astype(np.int64)[:, None])).reshape(len(x), 8, 4, 8)
    large, some = (v >= 2.0 ** 24).any(3), (v > 0).any(3)
    return (some.any(2) & ~large.any(2)).any(1) | ((large.sum((1, 2)) < 8) & (large != some).any((1, 2)))


@pytest.mark.parametrize("spread", [0.0, 3.0])
def test_activation_blocks_as_four_digits(orc, spread):
    rng = np.random.RandomState(8)
    tops = np.array([0x7EFEFE, 0x7EFEFF, 0x7FFFFF, 0], np.uint32)  # mantissas around the largest that four digits hold
    seen = []
    for i in range(50):
        x = (rng.randn(256) * np.exp(spread * rng.randn(256))).astype(np.float32)
        x[rng.randint(256)] *= -1.999
        at = np.argmax(np.abs(x))
        x[at] = np.copysign(((x[at:at + 1].view(np.uint32) & 0x7F800000) | tops[i % 4]).view(np.float32)[0], x[at])
        d, v, rest, s = _digits(x)
        assert d.min() >= -128 and d.max() <= 127
        assert np.array_equal(sum(256 ** j * d[j] for j in range(4)), v)
        left = x.astype(np.float64) - np.ldexp(v.astype(np.float64), -s)
        unit = 2.0 ** -30 * 1.01 * np.max(np.abs(x))  # at most, of it (or of 0.996 * 2^30)
        assert np.max(np.abs(left)) <= unit / 2
        left -= np.ldexp(rest / 15, -s)
        assert np.max(np.abs(left)) <= unit / 30
        seen.append(left / unit)
    assert abs(np.mean(seen)) < 4 * np.std(seen) / np.sqrt(50 * 256)  # no bias, which weights of one sign would add up


def test_which_activation_blocks_are_wide(orc):
    """Those with an outlier of 2^8 times the others or more, or with small sub-blocks; not normal ones, nor what the down projection meets
    (silu of one number times another, with half of them next to nothing where the first are large)."""
    rng = np.random.RandomState(9)
    f = lambda a: np.ascontiguousarray(a, np.float32)
    silu = lambda a: a / (1 + np.exp(-a))
    g, u = rng.randn(4000, 256), rng.randn(4000, 256)
    for x in (g, g + 3, silu(g) * u, silu(10 * g) * u, silu(100 * g) * u):
        assert _wide(f(x)).mean() < 1e-3
    for j, lo, hi in ((5, 0.0, 0.0), (8, 0.99, 1.0), (9, 1.0, 1.0), (20, 1.0, 1.0)):
        x = g.copy()
        x[:, 37] = 2.0 ** j * 1.5
        assert lo <= _wide(f(x)).mean() <= hi, j
    x = g.reshape(-1, 8, 32).copy()
    x[:, 5] *= 2.0 ** -8
    assert _wide(f(x.reshape(-1, 256))).mean() > 0.99
    x[:, 5] = 0.0
    assert not _wide(f(x.reshape(-1, 256))).any()  # zeros are exact


def test_integer_block_sums_fit(orc):
    """Largest sums of a 256-element block against a digit of 128: the arithmetic of the kernel's comments (test_largest_integer_sums runs such
    blocks through the kernels); the byte forms of the weights are the weights."""
    n = 32 * 128
    assert 8 * 16 * 63 * 15 * n < 2 ** 29 and 4 * 63 * (16 * 15 + 240) * n < 2 ** 29      # Q4_K: scales or nibbles 16 times as large
    assert 8 * 63 * 31 * n < 2 ** 26 and 8 * 31 * 62 * n < 2 ** 26                         # Q5_K, IQ3_XXS
    assert 16 * 128 * 16 * 128 * 128 < 2 ** 30 and 32 * 128 * 128 < 2 ** 22                # Q6_K; Q8_0 beside 1.5 * 2^23
    q = np.arange(64, dtype=np.uint32)                                                     # Q6_K: the upper pair of bits inverted in its upper bit
    byte = ((q & 15) << 2) | ((((q >> 4) ^ 2) & 3) << 6)
    assert np.array_equal(byte.astype(np.uint8).view(np.int8).astype(int), 4 * (q.astype(int) - 32))
    v = np.arange(4, 63, dtype=np.uint32)                                                  # IQ3_XXS: a negative byte is ~v + 1
    assert np.array_equal(((v ^ 255) + 1).astype(np.uint8).view(np.int8).astype(int), -v.astype(int))


def test_register_splits_fall_between_warpgroups():
    """csrc/grouped_tc.cu: setmaxnreg stands directly behind a condition on the warp's number that is the same for all four warps of a
    warpgroup, as PTX asks of it."""
    import denno_beta_b200

    with open(os.path.join(os.path.dirname(denno_beta_b200.__file__), "csrc", "grouped_tc.cu")) as f:
        src = f.read()
    value = {}
    for line in re.findall(r"^constexpr int ([A-Z_]+ = .*?);", src, re.M):
        for name, expr in re.findall(r"([A-Z_]+) = ([^,]+)", line):
            if re.fullmatch(r"[A-Z_0-9 +*]+", expr):
                value[name] = eval(expr, {}, value)
    calls = len(re.findall(r"^\s*reg_(?:inc|dec)<", src, re.M))
    sites = re.findall(r"if \(warp < ([A-Z_]+)\) \{\s*(?://[^\n]*\n\s*)*reg_(?:inc|dec)<", src)
    last = len(re.findall(r"\} else \{\s*(?://[^\n]*\n\s*)*reg_(?:inc|dec)<", src))
    assert calls >= 3 and last <= 1 and len(sites) + last == calls
    assert [value[s] for s in sites] == sorted(value[s] for s in sites)
    assert all(value[s] % 4 == 0 for s in sites), [(s, value[s]) for s in sites]
