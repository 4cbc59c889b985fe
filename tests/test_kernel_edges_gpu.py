"""The edges of the expert kernels' tiles and of the rules that choose between them, against the CPU oracle."""
import numpy as np
import pytest

from helpers import SEED, check_block, make_layer, rel_err
from test_hyper import hc_weights

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    from denno_beta_b200 import cuda as cu

    c = cu.CudaCtx(0)
    yield c
    assert c.device_status() == 0
    c.close()


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "IQ3_XXS"])
@pytest.mark.parametrize("k,n", [(256, 32), (768, 288), (2304, 544)])
def test_grouped_mma(orc, ctx, name, k, n):
    """grouped_mma.cu: row counts around its 8-token tiles, rows that end inside a 16-row tile group, K of 1, 3 and 9 blocks."""
    from denno_beta_b200 import cuda as cu

    ty, ne = orc.TYPE_BY_NAME[name], 6
    assert ctx.moe_config(1, k, n, ne, 2)
    w = orc.synth_blocks(ty, SEED, 40 + ty, ne * n * k // orc.blck_size(ty))
    assert ctx.register_experts(0, cu.GATE, ty, k, n, ne, w)
    segs, at = [], 0
    for ex, m in ((4, 17), (0, 9), (5, 8), (2, 7), (1, 1)):
        segs.append([ex, m, at, at])
        at += m
    segs = np.array(segs, np.uint32)
    x = orc.synth_normal(SEED, 41, 1.0, at * k).reshape(at, k)
    x[3] *= 1e-6  # rows are scaled one by one
    x[4] = 0.0
    got = cu.moe_grouped_gemm_layer(ctx, 0, cu.GATE, segs, x, n)
    want = orc.grouped_gemm(ty, w, k, n, segs, x)
    for lo, hi in ((0, 3), (3, 4), (5, at)):
        assert rel_err(got[lo:hi], want[lo:hi]) <= 2e-5
    assert not got[4].any()


@pytest.mark.parametrize("name", ["Q4_K", "IQ3_XXS"])
@pytest.mark.parametrize("e,ff,ne,k", [(256, 256, 8, 2), (768, 512, 16, 3), (2304, 256, 4, 1), (512, 1280, 24, 4)])
def test_block_between_kernels(orc, ctx, name, e, ff, ne, k):
    """Token counts on both sides of every hand-over (routing in two launches to 15, tensor-core router from 16, tcgen05 from 48),
    with experts of one token to several full tiles; K of 1 to 9
    blocks.  From 48 tokens on a token's bits do not depend on the size of its chunk."""
    assert ctx.moe_config(1, e, ff, ne, k)
    L = make_layer(orc, ctx, 0, orc.TYPE_BY_NAME[name], e, ff, ne, k, bias=True, gate_row=True)
    for nt in (2, 9, 15, 16, 47, 48, 49, 97, 256, 257):
        h = orc.synth_normal(SEED, 50 + nt, 1.0, nt * e).reshape(nt, e)
        out, sels, wts = ctx.moe_block(0, h, want_routing=True)
        err, _ = check_block(orc, L, h, out, sels, wts)
        assert err <= (5e-5 if nt < 16 else 2e-4), "nt %d: %.3g" % (nt, err)
        assert np.array_equal(out.view(np.uint32), ctx.moe_block(0, h).view(np.uint32)), "nt %d: bits of a replay" % nt
        if nt >= 256:
            part = ctx.moe_block(0, h[5:53])
            assert np.array_equal(part.view(np.uint32), out[5:53].view(np.uint32)), "nt %d: bits of a chunk of 48" % nt


@pytest.mark.parametrize("up,down", [("IQ3_XXS", "IQ3_XXS"), ("Q4_K", "Q4_K"), ("Q4_K", "Q6_K")])
def test_bits_do_not_depend_on_the_batch(orc, ctx, up, down):
    """Wide enough that a split of K pays for few tokens and not for many: a token has the same bits in every batch of 2 to 15, of
    16 to 47 and, in a layer of one format, from 48 on, routed by the layer or by the caller."""
    from denno_beta_b200 import cuda as cu

    e, ff, ne, k = 2048, 1024, 64, 8
    up, down = orc.TYPE_BY_NAME[up], orc.TYPE_BY_NAME[down]
    assert ctx.moe_config(1, e, ff, ne, k)
    for m, ty, ni, no, n in ((cu.GATE, up, e, ff, ne), (cu.UP, up, e, ff, ne), (cu.DOWN, down, ff, e, ne), (cu.SHARED_GATE, up, e, ff, 1),
                             (cu.SHARED_UP, up, e, ff, 1), (cu.SHARED_DOWN, down, ff, e, 1)):
        assert ctx.synth_experts(0, m, ty, ni, no, n, SEED)
    ctx.register_router(0, orc.synth_normal(SEED, 6, 0.02, ne * e).reshape(ne, e), None, np.ones(e, np.float32), None)
    h = orc.synth_normal(SEED, 95, 1.0, 96 * e).reshape(96, e)
    for large, small in ((15, 2), (9, 4), (47, 16)) + (((96, 48),) if up == down else ()):
        out, part = ctx.moe_block(0, h[:large]), ctx.moe_block(0, h[large - small:large])
        assert np.array_equal(out[large - small:].view(np.uint32), part.view(np.uint32)), (large, small)
    rng = np.random.RandomState(5)
    sels = np.sort(np.argsort(rng.rand(40, ne), axis=1)[:, :k], axis=1).astype(np.int32)
    wts = rng.rand(40, k).astype(np.float32)
    out, part = ctx.moe_experts(0, h[:40], sels, wts), ctx.moe_experts(0, h[7:8], sels[7:8], wts[7:8])
    assert np.array_equal(out[7:8].view(np.uint32), part.view(np.uint32))


def test_batch_with_a_long_k(orc, ctx):
    """Q8_0 rows of 6144: two warps' sums have no room beside the activations, so one warp takes all of K."""
    e, ff, ne, k, nt = 6144, 256, 4, 2, 9
    assert ctx.moe_config(1, e, ff, ne, k)
    L = make_layer(orc, ctx, 0, orc.Q8_0, e, ff, ne, k)
    h = orc.synth_normal(SEED, 97, 1.0, nt * e).reshape(nt, e)
    ctx.profile(True)
    out, sels, wts = ctx.moe_block(0, h, want_routing=True)
    launched = ctx.profile_read()
    ctx.profile(False)
    assert launched["mm_gate_up"]["launches"] == 1 and "combine" in launched
    assert check_block(orc, L, h, out, sels, wts)[0] <= 5e-5
    assert np.array_equal(ctx.moe_block(0, h[3:5]).view(np.uint32), out[3:5].view(np.uint32))


@pytest.mark.parametrize("up,down,e,ff", [("Q5_K", "Q8_0", 768, 288), ("Q4_K", "Q6_K", 512, 768), ("IQ3_XXS", "Q4_K", 512, 256)])
def test_experts_given_mixed(orc, ctx, up, down, e, ff):
    """A selection of the caller's own and two formats in a layer, one with an expert width (288) that the mma kernel leaves alone."""
    ne, k = 40, 5
    assert ctx.moe_config(1, e, ff, ne, k)
    L = make_layer(orc, ctx, 0, orc.TYPE_BY_NAME[up], e, ff, ne, k, ty_down=orc.TYPE_BY_NAME[down])
    rng = np.random.RandomState(3)
    for nt in (1, 4, 8, 9, 15, 16, 50):
        x = orc.synth_normal(SEED, 60 + nt, 1.0, nt * e).reshape(nt, e)
        sels = np.sort(np.argsort(rng.rand(nt, ne), axis=1)[:, :k], axis=1).astype(np.int32)
        wts = rng.rand(nt, k).astype(np.float32)
        for _ in range(3):  # the third one replays
            out = ctx.moe_experts(0, x, sels, wts)
            assert rel_err(out, orc.moe_experts_given(L, x, sels, wts)) <= 5e-5
            sels, wts = np.ascontiguousarray(sels[::-1]), np.ascontiguousarray(wts[::-1])


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "IQ3_XXS"])
@pytest.mark.parametrize("k,n,nvec", [(256, 1, 1), (768, 15, 2), (2304, 17, 3), (512, 2369, 8), (4096, 33, 1), (4352, 33, 1), (4864, 17, 2), (4864, 2400, 1),
                                      (5632, 371, 8), (8448, 15, 1), (2048, 2048, 4)])
def test_gemv_edges(orc, ctx, name, k, n, nvec):
    """Rows that end inside a group of 16, vectors in pairs and an odd one, K of 1 to 33 blocks: 17, 33 and (with more CTAs than SMs) 19 are two a stage
    with a last stage of one, 19 and 22 with few CTAs one a stage; 2048 x 2048 with four vectors is two CTAs an SM."""
    ty = orc.TYPE_BY_NAME[name]
    w = orc.synth_blocks(ty, SEED, 70 + ty, n * k // orc.blck_size(ty))
    x = orc.synth_normal(SEED, 71, 1.0, nvec * k).reshape(nvec, k)
    out = np.full((nvec + 1, n), 7.0, np.float32)
    dw, dx, do = ctx.dev_alloc(w.nbytes), ctx.dev_alloc(x.nbytes), ctx.dev_alloc(out.nbytes)
    try:
        ctx.upload(dw, w)
        ctx.upload(dx, x)
        ctx.upload(do, out)
        assert ctx.gemv_dev(ty, dw, k, n, dx, do, nvec)
        got = ctx.download(do, np.empty_like(out))
    finally:
        for p in (dw, dx, do):
            ctx.dev_free(p)
    assert np.all(got[nvec] == 7.0), "wrote behind the last row"
    want = np.stack([orc.gemv_scalar(ty, w, k, n, v) for v in x])
    assert rel_err(got[:nvec], want) <= 2e-5


def test_four_vectors_of_a_small_matrix(orc, ctx):
    """2048 x 2048 of IQ3_XXS: two CTAs fit an SM, so the two pairs of vectors are grid rows of the GEMV."""
    w = orc.synth_blocks(orc.IQ3_XXS, SEED, 75, 2048 * 8)
    dw, dx, do = ctx.dev_alloc(w.nbytes), ctx.dev_alloc(4 * 2048 * 4), ctx.dev_alloc(4 * 2048 * 4)
    try:
        ctx.upload(dw, w)
        ctx.upload(dx, orc.synth_normal(SEED, 76, 1.0, 4 * 2048))
        ctx.profile(True)
        assert ctx.gemv_dev(orc.IQ3_XXS, dw, 2048, 2048, dx, do, 4)
        assert list(ctx.profile_read()) == ["gemv_mma"]
        ctx.profile(False)
    finally:
        for p in (dw, dx, do):
            ctx.dev_free(p)


@pytest.mark.parametrize("base", [0, 2048])
def test_shared_memory_that_starts_elsewhere(orc, ctx, base):
    """IQ3_XXS where the tables of the mma.sync kernels would not be where their instructions look for them: other kernels serve every call.  A
    context that is told wrong learns it from the first tcgen05 call, which is declined, and the second one is served."""
    from denno_beta_b200 import cuda as cu

    e, ff, ne, k = 512, 256, 8, 2
    assert ctx.moe_config(1, e, ff, ne, k)
    L = make_layer(orc, ctx, 0, orc.IQ3_XXS, e, ff, ne, k)
    w = orc.synth_blocks(orc.IQ3_XXS, SEED, 190, 300 * e // 256)
    assert ctx.register_matrix(190, orc.IQ3_XXS, w, e, 300)
    h = orc.synth_normal(SEED, 191, 1.0, 64 * e).reshape(64, e)
    ctx.set_smem_base(base)
    ctx.profile(True)
    for nt in (1, 2, 9, 24):
        for _ in range(3):  # the third one replays
            out, sels, wts = ctx.moe_block(0, h[:nt], want_routing=True)
            assert check_block(orc, L, h[:nt], out, sels, wts)[0] <= 2e-4
    out = ctx.moe_experts(0, h[:4], sels[:4], wts[:4])
    assert rel_err(out, orc.moe_experts_given(L, h[:4], sels[:4], wts[:4])) <= 5e-5
    got = np.empty(300, np.float32)
    assert ctx.gemv(190, h[0], got)
    assert rel_err(got, orc.gemv_scalar(orc.IQ3_XXS, w, e, 300, h[0])) <= 2e-5
    assert not [n for n in ctx.profile_read() if n.startswith(("mm_", "gemv_mma"))]
    ctx.profile(False)
    if base:
        assert ctx.moe_block(0, h) is None
    out, sels, wts = ctx.moe_block(0, h, want_routing=True)
    assert check_block(orc, L, h, out, sels, wts)[0] <= 2e-4


@pytest.mark.parametrize("hc,lr,nts", [(1, 8, (1, 9)), (2, 33, (1, 8)), (3, 320, (2, 17))])
def test_hyper_edges(orc, ctx, hc, lr, nts):
    """Streams, ranks that end inside a CTA's rows, and more tokens than a CTA takes at once."""
    e, ff, ne, k = 512, 256, 8, 2
    assert ctx.moe_config(1, e, ff, ne, k)
    L = make_layer(orc, ctx, 0, orc.IQ3_XXS, e, ff, ne, k, norm=False)
    w_norm, w_down, w_up = hc_weights(orc, hc, e, lr, 1)
    ctx.register_hc(0, hc, lr, w_norm, w_down, w_up)
    for nt in nts:
        res = orc.synth_normal(SEED, 80 + nt, 1.0, nt * hc * e).reshape(nt, hc, e)
        mix = [orc.hc_mix(r, w_norm, w_down, w_up, lr, 1e-6)[:2] for r in res]
        blk = orc.moe_block(L, np.stack([m.reshape(-1) for m, _ in mix]))[0]
        want = np.stack([orc.hc_combine(r, b, inj) for r, b, (_, inj) in zip(res, blk, mix)])
        for _ in range(3):
            assert rel_err(ctx.hc_moe_block(0, res), want) <= 5e-5


@pytest.mark.parametrize("e,ff", [(512, 256), (1280, 1280), (2304, 512)])
@pytest.mark.parametrize("nt", [33, 64, 300])
def test_q4k_mins_of_any_size(orc, ctx, e, ff, nt):
    """Q4_K blocks whose dmin is fp16's largest number, or subnormal: dmin * m reaches 4e6, far outside fp16, in rows of all three
    matrices, on both expert kernels of a chunk and with one and two stages of mins.  The other rows do not feel it."""
    ne, k, row = 4, 2, 7

    def edit(name, blocks):
        n_out, n_in = (e, ff) if name == "down" else (ff, e)
        b = blocks.reshape(ne, n_out, n_in // 256, 144)
        b[:, row, :, 2:4] = np.array([65504.0], np.float16).view(np.uint8)
        b[:, row + 1, 0, 2:4] = np.array([65504.0], np.float16).view(np.uint8)  # beside blocks of ordinary size
        b[:, row + 2, :, 2:4] = np.array([6e-8], np.float16).view(np.uint8)

    assert ctx.moe_config(1, e, ff, ne, k)
    L = make_layer(orc, ctx, 0, orc.Q4_K, e, ff, ne, k, edit=edit)
    h = orc.synth_normal(SEED, 90 + nt, 1.0, nt * e).reshape(nt, e)
    out, sels, wts = ctx.moe_block(0, h, want_routing=True)
    assert np.isfinite(out).all()
    want = orc.moe_experts_given(L, orc.rmsnorm(h, np.ones(e, np.float32)), sels, wts)
    for rows in (slice(row, row + 2), slice(row + 2, e)):
        assert rel_err(out[:, rows], want[:, rows]) <= 2e-4


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "IQ3_XXS"])
@pytest.mark.parametrize("nvec", [1, 2, 5])
def test_activations_of_any_size(orc, ctx, name, nvec):
    """Activations are integers of their 256-element block: blocks from 1e-37 to 1e30, an element 2^20 times its neighbours, a block of
    zeros, and blocks with an infinity or a NaN, whose vector alone feels it."""
    ty, k, n = orc.TYPE_BY_NAME[name], 1024, 48
    w = orc.synth_blocks(ty, SEED, 110 + ty, n * k // orc.blck_size(ty))
    x = orc.synth_normal(SEED, 111, 1.0, 8 * nvec * k).reshape(8, nvec, k)
    for i, f in enumerate((1e-37, 1e-30, 1.0, 1e30)):
        x[i] *= np.float32(f)
    x[3, :, 256:512] = 0.0
    x[4, :, :256] *= np.float32(1e-20)
    x[5, :, 300] *= np.float32(2.0 ** 20)
    x[6, 0, 700] = np.inf
    x[7, 0, 5] = np.nan
    dw, dx, do = ctx.dev_alloc(w.nbytes), ctx.dev_alloc(x.nbytes), ctx.dev_alloc(8 * nvec * n * 4)
    try:
        ctx.upload(dw, w)
        ctx.upload(dx, x)
        for i in range(8):
            assert ctx.gemv_dev(ty, dw, k, n, dx + 4 * i * nvec * k, do + 4 * i * nvec * n, nvec)
        got = ctx.download(do, np.empty((8, nvec, n), np.float32))
    finally:
        for p in (dw, dx, do):
            ctx.dev_free(p)
    deq = orc.dequant_row(ty, w, n * k).reshape(n, k).astype(np.float64)
    for i in range(8):
        first = 1 if i > 5 else 0
        if first:
            assert not np.isfinite(got[i, 0]).any()
            if nvec == 1:
                continue
        want = x[i, first:].astype(np.float64) @ deq.T
        # fp32 sums, and what three fp16 parts would leave over of a block's largest element; 1e-37: an fp32 below 2^-126 keeps 2^-149
        tiny = k * 2.0 ** -149 * np.abs(deq).max() if i == 0 else 0.0
        bound = 2.0 ** -20 * np.sqrt((x[i, first:].astype(np.float64) ** 2) @ (deq ** 2).T) + 2.0 ** -34 * np.abs(x[i, first:]).max() * np.abs(deq).sum(1) + tiny
        assert np.all(np.abs(got[i, first:] - want) <= bound), (i, np.max(np.abs(got[i, first:] - want) / bound))


def _largest_weights(orc, name, n_blocks):
    """Blocks whose integers are as large as the format has them, of one sign."""
    if name == "Q8_0":
        b = np.full((n_blocks * 8, 34), 0x80, np.uint8)
        b[:, 0:2] = np.array([0.5], np.float16).view(np.uint8)
        return b
    b = np.full((n_blocks, {"Q4_K": 144, "Q5_K": 176, "Q6_K": 210, "IQ3_XXS": 98}[name]), 0xFF, np.uint8)
    if name in ("Q4_K", "Q5_K"):
        b[:, 0:4] = np.array([0.5, 0.25], np.float16).view(np.uint8)
    elif name == "Q6_K":
        b[:, :192] = 0     # q = -32
        b[:, 192:208] = 0x80
        b[:, 208:210] = np.array([0.5], np.float16).view(np.uint8)
    else:
        b[:, 0:2] = np.array([0.5], np.float16).view(np.uint8)
        b[:, 66:] = np.array([15 << 28], np.uint32).view(np.uint8).reshape(1, 4).repeat(8, 0).reshape(-1)
        sums = []
        for code in range(256):
            b[0, 2:66] = code
            sums.append(orc.dequant_row(orc.IQ3_XXS, b[0].copy(), 256).sum())
        b[:, 2:66] = int(np.argmax(sums))
    return b


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "IQ3_XXS"])
@pytest.mark.parametrize("nvec", [1, 2, 5])
def test_largest_integer_sums(orc, ctx, name, nvec):
    """Weights of the largest integers and scales against activations of the largest digits, all of one sign: 0x7e7f7f80 is the digits -128, -128,
    -128, 127 in base 256, -0x808080 in a block with one large element -128, -128, -128, 0.  Nothing leaves 32 bits."""
    ty, k, n = orc.TYPE_BY_NAME[name], 1024, 32
    w = _largest_weights(orc, name, n * k // 256)
    deq = orc.dequant_row(ty, w.reshape(-1), n * k).reshape(n, k).astype(np.float64)
    x = np.empty((3, nvec, 4, 256), np.float32)
    x[0] = 0x7E7F7F80 * 2.0 ** -23
    x[1] = -0x7E7F7F80 * 2.0 ** -23
    x[2] = -0x808080 * 2.0 ** -23
    x[2, ..., 100] = -128.0
    x = x.reshape(3, nvec, k)
    dw, dx, do = ctx.dev_alloc(w.nbytes), ctx.dev_alloc(x.nbytes), ctx.dev_alloc(3 * nvec * n * 4)
    try:
        ctx.upload(dw, w)
        ctx.upload(dx, x)
        for i in range(3):
            assert ctx.gemv_dev(ty, dw, k, n, dx + 4 * i * nvec * k, do + 4 * i * nvec * n, nvec)
        got = ctx.download(do, np.empty((3, nvec, n), np.float32))
    finally:
        for p in (dw, dx, do):
            ctx.dev_free(p)
    want = x.astype(np.float64) @ deq.T
    # at most a few dozen roundings of 2^-24 of sums of one sign; the mins (Q4_K, Q5_K) are a part of them
    assert np.all(np.abs(got - want) <= 40 * 2.0 ** -24 * np.abs(want)), np.max(np.abs(got / want - 1.0))


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "IQ3_XXS"])
@pytest.mark.parametrize("nvec", [1, 2, 5])
def test_subnormal_activations(orc, ctx, name, nvec):
    """Blocks whose elements are all below fp32's normal numbers are as exact as any: alone, beside zeros and beside small normal blocks."""
    ty, k, n = orc.TYPE_BY_NAME[name], 1024, 48
    w = orc.synth_blocks(ty, SEED, 120 + ty, n * k // orc.blck_size(ty))
    x = (orc.synth_normal(SEED, 121, 1.0, nvec * k).astype(np.float64) * 2e-39).reshape(nvec, 4, 256)
    x[-1, 1] = 0.0
    x[-1, 2] *= 3e4
    x = x.reshape(nvec, k).astype(np.float32)
    assert 0 < np.abs(x[0, :256]).max() < 2.0 ** -126
    dw, dx, do = ctx.dev_alloc(w.nbytes), ctx.dev_alloc(x.nbytes), ctx.dev_alloc(nvec * n * 4)
    try:
        ctx.upload(dw, w)
        ctx.upload(dx, x)
        assert ctx.gemv_dev(ty, dw, k, n, dx, do, nvec)
        got = ctx.download(do, np.empty((nvec, n), np.float32))
    finally:
        for p in (dw, dx, do):
            ctx.dev_free(p)
    deq = orc.dequant_row(ty, w, n * k).reshape(n, k).astype(np.float64)
    x64 = x.astype(np.float64)
    # fp32 sums; sums below the normal numbers round to 2^-149: four blocks, of a sum each for low and high digits, and their meeting
    bound = 2.0 ** -20 * np.sqrt((x64 ** 2) @ (deq ** 2).T) + 16 * 2.0 ** -149
    assert np.all(np.abs(got - x64 @ deq.T) <= bound), np.max(np.abs(got - x64 @ deq.T) / bound)


def _deaf(name, w):
    """Blocks of 256 elements whose weights do not hear element 37: zero, or (IQ3_XXS, which has no zero) the same as element 45's."""
    b = w.reshape(-1, {"Q4_K": 144, "Q5_K": 176, "Q6_K": 210, "Q8_0": 272, "IQ3_XXS": 98}[name])
    if name in ("Q4_K", "Q5_K"):
        b[:, 9] &= 0xC0  # the min of its sub-block
        b[:, (21 if name == "Q4_K" else 53)] &= 0x0F
        if name == "Q5_K":
            b[:, 21] &= 0xFD
    elif name == "Q6_K":
        b[:, 37] &= 0xF0
        b[:, 133] = (b[:, 133] & 0xF3) | 8
    elif name == "Q8_0":
        b[:, 41] = 0
    else:
        b[:, 12:14] = b[:, 10:12]
        signs = b[:, 70:74].copy().view(np.uint32)
        b[:, 70:74] = ((signs & ~np.uint32(0x3F80)) | ((signs & np.uint32(0x7F)) << np.uint32(7))).view(np.uint8)
    return w


def _beside_outliers(name, x, ratio):
    """x with element 37 of every block `ratio` times the others' size (IQ3_XXS: and element 45 its negative)."""
    x = x.copy()
    b = x.reshape(-1, 256)
    b[:, 37] = ratio * (1.0 + np.arange(len(b)) % 7 / 7.0)
    if name == "IQ3_XXS":
        b[:, 45] = -b[:, 37]
    return x


def _small_elements_bound(name, x, deq):
    """fp32 sums of what is heard, and 2^-34 of the row's largest element from each weight, as three fp16 parts of a row would have it."""
    y = x.astype(np.float64).reshape(len(x), -1, 256).copy()
    y[:, :, 37] = 0.0
    if name == "IQ3_XXS":
        y[:, :, 45] = 0.0
    norm = np.sqrt((deq ** 2).sum(1))
    return 2.0 ** -20 * np.sqrt((y.reshape(len(x), -1) ** 2) @ (deq ** 2).T) + 4 * 2.0 ** -34 * np.abs(x).max(1)[:, None] * norm


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "IQ3_XXS"])
@pytest.mark.parametrize("k,nvec", [(1024, 1), (1024, 2), (4352, 1), (768, 5)])
def test_small_elements_beside_large_ones_gemv(orc, ctx, name, k, nvec):
    """Blocks of x with an element far above the others that no weight hears: the others are as exact as three fp16 parts would hold them."""
    ty, n = orc.TYPE_BY_NAME[name], 48
    w = _deaf(name, np.array(orc.synth_blocks(ty, SEED, 170 + ty, n * k // orc.blck_size(ty))))
    deq = orc.dequant_row(ty, w, n * k).reshape(n, k).astype(np.float64)
    x = orc.synth_normal(SEED, 171, 1.0, nvec * k).reshape(nvec, k)
    dw, dx, do = ctx.dev_alloc(w.nbytes), ctx.dev_alloc(x.nbytes), ctx.dev_alloc(nvec * n * 4)
    try:
        ctx.upload(dw, w)
        for j in (8, 12, 16, 20):
            xs = _beside_outliers(name, x, 2.0 ** j)
            if j == 16:
                xs[0] = x[0]  # one vector without
            ctx.upload(dx, xs)
            assert ctx.gemv_dev(ty, dw, k, n, dx, do, nvec)
            got = ctx.download(do, np.empty((nvec, n), np.float32))
            off = np.abs(got - xs.astype(np.float64) @ deq.T) / _small_elements_bound(name, xs, deq)
            assert off.max() <= 1.0, (j, off.max())
    finally:
        for p in (dw, dx, do):
            ctx.dev_free(p)


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "IQ3_XXS"])
@pytest.mark.parametrize("sizes", [(1, 1, 2, 1, 1, 1), (3, 2, 4, 2, 1, 2), (1, 17, 8, 5, 3, 7)])
def test_small_elements_beside_large_ones_grouped(orc, ctx, name, sizes):
    """The same for items of one, two and four column tiles; tokens that have no such blocks do not feel their neighbours that do."""
    from denno_beta_b200 import cuda as cu

    ty, k, n, ne = orc.TYPE_BY_NAME[name], 768, 96, len(sizes)
    assert ctx.moe_config(1, k, n, ne, 2)
    w = _deaf(name, np.array(orc.synth_blocks(ty, SEED, 180 + ty, ne * n * k // orc.blck_size(ty))))
    assert ctx.register_experts(0, cu.GATE, ty, k, n, ne, w)
    deq = orc.dequant_row(ty, w, ne * n * k).reshape(ne, n, k).astype(np.float64)
    at = np.concatenate([[0], np.cumsum(sizes)])
    segs = np.array([[ne - 1 - i, m, at[i], at[i]] for i, m in enumerate(sizes)], np.uint32)
    x = orc.synth_normal(SEED, 181, 1.0, int(at[-1]) * k).reshape(-1, k)
    plain = cu.moe_grouped_gemm_layer(ctx, 0, cu.GATE, segs, x, n)
    for j in (8, 12, 16, 20):
        xs = _beside_outliers(name, x, 2.0 ** j)
        xs[1::3] = x[1::3]
        xs[2::5, 256:] = x[2::5, 256:]  # one wide block of three
        got = cu.moe_grouped_gemm_layer(ctx, 0, cu.GATE, segs, xs, n)
        same = np.all(xs == x, axis=1)
        assert np.array_equal(got[same].view(np.uint32), plain[same].view(np.uint32)), j
        for i, m in enumerate(sizes):
            rows, d = slice(at[i], at[i + 1]), deq[ne - 1 - i]
            off = np.abs(got[rows] - xs[rows].astype(np.float64) @ d.T) / _small_elements_bound(name, xs[rows], d)
            assert off.max() <= 1.0, (j, i, off.max())


@pytest.mark.parametrize("up,down", [("Q4_K", "Q6_K"), ("Q5_K", "Q8_0"), ("IQ3_XXS", "IQ3_XXS"), ("Q8_0", "Q4_K")])
def test_block_with_outliers(orc, ctx, up, down):
    """Tokens with an element far above the others in a block on the fused gate/up kernel; the other tokens do not feel them."""
    e, ff, ne, k = 1024, 512, 16, 3
    up, down = orc.TYPE_BY_NAME[up], orc.TYPE_BY_NAME[down]
    assert ctx.moe_config(1, e, ff, ne, k)
    L = make_layer(orc, ctx, 0, up, e, ff, ne, k, ty_down=down)
    for nt in (2, 9, 15, 40):
        h = orc.synth_normal(SEED, 210 + nt, 1.0, nt * e).reshape(nt, e)
        plain = ctx.moe_block(0, h)
        loud = h.copy()
        for i, at in ((1, 300), (4, 37), (7, 1000)):
            if i < nt:
                loud[i, at] = 2.0 ** (8 + 3 * i)
        out, sels, wts = ctx.moe_block(0, loud, want_routing=True)
        assert check_block(orc, L, loud, out, sels, wts)[0] <= 5e-5
        same = np.all(loud == h, axis=1)
        assert np.array_equal(out[same].view(np.uint32), plain[same].view(np.uint32)), nt


@pytest.mark.parametrize("name", ["Q4_K", "IQ3_XXS"])
@pytest.mark.parametrize("k,n", [(256, 256), (1024, 512), (1280, 256), (2304, 256)])
def test_tcgen05_items(orc, ctx, name, k, n):
    """grouped_tc.cu: experts whose tokens end on either side of 16, 32, 48 and 64 columns (N of the MMAs, loads of the sums) and of a second
    item, K of 1, 4, 5 and 9 blocks (the mins in one stage, in two, and a second time for the ninth).  Bound: an activation is 22 bits of its
    row's largest, a block's sum is rounded 16 times in 24 bits, rows of K / 256 blocks are summed in fp32: 2e-6 of the result's rms each, and up
    to 4 sigma of it over a row."""
    from denno_beta_b200 import cuda as cu

    ty, sizes = orc.TYPE_BY_NAME[name], (129, 128, 80, 65, 64, 63, 49, 48, 47, 33, 32, 31, 24, 17, 16, 15, 9, 8, 4, 1)
    ne = len(sizes)
    assert ctx.moe_config(1, k, n, ne, 1)
    w = orc.synth_blocks(ty, SEED, 140 + ty, ne * n * k // orc.blck_size(ty))
    assert ctx.register_experts(0, cu.GATE, ty, k, n, ne, w)
    at = np.concatenate([[0], np.cumsum(sizes)])
    segs = np.array([[ne - 1 - i, m, at[i], at[i]] for i, m in enumerate(sizes)], np.uint32)
    x = orc.synth_normal(SEED, 141, 1.0, int(at[-1]) * k).reshape(-1, k)
    x[5] *= 1e-6  # rows are scaled one by one
    x[6] = 0.0
    ctx.profile(True)
    got = cu.moe_grouped_gemm_layer(ctx, 0, cu.GATE, segs, x, n)
    launched = ctx.profile_read()
    ctx.profile(False)
    assert "tc_down" in launched, sorted(launched)
    want = orc.grouped_gemm(ty, w, k, n, segs, x)
    for i, m in enumerate(sizes):
        rows = slice(at[i] + (7 if i == 0 else 0), at[i + 1])
        assert rel_err(got[rows], want[rows]) <= 2e-5, m
    assert rel_err(got[5:6], want[5:6]) <= 2e-5 and not got[6].any()


@pytest.mark.parametrize("name", ["Q4_K", "IQ3_XXS"])
@pytest.mark.parametrize("k", [512, 2048])
def test_tcgen05_sums_are_not_short(orc, ctx, name, k):
    """One element of each block alone: nothing but the addition of hi and lo rounds, and it must not have a bias (a truncated one is 3e-8 of the
    result short).  The mean over 50,000 results of rounding errors of 6e-8 is known to 3e-10."""
    from denno_beta_b200 import cuda as cu

    ty, n, ne, m = orc.TYPE_BY_NAME[name], 256, 3, 64
    assert ctx.moe_config(1, k, n, ne, 1)
    w = orc.synth_blocks(ty, SEED, 200 + ty, ne * n * k // orc.blck_size(ty))
    assert ctx.register_experts(0, cu.GATE, ty, k, n, ne, w)
    deq = orc.dequant_row(ty, w, ne * n * k).reshape(ne, n, k).astype(np.float64)
    x = np.zeros((ne * m, k // 256, 256), np.float32)
    x[:, :, 37] = orc.synth_normal(SEED, 201, 1.0, ne * m * (k // 256)).reshape(ne * m, -1)
    x = x.reshape(ne * m, k)
    segs = np.array([[i, m, i * m, i * m] for i in range(ne)], np.uint32)
    ctx.profile(True)
    got = cu.moe_grouped_gemm_layer(ctx, 0, cu.GATE, segs, x, n)
    launched = ctx.profile_read()
    ctx.profile(False)
    assert "tc_down" in launched, sorted(launched)
    want = np.einsum("emk,enk->emn", x.reshape(ne, m, k).astype(np.float64), deq).reshape(ne * m, n)
    assert abs(np.sum((got - want) * want) / np.sum(want * want)) <= 1.5e-8


@pytest.mark.parametrize("k", [1, 8, 9, 12, 13, 25])
@pytest.mark.parametrize("nt", [5, 300])
def test_combine_slots(orc, ctx, k, nt):
    """combine_kernel: slots around the eight (large grids) and twelve (small ones) that are requested together, with a shared expert, its
    gate row and the residual of a block."""
    e, ff, ne = 256, 256, 32
    assert ctx.moe_config(1, e, ff, ne, k)
    L = make_layer(orc, ctx, 0, orc.Q4_K, e, ff, ne, k, bias=True, gate_row=True)
    h = orc.synth_normal(SEED, 160 + nt, 1.0, nt * e).reshape(nt, e)
    out, sels, wts = ctx.moe_block(0, h, want_routing=True)
    assert check_block(orc, L, h, out, sels, wts)[0] <= (5e-5 if nt < 16 else 2e-4)


@pytest.mark.parametrize("name,segments", [("Q4_K", 48), ("IQ3_XXS", 47)])
def test_tcgen05_many_items(orc, ctx, name, segments):
    """grouped_tc.cu: more items than a CTA has in its table (40 on 148 SMs), in a last round that is full or not; the same experts in turn."""
    from denno_beta_b200 import cuda as cu

    ty, k, n, m = orc.TYPE_BY_NAME[name], 256, 32768, 4
    assert ctx.moe_config(1, k, n, 2, 1)
    w = orc.synth_blocks(ty, SEED, 150 + ty, 2 * n * k // orc.blck_size(ty))
    assert ctx.register_experts(0, cu.GATE, ty, k, n, 2, w)
    segs = np.array([[i % 2, m, i * m, i * m] for i in range(segments)], np.uint32)
    x = orc.synth_normal(SEED, 151, 1.0, segments * m * k).reshape(-1, k)
    ctx.profile(True)
    got = cu.moe_grouped_gemm_layer(ctx, 0, cu.GATE, segs, x, n)
    launched = ctx.profile_read()
    ctx.profile(False)
    assert "tc_down" in launched, sorted(launched)
    assert rel_err(got, orc.grouped_gemm(ty, w, k, n, segs, x)) <= 2e-5


FIRST_CALLS = """
import threading
import numpy as np
from denno_beta_b200 import cuda as cu

k, n, threads = 1024, 512, 6
rng = np.random.default_rng(1)
w = rng.integers(0, 256, n * k // 256 * 98, dtype=np.uint8)
w.reshape(-1, 98)[:, :2] = np.array([0.01], np.float16).view(np.uint8)
x = rng.standard_normal(k).astype(np.float32)
start, got = threading.Barrier(threads), [None] * threads

def first_call(i):
    c = cu.CudaCtx(0)
    assert c.register_matrix(1, cu.IQ3_XXS, w, k, n)
    start.wait()
    outs = []
    for _ in range(2):
        outs.append(np.empty(n, np.float32))
        assert c.gemv(1, x, outs[-1])
    got[i] = outs
    c.close()

workers = [threading.Thread(target=first_call, args=(i,)) for i in range(threads)]
for t in workers:
    t.start()
for t in workers:
    t.join()
assert all(np.array_equal(o, got[0][1]) for outs in got for o in outs) and np.abs(got[0][1]).min() > 0
print("same")
"""


def test_first_calls_of_several_threads():
    """A process whose first IQ3_XXS calls come from several contexts at once: each finds the tables in place."""
    import subprocess
    import sys

    out = subprocess.run([sys.executable, "-c", FIRST_CALLS], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "same", out.stderr[-2000:]
