"""The edges of the tensor-core products' tiles: one and a few tokens, token tiles that are full, one over, or cut
into even parts, weight rows and K blocks that do not fill a tile, experts that another rank holds."""
import numpy as np
import pytest

import pelica_b200 as pb
from pelica_b200 import synth
from tests.helpers import SMALL, bits_equal, make_pair, mx_tile, tol_ok

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]


@pytest.fixture(scope="module")
def ctx():
    """A context that nobody has given a threshold: the default choice of kernels."""
    c = pb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("T", [2, 5, 33, 70, 300])
@pytest.mark.parametrize("shape", ["c6", "c7", "c8", "c7-shard", "c6-f16"])
def test_32_value_blocks(ctx, oracle, shape, T):
    """Q8_0 / IQ4_NL / IQ4_XS weights on int8 blocks of 32: the bits of the row kernels. ff = 160: five blocks a row (a
    last stage of one), 64-row tiles that the matrix half fills."""
    cfg = {"c7-shard": SMALL["c7"].scaled(first_local_expert=4, n_exp_local=8),
           "c6-f16": SMALL["c6"].scaled(act_quant=synth.AQ_Q8_32_F16, d=288)}.get(shape) or SMALL[shape]
    ol, gl, _ = make_pair(oracle, pb, ctx, cfg, 81)
    x = synth.make_activations(T, cfg.d, 900 + T)
    c0 = ctx.path_counts()
    got = gl.forward(x)
    c1 = ctx.path_counts()
    assert c1["tensor"] - c0["tensor"] == 2 and c1["general"] == c0["general"]
    assert bits_equal(got, ol.forward(x))
    gl.close()


@pytest.mark.parametrize("T", [1, 2, 5, 31, 32, 40, 150, 200])
@pytest.mark.parametrize("shape", ["c3", "c3-shard", "c3-wide", "c3-2048", "c3-2080"])
def test_mxfp4(ctx, oracle, shape, T):
    """MXFP4 weights and f32 activations: five (below 32 tokens) or four fp8 pieces in tiles of 16 or 32 tokens, two bf16 pieces in tiles
    of 128 (200 tokens; 150 too of a shard, which holds half of the experts, and of the widest shapes). ff = 160: a last stage of one block; the wider shapes cut the down products of a few tokens along K, into two parts
    (ff = 1120), four (2048: 16 stages) and three (2080: 17); calls of fewer than 32 tokens keep f32 precision."""
    cfg = {"c3-shard": SMALL["c3"].scaled(first_local_expert=2, n_exp_local=4),
           "c3-wide": SMALL["c3"].scaled(d=288, ff=1120), "c3-2048": SMALL["c3"].scaled(d=288, ff=2048),
           "c3-2080": SMALL["c3"].scaled(d=288, ff=2080)}.get(shape) or SMALL[shape]
    tile = mx_tile(pb, cfg, T)
    assert tile == (16 if T < 32 else 128 if T == 200 or (T == 150 and shape in ("c3-shard", "c3-2048", "c3-2080")) else 32)
    ol, gl, _ = make_pair(oracle, pb, ctx, cfg, 82)
    x = synth.make_activations(T, cfg.d, 950 + T)
    x[0, :32] *= 1e-12  # blocks of very different sizes, and one of zeros
    x[T - 1, 32:64] = 0.0
    c0 = ctx.path_counts()
    got = gl.forward(x)
    c1 = ctx.path_counts()
    assert c1["tensor"] - c0["tensor"] == 2 and c1["general"] == c0["general"]
    want = ol.forward(x)
    assert tol_ok(got, want), float(np.abs(got - want).max())
    # four pieces hold a value to 2^-19 = 1.9e-6 of its block's largest, 3e-6 of the RMS at most of N(0, 1) blocks: two products of independent errors of that
    # size spread over the sum, five deviations out, stay below 1e-5 (2.8e-6 seen); three pieces would be at 32 times that, two bf16 pieces at 2.4e-5
    if tile < 128:
        rms = float(np.sqrt((want.astype(np.float64) ** 2).mean()))
        assert float(np.abs(got - want).max()) < (4e-6 if T < 32 else 1e-5) * rms
    gl.close()


@pytest.mark.parametrize("T", [1, 7, 8, 9, 32, 33, 70, 130, 260])
@pytest.mark.parametrize("shape", ["c1", "c2", "c4", "c4-shard"])
def test_q8x_blocks_and_plan(ctx, oracle, shape, T):
    """Q4_K / Q6_K products in both shapes of the kernel (2 to 130 pairs a group: one to four passes, tiles that are
    full and one over), the shared expert as a group of the same launches; routing and plan on either side of
    8 tokens (one launch / a router of tiles) and of 32 (one segment / several): bits of the oracle."""
    cfg = SMALL["c4"].scaled(first_local_expert=8, n_exp_local=16) if shape == "c4-shard" else SMALL[shape]
    ol, gl, _ = make_pair(oracle, pb, ctx, cfg, 83)
    x = synth.make_activations(T, cfg.d, 970 + T)
    ids, w = gl.route(x)
    ids_o, w_o = ol.route(x)
    assert np.array_equal(ids, ids_o) and bits_equal(w, w_o)
    c0 = ctx.path_counts()
    got = gl.forward(x)
    c1 = ctx.path_counts()
    # one token takes the row kernels where no shared expert joins the launches
    kind, other = ("general", "tensor") if T == 1 and not cfg.shared else ("tensor", "general")
    assert c1[kind] - c0[kind] == 2 and c1[other] == c0[other]
    assert bits_equal(got, ol.forward(x))
    # rows that start 4 bytes off a 16-byte boundary take other loads, not other values
    xd, yd = ctx.alloc(x.nbytes + 16), ctx.alloc(x.nbytes + 16)
    xd.upload(np.concatenate([np.zeros(1, np.float32), x.ravel(), np.zeros(3, np.float32)]))
    pb._check(gl.lib.pm_moe_forward(gl.h, xd.ptr + 4, T, yd.ptr + 4, 0))
    ctx.sync()
    got = yd.download(np.float32, (x.size + 4,))[1:1 + x.size].reshape(x.shape)
    assert bits_equal(got, ol.forward(x))
    xd.free()
    yd.free()
    gl.close()


def test_workspace_of_a_long_mxfp4_prompt():
    """The pieces of a prompt take 4.25 bytes a value of workspace (four fp8 pieces and their scales; two bf16 pieces take
    4): the five pieces of short calls are not kept room for."""
    cfg, T = synth.C3_GPTOSS, 2048
    c = pb.Context(0)
    gl = pb.MoeLayer(c, cfg).fill_synthetic(5)
    x, y = c.alloc(4 * T * cfg.d), c.alloc(4 * T * cfg.d)
    before = c.device_free_bytes()
    gl.forward_dev(x, T, y)
    c.sync()
    used = before - c.device_free_bytes()
    P = T * cfg.top_k
    # h f32 and its quantised forms (5.5 bytes), pair outputs, the tokens' quantised forms, the pieces of whole 128-value stages, room to stage x and y
    need = P * cfg.ff * 5.5 + P * cfg.d * 4 + T * cfg.d * 2 + (P + 16 * cfg.n_exp) * 2944 * 4.25 + 2 * T * cfg.d * 4
    assert used < 1.125 * need + (8 << 20), (used, need)  # (the workspace grows by an eighth more than asked for)
    for b in (x, y):
        b.free()
    gl.close()
    c.close()


@pytest.mark.parametrize("shape", ["c2", "c4", "c8"])
def test_split_calls_choose_by_their_own_size(ctx, oracle, shape):
    """Rows and plans served for somebody else, and the shared expert alone: up to 16 pairs (4 tokens of the one shared
    expert) on the row kernels, more on the tensor cores; the same bits."""
    cfg = SMALL[shape]
    ol, gl, _ = make_pair(oracle, pb, ctx, cfg, 84)

    def kinds(call):
        c0 = ctx.path_counts()
        got = call()
        c1 = ctx.path_counts()
        return got, c1["general"] - c0["general"], c1["tensor"] - c0["tensor"]

    rng = np.random.default_rng(85)
    for R in (1, 16, 17):
        x = synth.make_activations(R, cfg.d, 980 + R)
        eids, w = rng.integers(0, cfg.n_exp, R).astype(np.uint32), rng.uniform(0.5, 1.5, R).astype(np.float32)
        got, row, tensor = kinds(lambda: gl.experts_rows(x, eids, w))
        assert (row, tensor) == ((0, 2) if R > 16 else (2, 0))
        for r in range(R):  # row r of a plan whose first pick is the row's expert
            ids = np.array([[eids[r]] + [e for e in range(cfg.n_exp) if e != eids[r]][:cfg.top_k - 1]], np.uint32)
            at = int(oracle.plan(ids, cfg.n_exp)["pair_pos"].ravel()[0])
            assert bits_equal(got[r], ol.experts(x[r:r + 1], ids, np.full(ids.shape, w[r], np.float32))[at])
    for T in (1, 2, 3, 9):
        x = synth.make_activations(T, cfg.d, 990 + T)
        ids, w = gl.route(x)
        got, row, tensor = kinds(lambda: gl.experts(x, ids, w))
        assert (row, tensor) == ((0, 2) if T * cfg.top_k > 16 else (2, 0))
        assert bits_equal(got, ol.experts(x, ids, w))
    if cfg.shared:
        for T in (1, 4, 5):
            x = synth.make_activations(T, cfg.d, 995 + T)
            got = gl.shared(x)
            ids, w = gl.route(x)
            assert bits_equal(gl.combine(gl.experts(x, ids, w), ids, w, got), ol.forward(x))
    gl.close()


@pytest.mark.parametrize("shape", ["q4q6", "q8_0"])
def test_split_calls_of_wide_layers(ctx, oracle, shape):
    """Up to 16 pairs the width decides: from 48 K pairs x (d + ff) on (here 8 pairs) rows and plans take the tensor cores; the same bits."""
    cfg = {"q4q6": SMALL["c2"], "q8_0": SMALL["c6"]}[shape].scaled(d=6144, ff=256, n_exp=6, top_k=2)
    ol, gl, _ = make_pair(oracle, pb, ctx, cfg, 86)
    rng = np.random.default_rng(87)
    for T, tensor in ((1, 0), (3, 0), (4, 2), (8, 2)):
        x = synth.make_activations(T, cfg.d, 940 + T)
        ids, w = gl.route(x)
        c0 = ctx.path_counts()
        got = gl.experts(x, ids, w)
        assert ctx.path_counts()["tensor"] - c0["tensor"] == tensor
        assert bits_equal(got, ol.experts(x, ids, w))
        x = synth.make_activations(2 * T, cfg.d, 945 + T)
        eids, w = rng.integers(0, cfg.n_exp, 2 * T).astype(np.uint32), rng.uniform(0.5, 1.5, 2 * T).astype(np.float32)
        c0 = ctx.path_counts()
        got = gl.experts_rows(x, eids, w)
        assert ctx.path_counts()["tensor"] - c0["tensor"] == tensor
        for r in range(2 * T):
            ids = np.array([[eids[r], (eids[r] + 1) % cfg.n_exp]], np.uint32)
            at = int(oracle.plan(ids, cfg.n_exp)["pair_pos"].ravel()[0])
            assert bits_equal(got[r], ol.experts(x[r:r + 1], ids, np.full(ids.shape, w[r], np.float32))[at])
    gl.close()
