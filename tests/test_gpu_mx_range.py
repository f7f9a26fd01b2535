"""MXFP4 products at the ends of the number range: each of the tensor-core kernels (five and four fp8 pieces, two bf16 pieces)
against the oracle and the row kernels."""
import numpy as np
import pytest

import pelica_b200 as pb
from pelica_b200 import synth
from tests.helpers import SMALL, mx_tile, tol_ok

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]


@pytest.fixture(scope="module")
def ctx():
    """A context that nobody has given a threshold: the default choice of kernels."""
    c = pb.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def rows_ctx():
    c = pb.Context(0)
    c.set_tensor_core_min_tokens(0)
    yield c
    c.close()


# tokens -> tokens of a tile of the kernel that a call of 8 experts, 4 a token, takes
TILES = {1: 16, 3: 16, 5: 16, 31: 16, 40: 32, 150: 32, 200: 128}


def codes(W, key, cfg):
    """[expert][row][block][17] of a matrix: the scale byte, then 16 bytes of codes."""
    rows, cols = (cfg.d, cfg.ff) if key == "down" else (cfg.ff, cfg.d)
    return W[key].reshape(cfg.n_exp, rows, cols // 32, 17)


def layers(oracle, ctx, rows_ctx, cfg, W):
    return (oracle.Layer(oracle.LayerDesc(**cfg.desc_fields()), W), pb.MoeLayer(ctx, cfg).load(W),
            pb.MoeLayer(rows_ctx, cfg).load(W))


def picks(T, cfg):
    """Expert ids spread evenly and weights that sum to one: the products without the router in front."""
    ids = (np.arange(T)[:, None] + np.arange(cfg.top_k)[None, :] * (cfg.n_exp // cfg.top_k)) % cfg.n_exp
    w = np.random.default_rng(T).uniform(0.5, 1.5, ids.shape).astype(np.float32)
    return ids.astype(np.uint32), w / w.sum(1, keepdims=True)


def agree(got, want):
    """Infinities and NaN where the reference has them, the rest within the layer tolerance."""
    fin = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
    assert tol_ok(got[fin], want[fin]), float(np.abs(got[fin] - want[fin]).max())


@pytest.mark.parametrize("T", [1, 5, 40, 200])
def test_activations_that_round_up_past_the_largest_float(ctx, rows_ctx, oracle, T):
    """|x| of 1.94 * 2^127 and more is 256 units of its first piece, 2^128: the pieces behind it still hold what is missing
    (3 % without them). The column meets codes of 0.5 in gate (no overflow in the row kernels either) and 0 in up."""
    cfg = SMALL["c3"].scaled(act_limit=3e38)
    assert mx_tile(pb, cfg, T) == TILES[T]
    W = synth.make_weights(cfg, 91)
    for key, code in (("gate", 1), ("up", 0)):
        c = codes(W, key, cfg)
        c[:, :, 2, 0] = 90                             # 2^-37: what comes out stays far from overflow
        c[:, :, 2, 1] = (c[:, :, 2, 1] & 0xF0) | code  # value 0 of block 2: the low nibble
    ol, gl, gr = layers(oracle, ctx, rows_ctx, cfg, W)
    x = synth.make_activations(T, cfg.d, 92)
    x[:, 64] = 3.4028234e38
    x[0, 64] = 3.31e38
    x[T // 2 + 1:, 64] *= -1
    ids, w = picks(T, cfg)
    want = ol.experts(x, ids, w)
    assert np.isfinite(want).all() and np.abs(want).max() > 1e20
    agree(gr.experts(x, ids, w), want)
    agree(gl.experts(x, ids, w), want)
    gl.close()
    gr.close()


@pytest.mark.parametrize("shape", ["c3", "c3-wide"])
@pytest.mark.parametrize("T", [1, 5, 31, 40, 150, 200])
def test_activations_that_are_no_finite_number(ctx, rows_ctx, oracle, T, shape):
    """One infinity (or NaN) in a 32-value block spoils the sums that f32 arithmetic spoils and no others: inf where it meets a
    weight, NaN where it meets a zero or its opposite. 0.03 of the codes of its column are zeros here, so most sums are
    infinite and the clamp of the activation makes them finite again."""
    cfg = SMALL["c3"] if shape == "c3" else SMALL["c3"].scaled(d=288, ff=1120)
    assert mx_tile(pb, cfg, T) == TILES[T]
    W = synth.make_weights(cfg, 93)
    rng = np.random.default_rng(94)
    for key in ("gate", "up"):
        c = codes(W, key, cfg)
        low = np.where(rng.random(c.shape[:2]) < 0.03, 0, rng.integers(1, 8, c.shape[:2]) | 8 * rng.integers(0, 2, c.shape[:2]))
        c[:, :, 1, 4] = (c[:, :, 1, 4] & 0xF0) | low  # value 3 of block 1: x[35]
    ol, gl, gr = layers(oracle, ctx, rows_ctx, cfg, W)
    x = synth.make_activations(T, cfg.d, 95)
    x[0, 35] = np.inf
    if T > 4:
        x[2, 35] = -np.inf
        x[2, 36] = np.inf
        x[3, 35] = np.nan
        x[T - 1, 35] = -np.inf
    ids, w = picks(T, cfg)
    with np.errstate(all="ignore"):
        want = ol.experts(x, ids, w)
        agree(gr.experts(x, ids, w), want)
        agree(gl.experts(x, ids, w), want)
        # the down products meet them in h
        h_inf = cfg.scaled(act_limit=np.inf)
        ol2, gl2, gr2 = layers(oracle, ctx, rows_ctx, h_inf, W)
        want = ol2.experts(x, ids, w)
        assert not np.isfinite(want).all()
        agree(gr2.experts(x, ids, w), want)
        agree(gl2.experts(x, ids, w), want)
    for g in (gl, gr, gl2, gr2):
        g.close()


@pytest.mark.parametrize("e", [0, 1, 2, 129, 249, 250, 253, 254, 255])
@pytest.mark.parametrize("T", [3, 40, 150, 200])
def test_scale_bytes_of_the_whole_range(ctx, rows_ctx, oracle, T, e):
    """A gate matrix whose blocks all have scale byte e, against activations that bring its sums back into range: fp8 products
    (3 tokens: five pieces, 40 and 150: four), bf16 products (200: a weight of 2^128 is none; an odd number of blocks a row). 255 is 2^128 as in
    the row kernels: codes of 1 and more are infinite, 0.5 is 2^127."""
    cfg = SMALL["c3"].scaled(act_limit=1e30, d=288 if T == 200 else 320)
    assert mx_tile(pb, cfg, T) == TILES[T]
    W = synth.make_weights(cfg, 96)
    c = codes(W, "gate", cfg)
    c[..., 0] = e
    if e == 255:  # finite sums: codes of 0 and 0.5 only
        c[..., 1:] &= 0x99
    ol, gl, gr = layers(oracle, ctx, rows_ctx, cfg, W)
    x = synth.make_activations(T, cfg.d, 97) * np.float32(2.0) ** int(np.clip(120 - e, -100, 60))
    ids, w = picks(T, cfg)
    want = ol.experts(x, ids, w)
    assert np.isfinite(want).all() and want.any()
    agree(gr.experts(x, ids, w), want)
    got = gl.experts(x, ids, w)
    agree(got, want)
    if T < 32:
        rms = float(np.sqrt((want.astype(np.float64) ** 2).mean()))
        assert float(np.abs(got - want).max()) < 4e-6 * rms
    gl.close()
    gr.close()
