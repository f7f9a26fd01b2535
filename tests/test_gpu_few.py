"""Tiles of at most 8 tokens (prefill_few.cu): Q4_K and Q6_K products whose sub-block scales are applied to the sums of
single product steps. Bits of the oracle at the edges of a tile (one column pair, one half, full, one over), for either
type in either place, on codes and scales of the whole range."""
import numpy as np
import pytest

import pelica_b200 as pb
from pelica_b200 import synth
from tests.helpers import SMALL, bits_equal, device_pair, make_pair

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]

Q4, Q6 = synth.Q4_K, synth.Q6_K
TYPES = {"q4q4": (Q4, Q4), "q4q6": (Q4, Q6), "q6q4": (Q6, Q4), "q6q6": (Q6, Q6)}


@pytest.fixture(scope="module")
def ctx():
    c = pb.Context(0)
    yield c
    c.close()


def random_blocks(w, ty, rng):
    """Every code, sub-scale and min of the blocks at random, some blocks with all bits set; small f16 scales."""
    b = w.reshape(-1, 144 if ty == Q4 else 210)
    b[:] = rng.integers(0, 256, b.shape, dtype=np.uint8)
    b[::7] = 255
    d = np.array([1e-4, 3e-5], np.float16).view(np.uint8)
    if ty == Q4:
        b[:, :4] = d
    else:
        b[:, 208:] = d[:2]
        b[1::9, 192:208] = 128  # sub-scales of -128


def layer(oracle, ctx, types, seed, **change):
    cfg = SMALL["c2"].scaled(n_exp=40, type_gate=types[0], type_up=types[0], type_down=types[1], **change)
    W = synth.make_weights(cfg, seed)
    rng = np.random.default_rng(seed)
    for key, ty in (("gate", types[0]), ("up", types[0]), ("down", types[1])):
        random_blocks(W[key], ty, rng)
    return cfg, oracle.Layer(oracle.LayerDesc(**cfg.desc_fields()), W), pb.MoeLayer(ctx, cfg).load(W), rng


@pytest.mark.parametrize("T", [2, 4, 5, 8])
@pytest.mark.parametrize("types", sorted(TYPES))
def test_whole_layers(ctx, oracle, types, T):
    cfg, ol, gl, rng = layer(oracle, ctx, TYPES[types], 60 + T)
    x = synth.make_activations(T, cfg.d, 61)
    x[0] = rng.choice([-1.0, 1.0], cfg.d)  # every activation at the end of its range
    c0 = ctx.path_counts()
    got = gl.forward(x)
    assert ctx.path_counts()["tensor"] - c0["tensor"] == 2
    assert bits_equal(got, ol.forward(x))
    gl.close()


@pytest.mark.parametrize("most", [1, 7, 8, 9, 16, 17, 32, 33, 48, 49, 64, 65])
@pytest.mark.parametrize("shape", ["c6", "c7", "c8"])
def test_folds_of_32_value_blocks(ctx, oracle, shape, most):
    """The same products' cousins on 32-value blocks (prefill_q32.cu): every width of a fold and a last stage of one block
    (ff = 160), one expert with `most` tokens and others with a few."""
    cfg = SMALL[shape].scaled(n_exp=32)
    W = synth.make_weights(cfg, 90)
    ol, gl = oracle.Layer(oracle.LayerDesc(**cfg.desc_fields()), W), pb.MoeLayer(ctx, cfg).load(W)
    T, rng = max(most, 20), np.random.default_rng(90 + most)
    x = synth.make_activations(T, cfg.d, 91)
    ids = np.stack([rng.choice(np.arange(4, cfg.n_exp), cfg.top_k, replace=False) for _ in range(T)]).astype(np.uint32)
    ids[:most, 0] = 2
    w = rng.uniform(0.5, 1.5, ids.shape).astype(np.float32)
    c0 = ctx.path_counts()
    got = gl.experts(x, ids, w)
    assert ctx.path_counts()["tensor"] - c0["tensor"] == 2
    assert bits_equal(got, ol.experts(x, ids, w))
    gl.close()


@pytest.mark.parametrize("most", [1, 3, 8, 9, 20])
@pytest.mark.parametrize("shard", [False, True])
@pytest.mark.parametrize("types", ["q4q4", "q6q6"])
def test_groups_of_every_size(ctx, oracle, types, shard, most):
    """A given plan: `most` tokens on one expert (above 8: several tiles), one to three on the others; a shard holds some."""
    change = dict(first_local_expert=1, n_exp_local=30) if shard else {}
    cfg, ol, gl, rng = layer(oracle, ctx, TYPES[types], 70 + most, **change)
    T = 20
    x = synth.make_activations(T, cfg.d, 71)
    ids = np.stack([rng.choice(np.arange(4, cfg.n_exp), cfg.top_k, replace=False) for _ in range(T)]).astype(np.uint32)
    ids[:most, 0] = 2
    w = rng.uniform(0.5, 1.5, ids.shape).astype(np.float32)
    c0 = ctx.path_counts()
    got = gl.experts(x, ids, w)
    assert ctx.path_counts()["tensor"] - c0["tensor"] == 2
    assert bits_equal(got, ol.experts(x, ids, w))
    gl.close()


@pytest.mark.parametrize("T", [8, 24])
@pytest.mark.parametrize("types", ["q4q6", "q6q4", "q6q6"])
def test_rings_go_round(ctx, oracle, types, T):
    """Rows of six and five blocks (more than any ring has stages) and more items than CTAs: about 28 experts x 20 tiles of gate and up rows,
    12 of down rows on two CTAs an SM, so a CTA takes a second item and its rings go round within an item and across two."""
    gu, down = TYPES[types]
    cfg = SMALL["c2"].scaled(d=1536, ff=1280, n_exp=32, type_gate=gu, type_up=gu, type_down=down)
    ol, gl = device_pair(oracle, pb, ctx, cfg, 95)
    x = synth.make_activations(T, cfg.d, 96 + T)
    used = len(np.unique(gl.route(x)[0]))
    assert used * (cfg.d // 128) > 2 * 148 and T * cfg.top_k // cfg.n_exp <= 6
    c0 = ctx.path_counts()
    got = gl.forward(x)
    assert ctx.path_counts()["tensor"] - c0["tensor"] == 2
    assert bits_equal(got, ol.forward(x))
    gl.close()


@pytest.mark.parametrize("T", [3, 9, 20])
def test_received_rows_of_q6k_layers(ctx, oracle, T):
    """Rows that arrive quantised (the expert-parallel call, a world of one) against Q6_K gate and up matrices: the record comes twice, each with
    every other sub-block zero (24 to 160 rows on 24 experts)."""
    cfg = SMALL["c2"].scaled(type_gate=Q6, type_up=Q6)
    ol, gl, _ = make_pair(oracle, pb, ctx, cfg, 97)
    x = synth.make_activations(T, cfg.d, 98 + T)
    ep = pb.ExpertParallel(ctx, pb.ep_unique_id(), 0, 1)
    c0 = ctx.path_counts()
    got = ep.forward(gl, x)
    assert ctx.path_counts()["tensor"] - c0["tensor"] == 2
    assert bits_equal(got, ol.forward(x))
    ep.close()
    gl.close()


@pytest.mark.parametrize("T", [1, 3, 40])
@pytest.mark.parametrize("d", [4096, 4352, 12544])
def test_wide_stacks(ctx, oracle, d, T):
    """The combine step that norms the rows for the next layer: one round of its 1,024 threads (4096 columns), a second one, and
    rows that need more than 48 KB of shared memory (12,544)."""
    cfg = SMALL["c2"].scaled(d=d, ff=256, n_exp=6, top_k=2)
    pairs = [device_pair(oracle, pb, ctx, cfg, 100 + l) for l in range(3)]
    st = pb.Stack(ctx, [p[1] for p in pairs], eps=1e-6)
    st.set_mode(True)  # (one token: not the decode kernel)
    x = np.random.default_rng(d + T).normal(0, 1, (T, d)).astype(np.float32)
    want = oracle.stack_forward([p[0] for p in pairs], 1e-6, x)
    for _ in range(3 if T <= 16 else 1):  # launch by launch, recorded, replayed
        assert bits_equal(st.forward(x), want)
    st.close()
    for p in pairs:
        p[1].close()
