"""MXFP4 products of small groups at the edges of their tiles: groups that fill one, two .. places of 8 tokens, one over,
and more than one tile, with five and with four pieces; rows of an odd number of blocks; a shard. Also whole calls on both
sides of the 8 tokens that one launch routes."""
import numpy as np
import pytest

import pelica_b200 as pb
from pelica_b200 import synth
from tests.helpers import SMALL, device_pair, make_pair, tol_ok

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]


@pytest.fixture(scope="module")
def ctx():
    c = pb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("T,most", [(30, 1), (30, 8), (30, 9), (30, 16), (30, 17), (70, 24), (70, 25), (70, 32), (70, 33), (70, 64)])
@pytest.mark.parametrize("shape", ["c3", "c3-odd", "c3-shard"])
def test_groups_of_every_size(ctx, oracle, shape, T, most):
    """A given plan: `most` tokens on one expert, a few on the others (f32 sums of another order below 32 tokens)."""
    cfg = {"c3": SMALL["c3"], "c3-odd": SMALL["c3"].scaled(d=288, ff=224),
           "c3-shard": SMALL["c3"].scaled(first_local_expert=1, n_exp_local=5)}[shape].scaled(n_exp=24 if shape != "c3-shard" else 8)
    ol, gl, _ = make_pair(oracle, pb, ctx, cfg, 86)
    rng = np.random.default_rng(T + most)
    x = synth.make_activations(T, cfg.d, 87)
    ids = np.stack([rng.choice(np.arange(3, cfg.n_exp), cfg.top_k, replace=False) for _ in range(T)]).astype(np.uint32)
    ids[:most, 0] = 2
    w = rng.uniform(0.5, 1.5, ids.shape).astype(np.float32)
    got, want = gl.experts(x, ids, w), ol.experts(x, ids, w)
    assert tol_ok(got, want), float(np.abs(got - want).max())
    if T < 32:
        assert float(np.abs(got - want).max()) < 4e-6 * float(np.sqrt((want.astype(np.float64) ** 2).mean()))
    gl.close()


@pytest.mark.parametrize("T", [3, 7, 8, 9])
@pytest.mark.parametrize("shape", ["c1", "c3", "c3-odd", "c4", "c4-q6", "c3-shard"])
def test_calls_around_the_one_launch_routing(ctx, oracle, shape, T):
    """Up to 8 tokens one launch routes and plans the call, above that two or more: the output is the oracle's either way."""
    cfg = {"c3-odd": SMALL["c3"].scaled(d=288, ff=224), "c4-q6": SMALL["c4"].scaled(type_gate=synth.Q6_K, type_up=synth.Q6_K),
           "c3-shard": SMALL["c3"].scaled(first_local_expert=2, n_exp_local=4)}.get(shape) or SMALL[shape]
    ol, gl, _ = make_pair(oracle, pb, ctx, cfg, 88)
    x = synth.make_activations(T, cfg.d, 89 + T)
    got, want = gl.forward(x), ol.forward(x)
    if shape.startswith("c3"):
        assert tol_ok(got, want)
        assert float(np.abs(got - want).max()) < 4e-6 * float(np.sqrt((want.astype(np.float64) ** 2).mean()))
    else:
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    gl.close()


@pytest.mark.parametrize("d", [4096, 4608, 12544])
def test_wide_stacks_of_parts(ctx, oracle, d):
    """One token through a stack: down products cut along K, whose parts the combine step adds before it norms the row for the next
    layer (one and two rounds of its threads, and more than 48 KB of shared memory)."""
    cfg = SMALL["c3"].scaled(d=d, ff=1120 if d < 8192 else 2080, n_exp=4, top_k=1)
    pairs = [device_pair(oracle, pb, ctx, cfg, 110 + l) for l in range(3)]
    st = pb.Stack(ctx, [p[1] for p in pairs], eps=1e-6)
    x = np.random.default_rng(d).normal(0, 1, (1, d)).astype(np.float32)
    got, want = st.forward(x), oracle.stack_forward([p[0] for p in pairs], 1e-6, x)
    assert tol_ok(got, want), float(np.abs(got - want).max())
    assert float(np.abs(got - want).max()) < 4e-6 * float(np.sqrt((want.astype(np.float64) ** 2).mean()))
    st.close()
    for p in pairs:
        p[1].close()
