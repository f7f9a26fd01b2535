"""The edges of the tensor-core products' tiles: one and a few tokens, token tiles that are full, one over, or cut
into even parts, weight rows and K blocks that do not fill a tile, experts that another rank holds."""
import numpy as np
import pytest

import pelica_b200 as pb
from pelica_b200 import synth
from tests.helpers import SMALL, bits_equal, make_pair, tol_ok

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]


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
