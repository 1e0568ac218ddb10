"""Steps of more than 128 rows in the serving precision: the kernels that only such steps reach, at the sizes where their tiles end.

Bars as in the design's own test files: the serving precision differs from the oracle (which rounds what it caches to bf16) by cached
elements that land on the other side of a rounding boundary, and a near-tied router may pick another expert after one (`allow`)."""
import numpy as np
import pytest

import test_nifunex_gpu as N
import test_rofetar_gpu as R
import test_tozarax_gpu as T

pytestmark = pytest.mark.gpu


def check(mod, cfg, n, seed, allow=0.02):
    oracle, model = mod.build(cfg, seed=seed, dtype="bf16")
    toks = mod.tokens(cfg, n, seed=seed + 1)
    got = model.new_device_cache(2, 512).forward_ragged([0], [toks], [list(range(n))])
    assert np.isfinite(got).all()
    assert mod.relerr(got, oracle.run(toks), *([allow] if allow else [])) < mod.TOL["bf16"]


# rows just above the border; runs of exactly one tile, of a tile and a row, of several; experts without a row; every expert picked;
# hidden widths that end inside a tile of 128 and inside 16 columns
@pytest.mark.parametrize("n,experts,top,ff,width", [(129, 4, 2, 24, 64), (128 * 2 + 1, 2, 2, 136, 64), (256, 1, 1, 128, 64), (300, 37, 2, 40, 72), (200, 5, 5, 264, 64),
                                                    (384, 3, 1, 8, 128)])
def test_expert_runs(n, experts, top, ff, width):
    cfg = N.config([N.gla(heads=2, dim=16, vdim=16, mlp=N.moe(ff=ff, experts=experts, top=top, shared=(24, 0.75)))], vocab=64, width=width)
    check(N, cfg, n, 31)


@pytest.mark.parametrize("n,ff", [(129, 24), (260, 136)])
def test_expert_runs_without_a_gate(n, ff):
    check(T, T.config([T.layer(mlp=T.moe(experts=8, top=2, ff=ff))], width=64), n, 33)


# the gated epilogue with biases: hidden widths of one tile, a tile and eight columns, less than a tile
@pytest.mark.parametrize("n,ff,width", [(129, 24, 64), (130, 128, 64), (257, 136, 72), (300, 520, 128)])
def test_gated_epilogue(n, ff, width):
    cfg = R.config([R.att(mlp=R.dense(ff=ff))], vocab=64, width=width)
    check(R, cfg, n, 35, 0.0)
