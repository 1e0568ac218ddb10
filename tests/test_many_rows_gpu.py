"""Steps of more than 128 rows in the serving precision: the kernels that only such steps reach, at the sizes where their tiles end.

Bars as in the design's own test files: the serving precision differs from the oracle (which rounds what it caches to bf16) by cached
elements that land on the other side of a rounding boundary, and a near-tied router may pick another expert after one (`allow`)."""
import os
import re
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import test_medulorn_gpu as M
import test_nifunex_gpu as N
import test_rofetar_gpu as R
import test_tozarax_gpu as T
import test_tufazen_gpu as U

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


@pytest.mark.parametrize("n", [60, 150])
def test_rows_that_are_not_numbers(n):
    """a token whose embedding overflows: its row's scores are no numbers, yet its choices are experts (they index the row
    lists); the other sequence does not notice"""
    def overflow(w):
        w["embed"][5, :] = np.inf
    cfg = N.config([N.gla(heads=2, dim=16, vdim=16, mlp=N.moe(ff=24, experts=5, top=3))], vocab=64, width=64)
    _, model = N.build(cfg, seed=97, dtype="bf16", tweak=overflow)
    good = [6 + t % 58 for t in N.tokens(cfg, n, seed=98)]
    bad = good[:n - 20] + [5] * 20
    cache = model.new_device_cache(2, 256)
    got = cache.forward_ragged([0, 1], [good, bad], [list(range(n)), list(range(n))])
    alone = N.run_cut(model, good, [100, 100], cache=model.new_device_cache(1, 256))
    assert N.relerr(got[:n], np.asarray(alone, dtype=np.float64)) < CHUNK_TOL
    assert np.isfinite(got[n:n + min(64, n - 20)]).all()


# expert results of one to four slices of K (hidden widths of 8 to 44 k blocks), k blocks that do not go evenly into them; one column tile of 256, three whole
# ones, two and a piece; runs of uneven length, an expert that few rows pick
@pytest.mark.parametrize("n,ff,experts,width", [(129, 520, 5, 64), (129, 1030 * 2, 8, 64), (300, 1536, 3, 64), (140, 2824, 2, 64), (260, 1536, 5, 768), (131, 2056, 19, 520)])
def test_expert_results_in_slices(n, ff, experts, width):
    cfg = N.config([N.gla(heads=2, dim=16, vdim=16, mlp=N.moe(ff=ff, experts=experts, top=2))], vocab=64, width=width)
    check(N, cfg, n, 37, 0.0)


@pytest.mark.parametrize("n,ff", [(129, 24), (260, 136)])
def test_expert_runs_without_a_gate(n, ff):
    check(T, T.config([T.layer(mlp=T.moe(experts=8, top=2, ff=ff))], width=64), n, 33)


# the gated epilogue with biases: hidden widths of one tile, a tile and eight columns, less than a tile
@pytest.mark.parametrize("n,ff,width", [(129, 24, 64), (130, 128, 64), (257, 136, 72), (300, 520, 128)])
def test_gated_epilogue(n, ff, width):
    cfg = R.config([R.att(mlp=R.dense(ff=ff))], vocab=64, width=width)
    check(R, cfg, n, 35, 0.0)


# ---- recurrences in chunks of 64 tokens (portions from LINE on) against the same model fed in portions that stay token by token ------
_LINE = {k: int(v) for k, v in re.findall(r"kCsMinTokens(\w+) = (\d+)", (Path(__file__).resolve().parent.parent / "fastllm_b200/csrc/chunk_scan.cuh").read_text())}
LINE = {"gla": _LINE["Gla"], "gla_fast_decay": _LINE["Gla"], "mamba": _LINE["One"], "lightning": _LINE["One"], "delta": _LINE["Delta"]}
SERIAL = 60                 # tokens of a portion that no recurrence takes in chunks
assert SERIAL < min(LINE.values())
# No cache is rounded in these models, so what is left between the two is the order of f32 sums in the recurrence and in the GEMMs around
# it: a few 1e-7 per sum, some tens of sums and norms behind one another.
CHUNK_TOL = 3e-5


def tags_of(run):
    """kernels that `run` launched, by the profiler's tags"""
    from fastllm_b200 import models
    models.prof_begin()
    out = run()
    return out, {p["kernel"] for p in models.prof_end()}


def in_portions(mod, model, toks, size=SERIAL):
    """token by token: portions below every line"""
    out, tags = tags_of(lambda: mod.run_cut(model, toks, [size] * (len(toks) // size + 1), cache=model.new_device_cache(2, max(512, len(toks) + 8))))
    assert not any("chunks" in t for t in tags)
    return np.asarray(out, dtype=np.float64)


def in_chunks(run):
    out, tags = tags_of(run)
    assert any("chunks" in t for t in tags)
    return out


def recurrent(kind, dim, vdim, heads=2):
    if kind == "gla":
        return N, N.config([N.gla(heads=heads, dim=dim, vdim=vdim, tau=2.0, rank=4)], width=64)
    if kind == "gla_fast_decay":
        return N, N.config([N.gla(heads=heads, dim=dim, vdim=vdim, tau=0.05, rank=4)], width=64)
    if kind == "mamba":
        return R, R.config([R.mamba(heads=2 * heads, vdim=vdim, state=dim, groups=heads)], width=64)
    return R, R.config([R.delta(heads=2 * heads, kv_heads=heads, dim=dim, vdim=vdim)], width=64)


# tokens behind the kind's line: whole chunks, a last one of 63 tokens, of one, of 57 to 9
@pytest.mark.parametrize("kind", ["gla", "gla_fast_decay", "mamba", "delta"])
@pytest.mark.parametrize("dim,vdim,more", [(16, 16, 0), (64, 64, 63), (68, 36, 1), (128, 68, 64), (100, 128, 121), (4, 132, 73)])
def test_chunks_equal_token_by_token(kind, dim, vdim, more):
    mod, cfg = recurrent(kind, dim, vdim)
    _, model = mod.build(cfg, seed=41, dtype="bf16")
    n = LINE[kind] + more
    toks = mod.tokens(cfg, n, seed=42)
    serial = in_portions(mod, model, toks)
    whole = in_chunks(lambda: mod.run_whole(model, toks, cache=model.new_device_cache(2, 512)))
    assert mod.relerr(whole, serial) < CHUNK_TOL
    if more >= 40:      # a portion of chunks behind a short one, and a short one behind it: the state passes both borders
        cut = in_chunks(lambda: mod.run_cut(model, toks, [30, n - 40], cache=model.new_device_cache(2, 512)))
        assert mod.relerr(cut, serial) < CHUNK_TOL


@pytest.mark.parametrize("kind", ["mamba", "delta"])
@pytest.mark.parametrize("dim,vdim", [(128, 64), (64, 40), (20, 36), (6, 10), (256, 32)])
def test_token_by_token_in_any_cut(kind, dim, vdim):
    """the serial recurrences bring four tokens at a time, rows of 16-byte pieces or not, heads of one to several pieces a lane: portions of every
    remainder give the bits of the whole prompt, in the exact mode, and the oracle's numbers"""
    mod, cfg = recurrent(kind, dim, vdim)
    oracle, model = mod.build(cfg, seed=57)
    toks = mod.tokens(cfg, 41, seed=58)
    whole = mod.run_whole(model, toks, cache=model.new_device_cache(2, 64))
    assert mod.relerr(whole, oracle.run(toks)) < mod.TOL["f32"]
    assert np.array_equal(whole, mod.run_cut(model, toks, [1, 2, 3, 4, 5, 12, 14], cache=model.new_device_cache(2, 64)))


# the first lengths that go in chunks and a token more, a last chunk of 63 tokens
@pytest.mark.parametrize("kind,more", [("gla", 0), ("gla", 1), ("gla", 63), ("gla_fast_decay", 127), ("mamba", 0), ("mamba", 1), ("delta", 0), ("delta", 63)])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (68, 132), (16, 20)])
def test_first_lengths_in_chunks(kind, more, dim, vdim):
    """against portions of 60 tokens, which no recurrence takes in chunks; a token less stays token by token"""
    mod, cfg = recurrent(kind, dim, vdim)
    _, model = mod.build(cfg, seed=81, dtype="bf16")
    n = LINE[kind] + more
    toks = mod.tokens(cfg, n, seed=82)
    whole = in_chunks(lambda: mod.run_whole(model, toks, cache=model.new_device_cache(2, 512)))
    assert mod.relerr(whole, in_portions(mod, model, toks)) < CHUNK_TOL
    if more == 0:
        _, tags = tags_of(lambda: mod.run_whole(model, toks[:-1], cache=model.new_device_cache(2, 512)))
        assert not any("chunks" in t for t in tags)


@pytest.mark.parametrize("groups,state,vdim", [(4, 128, 64), (1, 128, 68), (8, 64, 132), (4, 20, 36)])
def test_chunks_of_four_heads(groups, state, vdim):
    """heads that read the same queries and keys share a block by fours; 34 chunks: 32 at a time, whose 256 blocks of four heads go together in the last kernel too,
    then two, whose 16 blocks would leave SMs idle there and take one head each"""
    cfg = R.config([R.mamba(heads=32, vdim=vdim, state=state, groups=groups)], width=64)
    _, model = R.build(cfg, seed=83, dtype="bf16")
    toks = R.tokens(cfg, 2118, seed=84)
    whole = in_chunks(lambda: R.run_whole(model, toks, cache=model.new_device_cache(1, 2176)))
    assert R.relerr(whole, in_portions(R, model, toks)) < CHUNK_TOL


@pytest.mark.parametrize("kind", ["gla", "mamba", "delta"])
def test_chunks_of_several_sequences(kind):
    """two prompts of more chunks than are held at a time beside a short one and a decoded token; a reused slot starts from zero"""
    mod, cfg = recurrent(kind, 32, 32)
    _, model = mod.build(cfg, seed=43, dtype="bf16")
    lens = (1100, 3, 1090, 1)
    reqs = [mod.tokens(cfg, k, seed=50 + i) for i, k in enumerate(lens)]
    cache = model.new_device_cache(4, 1536)
    for round_ in range(2):
        got = in_chunks(lambda: cache.forward_ragged([2, 0, 3, 1], reqs, [list(range(k)) for k in lens]))
        at = 0
        for r, k in zip(reqs, lens):
            assert mod.relerr(got[at:at + k], in_portions(mod, model, r)) < CHUNK_TOL
            at += k
        for s in range(4):
            cache.slot_reset(s)


@pytest.mark.parametrize("kind", ["gla", "gla_fast_decay", "mamba", "delta"])
@pytest.mark.parametrize("dim,vdim,more", [(64, 64, 77), (100, 36, 8)])
def test_chunks_against_the_oracle(kind, dim, vdim, more):
    mod, cfg = recurrent(kind, dim, vdim)
    in_chunks(lambda: check(mod, cfg, LINE[kind] + more, 47, 0.0))


@pytest.mark.parametrize("dim,vdim,more", [(16, 24, 0), (128, 128, 8), (64, 72, 141)])
def test_lightning_chunks(dim, vdim, more):
    in_chunks(lambda: check(M, M.config([M.par_layer(b=M.lightning(heads=2, dim=dim, vdim=vdim))], width=64), LINE["lightning"] + more, 45, 0.0))


# ---- grouped-query attention of a portion in one kernel ----------------------------------------------------------------------------------
def both_ways(mod, cfg, n, cuts, seed):
    oracle, model = mod.build(cfg, seed=seed, dtype="bf16")
    toks = mod.tokens(cfg, n, seed=seed + 1)
    ref = oracle.run(toks)
    assert mod.relerr(mod.run_whole(model, toks, cache=model.new_device_cache(2, 1024)), ref) < mod.TOL["bf16"]
    assert mod.relerr(mod.run_cut(model, toks, cuts, cache=model.new_device_cache(2, 1024)), ref) < mod.TOL["bf16"]


# head sizes on both sides of 64 and up to 128, keys and values alike or not; portions of one page, a page and a row, a query tile and a row;
# portions that start inside a page
@pytest.mark.parametrize("dim,vdim,n", [(8, 8, 64), (16, 72, 65), (64, 64, 129), (72, 24, 200), (128, 128, 300), (120, 64, 257)])
def test_attention_of_a_portion(dim, vdim, n):
    cfg = R.config([R.att(heads=4, kv_heads=2, dim=dim, vdim=vdim, rot_dims=8), R.att(heads=2, kv_heads=2, dim=dim, vdim=vdim, rot_dims=4, kv_from=0)], width=64)
    both_ways(R, cfg, n, [30, n - 31] if n >= 95 else [n - 1], 61)


# windows with kept first keys (inside the window's first page, over two pages, none) and chunks, each longer than the 256 keys up to which
# the per-row kernel is taken
@pytest.mark.parametrize("window,keep,n", [(257, 2, 400), (300, 70, 520), (321, 0, 450)])
def test_attention_windows_of_a_portion(window, keep, n):
    both_ways(M, M.config([M.par_layer(M.windowed(dim=16, vdim=16, window=window, keep=keep), M.lightning(heads=2, dim=8, vdim=8))], width=64), n, [70, 201, 100], 63)


def test_attention_chunks_of_a_portion():
    both_ways(M, M.config([M.attn_layer(M.chunked(dim=16, vdim=16, chunk=270), mlp=None)], width=64), 600, [100, 300], 65)


@pytest.mark.parametrize("dim,dims", [(16, 8), (24, 24), (128, 40)])
def test_attention_with_gates_and_shared_values(dim, dims):
    both_ways(U, U.bare([U.alayer(U.grouped(dim=dim, dims=dims))], width=64), 200, [77, 100], 67)


def test_attention_sharp_scores():
    """scores far apart: the running maximum moves and the accumulator is rescaled"""
    both_ways(R, R.config([R.att(heads=2, kv_heads=1, dim=32, vdim=32, rot_dims=8, scale=6.0, softcap=None)], width=64), 300, [130, 100], 69)


# ---- the exact mode's GEMM -----------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("width,ff", [(64, 72), (50, 34), (36, 130), (33, 71)])
def test_exact_gemm_rows_stand_alone(width, ff):
    """f64 sums whose order depends on K alone: bitwise the same logits whether a token's row shares its tile with 7, 15, 16, 31, 32 others or
    with none, aligned rows or not"""
    cfg = R.config([R.delta(heads=4, kv_heads=2, dim=6, vdim=10, mlp=R.dense(ff=ff)), R.att(heads=4, kv_heads=2, dim=8, vdim=12, mlp=R.dense(ff=ff))], vocab=101, width=width)
    oracle, model = R.build(cfg, seed=71)
    toks = R.tokens(cfg, 110, seed=72)
    whole = R.run_whole(model, toks, cache=model.new_device_cache(2, 128))
    assert R.relerr(whole, oracle.run(toks)) < R.TOL["f32"]
    assert np.array_equal(whole, R.run_cut(model, toks, [1, 8, 9, 16, 17, 32, 2], cache=model.new_device_cache(2, 128)))


@pytest.mark.parametrize("width,ff", [(1032, 1544), (1028, 770), (550, 2050), (547, 1033), (1034, 1553)])
def test_exact_gemm_long_sums(width, ff):
    """sums of more chunks than a warp keeps on their way (above 512 columns), the last chunk a half or less, rows of W aligned for copies of 16, 8 or 4
    bytes or for none; tiles of 8 and of 16 rows"""
    cfg = R.config([R.delta(heads=4, kv_heads=2, dim=6, vdim=10, mlp=R.dense(ff=ff))], vocab=101, width=width)
    oracle, model = R.build(cfg, seed=73)
    toks = R.tokens(cfg, 48, seed=74)
    whole = R.run_whole(model, toks, cache=model.new_device_cache(2, 64))
    assert R.relerr(whole, oracle.run(toks)) < R.TOL["f32"]
    assert np.array_equal(whole, R.run_cut(model, toks, [1, 8, 16, 17, 6], cache=model.new_device_cache(2, 64)))


@pytest.mark.parametrize("width,ff", [(64, 72), (50, 34)])
def test_exact_expert_rows_stand_alone(width, ff):
    """the same for experts: 2, 8, 10, 16, 32, 34 and 128 picks in a step"""
    cfg = N.config([N.gla(heads=2, dim=6, vdim=10, mlp=N.moe(ff=ff, experts=5, top=2))], vocab=101, width=width)
    oracle, model = N.build(cfg, seed=75)
    toks = N.tokens(cfg, 64, seed=76)
    whole = N.run_whole(model, toks, cache=model.new_device_cache(2, 128))
    assert N.relerr(whole, oracle.run(toks)) < N.TOL["f32"]
    assert np.array_equal(whole, N.run_cut(model, toks, [1, 4, 5, 8, 16, 17], cache=model.new_device_cache(2, 128)))


def test_exact_head_rows_stand_alone():
    """the same for a matrix of so many columns that up to eight rows take other tiles than more"""
    cfg = R.config([R.delta(heads=4, kv_heads=2, dim=6, vdim=10)], vocab=8101, width=50)
    oracle, model = R.build(cfg, seed=77)
    toks = R.tokens(cfg, 40, seed=78)
    whole = R.run_whole(model, toks, cache=model.new_device_cache(2, 64))
    assert R.relerr(whole, oracle.run(toks)) < R.TOL["f32"]
    assert np.array_equal(whole, R.run_cut(model, toks, [1, 8, 9, 7, 14], cache=model.new_device_cache(2, 64)))


@pytest.mark.parametrize("dim", [8, 96])
def test_exact_attention_rows_stand_alone(dim):
    """the same for the preparation of heads (norm, rotation, cache append), in steps of more than 512 rows and of fewer"""
    cfg = R.config([R.att(heads=4, kv_heads=2, dim=dim, vdim=16, rot_dims=dim // 2)], vocab=64, width=64)
    oracle, model = R.build(cfg, seed=79)
    toks = R.tokens(cfg, 700, seed=80)
    whole = R.run_whole(model, toks, cache=model.new_device_cache(2, 768))
    assert R.relerr(whole, oracle.run(toks)) < R.TOL["f32"]
    assert np.array_equal(whole, R.run_cut(model, toks, [512, 3, 185], cache=model.new_device_cache(2, 768)))


# ---- convolutions in front of the recurrences, rows with a sliding window (blocks of 16 rows that fill the chip, four taps) -----------------------------------
@pytest.mark.parametrize("layer", [R.delta(heads=4, kv_heads=2, dim=32, vdim=24, conv=4), R.delta(heads=2, kv_heads=2, dim=128, vdim=132, conv=4),
                                   R.delta(heads=6, kv_heads=3, dim=64, vdim=8, conv=4), R.mamba(heads=4, vdim=12, state=20, groups=2, conv=4),
                                   R.mamba(heads=8, vdim=128, state=16, groups=1, conv=4)])
@pytest.mark.parametrize("long", [270, 2050])
def test_sliding_convolution(layer, long):
    """against the same model in portions that stay with the per-row kernel; several sequences per block, one that goes on, one of one token
    (270: the per-row kernel takes the mixed step too)"""
    cfg = R.config([layer], width=64)
    _, model = R.build(cfg, seed=81, dtype="bf16")
    reqs = [R.tokens(cfg, k, seed=82 + i) for i, k in enumerate((long, 5, 1, 33))]
    alone = [R.run_cut(model, r, [100] * 21, cache=model.new_device_cache(1, 2112)) for r in reqs]
    cache = model.new_device_cache(4, 2112)
    cache.forward_ragged([0], [reqs[0][:7]], [[]])
    got = cache.forward_ragged([3, 0, 2, 1], [reqs[1], reqs[0][7:], reqs[2], reqs[3]], [list(range(5)), list(range(long - 7)), [0], list(range(33))])
    want = np.concatenate([alone[1], alone[0][7:], alone[2], alone[3]])
    assert R.relerr(got, np.asarray(want, dtype=np.float64)) < CHUNK_TOL


@pytest.mark.parametrize("n,experts,top", [(130, 9, 4), (512, 3, 3)])
def test_expert_lists_of_many_picks(n, experts, top):
    """more than one round of 256 picks per list, lists that end on its border"""
    check(N, N.config([N.gla(heads=2, dim=16, vdim=16, mlp=N.moe(ff=24, experts=experts, top=top, shared=(24, 0.75)))], vocab=64, width=64), n, 91)


@pytest.mark.parametrize("scale", [-0.3, 0.0])
@pytest.mark.parametrize("softcap", [None, 4.0])
def test_attention_scale_of_any_sign(scale, softcap):
    """a scale of zero or below: masked scores stay masked, the maximum is that of the scaled scores"""
    both_ways(R, R.config([R.att(heads=2, kv_heads=1, dim=32, vdim=32, rot_dims=8, scale=scale, softcap=softcap)], width=64), 200, [130, 64], 73)
    both_ways(M, M.config([M.par_layer(M.windowed(dim=16, vdim=16, window=257, keep=2, scale=scale), M.lightning(heads=2, dim=8, vdim=8))], width=64), 400, [70, 201, 100], 74)


# ---- steps of single tokens, more than 128 of them: row runs inside a captured graph -----------------------------------------------------
def test_expert_runs_of_single_tokens():
    """run eagerly, captured, replayed and replayed with other tokens and routes; some sequences against the model alone"""
    n, cfg = 150, N.config([N.gla(heads=2, dim=16, vdim=16, mlp=N.moe(ff=24, experts=5, top=2))], vocab=64, width=64)
    _, model = N.build(cfg, seed=93, dtype="bf16")
    toks = [N.tokens(cfg, 5, seed=200 + i) for i in range(n)]
    cache = model.new_device_cache(n, 64)
    got = np.stack([cache.forward_ragged(list(range(n)), [t[k:k + 1] for t in toks], [[0]] * n) for k in range(5)], axis=1)
    for i in (0, 1, 77, 127, 128, 149):
        alone = N.run_cut(model, toks[i], [5], cache=model.new_device_cache(1, 64))
        assert N.relerr(got[i], np.asarray(alone, dtype=np.float64)) < CHUNK_TOL


# ---- dependent launch ------------------------------------------------------------------------------------------------------------------------
DEPENDENT_LAUNCH = r"""
import sys
import numpy as np
import test_many_rows_gpu as S
out = []
for mod, cfg in S.dependent_launch_cases():
    _, model = mod.build(cfg, seed=95, dtype="bf16")
    toks = [mod.tokens(cfg, k, seed=300 + k) for k in (1, 140, 30)]
    cache = model.new_device_cache(3, 256)
    out.append(cache.forward_ragged([0, 1, 2], toks, [[0], list(range(0, 140, 7)), [29]]).ravel())
    for k in range(4):                      # eager, captured, replayed
        out.append(cache.forward_ragged([2, 0, 1], [t[-1:] for t in toks], [[0]] * 3).ravel())
np.save(sys.argv[1], np.concatenate(out))
"""


def dependent_launch_cases():
    return [(N, N.hybrid_cfg()), (R, R.config([R.delta(heads=4, kv_heads=2, dim=32, vdim=24, conv=4, mlp=R.dense(ff=40)), R.att(heads=4, kv_heads=2, dim=16, vdim=16, rot_dims=8),
                                               R.mamba(heads=4, vdim=12, state=20, groups=2, conv=4)], width=64)),
            (T, T.config([T.layer(mlp=T.moe(experts=8, top=2, ff=24))], width=64)),
            (M, M.config([M.par_layer(M.windowed(dim=16, vdim=16, window=257, keep=2), M.lightning(heads=2, dim=8, vdim=8))], width=64)),
            (U, U.bare([U.alayer(U.grouped(dim=16, dims=8))], width=64))]


def test_dependent_launch_changes_nothing(tmp_path):
    """every kernel of a layered step waits for the one before: the same bits with and without dependent launch"""
    here = os.path.dirname(os.path.abspath(__file__))
    res = []
    for off in ("0", "1"):
        path = str(tmp_path / f"{off}.npy")
        env = {**os.environ, "FL_NO_PDL": off, "PYTHONPATH": os.pathsep.join([os.path.dirname(here), here])}
        subprocess.run([sys.executable, "-c", DEPENDENT_LAUNCH, path], check=True, env=env, cwd=here, timeout=300)
        res.append(np.load(path))
    assert np.isfinite(res[0]).all() and np.array_equal(res[0], res[1])


# ---- workspace: only what a step's path reads, grown between steps -----------------------------------------------------------------------------
@pytest.mark.parametrize("mod,cfg", [
    (N, N.config([N.gla(heads=2, dim=16, vdim=16, mlp=N.moe(ff=136, experts=5, top=2)), N.lat(mlp=N.dense(ff=1040))], vocab=64, width=64)),
    (N, N.config([N.gla(heads=2, dim=16, vdim=16, mlp=N.dense(ff=30)), N.gla(heads=2, dim=16, vdim=16, mlp=N.moe(ff=20, experts=5, top=2, shared=(30, 0.75)))], vocab=64, width=66)),
    (R, R.config([R.att(heads=4, kv_heads=2, dim=16, vdim=16, rot_dims=8, mlp=R.dense(ff=520)), R.delta(heads=4, kv_heads=2, dim=32, vdim=24, conv=4)], vocab=64, width=1024)),
    (T, T.config([T.layer(mlp=T.moe(experts=8, top=2, ff=136))], width=64, max_positions=1024))])
def test_steps_that_grow(mod, cfg):
    """a cache whose steps grow from one row to hundreds gives what a new one gives"""
    _, model = mod.build(cfg, seed=99, dtype="bf16")
    toks = mod.tokens(cfg, 700, seed=100)
    cache = model.new_device_cache(1, 1024)
    for n in (1, 40, 129, 300, 129, 700):
        cache.slot_reset(0)
        want = model.new_device_cache(1, 1024).forward_ragged([0], [toks[:n]], [[0, n - 1]])
        assert mod.relerr(cache.forward_ragged([0], [toks[:n]], [[0, n - 1]]), np.asarray(want, dtype=np.float64)) < CHUNK_TOL


# ---- GEMMs on pairs of SMs (gemm_pair.cuh): from 1024 rows on, where whole waves of pair tiles leave a few that are cut along K ------------------
def test_pairs_llama():
    """1290 rows: the last pair row ends inside its first half; o and gate|up leave 16 tiles to cut, which end inside a k block's run"""
    from fastllm_b200 import models
    from helpers import product_model
    from oracle import causal_lm as ocl
    from oracle import synth
    cfg = ocl.CausalLMConfig("llama", 3840, 1920, 1000, 1, 30, 5, 1e-5, 1e4, 1536)
    w = ocl.synth_weights(cfg, 0, 0.5 * 3840 ** -0.5)
    model = product_model(cfg, w)[0]
    ids = synth.token_ids(9, 1000, (1, 1290))
    cache = models.DeviceCache(model.dev, 1, 1536)
    want = ocl.CausalLM(cfg, w, kv_dtype="bf16").forward(ids, 0)
    for _ in range(2):                          # (the tiles' tickets are back at zero after a call)
        cache.reset()
        assert np.abs(cache.forward(ids, 0) - want).max() <= 3e-3


def test_pairs_gated_epilogue():
    """the gated epilogue on pairs (1290 rows) against the same tokens in portions that stay on single tiles"""
    cfg = R.config([R.mamba(heads=4, vdim=32, state=32, groups=2, mlp=R.dense(ff=1920))], vocab=64, width=3072)
    _, model = R.build(cfg, seed=71, dtype="bf16")
    toks = R.tokens(cfg, 1290, seed=72)
    cut = R.run_cut(model, toks, [650, 640], cache=model.new_device_cache(1, 1536))
    whole = R.run_whole(model, toks, cache=model.new_device_cache(1, 1536))
    assert R.relerr(whole, np.asarray(cut, dtype=np.float64)) < CHUNK_TOL


def test_a_step_does_not_depend_on_what_the_cache_has_seen():
    """heads above 128 channels: the value GEMM of a 1000-token portion has 19000 rows and K = 2560, a shape for pairs, in a step of fewer than 1024
    rows: the same kernels, hence the same bits, on a new cache and on one that has read a longer portion"""
    cfg = R.config([R.att(heads=19, kv_heads=1, dim=192, vdim=64, rot_dims=32, softcap=None)], vocab=64, width=64)
    _, model = R.build(cfg, seed=81, dtype="bf16")
    toks = R.tokens(cfg, 2540, seed=82)
    rows = []
    for used in (False, True):
        cache = model.new_device_cache(2, 2560)
        if used:
            cache.forward_ragged([1], [toks[:1100]], [[1099]])
        for a, b in ((0, 1000), (1000, 1540), (1540, 2540)):
            got = cache.forward_ragged([0], [toks[a:b]], [list(range(b - a))])
        rows.append(got)
    assert np.array_equal(*rows)


# rows and the tiles of 256 x 256 over 74 pairs: the last pair row ends inside its second half, 1 whole tile each and 16 cut ones (o, gate|up); 2 and 6
# (gate|up); 4 and none (gate|up).  Short sentences: a row of every tenth or eighth token is looked at
@pytest.mark.parametrize("batch,tokens,hidden,inter,heads,kv,paired", [(144, 10, 3840, 1920, 30, 5, {"o", "gateup"}), (170, 10, 2560, 2816, 20, 4, {"gateup"}),
                                                                       (250, 8, 512, 4736, 4, 2, {"gateup"})])
def test_pairs_all_over_the_rows(batch, tokens, hidden, inter, heads, kv, paired):
    from fastllm_b200 import models
    from helpers import product_model
    from oracle import causal_lm as ocl
    from oracle import synth
    cfg = ocl.CausalLMConfig("llama", hidden, inter, 500, 1, heads, kv, 1e-5, 1e4, 32)
    w = ocl.synth_weights(cfg, 0, 0.5 * hidden ** -0.5)
    model = product_model(cfg, w)[0]
    ids = synth.token_ids(11, 500, (batch, tokens))
    got, tags = tags_of(lambda: models.DeviceCache(model.dev, batch, 32).forward(ids, 0))
    assert {t for t in tags if t.endswith("_pairs")} == {f"gemm_tc_{p}_pairs" for p in paired}
    want = ocl.CausalLM(cfg, w, kv_dtype="bf16").forward(ids, 0)
    assert np.abs(got - want).max() <= 3e-3


def test_pairs_gated_rows():
    """the gated epilogue, 1440 rows (the last pair row ends inside its second half), every row against the same tokens in portions on single tiles"""
    cfg = R.config([R.mamba(heads=4, vdim=32, state=32, groups=2, mlp=R.dense(ff=1920))], vocab=64, width=3072)
    _, model = R.build(cfg, seed=71, dtype="bf16")
    toks = R.tokens(cfg, 1440, seed=73)
    cut = R.run_cut(model, toks, [720, 720], cache=model.new_device_cache(1, 1536))
    whole, tags = tags_of(lambda: R.run_whole(model, toks, cache=model.new_device_cache(1, 1536)))
    assert "gemm_ff_in_pairs" in tags
    assert R.relerr(whole, np.asarray(cut, dtype=np.float64)) < CHUNK_TOL
