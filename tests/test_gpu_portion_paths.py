"""Paths that only portions take, at their edges, against the float64 statement: the state-space recurrence in blocks of 16 tokens (ragged last
block, state sizes around the kernel's groups, heads sharing a group, a walk that continues a decoded state and is continued by one), narrow
products over many rows (router and token-input gate: 16 rows, 32 columns, slices of 16), and products on top of what they add to."""
import pytest

from test_gpu_hybrid import F32_TOL, ho, mk, rel, tokens_for  # noqa: F401
from test_gpu_netusun import in_portions
from test_gpu_netusun import mk as mk_netusun  # noqa: F401
from test_gpu_netusun import no  # noqa: F401
from test_gpu_zetivik import mk as mk_zetivik  # noqa: F401
from test_gpu_zetivik import zo  # noqa: F401

pytestmark = pytest.mark.gpu


def ssd(heads, vdim, state, groups, conv=3):
    return {"type": "mamba2", "mixer": {"heads": heads, "vdim": vdim, "state": state, "groups": groups, "conv": conv, "norm_groups": 1}, "mlp": None}


@pytest.mark.parametrize("heads,vdim,state,groups", [(3, 5, 3, 1), (4, 12, 33, 2), (6, 8, 130, 3), (2, 65, 256, 1), (9, 4, 16, 3)])
def test_recurrence_in_blocks(mk, ho, heads, vdim, state, groups):  # noqa: F811
    cfg = ho.small_config(layers=[ssd(heads, vdim, state, groups)] * 2, width=36, norm={"eps": 1e-5, "groups": 1})
    m, W = mk(cfg, seed=state, chunk=64)
    toks = tokens_for(cfg, 90, 11)
    exp = ho.run(cfg, W, toks)[0]
    for sizes in ([64, 26], [5, 17, 1, 1, 33], [4, 16, 32], [15, 49]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


# walks in segments on the tensor cores: 64 and 128 key entries, channels that end inside a group of 16 or need a second CTA, heads sharing a group, one to eight segments, the
# last one short or ragged; a portion that begins in a decoded state and is followed by tokens
@pytest.mark.parametrize("heads,vdim,state,groups", [(4, 4, 64, 2), (2, 68, 128, 1), (6, 60, 128, 3), (40, 16, 64, 1)])
def test_recurrence_in_segments(mk, ho, heads, vdim, state, groups):  # noqa: F811
    cfg = ho.small_config(layers=[ssd(heads, vdim, state, groups)] * 2, width=36, norm={"eps": 1e-5, "groups": 1})
    m, W = mk(cfg, seed=state + heads, chunk=600)
    toks = tokens_for(cfg, 600, 11)
    exp = ho.run(cfg, W, toks)[0]
    for sizes in ([600], [7, 577], [161, 1, 1, 437], [270, 329]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


# the same in one walk, which short portions of many heads take
@pytest.mark.parametrize("heads,vdim,state,groups", [(32, 64, 64, 4), (32, 128, 128, 2)])
def test_recurrence_in_one_walk(mk, ho, heads, vdim, state, groups):  # noqa: F811
    cfg = ho.small_config(layers=[ssd(heads, vdim, state, groups)], width=36, norm={"eps": 1e-5, "groups": 1})
    m, W = mk(cfg, seed=state + heads, chunk=80)
    toks = tokens_for(cfg, 130, 11)
    exp = ho.run(cfg, W, toks)[0]
    for sizes in ([48, 80], [7, 50, 73]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


@pytest.mark.parametrize("heads,dim,vdim", [(4, 64, 64), (3, 128, 60), (2, 64, 16), (2, 128, 12)])   # the normaliser's column: first of a CTA, last of a group, first of one, inside one
def test_matrix_memory_in_segments(mk_netusun, no, heads, dim, vdim):  # noqa: F811
    def edit(W):                                             # gates at the cap next to keeping everything
        W["l0.mix.f.b"][0] = -60.0
        W["l0.mix.i.b"][1] = 60.0
    cfg = no.model_config([no.mem(heads=heads, dim=dim, vdim=vdim, gate_cap=40.0), no.mem(heads=heads, dim=dim, vdim=vdim)], width=40, vocab=97)
    m, W = mk_netusun(cfg, seed=dim, chunk=500, edit=edit)
    toks = tokens_for(cfg, 500, 9)
    exp = no.run(cfg, W, toks)[0]
    for sizes in ([500], [9, 480], [290, 1, 209]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


@pytest.mark.parametrize("heads,dim,vdim", [(4, 64, 64), (3, 128, 100)])
def test_lightning_in_segments(mk_zetivik, zo, heads, dim, vdim):  # noqa: F811
    decay = [0.0, 1.0, 1e-20, 0.999][:heads]
    cfg = zo.model_config([zo.light(heads=heads, dim=dim, vdim=vdim, decay=decay)], width=40, vocab=97)
    m, W = mk_zetivik(cfg, seed=dim, chunk=500)
    toks = tokens_for(cfg, 500, 9)
    exp = zo.run(cfg, W, toks)[0]
    for sizes in ([500], [9, 480], [290, 1, 209]):
        assert rel(in_portions(m, toks, sizes), exp) < F32_TOL


@pytest.mark.parametrize("experts,side,width,tokens", [(5, 3, 36, 33), (33, 32, 40, 48), (96, 90, 72, 65), (7, 64, 130, 100)])
def test_narrow_products(mk, ho, experts, side, width, tokens):  # noqa: F811
    moe = {"kind": "moe", "router": {"experts": experts, "top": 2, "scale": 1.0}, "expert": {"ff": 12, "limit": 3.0}}
    cfg = ho.small_config(layers=[dict(ssd(2, 6, 4, 1), mlp=moe)], width=width, norm={"eps": 1e-5, "groups": 1}, token_side={"dim": side})
    m, W = mk(cfg, seed=experts, chunk=128)
    toks = tokens_for(cfg, tokens, 12)
    assert rel(m.forward_chunk(toks, 0, range(tokens)), ho.run(cfg, W, toks)[0]) < F32_TOL


@pytest.mark.parametrize("experts,side,width,tokens", [(5, 3, 36, 448), (33, 32, 40, 449), (96, 90, 72, 513), (7, 64, 130, 463)])
def test_narrow_products_of_many_rows(mk, ho, experts, side, width, tokens):  # noqa: F811
    moe = {"kind": "moe", "router": {"experts": experts, "top": 2, "scale": 1.0}, "expert": {"ff": 12, "limit": 3.0}}
    cfg = ho.small_config(layers=[dict(ssd(2, 6, 4, 1), mlp=moe)], width=width, norm={"eps": 1e-5, "groups": 1}, token_side={"dim": side})
    m, W = mk(cfg, seed=experts, chunk=600)
    toks = tokens_for(cfg, tokens, 12)
    assert rel(m.forward_chunk(toks, 0, range(tokens)), ho.run(cfg, W, toks)[0]) < F32_TOL


def test_large_windows_take_the_fused_kernel(mk_netusun, no, monkeypatch, capfd):  # noqa: F811
    """What switches the attention of portions on is the memory of the layers that use it: 64 heads x 256 queries x 70000 keys are 4.6 GB of scores, which
    only the products between which scores lie in memory would have."""
    monkeypatch.setenv("DSK_HY_TIMELINE", "1")
    cfg = no.model_config([no.att(heads=64, kv_heads=1, dim=8, vdim=8, size=None)], width=40, vocab=97)
    m, W = mk_netusun(cfg, seed=3, chunk=64, context=70000)
    toks = tokens_for(cfg, 100, 9)
    got = in_portions(m, toks, [60, 40])
    assert rel(got, no.run(cfg, W, toks)[0]) < F32_TOL
    assert capfd.readouterr().err.count("att.fused") == 2
