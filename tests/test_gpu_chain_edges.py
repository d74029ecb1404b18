"""The token chain (csrc/dsk_decode.cuh) against the interpreter that runs the models it refuses, where a call leaves the ordinary: values that are not finite, cache rows behind
those that are read, launches of like sizes.

K-quants have one order of sums in both and are equal bit for bit; of the other formats the places that are not finite are equal, and the rest within 2^-11 (a cached
key or value that rounds to fp16 the other way)."""
import os
import pickle
import subprocess
import sys
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [os.path.join(HERE, "..", "deepseek.cpp_b200"), os.path.join(HERE, "..", "oracle")]
pytestmark = pytest.mark.gpu

PRESET = {"q2_k": "tiny_v2", "q3_k": "tiny_v3", "f8e5m2": "tiny_v2", "fp16": "tiny_v3", "fp32": "tiny_v2"}
NAN = {"q2_k": (slice(84 + 80, 84 + 82), (0, 0x7E)), "q3_k": (slice(110 + 108, 110 + 110), (0, 0x7E)), "f8e5m2": (300, 0x7F), "fp16": (300, np.nan), "fp32": (300, np.nan)}
INF = {"q2_k": (slice(84 + 80, 84 + 82), (0, 0x7C)), "q3_k": (slice(110 + 108, 110 + 110), (0, 0x7C)), "f8e5m2": (300, 0x7C), "fp16": (300, np.inf), "fp32": (300, np.inf)}


def load(quant, edit=None, seed=5, **sizes):
    """A small model; `edit` changes copies of its tensors."""
    import dseek
    import dsk
    import mint
    with tempfile.TemporaryDirectory() as d:
        mint.mint(d, PRESET[quant], quant, fast=True, seed=seed, **sizes)
        md, tensors = dseek.read_dir(d)
        m = dsk.Model(dsk.Config.from_metadata(md, 0))
        for name, t in tensors.items():
            data = np.array(t.data)
            if edit:
                edit(name, data)
            m.upload(name, t.dtype, t.shape, data)
        m.finalize()
    return m


def not_finite(quant):
    """Embedding rows with a block (K-quants) or a value that is NaN, infinite; then cached values that are, which attention hands on to a product without a norm."""
    def edit(name, data):
        if name == "model.embed.weight":
            for row, (at, v) in ((7, NAN[quant]), (9, INF[quant])):
                data.reshape(1024, -1)[row, at] = v
    m = load(quant, edit)
    got = {}
    for pos, token in enumerate((3, 7, 9, 4)):
        logits, best = m.forward(token, pos)
        got[f"token {token}"] = [np.array(logits), np.array([best])]
    for pos in range(4):
        m.forward(3 + 2 * pos + (pos > 1), pos)   # (finite rows again)
    clean = m.kv_cache(0, 1).copy()
    c = m.cfg
    for name, heads, value in (("NaN", 1, np.nan), ("inf", 1, np.inf), ("-inf", 1, -np.inf), ("NaN heads", 4, np.nan)):
        kv = clean.view(np.float16).reshape(-1, c.n_heads, c.v_head_dim).copy()
        kv[1, :heads, 5 if heads == 1 else slice(None)] = value
        m.set_kv_cache(0, 1, kv.view(np.uint16).reshape(-1))
        m.copy_embedding(3)
        m.block(0, 3, 0, 3, 4)
        got["cached " + name] = [m.buffer("x")]
    m.close()
    return got


def row_behind(quant):
    """Block calls whose new row lies behind the rows that are read: inside and outside of what the attention holds in shared memory (about 90 rows of these heads)."""
    m = load(quant, qk_nope_head_dim=256, qk_rope_head_dim=64, v_head_dim=256)
    for pos in range(10):
        m.forward(5 + 31 * pos, pos)
    got = {}
    for kv_pos in (9, 10, 60, 89, 130, 255):
        for layer in (0, 1):
            m.copy_embedding(40 + kv_pos)
            m.block(layer, kv_pos, 0, kv_pos, 10)
            got[f"row {kv_pos}, layer {layer}"] = [m.buffer("x")] + [m.kv_cache(layer, which).view(np.float16).astype(np.float32) for which in (0, 1)]
    m.close()
    return got


def like_sizes(quant):
    """The output projection of attention and the LM head have the same sizes; only the second one's input has a norm (they run in launches of the same form)."""
    m = load(quant, dim=512, vocab_size=512, n_heads=4, v_head_dim=128, n_layers=1, first_k_dense_replace=0)
    got = {f"position {pos}": [np.array(m.forward(5 + 31 * pos, pos)[0])] for pos in range(4)}
    m.close()
    return got


SCENARIOS = {(n, q): (f, q) for n, f in (("not finite", not_finite), ("row behind", row_behind), ("like sizes", like_sizes)) for q in PRESET}


def _run(out):
    import dsk
    dsk.init(0)
    with open(out, "wb") as f:
        pickle.dump({k: fn(*args) for k, (fn, *args) in SCENARIOS.items()}, f)


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    out = []
    for engine in ("chain", "mega"):
        p = str(tmp_path_factory.mktemp(engine) / "out")
        subprocess.run([sys.executable, __file__, p], env={**os.environ, "DSK_ENGINE": engine}, check=True, timeout=300)
        with open(p, "rb") as f:
            out.append(pickle.load(f))
    return out


@pytest.mark.parametrize("scenario", SCENARIOS, ids=str)
def test_chain_against_interpreter(both, scenario):
    chain, mega = (b[scenario] for b in both)
    assert chain.keys() == mega.keys()
    for what in chain:
        for a, b in zip(chain[what], mega[what]):
            if scenario[1] in ("q2_k", "q3_k") or a.dtype.kind == "i":
                assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), what
            else:
                f = np.isfinite(b)
                assert np.array_equal(np.isfinite(a), f) and np.array_equal(np.isnan(a), np.isnan(b)), what
                assert np.linalg.norm((a - b)[f]) <= 2.0 ** -11 * np.linalg.norm(b[f]), what


@pytest.mark.parametrize("row", [0, 1])
def test_new_row_is_a_sink(row):
    """A block call whose new row is one of the rows that turn: it is rotated, written and then turned with them.  Against the oracle (fp32; a cached value may round
    to fp16 the other way)."""
    import dsk
    import mint
    import oracle
    with tempfile.TemporaryDirectory() as d:
        mint.mint(d, "tiny_v2", "fp32", fast=True, seed=5)
        m, o = dsk.Model.from_dir(d), oracle.open_session(d)
        for pos in range(6):
            m.forward(5 + 31 * pos, pos)
        for which in (0, 1):
            o.kv_cache(0, which)[:] = m.kv_cache(0, which)
        for s in (m, o):
            s.copy_embedding(40)
            s.block(0, 9, 2, row, 6)
        exp = o.buffer("x")
        assert np.linalg.norm(m.buffer("x") - exp) <= 2.0 ** -11 * np.linalg.norm(exp)
        a, b = (s.kv_cache(0, 0)[:6 * 4 * 96].view(np.float16).astype(np.float32) for s in (m, o))
        assert np.abs(a - b).max() <= 2.0 ** -10 * np.abs(b).max()
        m.close()
        o.close()


@pytest.mark.parametrize("quant", PRESET)
def test_tensors_from_host_and_device(quant):
    """A model whose tensors come by turns from the host, each a larger one, and from device addresses that no vector load may take, each a smaller one."""
    import dseek
    import dsk
    import mint
    import torch
    logits = []
    with tempfile.TemporaryDirectory() as d:
        mint.mint(d, PRESET[quant], quant, fast=True, seed=5, hidden_dim=8192)
        md, tensors = dseek.read_dir(d)
        names = sorted((n for n in tensors if n != "tokenizer.tokens"), key=lambda n: tensors[n].data.nbytes)
        big, small = names[len(names) // 2:][::-1], names[:len(names) // 2]
        turns = [n for pair in zip(big, small + [None]) for n in pair if n]
        assert sorted(turns) == sorted(names)
        for mixed in (False, True):
            m = dsk.Model(dsk.Config.from_metadata(md, 0))
            for i, name in enumerate(turns):
                t = tensors[name]
                data = np.ascontiguousarray(t.data)
                if mixed and name in small:
                    buf = torch.zeros(data.nbytes + 16, dtype=torch.uint8, device="cuda")
                    at = 2 if data.dtype.itemsize <= 2 else 4
                    buf[at:at + data.nbytes] = torch.from_numpy(data.reshape(-1).view(np.uint8).copy()).cuda()
                    torch.cuda.synchronize()
                    m.upload_device(name, t.dtype, t.shape, buf.data_ptr() + at, data.nbytes)
                else:
                    m.upload(name, t.dtype, t.shape, data)
            m.finalize()
            logits.append(np.stack([np.array(m.forward(5 + 31 * pos, pos)[0]) for pos in range(4)]))
            m.close()
    assert np.array_equal(*logits)


@pytest.mark.parametrize("quant", PRESET)
def test_state_before_finalize(quant):
    """A state that is made when all tensors have come, but before the model is finished."""
    import dseek
    import dsk
    import mint
    logits = []
    with tempfile.TemporaryDirectory() as d:
        mint.mint(d, PRESET[quant], quant, fast=True, seed=5)
        md, tensors = dseek.read_dir(d)
    for early in (False, True):
        m = dsk.Model(dsk.Config.from_metadata(md, 0))
        for name, t in tensors.items():
            m.upload(name, t.dtype, t.shape, t.data)
        state = m.new_state() if early else None
        m.finalize()
        if early:
            m.s, m._extra_states = state, [m.s]
        logits.append(np.stack([np.array(m.forward(5 + 31 * pos, pos)[0]) for pos in range(4)]))
        m.close()
    assert np.array_equal(*logits)


@pytest.mark.parametrize("missing", ["model.output.scale", "model.output.weight", "model.embed.scale", "model.layers.1.moegate.weight", "model.layers.1.mlp.w2.scale",
                                     "model.layers.0.attn.norm.weight", "model.layers.2.shared_mlp.w1.weight"])
def test_state_of_an_incomplete_model_is_refused(missing):
    import dseek
    import dsk
    import mint
    with tempfile.TemporaryDirectory() as d:
        mint.mint(d, "tiny_v2", "f8e5m2", fast=True, seed=5)
        md, tensors = dseek.read_dir(d)
    m = dsk.Model(dsk.Config.from_metadata(md, 0))
    for name, t in tensors.items():
        if name != missing and not (missing == "model.output.weight" and name == "model.output.scale"):
            m.upload(name, t.dtype, t.shape, t.data)
    with pytest.raises(dsk.DskError):
        m.new_state()
    if missing == "model.output.weight":   # (tied embeddings: once the model is finished)
        m.finalize()
        assert np.isfinite(m.forward(3, 0)[0]).all()
    else:
        with pytest.raises(dsk.DskError):
            m.finalize()
    m.close()


@pytest.mark.parametrize("vocab,chain", [(1000003, True), (2000003, False)])
def test_large_vocabulary(vocab, chain):
    """The sums of an LM head's rows (64 floats a tile of 16 rows) fit a CTA's shared memory up to about 1.5 million rows; the interpreter runs what does not."""
    import dseek
    import dsk
    import mint
    import torch
    logits = []
    with tempfile.TemporaryDirectory() as d:
        mint.mint(d, "tiny_v2", "q2_k", fast=True, seed=5, dim=256)
        md, tensors = dseek.read_dir(d)
    for rows in (1024, vocab):
        cfg = dsk.Config.from_metadata(md, 0)
        cfg.vocab_size = rows
        m = dsk.Model(cfg)
        for name, t in tensors.items():
            if name in ("model.embed.weight", "model.output.weight"):
                q = torch.from_numpy(np.array(t.data)).cuda()
                q = q.repeat(-(-rows // 1024), 1)[:rows].contiguous()
                torch.cuda.synchronize()
                m.upload_device(name, t.dtype, q.shape, q.data_ptr(), q.numel())
            else:
                m.upload(name, t.dtype, t.shape, t.data)
        m.finalize()
        assert (m.launches_per_forward() > 1) == (chain or rows == 1024)
        logits.append(np.stack([np.array(m.forward(5 + 31 * pos, pos)[0]) for pos in range(3)]))
        m.close()
    assert np.array_equal(logits[1], np.tile(logits[0], (1, -(-vocab // 1024)))[:, :vocab])


@pytest.mark.parametrize("quant,sizes", [("q3_k", dict(moe_intermediate_size=5120, n_routed_experts=256, n_layers=2)),   # 288 MB a stack of experts
                                         ("fp32", dict(dim=1036, n_heads=5, v_head_dim=64, vocab_size=66003, n_layers=2))])   # 274 MB of vocabulary, the last piece ragged
def test_uploads_in_pieces(quant, sizes):
    """Tensors from the host pass through a buffer of 256 MB: stacks of experts in whole matrices, one large matrix in whole row tiles.  Against one copy on the device."""
    import dseek
    import dsk
    import mint
    import torch
    logits = []
    with tempfile.TemporaryDirectory() as d:
        mint.mint(d, PRESET[quant], quant, fast=True, seed=5, **sizes)
        md, tensors = dseek.read_dir(d)
        for host in (True, False):
            m = dsk.Model(dsk.Config.from_metadata(md, 0))
            assert m.launches_per_forward() > 1
            for name, t in tensors.items():
                if host or name == "tokenizer.tokens":
                    m.upload(name, t.dtype, t.shape, t.data)
                else:
                    q = torch.from_numpy(np.array(t.data).reshape(-1).view(np.uint8)).cuda()
                    torch.cuda.synchronize()
                    m.upload_device(name, t.dtype, t.shape, q.data_ptr(), q.numel())
            m.finalize()
            logits.append(np.stack([np.array(m.forward(5 + 31 * pos, pos)[0]) for pos in range(3)] + [np.array(m.forward(m.cfg.vocab_size - 1, 3)[0])]))
            m.close()
    assert np.array_equal(*logits)


if __name__ == "__main__":
    _run(sys.argv[1])
