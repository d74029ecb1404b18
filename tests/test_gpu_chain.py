"""The token chain (csrc/dsk_decode.cuh) against the interpreter that runs the models it refuses: sizes that fill no row tile, no unit of columns and no
CTA's warps, an odd number of K-quant blocks, contexts on both sides of what the attention holds in shared memory, sinks, and its captured graphs.

K-quants have one order of sums in both and are equal bit for bit.  The other formats sum in another order (2^-24 a step); what that can turn the other way is
the rounding of a cached key or value to fp16, 2^-11 of that element, so 2^-11 of the logits bounds their difference."""
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

CASES = {
    "q2_k": ("tiny_v2", dict(dim=768, hidden_dim=2816, n_heads=3, vocab_size=1003, qk_nope_head_dim=256, qk_rope_head_dim=64, v_head_dim=256, kv_lora_rank=256,
                             q_lora_rank=1280, moe_intermediate_size=1280)),
    "q3_k": ("tiny_v3", dict(dim=1792, hidden_dim=256, n_heads=2, vocab_size=33, v_head_dim=128, n_active_routed=8, n_routed_experts=24, moe_intermediate_size=2304)),
    "f8e5m2": ("tiny_v2lite", dict(dim=448, hidden_dim=704, n_heads=5, vocab_size=1003, qk_nope_head_dim=56, qk_rope_head_dim=24, kv_lora_rank=192,
                                   moe_intermediate_size=192)),
    "fp16": ("tiny_v3", dict(dim=336, hidden_dim=432, n_heads=2, vocab_size=997, v_head_dim=40, kv_lora_rank=112, q_lora_rank=48, moe_intermediate_size=80)),
    "fp32": ("tiny_v2lite", dict(dim=132, hidden_dim=76, n_heads=3, vocab_size=131, qk_nope_head_dim=16, qk_rope_head_dim=8, v_head_dim=8, kv_lora_rank=36,
                                 moe_intermediate_size=20)),
}
WANTED = (0, 1, 7, 8, 90, 130, 199, 200, 230)   # 200 positions, then sinks


def _run(out):
    import dsk
    import mint
    dsk.init(0)
    got = {}
    for quant, (preset, sizes) in CASES.items():
        with tempfile.TemporaryDirectory() as d:
            mint.mint(d, preset, quant, fast=True, seed=11, original_max_position=200, **sizes)
            m = dsk.Model.from_dir(d)
        for pos in range(WANTED[-1] + 1):
            logits, best = m.forward(pos * 31 % sizes["vocab_size"], pos, want_logits=pos in WANTED)
            if pos in WANTED:
                got[quant, pos] = np.array(logits), best
        m.forward(3, 0)
        got[quant, "greedy"] = [m.decode_greedy(s, 6)[0].tolist() for s in (1, 7)]
        got[quant, "launches"] = m.launches_per_forward()
        m.close()
    with open(out, "wb") as f:
        pickle.dump(got, f)


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    out = []
    for engine in ("chain", "mega"):
        p = str(tmp_path_factory.mktemp(engine) / "out")
        subprocess.run([sys.executable, __file__, p], env={**os.environ, "DSK_ENGINE": engine}, check=True, timeout=300)
        with open(p, "rb") as f:
            out.append(pickle.load(f))
    return out


@pytest.mark.parametrize("quant", CASES)
def test_chain_against_interpreter(both, quant):
    chain, mega = both
    assert chain[quant, "launches"] > 1 and mega[quant, "launches"] == 1
    assert chain[quant, "greedy"] == mega[quant, "greedy"]
    for pos in WANTED:
        (a, ia), (b, ib) = chain[quant, pos], mega[quant, pos]
        if quant in ("q2_k", "q3_k"):
            assert np.array_equal(a, b) and ia == ib, pos
        else:
            assert np.linalg.norm(a - b) <= 2.0 ** -11 * np.linalg.norm(b), pos


if __name__ == "__main__":
    _run(sys.argv[1])
