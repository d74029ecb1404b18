"""Sharded decode on >= 2 GPUs of one node: every rank loads the same checkpoint and keeps its slices —
routed experts always; with peer memory (DSK_P2P=1, the default) and head dims that allow it also the attention heads, wo
columns, shared-expert / dense-FFN hidden units and LM-head rows (tensor parallel).  Partial sums, logits and arg-max keys
are exchanged inside the persistent kernel over CUDA-IPC-mapped peer memory; DSK_P2P=0 = expert-only sharding with
ncclAllReduce between kernel segments.  Rank 0 checks teacher-forced logits and the device-resident greedy loop against
the reference (or its C restatement) on the full checkpoint; the "_tp" cases use real head dims (128 + 64 / 128) so that
two heads fill a 256-column K-quant block and assert that the tensor-parallel plan is actually active; the "_mla" case runs a
true-MLA checkpoint (experts sharded, attention replicated).

Skipped on a single GPU.
"""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

WORKER = textwrap.dedent("""
    import os, sys, json
    import numpy as np
    repo = sys.argv[1]; ckpt = sys.argv[2]
    sys.path[:0] = [os.path.join(repo, "oracle"), os.path.join(repo, "deepseek.cpp_b200"), repo]
    import torch, torch.distributed as dist
    import dsk
    rank, world = int(os.environ["RANK"]), int(os.environ["WORLD_SIZE"])
    torch.cuda.set_device(rank)
    dist.init_process_group("nccl", device_id=torch.device("cuda", rank))
    dsk.init(rank)
    m = dsk.Model.from_dir(ckpt, rank=rank, n_ranks=world, device=rank)
    uid = torch.zeros(128, dtype=torch.uint8, device="cuda")
    if rank == 0:
        uid = torch.frombuffer(bytearray(dsk.Model.comm_unique_id()), dtype=torch.uint8).cuda()
    dist.broadcast(uid, 0)
    m.comm_init(bytes(uid.cpu().numpy().tobytes()))
    toks = [0, 9, 400, 33, 1001, 77, 5, 640]
    errs = []
    if rank == 0:
        import oracle as O
        o = O.open_session(ckpt)
    am = 0
    for pos, t in enumerate(toks):
        logits, am = m.forward(t, pos)
        if rank == 0:
            o.forward(t, pos)
            exp = o.buffer("logits")
            errs.append(float(np.linalg.norm(logits - exp) / np.linalg.norm(exp)))
    dev, _ = m.decode_greedy(len(toks), 6)       # every rank replays the same device-resident loop
    host = []
    if rank == 0:
        pos = len(toks)
        tok = am
        for _ in range(6):
            host.append(int(tok))
            o.forward(int(tok), pos)
            tok = o.argmax()
            pos += 1
        print("RESULT " + json.dumps({"errs": errs, "dev": [int(x) for x in dev], "host": host, "tp": bool(m.sharding()[0]),
                                      "launches": m.launches_per_forward(dsk.OUTPUT_LOGITS)}), flush=True)
    dist.barrier()
    m.close()
    dist.destroy_process_group()
""")


def _gpus():
    try:
        import torch
        return torch.cuda.device_count()
    except Exception:
        return 0


@pytest.mark.skipif(_gpus() < 2, reason="needs 2 GPUs on one node")
@pytest.mark.parametrize("p2p", ["1", "0"])
@pytest.mark.parametrize("preset,quant,tol", [("tiny_v2lite", "fp32", 2e-4), ("tiny_v2lite", "f8e5m2", 5e-4),
                                              ("tiny_v3", "f8e5m2", 5e-4), ("tiny_v2", "q2_k", 8e-2), ("tiny_v3", "q3_k", 8e-2),
                                              ("tiny_v2lite_tp", "fp32", 2e-4), ("tiny_v2_tp", "f8e5m2", 5e-4),
                                              ("tiny_v3_tp", "f8e5m2", 5e-4), ("tiny_v2_tp", "q2_k", 8e-2), ("tiny_v3_tp", "q2_k", 8e-2),
                                              ("tiny_v3_mla", "f8e5m2", 5e-4)])
def test_sharded_decode_matches_reference(repo, ckpt, tmp_path, p2p, preset, quant, tol):
    import json
    want_tp = preset.endswith("_tp") and p2p == "1"
    if preset.endswith("_mla"):  # true-MLA blocks: experts sharded, attention replicated (no tensor-parallel plan for BlockMLA)
        d = ckpt(preset[:-4], quant, use_mla=True, v_head_dim=128)
    elif preset.endswith("_tp"):   # real head dims: 2 local heads x 128 = one 256-column block of wo; f8 scale rows stay aligned
        d = ckpt(preset[:-3], quant, qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128)
    else:
        d = ckpt(preset, quant)
    script = tmp_path / "worker.py"
    script.write_text(WORKER)
    env = dict(os.environ, DSK_P2P=p2p)
    r = subprocess.run([sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node", "2",
                        "--master-addr", "127.0.0.1", "--master-port", str(29541 + (hash((preset, quant, p2p)) % 400)),
                        str(script), repo, d], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    line = [ln for ln in r.stdout.splitlines() if ln.startswith("RESULT ")][-1]
    res = json.loads(line[len("RESULT "):])
    assert max(res["errs"]) < tol, res
    assert res["tp"] == want_tp, res
    if quant in ("fp32", "f8e5m2"):
        assert res["dev"] == res["host"], res      # greedy tokens identical to the reference for the dense quants
    else:
        # K-quants: the sharded sum order differs from the CPU's expert loop, so a Q8_K rounding may flip downstream
        # (the reference does the same against itself); the bound is the reference-vs-reference floor and the median must sit far below it
        import numpy as np
        assert np.median(res["errs"]) < 2e-2, res
    assert res["launches"] == (1 if p2p == "1" else res["launches"])   # peer-memory mode: one kernel per token
