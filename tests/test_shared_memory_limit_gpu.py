"""Rows whose dynamic shared memory is 48 KB to the byte: the kernels' static arrays come on top, so the launch has to opt in. Each
kernel's first launch is the one that counts (the opt-in stays), hence a process of its own."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

CHILD = r"""
import sys
import torch
from pocketllm_b200 import ops
from pocketllm_b200.formats import gguf_quants as gq
from pocketllm_b200.ops import gguf_ops as go

rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
r = lambda *s: torch.randn(*s, device="cuda", generator=torch.Generator("cuda").manual_seed(sum(s)))


def staging():
    blocks = gq.quantize(r(40, 12288).cpu().numpy() * 0.02, "q4_k")
    w = torch.from_numpy(gq.dequantize(blocks, "q4_k").reshape(40, 12288)).cuda().double()
    x = r(9, 12288).to(torch.bfloat16)
    assert rel(go.gguf_linear(x, torch.from_numpy(blocks).cuda().view(-1), "q4_k", 40, epi=2), x.double() @ w.T) < 1e-6


def rmsnorm():
    x, g = r(3, 12288).to(torch.bfloat16), r(12288)
    want = x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-6) * (1 + g.double())
    assert rel(ops.rmsnorm(x, g), want) < 2 ** -8


def residual():
    x, y = r(3, 12288).to(torch.bfloat16), r(3, 12288)
    assert torch.equal(ops.residual_add(x, y), (x + y).to(torch.bfloat16))


def groups():
    ids = torch.randint(0, 384, (128, 8), generator=torch.Generator().manual_seed(1), dtype=torch.int32)
    routes = go.group_routes(ids.cuda(), torch.ones(128, 8, device="cuda"), 384)
    assert torch.equal(routes.src.cpu().long(), torch.sort(ids.view(-1), stable=True).indices)


def heads():
    T, Hq, Hkv = 2, 96, 8
    q, k, v = (r(T, h * 128).to(torch.bfloat16) for h in (Hq, Hkv, Hkv + 1))
    gq_, gk, one = r(Hq * 128), r(Hkv * 128), torch.ones(16, 16, device="cuda")
    kc = torch.zeros(Hkv, 16, 128, device="cuda", dtype=torch.bfloat16)
    out = ops.full_qk_norm_rope_append(q, k, v, torch.arange(T, device="cuda", dtype=torch.int32), gq_, gk, one, 0 * one, kc, kc.clone(), n_heads=Hq,
                                       n_kv_heads=Hkv, rope_dim=32)
    want = q.double() * torch.rsqrt((q.double() ** 2).mean(-1, keepdim=True) + 1e-6) * gq_.double()
    assert rel(out.view(T, -1), want) < 2 ** -8


globals()[sys.argv[1]]()
print("ok")
"""


@pytest.mark.parametrize("what", ["staging", "rmsnorm", "residual", "groups", "heads"])
def test_first_launch_at_the_limit(what):
    p = subprocess.run([sys.executable, "-c", CHILD, what], capture_output=True, text=True, timeout=300, cwd=str(ROOT))
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout + p.stderr
