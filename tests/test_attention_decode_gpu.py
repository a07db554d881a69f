"""Attention of decoded tokens by TMA: slices from one to eight, tiles that end inside a page, pages of every size, requests
of one key, several new tokens per request, slices that are empty, pages that hold NaN where no key is; pages larger than a tile
stay on the kernel that gathers."""
import math
import types

import pytest
import torch

import plain_llama as pl
from test_kernels_gpu import launched, paged_setup, tol

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("hd,nq,nkv,q_len,page", [(64, 32, 4, 1, 16), (64, 16, 1, 1, 64), (64, 6, 2, 5, 8), (64, 3, 3, 16, 32),
                                                  (128, 32, 8, 1, 16), (128, 7, 1, 2, 8), (128, 4, 4, 1, 32),
                                                  (128, 4, 4, 1, 64)])
@pytest.mark.parametrize("slices", [1, 2, 5, 8])
@pytest.mark.parametrize("few", [True, False])
def test_decoded_tokens_in_slices_of_keys(hd, nq, nkv, q_len, page, slices, few, monkeypatch):
    from tiny_llm_b200 import ops
    from tiny_llm_b200.engine import Workspace
    monkeypatch.setattr(ops, "_decode_slices", lambda *_: (slices, few))
    lens = [max(n, q_len) for n in (1, 2, 31, 32, 33, 63, 64, 65, 127, 385, 1000, 1537)]
    n = len(lens)
    table, kc, vc, ks, vs = paged_setup("bfloat16", n, lens, nkv, hd, page, seed=hd + nq + page)
    g = torch.Generator().manual_seed(slices)
    t = n * q_len
    qkv = (torch.randn(t, (nq + 2 * nkv) * hd, generator=g) * 2).to(torch.bfloat16)
    pos = torch.cat([torch.arange(l - q_len, l, dtype=torch.int32) for l in lens])
    batch = types.SimpleNamespace(
        token_request=torch.arange(n, dtype=torch.int32).repeat_interleave(q_len).to(DEV), positions=pos.to(DEV),
        cu_q=torch.arange(0, t + 1, q_len, dtype=torch.int32).to(DEV),
        q_start=torch.tensor([l - q_len for l in lens], dtype=torch.int32).to(DEV), num_requests=n, max_q_len=q_len, max_kv_len=max(lens))
    out = torch.full((t, nq * hd), math.nan, dtype=torch.bfloat16, device=DEV)
    names = launched(ops, lambda: ops.paged_attention(qkv.to(DEV), nq, nkv, hd, kc.to(DEV), vc.to(DEV), table.to(DEV), batch, out,
                                                      hd ** -0.5, None, Workspace(DEV)))
    ops.check_status()
    assert names == ["tllm_attention_decode" if page * hd <= 4096 else "tllm_attention_mma"]
    out = out.float().cpu()
    for r, l in enumerate(lens):
        q = qkv[r * q_len: (r + 1) * q_len, : nq * hd].float().view(q_len, nq, hd)
        ref = pl.attention(q, ks[r].float(), vs[r].float(), pos[r * q_len: (r + 1) * q_len], quant=pl.bf16_quant).reshape(q_len, nq * hd)
        d = float((out[r * q_len: (r + 1) * q_len] - ref).abs().max())
        assert d <= tol("bfloat16", max(1.0, float(ref.abs().max()))), (r, l, d)
