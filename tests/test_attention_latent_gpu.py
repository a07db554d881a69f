"""Latent attention of prompt portions (keys of 256 values, values of 192), whose softmax weights must reach the product with
at least 16 bits: portions that start in the middle of a sequence and end inside a page, tiles with rows of several tokens, a
sink, pages of every size, unwritten slots that are NaN."""
import math
import types

import pytest
import torch

from test_kernels_gpu import launched

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
KD, VD = 256, 192


@pytest.mark.parametrize("nq,nkv,page", [(16, 1, 16), (16, 1, 8), (4, 2, 64), (128, 1, 32), (8, 8, 16)])
@pytest.mark.parametrize("sink", [False, True])
def test_portions_with_latent_keys(nq, nkv, page, sink):
    from tiny_llm_b200 import ops
    from tiny_llm_b200.engine import Workspace
    g = torch.Generator().manual_seed(nq + page + sink)
    lens, q_lens = [900, 333, 129, 65, 64, 1], [389, 333, 17, 2, 64, 1]
    blocks = [-(-n // page) for n in lens]
    table, ids = torch.full((len(lens), max(blocks) + 1), -1, dtype=torch.int32), torch.randperm(sum(blocks) + 2, generator=g)
    kc = torch.full((sum(blocks) + 2, nkv, page, KD), math.nan, dtype=torch.bfloat16)
    vc = torch.full((sum(blocks) + 2, nkv, page, VD), math.nan, dtype=torch.bfloat16)
    ks, vs = [torch.randn(n, nkv, KD, generator=g).bfloat16() for n in lens], [torch.randn(n, nkv, VD, generator=g).bfloat16() for n in lens]
    for r, n in enumerate(lens):
        table[r, :blocks[r]], ids = ids[:blocks[r]].int(), ids[blocks[r]:]
        for j in range(n):
            kc[table[r, j // page], :, j % page], vc[table[r, j // page], :, j % page] = ks[r][j], vs[r][j]
    t = sum(q_lens)
    q = (torch.randn(t, nq * KD + 8, generator=g) * 1.5).bfloat16()
    ks[0][5, 0] = kc[table[0, 5 // page], 0, 5 % page] = (q[388, :KD].float() / q[388, :KD].float().norm() * 40).bfloat16()   # a far key that carries a query
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    batch = types.SimpleNamespace(
        token_request=torch.arange(len(lens), dtype=torch.int32).repeat_interleave(torch.tensor(q_lens)).to(DEV),
        positions=torch.cat([torch.arange(n - m, n, dtype=torch.int32) for n, m in zip(lens, q_lens)]).to(DEV), cu_q=cu.to(DEV),
        q_start=torch.tensor([n - m for n, m in zip(lens, q_lens)], dtype=torch.int32).to(DEV), num_requests=len(lens),
        max_q_len=max(q_lens), max_kv_len=max(lens))
    extra = torch.randn(nq, generator=g) * 2 if sink else None
    out = torch.full((t, nq * VD), math.nan, dtype=torch.bfloat16, device=DEV)
    assert launched(ops, lambda: ops.paged_attention_maps(
        q.to(DEV)[:, :nq * KD], nq, nkv, 1, KD, VD, kc.to(DEV), vc.to(DEV), table.to(DEV), batch, out, KD ** -0.5,
        sink=None if extra is None else extra.to(DEV), workspace=Workspace(DEV))) == ["tllm_attention_maps_mma"]
    ops.check_status()
    out, group = out.double().cpu().view(t, nq, VD), nq // nkv
    for r, (n, m) in enumerate(zip(lens, q_lens)):
        rows = q[cu[r]:cu[r + 1], :nq * KD].double().view(m, nkv, group, KD)
        scores = torch.einsum("tkgd,jkd->tkgj", rows, ks[r].double()) * KD ** -0.5
        scores.masked_fill_((torch.arange(n) > torch.arange(n - m, n)[:, None])[:, None, None], -math.inf)
        if extra is not None:
            scores = torch.cat([scores, extra.double().view(1, nkv, group, 1).expand(m, -1, -1, 1)], -1)
        p = torch.softmax(scores, -1)[..., :n]
        ref = torch.einsum("tkgj,jkd->tkgd", p, vs[r].double()).reshape(m, nq, VD)
        # The result's rounding, 2^-8 of it.  Weights: two bfloat16 parts leave 2^-17 out; scores are sums of 16 additions of 16
        # products, each within 2^-23 of the sizes added up (|q k| of about 22 in units of log2 e): 2^-14 of a weight in all.
        # (One bfloat16 part would leave 2^-9.)
        most = torch.einsum("tkgj,jkd->tkgd", p, vs[r].double().abs()).reshape(m, nq, VD) * 2.0 ** -14 + ref.abs() * 2.0 ** -8 + 1e-6
        assert bool(((out[cu[r]:cu[r + 1]] - ref).abs() <= most).all()), r
