"""The latent attention over prompts on tcgen05 (a cluster of two blocks per 128 query rows) against 64 bits and beside the
mma.sync kernel: tiles' and pages' edges, cached prefixes, unequal batches, pages that start as NaN, large scores."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def case(heads, rank, seqs, seed, loud=1.0):
    """seqs: (tokens already cached, new tokens).  Returns the step, the queries, the cache and every sequence's rows."""
    from builderforce_inference_b200.cache import KVView
    from builderforce_inference_b200.engine.context import Workspace
    g = torch.Generator(device=DEV).manual_seed(seed)
    d = rank + 64
    blocks = max((s + n + 63) // 64 for s, n in seqs)
    perm = torch.randperm(len(seqs) * blocks + 2, generator=torch.Generator().manual_seed(seed))[:len(seqs) * blocks]
    table = perm.int().view(len(seqs), blocks)
    pages = torch.full((len(seqs) * blocks + 2, 1, 64, d), float("nan"), dtype=torch.bfloat16, device=DEV)
    rows = []
    for i, (s, n) in enumerate(seqs):
        x = torch.randn(s + n, d, generator=g, device=DEV).bfloat16()
        rows.append(x)
        flat = torch.full((blocks * 64, d), float("nan"), dtype=torch.bfloat16, device=DEV)
        flat[:s + n] = x
        pages[table[i].long().to(DEV), 0] = flat.view(blocks, 64, d)
    total = sum(n for _, n in seqs)
    q = (loud * torch.randn(total + 1, heads * d, generator=g, device=DEV)).bfloat16()
    q[-1] = float("nan")                                     # a padding row
    cu = [0]
    for _, n in seqs:
        cu.append(cu[-1] + n)
    view = KVView(pages, pages, table.to(DEV), 1, d, None, v_dim=rank, values_in_keys=True)
    ctx = SimpleNamespace(n_seqs=len(seqs), max_seq_tokens=max(n for _, n in seqs), cu_seqlens=i32(cu), seq_slot=i32(list(range(len(seqs)))),
                          seq_start=i32([s for s, _ in seqs]), workspace=Workspace(DEV), pages_bucket=0)
    return ctx, q, view, rows, cu


def plain(q, rows, seqs, cu, heads, rank, scale, sinks, gate):
    out = []
    for i, (s, n) in enumerate(seqs):
        k = rows[i].double()
        qq = q[cu[i]:cu[i + 1]].double().view(n, heads, -1)
        x = torch.einsum("thd,kd->thk", qq, k) * scale
        mask = torch.arange(s + n, device=DEV)[None] > torch.arange(s, s + n, device=DEV)[:, None]
        x = x.masked_fill(mask[:, None], float("-inf"))
        m = x.amax(-1, keepdim=True)
        e = torch.exp(x - m)
        z = e.sum(-1, keepdim=True)
        if sinks is not None:
            z = z + torch.exp(sinks.double()[None, :, None] - m)
        o = torch.einsum("thk,kd->thd", e / z, k[:, :rank])
        if gate is not None:
            o = o * torch.sigmoid(gate[cu[i]:cu[i + 1]].double())[..., None]
        out.append(o.reshape(n, -1))
    return torch.cat(out)


@pytest.mark.parametrize("heads,rank,seqs", [
    (1, 128, [(0, 300)]), (3, 256, [(0, 130), (63, 100), (64, 128)]), (16, 512, [(0, 17), (200, 40)]), (5, 384, [(0, 1), (5, 64), (190, 129)]),
    (16, 512, [(0, 200)]), (12, 256, [(1000, 65)]), (128, 128, [(0, 3), (61, 5)])])
@pytest.mark.parametrize("loud,extras", [(1.0, True), (6.0, False)])
def test_prompts(heads, rank, seqs, loud, extras):
    from builderforce_inference_b200.kernels import fast_ops
    ctx, q, view, rows, cu = case(heads, rank, seqs, heads + rank, loud)
    scale = (rank + 64) ** -0.5
    g = torch.Generator(device=DEV).manual_seed(9)
    sinks = 3.0 * torch.randn(heads, generator=g, device=DEV) if extras else None
    wide = torch.randn(q.shape[0], heads + 8, generator=g, device=DEV).bfloat16()
    gate = wide[:, 3:3 + heads] if extras else None
    assert ctx.max_seq_tokens * heads >= fast_ops.LATENT_TCGEN05_MIN_ROWS
    out = torch.full((q.shape[0], heads * rank), 9.0, dtype=torch.bfloat16, device=DEV)
    assert fast_ops.attention_latent_bf16(ctx, q, out, view, heads, scale, sinks, gate=gate)
    assert int(fast_ops.tc_status(DEV)[0].item()) == 0
    other = torch.empty_like(out)
    assert fast_ops.attention_latent_bf16(ctx, q, other, view, heads, scale, sinks, splits=1, gate=gate)
    ref = plain(q, rows, seqs, cu, heads, rank, scale, sinks, gate)
    err = lambda x: float((x[:-1].double() - ref).norm() / ref.norm())  # noqa: E731
    # bfloat16 outputs of float32 sums: half a unit in the last place, uniformly 2^-9 / sqrt(3) and a little
    assert err(out) < 2.0 ** -8 and err(out) <= 1.02 * err(other)
    assert bool((out[-1] == 9.0).all())


def test_sizes_it_leaves_to_the_other_kernel():
    from builderforce_inference_b200.kernels.library import library
    from ctypes import c_float, c_int, c_long, c_void_p
    z, st = c_void_p(0), torch.zeros(4, dtype=torch.int32, device=DEV)
    x = torch.zeros(8, dtype=torch.bfloat16, device=DEV)
    p = c_void_p(x.data_ptr())

    def taken(d, dv, q_stride, scale):
        return library("fast").call_optional("bfi_attention_latent_tcgen05_bf16", p, c_long(q_stride), p, c_long(8), p, c_long(1), z, c_int(1), z, z, z,
                                             c_int(1), c_int(1), c_int(1), c_int(1), c_int(d), c_int(dv), c_float(scale), z, z, c_long(0),
                                             c_void_p(st.data_ptr()), z)

    assert not taken(544, 512, 544, 0.1) and not taken(160, 96, 160, 0.1) and not taken(704, 640, 704, 0.1)     # rotated part, values
    assert not taken(192, 128, 200, 0.1) and not taken(192, 128, 192, -0.1)                                     # rows with gaps, a scale that turns the order
