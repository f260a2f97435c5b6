"""The float32 attention by tiles of 64 rows and 64 keys (heads of 64 or 128) against 64 bits with every mask and option."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def make(n_q, n_kv, d, seqs, seed, **mask):
    from builderforce_inference_b200.cache import KVView
    g = torch.Generator(device=DEV).manual_seed(seed)
    blocks = max((s + n + 63) // 64 for s, n in seqs)
    table = torch.randperm(len(seqs) * blocks + 1, generator=torch.Generator().manual_seed(seed))[:len(seqs) * blocks].int().view(len(seqs), blocks)
    k = torch.full((len(seqs) * blocks + 1, n_kv, 64, d), float("nan"), device=DEV)
    v = k.clone()
    rows = []
    for i, (s, n) in enumerate(seqs):
        x = torch.randn(2, s + n, n_kv, d, generator=g, device=DEV)
        rows.append(x)
        for t, store in ((x[0], k), (x[1], v)):
            flat = torch.full((blocks * 64, n_kv, d), float("nan"), device=DEV)
            flat[:s + n] = t
            store[table[i].long().to(DEV)] = flat.view(blocks, 64, n_kv, d).transpose(1, 2)
    q = torch.randn(sum(n for _, n in seqs), n_q * d, generator=g, device=DEV)
    return q, KVView(k, v, table.to(DEV), n_kv, d, mask.get("window"), chunk=mask.get("chunk"), keep_first=mask.get("keep_first", 0)), rows


def run(q, view, seqs, n_q, scale, sink=None, softcap=None, max_tokens=None):
    from builderforce_inference_b200.kernels import ops
    cu = [0]
    for _, n in seqs:
        cu.append(cu[-1] + n)
    out = torch.full_like(q, float("nan"))
    ops.attention_paged(q, q.stride(0), out, view, i32(cu), i32(list(range(len(seqs)))), i32([s for s, _ in seqs]), len(seqs),
                        max_tokens or max(n for _, n in seqs), n_q, scale, sink, softcap)
    return out


def plain(q, rows, seqs, n_q, n_kv, d, scale, sink=None, softcap=None, window=None, keep_first=0, chunk=None):
    out, at = [], 0
    for (s, n), kv in zip(seqs, rows):
        k, v = (t.double().repeat_interleave(n_q // n_kv, 1) for t in kv)
        x = torch.einsum("thd,khd->htk", q[at:at + n].double().view(n, n_q, d), k) * scale
        if softcap:
            x = softcap * torch.tanh(x / softcap)
        p, j = torch.arange(s, s + n, device=DEV)[:, None], torch.arange(s + n, device=DEV)[None]
        seen = j <= p
        if window:
            seen &= (j > p - window) | (j < keep_first)
        if chunk:
            seen &= j >= p // chunk * chunk
        x = x.masked_fill(~seen, float("-inf"))
        m = x.amax(-1, keepdim=True)
        e = torch.exp(x - m)
        z = e.sum(-1, keepdim=True)
        if sink is not None:
            z = z + torch.exp((sink.double()[:, None, None] if torch.is_tensor(sink) else sink) - m)
        out.append(torch.einsum("htk,khd->thd", e / z, v).reshape(n, -1))
        at += n
    return torch.cat(out)


@pytest.mark.parametrize("n_q,n_kv,d,seqs", [(4, 1, 128, [(0, 70), (63, 8), (128, 1)]), (6, 1, 64, [(0, 130), (5, 33)]), (3, 3, 128, [(0, 65)]),
                                             (64, 1, 64, [(0, 9), (60, 10)]), (8, 2, 64, [(300, 1), (0, 1)]), (5, 1, 128, [(100, 64), (0, 1)])])
@pytest.mark.parametrize("opt", [{}, {"window": 30, "keep_first": 5}, {"chunk": 48}, {"sink": 1.5, "softcap": 2.0}, {"sink": "each", "window": 64}])
def test_tiles(n_q, n_kv, d, seqs, opt):
    mask = {k: v for k, v in opt.items() if k in ("window", "keep_first", "chunk")}
    q, view, rows = make(n_q, n_kv, d, seqs, n_q + d, **mask)
    sink = opt.get("sink")
    if sink == "each":
        sink = torch.linspace(-2.0, 3.0, n_q, device=DEV)
    scale = d ** -0.5
    got = run(q, view, seqs, n_q, scale, sink, opt.get("softcap"))
    ref = plain(q, rows, seqs, n_q, n_kv, d, scale, sink, opt.get("softcap"), **mask)
    assert float((got.double() - ref).norm() / ref.norm()) < 1e-6


def test_a_value_that_is_not_finite_reaches_only_the_tokens_that_see_it():
    q, view, rows = make(4, 2, 64, [(0, 40)], 3)
    page = int(view.block_table[0, 0])
    view.v[page, 0, 20, 3] = float("inf")
    got = run(q, view, [(0, 40)], 4, 0.125).view(40, 4, 64)
    assert bool(torch.isfinite(got[:20]).all()) and bool(torch.isinf(got[20:, :2, 3]).all())
    got[20:, :2, 3] = 0.0
    assert bool(torch.isfinite(got).all())
