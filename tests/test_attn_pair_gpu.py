"""Prompt attention of two query tiles per block and of keys split over blocks (csrc/attention_pair.cu) against 64-bit attention."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(q_lens, ctx, Hq, Hkv, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    lens = [q + c for q, c in zip(q_lens, ctx)]
    pages = [-(-n // 64) for n in lens]
    kc = torch.randn(sum(pages) + 1, Hkv, 64, 128, generator=g, device="cuda").to(torch.bfloat16)
    vc = torch.randn(kc.shape, generator=g, device="cuda").to(torch.bfloat16)
    kc[0], vc[0] = 0, 0
    perm = torch.randperm(sum(pages), generator=g, device="cuda").to(torch.int32) + 1
    table = torch.zeros(len(lens), max(pages) + 1, dtype=torch.int32, device="cuda")
    for i, n in enumerate(pages):
        table[i, :n] = perm[sum(pages[:i]):sum(pages[:i + 1])]
    q = (2 * torch.randn(sum(q_lens), Hq, 128, generator=g, device="cuda")).to(torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    starts = [sum(q_lens[:i]) for i in range(len(q_lens) + 1)]
    return q, kc, vc, table, i32(lens), i32(starts), lens, starts


def _ref(q, kc, vc, table, lens, starts, window, keep, sink, gate):
    Hq, Hkv = q.shape[1], kc.shape[1]
    out = torch.zeros(q.shape, dtype=torch.float64, device="cuda")
    for i, n in enumerate(lens):
        a, b = starts[i], starts[i + 1]
        pg = table[i, :-(-n // 64)].long()
        k, v = (c[pg].transpose(0, 1).flatten(1, 2)[:, :n].double() for c in (kc, vc))
        pos, key = torch.arange(n - (b - a), n, device="cuda")[:, None], torch.arange(n, device="cuda")[None]
        see = key <= pos
        if window:
            see &= (key > pos - window) | (key < keep)
        for h in range(Hq):
            s = (q[a:b, h].double() @ k[h // (Hq // Hkv)].T / math.sqrt(128)).masked_fill(~see, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].double().expand(b - a, 1)], 1)
            w = torch.softmax(s, -1)[:, :n]
            o = w @ v[h // (Hq // Hkv)]
            out[a:b, h] = o * torch.sigmoid(gate[a:b, h].double())[:, None] if gate is not None else o
    return out


def _close(out, ref, mass):
    # every weight w is rounded to bf16 (eight bits: within 2^-8 of it) and so is the result, which is 2^-8 sum w |v| each at most; an eighth
    # more for sums and exponentials in fp32
    assert ((out.double() - ref).abs() <= 1.125 * 2.0 ** -7 * mass).all()


@pytest.mark.parametrize("q_lens,ctx", [([1], [0]), ([127], [1]), ([128], [128]), ([129], [700]), ([300, 1, 65], [0, 513, 40]), ([700], [1300])])
@pytest.mark.parametrize("heads", [(8, 4), (16, 2), (6, 1)])
@pytest.mark.parametrize("splits", [1, 2, 3, 8])
def test_pairs_and_shares(q_lens, ctx, heads, splits):
    from cuteafd_b200.ops import kernels as K
    q, kc, vc, table, sl, qs, lens, starts = _case(q_lens, ctx, *heads)
    out = torch.full_like(q, float("nan"))
    scratch = torch.full((K.attn_prefill_scratch_floats(q.shape[0], heads[0], splits),), float("nan"), device="cuda") if splits > 1 else None
    K.attn_prefill(q, kc, vc, table, sl, qs, out, max(q_lens), splits=splits, scratch=scratch)
    assert K.read_status() == 0
    _close(out, *(_ref(q, kc, c, table, lens, starts, 0, 0, None, None) for c in (vc, vc.abs())))


@pytest.mark.parametrize("window,keep", [(0, 0), (100, 0), (300, 130), (1000, 4)])
@pytest.mark.parametrize("splits", [1, 4])
def test_windows_sinks_gates(window, keep, splits):
    from cuteafd_b200.ops import kernels as K
    q, kc, vc, table, sl, qs, lens, starts = _case([260, 40], [1500, 3000], 4, 2, seed=3)
    sink, gate = torch.randn(4, device="cuda"), torch.randn(300, 4, device="cuda").to(torch.bfloat16)
    out = torch.full_like(q, float("nan"))
    scratch = torch.full((K.attn_prefill_scratch_floats(300, 4, splits),), float("nan"), device="cuda") if splits > 1 else None
    K.attn_prefill(q, kc, vc, table, sl, qs, out, 260, window=window, keep=keep, sink=sink, gate=gate, splits=splits, scratch=scratch)
    assert K.read_status() == 0
    _close(out, *(_ref(q, kc, c, table, lens, starts, window, keep, sink, gate) for c in (vc, vc.abs())))


@pytest.mark.parametrize("T", [129, 256, 257, 640])
def test_rows_of_one_head(T):
    """Expanded MLA: two row tiles of a head, the second without rows, ragged or full."""
    from cuteafd_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(T)
    heads, pages = 3, -(-T // 64)
    q = torch.randn(T, heads * 192, generator=g, device="cuda").to(torch.bfloat16)
    qr = torch.randn(T, heads, 576, generator=g, device="cuda").to(torch.bfloat16)
    k, v = (torch.randn(pages * 64, heads * 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    cache = torch.randn(pages + 1, 64, 576, generator=g, device="cuda").to(torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    table = torch.arange(1, pages + 1, dtype=torch.int32, device="cuda")[None].contiguous()
    out = torch.full((T, heads, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    K.attn_prefill_mla(q, qr, k, v, i32([0]), cache, table, i32([T]), i32([0, T]), out, T, heads, 192 ** -0.5)
    assert K.read_status() == 0
    kr = cache[1:].flatten(0, 1)[:T, 512:].double()
    ref, mass = torch.empty(2, T, heads, 128, dtype=torch.float64, device="cuda")
    for h in range(heads):
        s = q[:, h * 192:h * 192 + 128].double() @ k[:T, h * 128:(h + 1) * 128].double().T + qr[:, h, 512:].double() @ kr.T
        s = (s * 192 ** -0.5).masked_fill(~torch.ones(T, T, dtype=torch.bool, device="cuda").tril(), -math.inf)
        w, vh = torch.softmax(s, -1), v[:T, h * 128:(h + 1) * 128].double()
        ref[:, h], mass[:, h] = w @ vh, w @ vh.abs()
    _close(out, ref, mass)


@pytest.mark.parametrize("T,ctx,window", [(777, 0, 0), (130, 400, 0), (513, 200, 300)])
def test_bits_of_the_one_tile_kernel(T, ctx, window):
    """A kv head of two heads (two tiles per block) and the same head given twice (one tile per block)."""
    from cuteafd_b200.ops import kernels as K
    q, kc, vc, table, sl, qs, _, _ = _case([T], [ctx], 2, 1, seed=T)
    one, two = torch.empty_like(q), torch.empty_like(q)
    K.attn_prefill(q, kc, vc, table, sl, qs, two, T, window=window)
    K.attn_prefill(q, kc.repeat(1, 2, 1, 1), vc.repeat(1, 2, 1, 1), table, sl, qs, one, T, window=window)
    assert torch.equal(one, two)
