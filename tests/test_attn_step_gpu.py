"""One-launch attention of a decode step (csrc/attention_step.cu): caches against the rotation kernel's bits, outputs against 64-bit attention."""
import pytest
import torch

from .test_attn_pair_gpu import _case, _close, _ref

pytestmark = pytest.mark.gpu


def _step(lens, Hq, Hkv, splits, window=0, rot=128, interleaved=False, norm=True, bias=False, early=False):
    from cuteafd_b200.ops import kernels as K
    n = len(lens)
    _, kc, vc, table, sl, qs, _, starts = _case([1] * n, [x - 1 for x in lens], Hq, Hkv, seed=sum(lens))
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    qkv, b = 2 * r(n, (Hq + 2 * Hkv) * 128), r((Hq + 2 * Hkv) * 128) if bias else None
    qn, kn = (1 + r(128) / 8, 1 + r(128) / 8) if norm else (None, None)
    inv = 10000.0 ** (-torch.arange(rot // 2, device="cuda").float() * 2 / rot)
    pos = sl - 1
    slots = (table[torch.arange(n, device="cuda"), (pos // 64).long()] * 64 + pos % 64).to(torch.int32)
    k1, v1, q = kc.clone(), vc.clone(), torch.empty(n, Hq, 128, dtype=torch.bfloat16, device="cuda")
    K.qk_rope_kv(qkv, qn, kn, inv, pos, slots, q, k1, v1, Hq, Hkv, 128, 1e-6, interleaved, bias=b)
    out = torch.full((n, Hq, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    K.attn_step(qkv, qn, kn, inv, pos, slots, kc, vc, table, sl, qs, out, Hq, 1e-6, interleaved, splits, bias=b, window=window, resident=early)
    torch.cuda.synchronize()
    assert torch.equal(kc, k1) and torch.equal(vc, v1)
    _close(out, *(_ref(q, k1, c, table, lens, starts, window, 0, None, None) for c in (v1, v1.abs())))


@pytest.mark.parametrize("lens", [[1], [64], [65], [1000], [1, 63, 64, 65, 128, 129, 700, 2111]])
@pytest.mark.parametrize("heads", [(4, 4), (8, 4), (16, 2), (6, 2), (32, 2)])
@pytest.mark.parametrize("splits", [1, 2, 5, 10, 16])
def test_lengths_heads_splits(lens, heads, splits):
    _step(lens, *heads, splits)


@pytest.mark.parametrize("kw", [dict(rot=64), dict(rot=64, interleaved=True), dict(interleaved=True), dict(norm=False), dict(bias=True), dict(early=True),
                                dict(window=1), dict(window=64), dict(window=100), dict(window=600)])
def test_options(kw):
    _step([3, 130, 1025], 8, 2, 4, **kw)


def test_many_blocks():
    """More blocks than run at once, and every stage of the rings."""
    _step([64 * (i % 9) + 1 + i for i in range(60)], 8, 4, 8)


def test_rows_without_slot_and_sequences_without_row():
    from cuteafd_b200.ops import kernels as K
    _, kc, vc, table, sl, _, _, _ = _case([1, 1, 1], [99, 199, 299], 8, 2)
    qs = torch.tensor([0, 1, 1, 2], dtype=torch.int32, device="cuda")           # the second sequence has no row
    qkv = torch.randn(2, 12 * 128, device="cuda").to(torch.bfloat16)
    inv = 10000.0 ** (-torch.arange(64, device="cuda").float() / 64)
    pos = torch.tensor([99, 299], dtype=torch.int32, device="cuda")
    slots = torch.tensor([-1, int(table[2, 4]) * 64 + 43], dtype=torch.int32, device="cuda")
    k0 = kc.clone()
    out = torch.full((2, 8, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    K.attn_step(qkv, None, None, inv, pos, slots, kc, vc, table, sl, qs, out, 8, 1e-6, False, 4)
    changed = (kc != k0).flatten(2).any(2).nonzero()[:, 0].unique().tolist()
    assert changed == [int(table[2, 4])] and bool(torch.isfinite(out.float()).all())
