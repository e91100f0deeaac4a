"""Few-row products (dense projections and routed experts of a decode step) against fp64 products of the same bf16 values."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def _close(got, want, scale):
    """One rounding to bf16 (2^-9 of the value) plus fp32 sums of ``scale``-sized terms in another order."""
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * scale).all()


@pytest.mark.parametrize("T", [1, 7, 8, 9, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("N,K", [(1, 64), (17, 768), (40, 1024), (24, 1088), (5120, 2048), (2048, 4096), (37, 7168)])
def test_dense_rows(T, N, K):
    from cuteafd_b200.ops import kernels as k
    g = torch.Generator(device=DEV).manual_seed(T * N + K)
    x, w = (torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for s in ((T, K), (N, K)))
    up = torch.randn(N, K, device=DEV, generator=g).to(torch.bfloat16)
    torch.cuda.synchronize()
    a = x.double() @ w.double().T
    scale = K ** 0.5
    _close(k.linear(x, w, out_f32=True), a, scale)
    # in rows of their own pitch, the columns between left alone
    full, hs = torch.full((T, N + 8), 7.0, dtype=torch.bfloat16, device=DEV), torch.randn(T, N + 8, device=DEV, generator=g).to(torch.bfloat16)[:, :N]
    _close(k.linear(x, w, out=full[:, :N]), a, scale)
    assert (full[:, N:] == 7.0).all()
    _close(k.linear(x, w, out=full[:, :N], residual=hs), a + hs.double(), scale)
    assert (full[:, N:] == 7.0).all()
    h = torch.randn(T, N, device=DEV, generator=g).to(torch.bfloat16)
    want = a + h.double()                         # in place, as the engines add to the residual stream
    _close(k.linear(x, w, out=h, residual=h, resident=True), want, scale)
    xs = x / scale
    b = xs.double() @ up.double().T
    c = xs.double() @ w.double().T
    _close(k.linear(xs, w, w_up=up, resident=True), torch.nn.functional.silu(c) * b, 1.0 + c.abs() + b.abs())


@pytest.mark.parametrize("N,K", [(2048, 4096), (4096, 4096), (2176, 7168), (5120, 2048)])
def test_sums_of_few_rows_lose_no_more_than_split_ones(N, K):
    """fp32 results of up to eight rows are no further from fp64 than those of the kernel that the batch-invariant mode keeps, whose blocks
    share K out (2-norms over eight draws: one and a half thousand to forty thousand values each, so the comparison is no coin's toss)."""
    from cuteafd_b200.ops import kernels as k
    off = []
    for split in (0, 64):
        k.set_fixed_kv_split(split)
        try:
            total = 0.0
            for seed in range(8):
                g = torch.Generator(device=DEV).manual_seed(seed)
                x, w = (torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for s in ((seed + 1, K), (N, K)))
                total += (k.linear(x, w, out_f32=True).double() - x.double() @ w.double().T).pow(2).sum().item()
        finally:
            k.set_fixed_kv_split(0)
        off.append(total ** 0.5)
    assert off[0] <= 1.02 * off[1]


@pytest.mark.parametrize("T,top_k,E,I,H,spread", [(1, 8, 128, 768, 2048, "random"), (3, 2, 8, 64, 128, "one"), (8, 8, 256, 192, 1088, "random"),
                                                  (11, 8, 512, 256, 512, "random"), (12, 8, 128, 768, 2048, "random"), (12, 8, 16, 128, 2048, "one"),
                                                  (5, 4, 9, 128, 1024, "outside"), (12, 8, 9, 128, 1024, "same"), (8, 8, 9, 64, 128, "same")])
def test_experts_of_a_step(T, top_k, E, I, H, spread):
    """Both expert products from the routes: spread routes, every token on the same experts, every slot on one expert (what scores that
    are no numbers give), and routes outside the stored ids."""
    from cuteafd_b200.ops import kernels as k
    g = torch.Generator(device=DEV).manual_seed(T * E)
    x = torch.randn(T, H, device=DEV, generator=g).to(torch.bfloat16)
    gate, up = ((torch.randn(E, I, H, device=DEV, generator=g) * H ** -0.5).to(torch.bfloat16) for _ in range(2))
    down = (torch.randn(E, H, I, device=DEV, generator=g) * I ** -0.5).to(torch.bfloat16)
    if spread == "same":
        idx = torch.full((T, top_k), 3, device=DEV)
        idx[1, 2] = 5
    elif spread == "one":
        idx = torch.arange(top_k, device=DEV).expand(T, top_k)
    else:
        idx = torch.rand(T, E + (2 if spread == "outside" else 0), device=DEV, generator=g).topk(top_k).indices
    idx = idx.to(torch.int32).contiguous()
    torch.cuda.synchronize()
    hbuf = torch.full((T * top_k, I), 3.0, dtype=torch.bfloat16, device=DEV)
    out = torch.full((T * top_k, H), 3.0, dtype=torch.bfloat16, device=DEV)
    count = torch.arange(E, dtype=torch.int32, device=DEV)        # added to
    assert k.moe_skinny_ok(T * top_k, T, gate, x)
    k.moe_skinny(x, top_k, gate, up, idx, hbuf, expert_count=count)
    k.moe_skinny(hbuf, 1, down, None, idx, out, early=True)
    torch.cuda.synchronize()
    flat = idx.flatten().tolist()
    for e, ex in enumerate(flat):
        if ex >= E:
            assert (hbuf[e] == 3.0).all() and (out[e] == 3.0).all()
            continue
        xe = x[e // top_k].double()
        c, b = gate[ex].double() @ xe, up[ex].double() @ xe
        _close(hbuf[e], torch.nn.functional.silu(c) * b, 1.0 + c.abs() + b.abs())
        _close(out[e], down[ex].double() @ hbuf[e].double(), 1.0)
    assert (count.cpu() - torch.arange(E)).tolist() == torch.bincount(idx.flatten()[idx.flatten() < E], minlength=E).tolist()


@pytest.mark.parametrize("fmt", ["bf16", "fp8"])
def test_expert_counts_add_up_over_steps_of_any_size(fmt):
    """A prompt-sized step, a few-row step and a prompt-sized one again: the exchange's counter holds the routes of all three."""
    from cuteafd_b200.parallel.moe_exchange import ExchangeGeometry, LocalExchange
    E, I, H, top_k = 16, 128, 256, 4
    g = torch.Generator(device=DEV).manual_seed(3)
    if fmt == "bf16":
        ws = [torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for s in ((E, I, H), (E, I, H), (E, H, I))]
    else:
        ws = [_e4m3(s, g)[:2] for s in ((E, I, H), (E, I, H), (E, H, I))]
    ex = LocalExchange(ExchangeGeometry(H, I, E, top_k, 64, 1), DEV)
    seen = []
    for T in (40, 5, 1, 40):
        idx = torch.rand(T, E, device=DEV, generator=g).topk(top_k).indices.to(torch.int32)
        ex.att.idx[:T], ex.att.w[:T] = idx, 1.0 / top_k
        seen.append(idx.flatten())
        x = torch.randn(T, H, device=DEV, generator=g).to(torch.bfloat16)
        (ex.forward if fmt == "bf16" else ex.forward_fp8)(x, None, {}, *ws, torch.empty_like(x))
    assert torch.equal(ex.att.expert_count.long(), torch.bincount(torch.cat(seen).long(), minlength=E))


def _e4m3(shape, g):
    """E4M3 values over the whole finite range (subnormals and zeros among them), a scale for every 128 x 128 block, and the fp64 weights."""
    byte = torch.randint(0, 256, shape, device=DEV, generator=g).to(torch.uint8)
    byte[(byte & 0x7f) == 0x7f] = 0                               # the two NaN codes
    q = byte.view(torch.float8_e4m3fn)
    s = (0.5 + torch.rand(*shape[:-2], shape[-2] // 128, shape[-1] // 128, device=DEV, generator=g)) * 2.0 ** -9
    return q, s, q.double() * s.double().repeat_interleave(128, -2).repeat_interleave(128, -1)


@pytest.mark.parametrize("T", [1, 5, 8])
@pytest.mark.parametrize("N,K", [(128, 128), (256, 384), (384, 2048), (1536, 7168), (7168, 2304)])
def test_e4m3_rows(T, N, K):
    from cuteafd_b200.ops import kernels as k
    g = torch.Generator(device=DEV).manual_seed(N + K + T)
    x = (torch.randn(T, K, device=DEV, generator=g) * K ** -0.5).to(torch.bfloat16)
    (q, s, w), (qu, su, wu) = _e4m3((N, K), g), _e4m3((N, K), g)
    h = torch.randn(T, N, device=DEV, generator=g).to(torch.bfloat16)
    torch.cuda.synchronize()
    a, b = x.double() @ w.T, x.double() @ wu.T
    want = a + h.double()
    _close(k.linear_w8(x, q, s, torch.empty_like(h)), a, 1.0)
    _close(k.linear_w8(x, q, s, h, residual=h, resident=True), want, 1.0)
    _close(k.linear_w8(x, q, s, torch.empty_like(h), w_up=qu, ws_up=su), torch.nn.functional.silu(a) * b, 1.0 + a.abs() + b.abs())


@pytest.mark.parametrize("T,top_k,E,I,H,spread", [(1, 8, 256, 256, 384, "random"), (8, 8, 256, 128, 2304, "random"), (3, 2, 4, 384, 128, "random"),
                                                  (8, 8, 5, 128, 384, "same"), (8, 4, 6, 256, 256, "outside")])
def test_e4m3_experts_of_a_step(T, top_k, E, I, H, spread):
    """Spread routes, more routes on one expert than a column tile holds, and routes outside the stored ids."""
    from cuteafd_b200.ops import kernels as k
    g = torch.Generator(device=DEV).manual_seed(T + E)
    x = (torch.randn(T, H, device=DEV, generator=g) * H ** -0.5).to(torch.bfloat16)
    (qg, sg, gate), (qu, su, up), (qd, sd, down) = _e4m3((E, I, H), g), _e4m3((E, I, H), g), _e4m3((E, H, I), g)
    if spread == "same":
        idx = torch.full((T, top_k), 3, device=DEV)
        idx[1, 2] = 4
    else:
        idx = torch.rand(T, E + (2 if spread == "outside" else 0), device=DEV, generator=g).topk(top_k).indices
    idx = idx.to(torch.int32).contiguous()
    torch.cuda.synchronize()
    hbuf, out = (torch.full((T * top_k, n), 3.0, dtype=torch.bfloat16, device=DEV) for n in (I, H))
    assert k.moe_skinny_w8_ok(T * top_k, T, qg, x) and k.moe_skinny_w8_ok(T * top_k, T, qd, x)
    k.moe_skinny(x, top_k, qg, qu, idx, hbuf, scale=sg, scale_up=su)
    k.moe_skinny(hbuf, 1, qd, None, idx, out, scale=sd, early=True)
    for e, ex in enumerate(idx.flatten().tolist()):
        if ex >= E:
            assert (hbuf[e] == 3.0).all() and (out[e] == 3.0).all()
            continue
        c, b = gate[ex] @ x[e // top_k].double(), up[ex] @ x[e // top_k].double()
        _close(hbuf[e], torch.nn.functional.silu(c) * b, 1.0 + c.abs() + b.abs())
        _close(out[e], down[ex] @ hbuf[e].double(), I ** 0.5 * float(hbuf[e].abs().max()))


def test_e4m3_rows_of_any_size():
    """Values from bf16 subnormals to near its largest number, alone in a row and side by side in one 128-wide block: off the fp64 product by
    what fp32 sums lose (a few 2^-24 of the terms' absolute sum) and one rounding to bf16; infinities and NaN come through."""
    from cuteafd_b200.ops import kernels as k
    g = torch.Generator(device=DEV).manual_seed(11)
    N, K = 256, 512
    q, s, w = _e4m3((N, K), g)
    x = torch.randn(8, K, device=DEV, generator=g).double()
    x[0] *= 2.0 ** -130
    x[1] *= 2.0 ** 112
    x[2] *= 2.0 ** torch.randint(-60, 60, (K,), device=DEV, generator=g)
    x[3] *= 2.0 ** torch.randint(-24, 1, (K,), device=DEV, generator=g)
    x[4, 128:] = 0
    x[5] = 0
    x[6] *= 70000.0
    x = x.to(torch.bfloat16)
    want, size = x.double() @ w.T, x.double().abs() @ w.abs().T
    got = k.linear_w8(x, q, s, torch.empty(8, N, dtype=torch.bfloat16, device=DEV)).double()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * size + 2.0 ** -133).all()
    x[0, 7], x[1, 300] = float("inf"), float("nan")
    got = k.linear_w8(x, q, s, torch.empty(8, N, dtype=torch.bfloat16, device=DEV))
    assert torch.equal(got[2:].double(), k.linear_w8(x[2:], q, s, torch.empty(6, N, dtype=torch.bfloat16, device=DEV)).double())
    assert not got[:2].isfinite().any() and got[1].isnan().all()


def test_e4m3_nan_codes_stay_nan():
    """A weight row that holds one of the two NaN codes gives NaN in its feature for every row of x, zero rows included, as the tensor-core
    products of larger steps do; every other feature is untouched."""
    from cuteafd_b200.ops import kernels as k
    g = torch.Generator(device=DEV).manual_seed(5)
    T, N, K, E = 6, 256, 1152, 4
    x = (torch.randn(T, K, device=DEV, generator=g) * K ** -0.5).to(torch.bfloat16)
    x[2] = 0
    q, s, _ = _e4m3((N, K), g)
    clean = k.linear_w8(x, q, s, torch.empty(T, N, dtype=torch.bfloat16, device=DEV))
    bad = {0: (0, 0x7f), 5: (K - 1, 0xff), 8: (77, 0x7f), 130: (640, 0xff), N - 1: (3, 0xff)}
    qb = q.clone()
    for row, (col, code) in bad.items():
        qb.view(torch.uint8)[row, col] = code
    rows = torch.zeros(N, dtype=torch.bool, device=DEV)
    rows[list(bad)] = True
    for up in (None, q):
        got = k.linear_w8(x, qb, s, torch.empty_like(clean), w_up=up, ws_up=s if up is not None else None)
        assert got[:, rows].isnan().all() and got[:, ~rows].isfinite().all()
        assert up is not None or torch.equal(got[:, ~rows], clean[:, ~rows])
    assert k.linear_w8(x, q, s, torch.empty_like(clean), w_up=qb, ws_up=s)[:, rows].isnan().all()
    (qe, se, _), (qu, su, _) = _e4m3((E, N, K), g), _e4m3((E, N, K), g)
    qe.view(torch.uint8)[2, 9, 200] = 0x7f
    idx = torch.tensor([[0, 1], [2, 3], [3, 0], [1, 2], [0, 3], [1, 0]], dtype=torch.int32, device=DEV)
    h = torch.empty(T * 2, N, dtype=torch.bfloat16, device=DEV)
    k.moe_skinny(x, 2, qe, qu, idx, h, scale=se, scale_up=su)
    want = torch.zeros(T * 2, N, dtype=torch.bool, device=DEV)
    want[:, 9] = idx.flatten() == 2
    assert torch.equal(h.isnan(), want)
