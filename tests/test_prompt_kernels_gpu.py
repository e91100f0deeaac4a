"""Kernels of prompt-sized steps at the sizes where their variants change over."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("T", [129, 256, 500, 777, 2300])
@pytest.mark.parametrize("N", [8, 128, 200, 2048])
def test_projections_of_chat_sized_prompts(T, N):
    """Tiles of 64, 128 and 256 features, whole and ragged, against fp64 products of the same bf16 values: one rounding to bf16 and fp32
    sums of K terms of size one."""
    from cuteafd_b200.ops import kernels as k
    K = 512
    g = torch.Generator(device=DEV).manual_seed(T + N)
    x, w, h = (torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for s in ((T, K), (N, K), (T, N)))
    want = x.double() @ w.double().T
    for got, ref in ((k.linear(x, w, out_f32=True), want), (k.linear(x, w), want), (k.linear(x, w, residual=h), want + h.double())):
        assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * K ** 0.5).all()


@pytest.mark.parametrize("K", [1408, 4096, 7168])
def test_projections_do_not_depend_on_the_tile_width(K):
    """The same rows in prompts that take tiles of 64 (up to 512 rows), 128 (777) and 256 features (2300): the same bits."""
    from cuteafd_b200.ops import kernels as k
    N = 2048
    g = torch.Generator(device=DEV).manual_seed(K)
    x, w = (torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for s in ((2300, K), (N, K)))
    wide = k.linear(x, w, out_f32=True)
    widths = [256]
    for T in (129, 512, 777):
        widths.append(k._n.cuda_lib().cafd_gemm_prompt_tile(T, N, k.num_sms()))
        assert torch.equal(k.linear(x[:T], w, out_f32=True), wide[:T])
    assert k._n.cuda_lib().cafd_gemm_prompt_tile(2300, N, k.num_sms()) == 256 and set(widths) == {64, 128, 256}


@pytest.mark.parametrize("Hq,Hkv", [(32, 4), (8, 2), (5, 1), (13, 2)])
@pytest.mark.parametrize("interleaved,rot,bias", [(False, 128, False), (True, 128, True), (False, 64, False), (True, 64, False)])
def test_rope_of_a_prompt_is_that_of_its_tokens(Hq, Hkv, interleaved, rot, bias):
    """Up to eight heads per warp and one: the same bits, head counts that share out evenly and not, dropped slots included."""
    from cuteafd_b200.ops import kernels as k
    heads, D = Hq + 2 * Hkv, 128
    T = 12 * k.num_sms() // -(-heads // 8) + 11
    per = k._n.cuda_lib().cafd_rope_heads_per_warp
    assert per(T, heads, k.num_sms()) == 8 and per(100, heads, k.num_sms()) == 1
    g = torch.Generator(device=DEV).manual_seed(Hq)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, generator=g).to(torch.bfloat16)
    qn, kn = (1 + torch.rand(D, device=DEV, generator=g)).to(torch.bfloat16), (1 + torch.rand(D, device=DEV, generator=g)).to(torch.bfloat16)
    b = torch.randn((Hq + 2 * Hkv) * D, device=DEV, generator=g).to(torch.bfloat16) if bias else None
    inv = (1e6 ** (-torch.arange(0, rot, 2, device=DEV).float() / rot)).contiguous()
    pos = torch.arange(8000, 8000 + T, dtype=torch.int32, device=DEV)
    pages = T // 64 + 2
    slots = torch.randperm(pages * 64, device=DEV, generator=g)[:T].to(torch.int32)
    slots[7] = -1
    outs = []
    for step in (T, 100):
        q = torch.zeros(T, Hq, D, dtype=torch.bfloat16, device=DEV)
        kc, vc = (torch.zeros(pages, Hkv, 64, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        for a in range(0, T, step):
            k.qk_rope_kv(qkv[a:a + step], qn, kn, inv, pos[a:a + step], slots[a:a + step], q[a:a + step], kc, vc, Hq, Hkv, D, 1e-6, interleaved, bias=b)
        outs.append((q, kc, vc))
    assert all(torch.equal(x, y) for x, y in zip(*outs))
