"""E4M3 experts expanded in the tile (csrc/gemm_w8_tcgen05.cu) against the same weights expanded in memory."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weights(E, N, Kd, seed, wild=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    codes = torch.randint(0, 256, (E, N, Kd), generator=g, device="cuda", dtype=torch.uint8)
    codes[(codes & 0x7F) == 0x7F] = 0x38                          # no NaN here
    s = torch.exp2(torch.randint(-9, -5, (E, N // 128, Kd // 128), generator=g, device="cuda").float())
    s = s * (1 + torch.rand(s.shape, generator=g, device="cuda"))
    if wild:
        s = s * torch.exp2(torch.randint(-100, 100, s.shape, generator=g, device="cuda").float())
    return codes.view(torch.float8_e4m3fn), s.contiguous()


def _exchange(E, k, H, I, counts):
    """An exchange whose routes give expert e ``counts[e]`` rows, and the rows."""
    from cuteafd_b200.parallel.moe_exchange import ExchangeGeometry, LocalExchange
    T = sum(counts)
    ex = LocalExchange(ExchangeGeometry(H, I, E, 1, T, 1), torch.device("cuda", 0))
    order = torch.randperm(T, generator=torch.Generator().manual_seed(1))
    ids = torch.tensor([e for e, n in enumerate(counts) for _ in range(n)], dtype=torch.int32)[order]
    ex.att.idx[:T, 0], ex.att.w[:T] = ids.cuda(), 1.0
    x = torch.randn(T, H, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").to(torch.bfloat16)
    return ex, x, ids.cuda()


@pytest.mark.parametrize("tile", [32, 64, 128])
@pytest.mark.parametrize("H,I", [(128, 128), (384, 256), (640, 384), (256, 1152)])
def test_expanded_in_the_tile(tile, H, I):
    """Empty, single-row, tile-edge and several-tile segments; one K block and several; odd counts of feature tiles."""
    from cuteafd_b200.ops import kernels as K
    counts = [0, 1, 31, 32, 33, 0, 63, 64, 65, 127, 128, 129, 3, 260, 0]
    E = len(counts)
    ex, x, ids = _exchange(E, 1, H, I, counts)
    wg, wu, wd = _weights(E, I, H, 3), _weights(E, I, H, 4), _weights(E, H, I, 5)
    out = torch.full_like(x, float("nan"))
    ex.att.dispatch(x, None, {}, tile, 0, ex.epoch)
    ex.exp.run_w8(wg, wu, wd, tile, 0, ex.epoch, ex.att.combine.data_ptr(), None, wait=False)
    ex.att.combine_into(out, x.shape[0], 0, ex.epoch, shared=None, residual=None, wait=False)
    assert K.read_status() == 0
    deq = [K.fp8_dequant_block128(*w).float() for w in (wg, wu, wd)]
    for e, n in enumerate(counts):
        if not n:
            continue
        rows = x[ids == e].float()
        a, b = rows @ deq[0][e].T, rows @ deq[1][e].T
        h = (torch.nn.functional.silu(a.double()) * b).to(torch.bfloat16).float()
        ref = h.double() @ deq[2][e].double().T
        # the rounding of the result (2^-8 of it), and the fc1 outputs that fp32 sums in another order round the other way: a unit of bf16 (2^-7)
        # of a few of them, taken as half of the largest term
        bound = 2.0 ** -8 * ref.abs() + 2.0 ** -8 * (h.double().abs().max() * deq[2][e].abs().max())
        assert ((out[ids == e].double() - ref).abs() <= bound).all(), e


def test_codes_and_scales_keep_their_bits():
    """One row of ones against unit columns reads single weights: the values of the expansion in memory, over scales of all sizes."""
    from cuteafd_b200.ops import kernels as K
    ex, x, _ = _exchange(2, 1, 256, 256, [128, 128])
    w = _weights(2, 256, 256, 7, wild=True)
    x.zero_()
    x[torch.arange(256), torch.arange(256)] = 1.0
    # token t is row t of an identity; expert e gets the tokens of its routes
    ex.att.dispatch(x, None, {}, 128, 0, ex.epoch)
    e = ex.exp
    K.grouped_linear_w8(e.slab, w, e.hbuf, e.tile_expert, e.tile_row0, e.num_tiles, ex.geo.max_tiles, 128, row_dst=e.row_dst,
                        out_ptr=ex.att.combine.data_ptr(), ldo=256)
    deq = K.fp8_dequant_block128(*w)
    ref = deq[ex.att.idx[:256, 0].long(), :, torch.arange(256, device="cuda")]
    assert torch.equal(ex.att.combine[:256].float(), ref.float())


def test_nan_codes_stay_nan():
    from cuteafd_b200.ops import kernels as K
    ex, x, ids = _exchange(2, 1, 256, 256, [5, 40])
    q, s = _weights(2, 256, 256, 8)
    q.view(torch.uint8)[1, 17, 33], q.view(torch.uint8)[1, 200, 255] = 0x7F, 0xFF
    ex.att.dispatch(x, None, {}, 64, 0, ex.epoch)
    e = ex.exp
    K.grouped_linear_w8(e.slab, (q, s), e.hbuf, e.tile_expert, e.tile_row0, e.num_tiles, ex.geo.max_tiles, 64, row_dst=e.row_dst,
                        out_ptr=ex.att.combine.data_ptr(), ldo=256)
    bad = torch.isnan(ex.att.combine[:45].float())
    want = torch.zeros_like(bad)
    want[:, 17] = want[:, 200] = ids == 1
    assert torch.equal(bad, want)


@pytest.mark.parametrize("T", [40, 300, 700, 2500])
def test_exchange_takes_it(T):
    """The exchange of steps past the few-row kernel, by its own rule, against the experts' formula with bf16 rows."""
    from cuteafd_b200.ops import kernels as K
    from cuteafd_b200.parallel.moe_exchange import ExchangeGeometry, LocalExchange
    H, I, E, k = 256, 128, 16, 2
    ex = LocalExchange(ExchangeGeometry(H, I, E, k, T, 1), torch.device("cuda", 0))
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    wg, wu, wd = _weights(E, I, H, 3), _weights(E, I, H, 4), _weights(E, H, I, 5)
    logits, out, res = torch.randn(T, E, device="cuda"), torch.empty_like(x), torch.empty_like(x)
    ex.forward_fp8(x, logits, dict(scoring="softmax"), wg, wu, wd, out)
    ex.forward(x, logits, dict(scoring="softmax"), *[K.fp8_dequant_block128(*w) for w in (wg, wu, wd)], res)
    assert K.read_status() == 0
    assert (out.float() - res.float()).norm() <= 2.0 ** -8 * res.float().norm()        # fp32 sums in another order, then bf16
