"""Dense products of up to 128 rows whose K range is cut over a cluster of blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from cuteafd_b200.ops import kernels
    return kernels


@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("N,Kd", [(128, 512), (200, 1000), (2048, 4096), (5120, 2048), (896, 7168), (256, 7168), (7168, 9216), (9472, 256)])
@pytest.mark.parametrize("form", ["plain", "residual", "f32", "resident"])
def test_split_product(K, T, N, Kd, form):
    """Token tiles in and out of whole ones, ragged features and K, 2 to 16 parts and shapes that stay with the other kernels (one part,
    long parts, few rows).  Twice: the partial sums' room is the ring's."""
    g = torch.Generator().manual_seed(T + N)
    dev = torch.device("cuda", 0)
    x = torch.randn(T, Kd, generator=g).to(torch.bfloat16).to(dev)
    w = (torch.randn(N, Kd, generator=g) * 0.05).to(torch.bfloat16).to(dev)
    res = torch.randn(T, N, generator=g).to(torch.bfloat16).to(dev) if form == "residual" else None
    outs = []
    for _ in range(2):
        out = torch.full((T + 1, N), 7.0, dtype=torch.float32 if form == "f32" else torch.bfloat16, device=dev)
        K.linear(x, w, out=out[:T], residual=res, out_f32=form == "f32", swap=True, resident=form == "resident")
        torch.cuda.synchronize()
        assert K.read_status() == 0 and (out[T] == 7.0).all()
        outs.append(out[:T])
    assert torch.equal(*outs)
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # fp32 sums of Kd products, an ulp each at the most (the tensor core may cut instead of round); the result's rounding to bf16
    bound = Kd * 2.0 ** -23 * size
    if res is not None:
        ref = ref + res.double()
    if form != "f32":
        bound = bound + 2.0 ** -8 * ref.abs()
    assert ((outs[0].double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("E,H,scoring", [(256, 7168, "sigmoid"), (64, 4104, "softmax")])
def test_router_apart_from_the_norm(K, E, H, scoring):
    """Rows and widths where the router's scores come from a dense product of their own: the routes are those of the one-launch form wherever
    no score is within the two sums' rounding of another."""
    assert K.norm_route_rows(E, H) == 0 and K.norm_route_rows(128, 2048) == 64 and K.norm_route_rows(256, 4096) == 16
    T, k, dev, g = 8, 6, torch.device("cuda", 0), torch.Generator().manual_seed(3)
    h, lw = torch.randn(T, H, generator=g).bfloat16().to(dev), torch.ones(H, dtype=torch.bfloat16, device=dev)
    w = (torch.randn(E, H, generator=g) * 0.05).bfloat16().to(dev)
    x = torch.empty_like(h)
    idx, wt = torch.empty(T, k, dtype=torch.int32, device=dev), torch.empty(T, k, device=dev)
    one = torch.empty(T, E, device=dev)
    K.norm_route(h, lw, 1e-6, w, x, idx, wt, k, scoring=scoring, logits_out=one)
    two = K.linear(x, w, out_f32=True, resident=True)
    idx2, wt2 = K.route_topk(two, k, scoring)
    size = x.double().abs() @ w.double().abs().T
    assert ((one - two).abs() <= 2 * H * 2.0 ** -23 * size).all()
    top = two.double().sort(1, descending=True).values[:, :k + 1]
    clear = (top[:, :-1] - top[:, 1:]).min(1).values > 4 * (one - two).abs().max()
    assert clear.any() and torch.equal(idx[clear], idx2[clear])
