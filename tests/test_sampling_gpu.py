"""GPU target sampler and accept-prefix scan against the CPU oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_sample_rows_match_oracle():
    from cuteafd_b200.ops import kernels as K
    from cuteafd_b200.runtime.sampling import SamplingParams, select_rows
    dev = torch.device("cuda", 0)
    V = 5003
    g = torch.Generator().manual_seed(0)
    cases = [SamplingParams(), SamplingParams(temperature=0.7, seed=1), SamplingParams(temperature=1.0, top_k=5, seed=2),
             SamplingParams(temperature=1.3, top_p=0.9, seed=3), SamplingParams(temperature=0.9, min_p=0.05, seed=4),
             SamplingParams(temperature=1.0, top_k=50, top_p=0.8, min_p=0.01, seed=5), SamplingParams(temperature=2.0, top_k=1, seed=6),
             SamplingParams(temperature=0.3, top_p=0.5, seed=7), SamplingParams(temperature=1.0, top_k=V + 10, seed=8)]
    params, positions = [], []
    for rep in range(6):
        for c in cases:
            params.append(SamplingParams(c.temperature, c.top_p, c.top_k, c.min_p, c.seed + 100 * rep))
            positions.append(17 + 1000 * rep + len(params))
    n = len(params)
    logits = torch.randn(n, V, generator=g) * 3.0
    logits[3, 100:110] = logits[3].max() + 1.0            # a block of exact ties at the top
    logits[5, ::7] = 2.5                                  # many ties in the middle
    masks = [None] * n
    words = (V + 31) // 32
    mask_bits = torch.zeros(n, words, dtype=torch.int32)
    mask_word0 = [None] * n
    for i in range(0, n, 4):
        m = torch.rand(V, generator=g) < 0.3
        m[int(torch.randint(0, V, (1,), generator=g))] = True
        masks[i] = m
        padded = torch.zeros(words * 32, dtype=torch.bool); padded[:V] = m
        w = (padded.view(words, 32).long() << torch.arange(32)).sum(1)
        mask_bits[i] = torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32)
        mask_word0[i] = i * words
    want, want_status = select_rows(logits, params, positions, masks)
    rows = K.pack_sample_rows(params, positions, mask_word0=mask_word0).to(dev)
    tok = torch.full((n,), -7, dtype=torch.int32, device=dev)
    st = torch.full((n,), -7, dtype=torch.int32, device=dev)
    for _ in range(2):
        K.sample_rows(logits.to(dev), rows, tok, st, mask_bits.to(dev))
    torch.cuda.synchronize()
    assert st.tolist() == want_status
    got = tok.tolist()
    bad = [i for i in range(n) if got[i] != want[i]]
    assert not bad, [(i, got[i], want[i], params[i]) for i in bad[:5]]


def test_sample_row_errors_and_accept_prefix():
    from cuteafd_b200.ops import kernels as K
    from cuteafd_b200.runtime.sampling import STATUS_EMPTY_MASK, STATUS_NONFINITE, SamplingParams, accept_prefix
    dev = torch.device("cuda", 0)
    V = 300
    logits = torch.randn(3, V)
    logits[1, 5] = float("nan")
    mask_bits = torch.zeros(3, (V + 31) // 32, dtype=torch.int32)
    params = [SamplingParams(temperature=1.0)] * 3
    rows = K.pack_sample_rows(params, [0, 1, 2], mask_word0=[None, None, 2 * mask_bits.shape[1]]).to(dev)
    tok = torch.zeros(3, dtype=torch.int32, device=dev); st = torch.zeros(3, dtype=torch.int32, device=dev)
    K.sample_rows(logits.to(dev), rows, tok, st, mask_bits.to(dev))
    assert st.tolist() == [0, STATUS_NONFINITE, STATUS_EMPTY_MASK] and tok.tolist()[1:] == [-1, -1]
    # accept-prefix: three sequences with 4, 1 and 3 rows
    selected = [5, 6, 7, 8, 9, 1, 2, 3]
    draft = [5, 6, 0, 0, 0, 1, 2, 0]
    row_start = [0, 4, 5, 8]
    i32 = dict(dtype=torch.int32, device=dev)
    acc = torch.zeros(3, **i32); bonus = torch.zeros(3, **i32)
    K.accept_prefix(torch.tensor(selected, **i32), torch.tensor(draft, **i32), torch.tensor(row_start, **i32), acc, bonus)
    want = [accept_prefix(selected[a:b], draft[a:b - 1]) for a, b in zip(row_start[:-1], row_start[1:])]
    assert list(zip(acc.tolist(), bonus.tolist())) == want


@pytest.mark.parametrize("V", [1, 7, 8, 1023, 8 * 1024 + 5, 131071, 262147, 8 * 48 * 1024 - 3, 8 * 48 * 1024 + 11])
@pytest.mark.parametrize("shape", ["peaked", "flat", "ties"])
def test_sample_rows_over_vocabularies(V, shape):
    """Slices that are empty, ragged, in shared memory and too long for it; tokens above the line that fit the sorted list (peaked) and
    that do not (flat, ties).  Values lie on a grid of 1/64, so that the oracle's fp64 masses and the kernel's differ by rounding alone."""
    from cuteafd_b200.ops import kernels as K
    from cuteafd_b200.runtime.sampling import SamplingParams, select_rows
    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(V)
    params = [SamplingParams(temperature=1.0, seed=1), SamplingParams(temperature=0.5, top_p=0.9, seed=2), SamplingParams(temperature=1.0, top_k=50, top_p=0.95, seed=3),
              SamplingParams(temperature=2.0, top_k=3000, seed=4), SamplingParams(temperature=1.0, min_p=0.02, top_p=0.8, seed=5), SamplingParams()]
    n = len(params)
    logits = torch.randn(n, V, generator=g)
    if shape == "peaked":
        logits = logits * 2
        logits[:, :: max(1, V // 100)] += 12.0
    logits = (logits * 64).round() / 64 if shape != "ties" else (logits * 2).round() / 2              # zeros of both signs among them
    positions = [11 * i + V for i in range(n)]
    want, status = select_rows(logits, params, positions, [None] * n)
    tok = torch.full((n,), -7, dtype=torch.int32, device=dev)
    st = torch.full((n,), -7, dtype=torch.int32, device=dev)
    K.sample_rows(logits.to(dev), K.pack_sample_rows(params, positions).to(dev), tok, st)
    assert st.tolist() == status and tok.tolist() == want


@pytest.mark.parametrize("n,V,blocks", [(74, 32003, 4), (148, 32003, 2), (150, 20481, 2), (300, 1, 1), (300, 9, 1), (300, 2500, 1), (300, 20479, 1)])
@pytest.mark.parametrize("shape", ["flat", "ties"])
def test_sample_many_rows(n, V, blocks, shape):
    """Batches whose rows get four, two and one block each, every third row under a mask of allowed tokens."""
    from cuteafd_b200.ops import kernels as K
    from cuteafd_b200.runtime.sampling import SamplingParams, select_rows
    dev = torch.device("cuda", 0)
    kinds = [dict(temperature=1.0), dict(temperature=0.5, top_p=0.9), dict(temperature=1.0, top_k=50, top_p=0.95), dict(temperature=2.0, top_k=3000),
             dict(temperature=1.0, min_p=0.02, top_p=0.8), dict()]
    params = [SamplingParams(seed=i, **kinds[i % 6]) for i in range(n)]
    positions = [7 * i for i in range(n)]
    g = torch.Generator().manual_seed(n + V)
    logits = torch.randn(n, V, generator=g)
    logits = (logits * 64).round() / 64 if shape == "flat" else (logits * 2).round() / 2
    words = (V + 31) // 32
    allowed = torch.rand(words * 32, generator=g) < 0.3
    allowed[0] = True
    w = (allowed.view(words, 32).long() << torch.arange(32)).sum(1)
    bits = torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32)
    assert K._n.cuda_lib().cafd_sample_cluster(n, V, 148) == blocks
    tok, st = (torch.full((n,), -7, dtype=torch.int32, device=dev) for _ in range(2))
    rows = K.pack_sample_rows(params, positions, mask_word0=[0 if i % 3 == 0 else None for i in range(n)]).to(dev)
    K.sample_rows(logits.to(dev), rows, tok, st, masks=bits.to(dev))
    some = list(range(0, n, 11))
    want, status = select_rows(logits[some], [params[i] for i in some], [positions[i] for i in some],
                               [allowed[:V] if i % 3 == 0 else None for i in some])
    assert not st.any() and tok[some].tolist() == want and status == [0] * len(some)


@pytest.mark.parametrize("V", [40, 6000])
def test_zeros_of_both_signs_are_one_value(V):
    """The lowest id wins a tie also between 0.0 and -0.0: at the top-k boundary, in the nucleus and in the draw, with few tokens above the
    line and with many."""
    from cuteafd_b200.ops import kernels as K
    from cuteafd_b200.runtime.sampling import SamplingParams, select_rows
    dev = torch.device("cuda", 0)
    kinds = [dict(top_k=5), dict(top_k=V - 7), dict(top_p=0.5), dict(), dict(min_p=0.9, top_k=3)]
    params = [SamplingParams(temperature=1.0 + 0.1 * (i % 3), seed=i, **kinds[i % len(kinds)]) for i in range(40)]
    logits = torch.zeros(40, V)
    logits[:, ::2] = -0.0
    logits[::2, V // 2] = 1.0
    logits[:, V - 4:] = -3.0
    positions = list(range(40))
    want, status = select_rows(logits, params, positions, [None] * 40)
    tok, st = (torch.full((40,), -7, dtype=torch.int32, device=dev) for _ in range(2))
    K.sample_rows(logits.to(dev), K.pack_sample_rows(params, positions).to(dev), tok, st)
    assert st.tolist() == status and tok.tolist() == want


@pytest.mark.parametrize("n", [6, 300])
@pytest.mark.parametrize("V,ld", [(3, 4), (2047, 2050), (2048, 2048), (2050, 2052), (16387, 16389), (16388, 16392)])
@pytest.mark.parametrize("first", [0, 1])
def test_sample_rows_of_any_alignment(n, V, ld, first):
    """Rows that start on a 16-byte boundary and rows that don't, whole and broken groups of four tokens, with and without a mask."""
    from cuteafd_b200.ops import kernels as K
    from cuteafd_b200.runtime.sampling import SamplingParams, select_rows
    dev = torch.device("cuda", 0)
    kinds = [dict(), dict(temperature=0.7, top_k=50, top_p=0.95), dict(temperature=1.0, top_p=0.8)]
    params = [SamplingParams(seed=i, **kinds[i % 3]) for i in range(n)]
    g = torch.Generator().manual_seed(V + ld)
    whole = torch.full((n * ld + 8,), float("nan"))                     # what lies between rows is nobody's token
    on_host = whole[first:].as_strided((n, V), (ld, 1))
    on_host.copy_((torch.randn(n, V, generator=g) * 128).round() / 64)
    logits = whole.to(dev)[first:].as_strided((n, V), (ld, 1))
    words = (V + 31) // 32
    allowed = torch.rand(words * 32, generator=g) < 0.4
    allowed[V - 1] = True
    w = (allowed.view(words, 32).long() << torch.arange(32)).sum(1)
    bits = torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32).to(dev)
    tok, st = (torch.full((n,), -7, dtype=torch.int32, device=dev) for _ in range(2))
    rows = K.pack_sample_rows(params, list(range(n)), mask_word0=[0 if i % 2 else None for i in range(n)]).to(dev)
    K.sample_rows(logits, rows, tok, st, masks=bits)
    some = list(range(0, n, 1 if n < 10 else 23))
    want, status = select_rows(on_host[some].contiguous(), [params[i] for i in some], some, [allowed[:V] if i % 2 else None for i in some])
    assert not st.any() and status == [0] * len(some) and tok[some].tolist() == want


@pytest.mark.parametrize("V", [4097, 60011, 151936])
@pytest.mark.parametrize("shape", ["peaked", "flat", "steps", "one thread", "negative"])
def test_lines_from_the_threads_best_tokens(V, shape):
    """Rows whose candidates are few and near, too many, tied over whole bins, or all in neighbouring tokens, under every order of filters."""
    from cuteafd_b200.ops import kernels as K
    from cuteafd_b200.runtime.sampling import SamplingParams, select_rows
    g = torch.Generator().manual_seed(V)
    params = [SamplingParams(temperature=t, top_k=k, top_p=p, min_p=m, seed=7 * i)
              for i, (t, k, p, m) in enumerate([(1.0, None, 0.9, 0.0), (0.7, 50, 0.95, 0.0), (0.6, 1000, 1.0, 0.0), (1.0, 4000, 0.9, 0.0), (1.5, None, 1.0, 0.0),
                                                (0.8, 20, 0.8, 0.05), (1.0, None, 0.99, 0.1), (0.05, 50, 0.9, 0.0), (2.0, None, 0.3, 0.0)])]
    n = len(params)
    x = torch.randn(n, V, generator=g) * 2
    if shape == "peaked":
        x[:, torch.randperm(V, generator=g)[:300]] += 9
    elif shape == "flat":
        x *= 0.05
    elif shape == "steps":
        x = (x * 2).round() / 2                                   # values on the bins' edges, ties everywhere
    elif shape == "one thread":
        x[:, 1000:3000] += 8                                      # 2000 neighbours: more than a block notes
    else:
        x = x.abs().neg() * 50 - 1000
    want, status = select_rows(x, params, list(range(n)), [None] * n)
    rows = K.pack_sample_rows(params, list(range(n))).cuda()
    tok, st = torch.full((n,), -7, dtype=torch.int32, device="cuda"), torch.full((n,), -7, dtype=torch.int32, device="cuda")
    K.sample_rows(x.cuda(), rows, tok, st)
    assert st.tolist() == status and tok.tolist() == want
