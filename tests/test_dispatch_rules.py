"""Rules that pick a kernel's form from sizes alone, checked on the host."""
import ctypes as C

import pytest
import torch

from cuteafd_b200._native import lib as _n


@pytest.mark.parametrize("sms", [20, 148, 160])
def test_prompt_tiles_are_narrow_only_while_they_all_run_at_once(sms):
    """A narrow tile takes more than half a wide one's time: one wave of them at most, the narrowest such width, else the wide one."""
    tile = _n.cuda_lib().cafd_gemm_prompt_tile
    for rows in (1, 128, 129, 300, 640, 777, 1300, 8192, 2 ** 31 - 1):
        for n in (1, 64, 65, 128, 2048, 4096, 5120, 37984, 2 ** 31 - 1):
            blocks = {w: -(-rows // 128) * -(-n // w) for w in (64, 128)}
            want = next((w for w in (64, 128) if blocks[w] <= sms), 256)
            assert tile(rows, n, sms) == want, (rows, n)


def test_sampler_blocks_per_row():
    """Eight blocks for a row, fewer while that makes the whole batch resident at once (two blocks to an SM) and a slice's keys still fit
    beside another block's."""
    blocks = _n.cuda_lib().cafd_sample_cluster
    for sms in (20, 148):
        for n in (1, 2, 5, 37, 38, 74, 75, 148, 149, 296, 297, 4096):
            for V in (0, 1, 1000, 20479, 20480, 40960, 151936, 262144, 2 ** 31 - 1):
                c = blocks(n, V, sms)
                assert c in (1, 2, 4, 8)
                assert c == 8 or (2 * n * c > 2 * sms and V // c < 20480)                      # the next larger size isn't resident, the slice fits
                assert c == 1 or n * c <= 2 * sms or V // (c // 2) >= 20480


def _few(rows, n, k, sms, dual=False, **kw):
    a = _n.GemmArgs()
    a.w0, a.x, a.out, a.w1 = 1 << 20, 1 << 21, 1 << 22, (1 << 23) if dual else None
    a.k, a.n_features, a.x_rows, a.ldo, a.swap, a.dual, a.bx, a.num_sms = k, n, rows, n, 1, int(dual), 32, sms
    for name, v in kw.items():
        setattr(a, name, v)
    return bool(_n.cuda_lib().cafd_gemm_few_rows(C.byref(a)))


def test_few_row_products_count_tiles_against_the_sms_that_they_get():
    for sms in (40, 148):
        for rows, waves in ((16, 4), (17, 1), (32, 1)):
            assert _few(rows, 16 * waves * sms, 2048, sms) and not _few(rows, 16 * waves * sms + 1, 2048, sms)
            assert _few(rows, 8 * waves * sms, 2048, sms, dual=True) and not _few(rows, 8 * waves * sms + 1, 2048, sms, dual=True)
        assert _few(8, 32 * sms, 7168, sms) and not _few(8, 32 * sms + 1, 7168, sms)
    assert not _few(33, 64, 2048, 148)


def test_few_row_products_end_where_the_weights_outgrow_their_advantage():
    """Both kernels timed at these sizes: the largest that the few-row one wins, the smallest that it loses."""
    assert _few(1, 65536, 1024, 148) and _few(8, 32000, 4096, 148) and not _few(1, 151936, 2048, 148)
    assert _few(8, 10944, 4096, 148, dual=True) and not _few(1, 14336, 4096, 148, dual=True)


def test_few_row_products_leave_every_other_form_alone():
    ok = dict(rows=8, n=1024, k=2048, sms=148)
    assert _few(**ok)
    for kw in (dict(swap=0), dict(fp8=1), dict(k=2056), dict(tile_expert=1), dict(row_dst=1), dict(row_scale=1), dict(wait_flag=1), dict(signal_flag=1),
               dict(rs_ranks=2), dict(n_signal_flags=1), dict(w0=8), dict(x=8), dict(x_rows=0)):
        assert not _few(**{**ok, **{k: v for k, v in kw.items() if k in ok}}, **{k: v for k, v in kw.items() if k not in ok}), kw
    assert not _few(dual=True, glu=1, **ok) and not _few(dual=True, w1_row_offset=8, **ok)


def test_few_row_experts_by_the_size_of_a_matrix():
    from cuteafd_b200.ops import kernels as K
    for (E, I, H), most in (((128, 768, 2048), 12), ((64, 1024, 2048), 12), ((56, 1536, 4096), 12), ((128, 1408, 4096), 8), ((256, 2048, 7168), 8), ((8, 14336, 4096), 12)):
        for shape in ((E, I, H), (E, H, I)):
            w = torch.empty(shape, dtype=torch.bfloat16, device="meta")
            x = torch.empty(16, shape[2], dtype=torch.bfloat16, device="meta")
            assert [K.moe_skinny_ok(2 * T, T, w, x) for T in range(1, 17)] == [T <= most for T in range(1, 17)]


# us of a whole exchange with row tiles of 16 / 32 / 64 / 128, by geometry and mean segment length
TILE_TIMES = {
    (64, 1024, 2048): {9: (179, 196, 251, 229), 12: (179, 197, 252, 230), 15: (190, 198, 245, 225), 16: (202, 191, 246, 225), 20: (223, 201, 255, 229), 24: (221, 202, 257, 232),
                       26: (247, 206, 258, 231), 32: (276, 243, 249, 226), 48: (352, 273, 262, 228)},
    (56, 1536, 4096): {8.04: (380, 398, 462, 419), 11: (375, 399, 464, 420), 16: (424, 400, 470, 423), 20.1: (487, 400, 474, 426), 24: (531, 397, 477, 424), 26: (531, 396, 483, 426), 32: (616, 448, 479, 423)},
    (8, 14336, 4096): {10: (488, 501, 536, 523), 14: (540, 504, 533, 519), 16: (556, 508, 535, 526), 21: (668, 506, 538, 529), 24: (688, 504, 539, 529), 26: (688, 509, 539, 529), 44: (987, 681, 538, 527)},
    (128, 768, 2048): {9: (241, 284, 381, 305), 12: (250, 293, 395, 313), 16: (274, 297, 396, 317), 21: (311, 301, 401, 317), 26: (328, 308, 400, 309), 32: (382, 358, 413, 317)},
    (128, 1408, 4096): {9: (738, 789, 966, 792), 11: (732, 791, 953, 785), 16: (838, 792, 963, 795), 22: (1025, 789, 983, 800), 24: (1061, 816, 975, 799), 32: (1231, 944, 995, 806)},
    (256, 2048, 7168): {8: (3860, 4028, 4306, 3570), 16: (4881, 3815, 4328, 3628), 20: (6120, 3855, 4353, 3605), 24: (5436, 3892, 4434, 3622), 32: (7534, 4247, 4413, 3625)},
}


def test_row_tiles_are_the_faster_ones_at_every_geometry_measured():
    """Within 3 % of the better of the two rules that knew the mean segment alone (16 / 32 / 64 / 128 up to 8 / 24 / 48 rows, and 16 / 32 / 128
    up to 16 / 20), which lost up to a third of each other's time."""
    from cuteafd_b200.parallel.moe_exchange import pick_tile_rows, plan_tile_rows
    for (E, ffn, hidden), rows in TILE_TIMES.items():
        for avg, us in rows.items():
            took = dict(zip((16, 32, 64, 128), us))
            a, b = 16 if avg <= 8 else 32 if avg <= 24 else 64 if avg <= 48 else 128, 16 if avg <= 16 else 32 if avg <= 20 else 128
            got = pick_tile_rows(round(avg * E), 1, E, ffn, hidden)
            assert took[got] <= 1.03 * min(took[a], took[b]), (E, ffn, hidden, avg, got)
            assert plan_tile_rows("bf16", round(avg * E), 1, E, ffn, hidden) == got
    assert [plan_tile_rows("fp32", 16 * n, 1, 16) for n in (8, 9, 24, 25, 47, 48)] == [16, 32, 32, 64, 64, 128]


def test_rotation_shares_angles_once_there_are_warps_enough():
    """By the warps that the step has, not by its tokens: a shard with few heads needs more of them."""
    per = _n.cuda_lib().cafd_rope_heads_per_warp
    for sms in (40, 148):
        for heads in (3, 6, 10, 40, 112):
            T = -(-12 * sms // -(-heads // 8))
            assert per(1, heads, sms) == per(T - 1, heads, sms) == 1 and per(T, heads, sms) == per(1 << 20, heads, sms) == 8


def test_few_row_operands_are_checked_before_their_addresses_are_used():
    """Shapes, types and layouts that the kernel doesn't look at are refused by the wrappers; nothing here reaches a device."""
    from cuteafd_b200.ops import kernels as K
    bf, f8 = torch.bfloat16, torch.float8_e4m3fn
    E, N, Kd, T, k = 4, 128, 256, 3, 2

    def t(*shape, dtype=bf):
        return torch.zeros(*shape, dtype=dtype)
    ok = dict(x=t(T, Kd), row_div=k, w=t(E, N, Kd), w_up=t(E, N, Kd), idx=t(T, k, dtype=torch.int32), out=t(T * k, N))
    f8s = dict(ok, w=t(E, N, Kd, dtype=f8), w_up=t(E, N, Kd, dtype=f8), scale=t(E, 1, 2, dtype=torch.float32), scale_up=t(E, 1, 2, dtype=torch.float32))
    for base, bad in ((ok, dict(idx=t(T, k, dtype=torch.int64))), (ok, dict(w_up=t(E, N, Kd // 2))), (ok, dict(w_up=t(E, N, Kd, dtype=f8))), (ok, dict(w_up=t(E, Kd, N).mT)),
                      (ok, dict(out=t(T * k - 1, N))), (ok, dict(out=t(T * k, N, dtype=torch.float32))), (ok, dict(out=t(T * k, N - 1))), (ok, dict(x=t(T - 1, Kd))),
                      (ok, dict(x=t(T, Kd, dtype=torch.float16))), (ok, dict(x=t(T, 2 * Kd)[:, ::2])), (ok, dict(w=t(E, N, Kd, dtype=f8))), (ok, dict(scale_up=t(E, 1, 2, dtype=torch.float32))),
                      (ok, dict(expert_count=t(E - 1, dtype=torch.int32))), (ok, dict(expert_count=t(E, dtype=torch.int64))), (f8s, dict(scale_up=None)),
                      (f8s, dict(scale_up=t(E, 2, 1, dtype=torch.float32))), (f8s, dict(scale_up=t(E, 1, 2))), (f8s, dict(scale=t(E, 1, 1, dtype=torch.float32))), (f8s, dict(w_up=t(E, N, Kd)))):
        with pytest.raises(AssertionError):
            K.moe_skinny(**{**base, **bad})
    lin = dict(x=t(T, Kd), w=t(N, Kd, dtype=f8), ws=t(1, 2, dtype=torch.float32), out=t(T, N), w_up=t(N, Kd, dtype=f8), ws_up=t(1, 2, dtype=torch.float32), residual=t(T, N))
    for bad in (dict(ws=t(2, 1, dtype=torch.float32)), dict(ws=t(1, 2)), dict(w=t(N, Kd)), dict(w_up=t(N, Kd)), dict(w_up=t(N // 2, Kd, dtype=f8)), dict(ws_up=None),
                dict(ws_up=t(1, 1, dtype=torch.float32)), dict(w_up=None), dict(out=t(T, N, dtype=torch.float32)), dict(out=t(T - 1, N)), dict(residual=t(T, N, dtype=torch.float32)),
                dict(residual=t(T, 2 * N)[:, :N]), dict(x=t(T, Kd // 2))):
        with pytest.raises((AssertionError, AttributeError)):
            K.linear_w8(**{**lin, **bad})


def test_w8_rules():
    from cuteafd_b200.parallel.moe_exchange import w8_expands, w8_tile_rows
    assert [w8_tile_rows(n * 32, 8, 256) for n in (1, 20, 21, 48, 49, 300)] == [32, 32, 64, 64, 128, 128]
    assert not w8_expands(512 * 16, 16) and w8_expands(512 * 16 + 1, 16)


def test_prompt_share_rules():
    from cuteafd_b200._native import lib as n
    f = n.cuda_lib().cafd_attn_prefill_splits
    assert f(1, 512, 16896, 32, 4, 148) == 2 and f(1, 65, 16449, 32, 4, 148) == 8
    assert f(1, 300, 1300, 32, 4, 148) == 1 and f(1, 8192, 8192, 32, 4, 148) == 1 and f(1, 777, 777, 32, 4, 148) == 1
    assert f(1, 512, 16896, 24, 8, 148) == 1                        # an odd number of heads shares a kv head
    assert f(1, 512, 0, 32, 4, 148) == 1                            # the host doesn't know the lengths


def test_step_attention_rules():
    from cuteafd_b200._native import lib as n
    f = n.cuda_lib().cafd_attn_step_splits
    for s, pages, hkv in ((1, 129, 4), (8, 129, 4), (32, 129, 4), (3, 8, 4), (1, 1, 1), (300, 3, 8)):
        got = f(s, pages, 4 * hkv, hkv, 0, 148)
        assert 1 <= got <= min(16, pages)
    assert [f(r, 129, 32, 4, 0, 148) for r in (1, 4, 8, 16, 32)] == [16, 16, 10, 5, 6] and f(32, 8, 32, 4, 0, 148) == 2
    assert f(1, 4000, 32, 4, 0, 148) == 0 and f(1, 4000, 32, 4, 512, 148) > 0           # a long context of one row; a window of it
    assert f(1, 129, 136, 4, 0, 148) == 0                                               # 34 heads to a kv head
