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
