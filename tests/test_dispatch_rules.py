"""Rules that pick a kernel's form from sizes alone, checked on the host."""
import pytest

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
