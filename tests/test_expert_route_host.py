"""The host rules that choose between the large-batch expert kernels (csrc/expert_route.h), on the CPU."""
import pytest

from tests import hostcheck as hc


def cut(rows, most):
    """Even blocks of whole groups of 8 rows, as the kernels deal a slot's rows."""
    n = -(-rows // most)
    per = 8 * -(-(-(-rows // 8)) // n)
    return [min(per, rows - at) for at in range(0, rows, per)]


def test_rows_are_cut_as_the_kernels_cut_them():
    for rows in list(range(1, 300)) + [1000, 4095, 4096, 4097]:
        fold, units = cut(rows, 64), cut(rows, 32)
        want = [sum(r <= 32 for r in fold), len(fold)] + [sum(-(-r // 8) == g for r in units) for g in (1, 2, 3, 4)]
        assert hc.row_blocks(rows) == want, rows


# (mode, O, K, group size, rows per slot, us with the small-batch kernel, us with the fold kernel), B200.  Groups are
# whole calls, so their figures hold the other phase too (RAMP40: 40 experts with 1 to 40 rows).
RAMP40 = [1 + (i * 7) % 40 for i in range(39)] + [40]
MEASURED = [
    (1, 16000, 6144, 32, [128], 144, 97), (1, 16000, 6144, 32, [129], 145, 170), (1, 16000, 6144, 32, [64], 89, 95),
    (1, 16000, 3072, 32, [129], 79, 95), (1, 8192, 6144, 32, [129], 82, 95), (1, 8192, 6144, 32, [200], 136, 95),
    (1, 4096, 2048, 32, [64], 28, 44), (1, 33000, 6144, 32, [32], 92, 85), (1, 33000, 6144, 32, [1200], 1804, 1322),
    (1, 33000, 2048, 0, [32], 38, 32), (1, 16000, 6144, 0, [129], 135, 102), (1, 8192, 6144, 0, [32], 46, 58),
    (1, 32000, 6144, 32, [100], 199, 172),
    (0, 1600, 4000, 32, RAMP40, 250, 311), (0, 2048, 6144, 32, RAMP40, 402, 499), (0, 1024, 2048, 32, RAMP40, 124, 146),
    (1, 6144, 2048, 32, RAMP40, 402, 451), (0, 1024, 2048, 32, [150] * 40, 475, 437), (0, 2048, 6144, 0, [28] * 39 + [32], 486, 403),
]


@pytest.mark.parametrize("mode,o,k,gs,rows,block,fold", MEASURED)
def test_the_faster_kernel_is_chosen(mode, o, k, gs, rows, block, fold):
    assert hc.fold_beats_block(o, k, gs, mode, rows) == (fold < block)


def test_what_the_fold_kernel_is_not_given():
    assert hc.fold_beats_block(33000, 2048, 32, 1, 1000)
    assert not hc.fold_beats_block(33000, 1792, 32, 1, 1000)      # 7 chunks
    assert not hc.fold_beats_block(33000, 2048, 0, 1, 31)         # fewer than 32 rows
    assert hc.fold_beats_block(33000, 16384, 0, 1, 1000)
    assert not hc.fold_beats_block(33000, 16385, 0, 1, 1000)      # per-row dots beyond the accumulator's 24 bits
    assert hc.fold_beats_block(33000, 16385, 32, 1, 1000)         # (a group's dot stays far below)
