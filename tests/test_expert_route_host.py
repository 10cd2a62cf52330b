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
    (1, 32000, 6144, 32, [100], 199, 172), (1, 10222, 4728, 32, [216], 113, 139), (1, 11116, 5192, 32, [203], 130, 150),
    (1, 9822, 1808, 32, [229], 60, 72),
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


FULL, SMALL = (6144, 2048, 256, 8), (2048, 1024, 64, 4)  # hidden, inter, experts, top-k
# ((hidden, inter, experts, top-k), group size, tokens, us of gate/up and down with the tiles, with the fold kernel).  Only
# launches with a clear difference: the others may go either way.
LAYERS = [
    (FULL, 32, 64, (436, 278), (414, 198)), (FULL, 32, 2000, (3252, 1787), (2988, 1520)),
    (FULL, 0, 48, (374, 213), (268, 151)), (SMALL, 0, 512, (104, 65), (83, 50)),
    ((2048, 768, 16, 4), 32, 48, (34, 29), (50, 31)), ((2048, 256, 8, 2), 32, 64, (35, 19), (51, 25)),
    ((2816, 128, 16, 8), 32, 128, (57, 30), (61, 34)), ((2560, 1600, 8, 1), 32, 48, (38, 34), (60, 44)),
    ((1416, 616, 48, 6), 64, 301, (65, 45), (81, 44)),
]


def test_each_phase_of_a_layer_chooses_for_itself():
    for (d, i, e, k), gs, m, tiles, fold in LAYERS:
        got = hc.layer_route(d, i, gs, m, e, k)
        for phase in (0, 1):
            if abs(tiles[phase] - fold[phase]) > 0.03 * tiles[phase]:
                assert got[phase] == ("fold" if fold[phase] < tiles[phase] else "tiles"), (d, i, gs, m, phase)
    assert hc.layer_route(2048, 256, 0, 160, 100, 2) == ("fold", "tiles")     # one chunk of inter
    # 136 rows: two blocks of 128 against three of 64 (a layer of 452 us with the tiles, 502 with gate/up on the fold kernel)
    assert hc.layer_route(2184, 136, 128, 1576, 40, 8) == ("tiles", "tiles")
    assert hc.layer_route(2184, 256, 128, 1576, 40, 8) == ("fold", "tiles")
    assert hc.layer_route(1024, 2048, 0, 300, 36, 4) == ("tiles", "fold")    # four chunks of hidden


def test_more_tokens_never_leave_the_fold_kernel():
    # a layer's scratch is sized by the most tokens it has seen
    for d, i, e, k in (FULL, SMALL, (2048, 256, 8, 2), (1416, 616, 48, 6), (3200, 1600, 100, 8), (2816, 128, 16, 8)):
        for gs in (0, 32, 64, 128, 256):
            seen = [False, False]
            for m in list(range(3, 700)) + [1000, 2000, 3000, 4096, 8192]:
                got = hc.layer_route(d, i, gs, m, e, k)
                for phase in (0, 1):
                    assert not (seen[phase] and got[phase] != "fold"), (d, i, e, k, gs, m, phase)
                    seen[phase] |= got[phase] == "fold"


def test_forced_layer_kernels_and_limits():
    assert hc.layer_route(*FULL[:2], 32, 32, *FULL[2:]) == ("small", "small")
    assert hc.layer_route(256, 96, 32, 4, 12, 3, want=2) == ("fold", "fold")
    assert hc.layer_route(256, 96, 32, 4, 12, 3, want=1) == ("tiles", "tiles")
    assert hc.layer_route(*FULL[:2], 32, 4096, *FULL[2:], want=0) == ("small", "small")
    assert hc.layer_route(16385, 2048, 0, 512, 16, 4, want=2) == ("tiles", "fold")  # per-row rows too long for it
    assert hc.layer_route(2048, 1024, 32, 4096, 1024, 8) == ("tiles", "tiles")      # 1025 slots: one too many
