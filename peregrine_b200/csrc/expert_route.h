// Which expert kernel a large launch is given: rules on sizes and weight format, plain host code that the CPU
// tests compile too.
#pragma once
#include <cmath>

#include "w4_layout.h"

namespace pgb {

constexpr int kFoTok = 64;         // activation rows of a fold-kernel item
constexpr int kFoMaxSlots = 1024;  // slots of its launches

// Can the fold kernel hold the launch at all: its slot table, and for per-row scales the whole row's integer dot,
// which has to stay exact in the fp32 accumulator (8 * 128 * K <= 2^24).
inline bool fold_fits(const W4Layout &L, int slots_max) {
    return slots_max <= kFoMaxSlots && (L.grouped || L.kp <= 16384);
}

// The rows of a launch whose slots the host knows, as the two kernels cut them.
struct RowBlocks {
    int slots = 0, max_rows = 0;
    long long narrow = 0, wide = 0;           // fold kernel: row blocks of at most 32 and of up to 64 rows
    long long units[5] = {0, 0, 0, 0, 0};     // small-batch kernel: units of 8, 16, 24 and 32 rows
    void add(int rows) {
        if (rows < 1) return;
        ++slots;
        max_rows = rows > max_rows ? rows : max_rows;
        cut(rows, kFoTok, [this](int r, long long n) { (r <= 32 ? narrow : wide) += n; });
        cut(rows, 32, [this](int r, long long n) { units[(r + 7) / 8] += n; });
    }

  private:
    template <typename F>
    static void cut(int rows, int most, F use) {  // even blocks of whole groups of 8 rows
        const int blocks = (rows + most - 1) / most, per = 8 * (((rows + 7) / 8 + blocks - 1) / blocks);
        use(per < rows ? per : rows, rows / per > 0 ? rows / per : 1);
        if (rows > per && rows % per) use(rows % per, 1);
    }
};

// Rounds of a launch's items over `sms` CTAs that take the longest first: `wide` items of length 1, then `narrow` ones
// of length w.
inline double item_rounds(long long wide, long long narrow, double w, int sms) {
    const long long late = wide % sms, early = sms - late;  // CTAs with one wide item more, and the others
    const long long whole = narrow / sms > 4 ? narrow / sms - 4 : 0;
    double a = (double)(wide / sms) + whole * w, b = a + 1.0;  // when they are free
    double end = late ? b : a;
    for (narrow -= whole * sms; narrow > 0;) {
        const bool first = late == 0 || a <= b;
        (first ? a : b) += w;
        narrow -= first ? early : late;
        if ((first ? a : b) > end) end = first ? a : b;
    }
    return end;
}

// Is the fold kernel faster than the shared-row small-batch kernel for these rows?  Both are given the time of
// their rounds of items over the SMs.  The constants (us) are fitted to 7215 measured launches with 8+ chunks of K and
// 32+ rows in some slot (B200; single matrices of O 200..33000 and K up to 6144 with up to 1200 rows, both phases
// of groups of up to 40 experts with up to 150 rows, five formats).  Over these the choice is 0.1 % behind the faster
// kernel of each; 44 lose over 2 %, at most 18 %.
//   * fold: an item is 256 weight rows x up to 64 rows and always costs its whole width (or half of it); a last
//     round that few items fill costs like a full one.  6144 x 16000, group 32: 128 rows 144 -> 97 us, 129 rows
//     (three blocks of 43, 189 items) 145 against 170.
//   * small batch: units of 32 rows whose cost goes with their groups of 8 rows; cut finer when items are few.
//     2048 x 4096, 64 rows: 28 us against 44.
// Below 8 chunks of K and below 32 rows the small-batch kernel stays: nothing was settled there.
inline bool fold_may_beat_block(const W4Layout &L, int max_rows) { return L.nchunk >= 8 && max_rows >= 32; }
inline bool fold_beats_block(const W4Layout &L, int mode, const RowBlocks &R, int sms) {
    if (!fold_fits(L, R.slots) || !fold_may_beat_block(L, R.max_rows)) return false;
    struct Cost {
        double fold, narrow, block;  // us per chunk and round; narrow items relative to wide ones
    };
    const Cost per_row{1.75, 0.85, 2.05};
    const Cost by_bpg[4] = {{3.20, 0.80, 2.30}, {2.60, 0.85, 2.15}, {2.05, 0.95, 2.30}, {1.90, 0.95, 2.20}};
    const Cost &c = !L.grouped ? per_row : by_bpg[L.bpg == 1 ? 0 : L.bpg == 2 ? 1 : L.bpg == 4 ? 2 : 3];
    const long long n_ob = mode == 0 ? (L.ntile + 7) / 8 : (L.ntile + 15) / 16;
    const double fold_rounds = item_rounds(n_ob * R.wide, n_ob * R.narrow, c.narrow, sms);
    double units = 0, weight = 0;
    for (int g = 1; g <= 4; ++g) {
        units += (double)n_ob * R.units[g];
        weight += (double)n_ob * R.units[g] * (0.12 + 0.22 * g);
    }
    const double block_rounds = weight / sms + (units > sms ? 0.45 : 0.42);
    // (the epilogues count as chunks: gate/up's holds the SwiGLU)
    const double fold_us = 17.0 + c.fold * (L.nchunk + (mode == 0 ? 1.5 : 0.0)) * fold_rounds;
    const double block_us = 14.0 + c.block * (L.nchunk + (mode == 0 ? 2.0 : 0.5)) * block_rounds;
    return fold_us < block_us;
}

// The same against the CTA-tiled mma.sync kernel, for one phase of a layer of M tokens, top-k of E experts, whose rows
// per expert only the device knows: an even spread is assumed.  Items come in rounds over the SMs; the fold kernel
// needs a full round or more, and enough chunks in all for its long pipelines to pay for their start.  Measured at
// 13 shapes x 5 formats x 48..4000 tokens (gate/up and down separately, us tiles -> fold): gate/up of 24 chunks
// group 32 3252 -> 2988, of 8 chunks 371 -> 380 at 2000 tokens and 80 -> 67 at 128; down of 8 chunks 1787 -> 1520,
// of 4 chunks 205 -> 192; where items are few (768 x 2048, 16 experts, 48 tokens: 102 items) 34 -> 50.  Per-row
// scales, without a fold per group, are ahead from one round on (1600 x 2560, 8 experts, 200 tokens: 53 -> 47).  Below 8 chunks
// gate/up, whose epilogue is the longer one, stays with the tiles (6 chunks group 64: 137 -> 146); grouped down of
// one chunk too (58 -> 63); so does gate/up whose blocks of 128 weight rows hold over a tenth more padding than the
// tiles' of 64 (inter 136: layer of 1576 tokens 452 -> 502).  Over 2060 layers, 1449 of them drawn at random, the
// choice is 5.1 % ahead of the tiles alone and 0.5 % behind the better kernel of each phase; 59 lose over 2 %, at most
// 8 %.
// (More tokens never take a layer back to the tiles: its scratch is sized by the most tokens it has seen.)
inline bool fold_beats_tiles(const W4Layout &L, int mode, int M, int E, int k, int sms) {
    if (!fold_fits(L, E + 1) || L.nchunk < (mode == 0 ? 8 : L.grouped ? 2 : 1)) return false;
    const int ob = mode == 0 ? (L.ntile + 7) / 8 : (L.ntile + 15) / 16;
    const double n_ob = ob;
    if (mode == 0 && 20 * ob > 11 * ((L.ntile + 3) / 4)) return false;  // blocks of 128 rows against 64
    const double touched = E * (1.0 - std::pow(1.0 - (double)(k < E ? k : E) / E, M));
    const double full = (double)M * k / kFoTok;
    const double rounds = n_ob * ((touched > full ? touched : full) + (M + kFoTok - 1) / kFoTok) / sms;
    if (!L.grouped) return rounds >= 1.0 && rounds * L.nchunk >= (mode == 0 ? 8.0 : 6.0);
    return rounds >= 1.5 && rounds * L.nchunk >= (mode == 0 ? 24.0 : 8.0);
}

// The expert kernels of a layer call of 3 or more tokens.  Batches of 48+ tokens with on average 1.5+ rows per routed
// expert (measured crossover between 32 and 64 tokens at 256 experts top-8: 255 us against 378, 575 against 477)
// leave the small-batch kernels.  `want` (-1: none) forces a choice: 0 small batch, 1 tiles, 2 fold kernel.
struct LayerRoute {
    bool tiles_gu, tiles_dn, fold_gu, fold_dn;
};
inline LayerRoute layer_route(const W4Layout &Lgu, const W4Layout &Ldn, int M, int E, int k, int sms, int want) {
    LayerRoute r{};
    const bool large = want < 0 ? M >= 48 && 2LL * M * k >= 3LL * E : want > 0;
    if (!large) return r;
    r.fold_gu = want == 2 ? fold_fits(Lgu, E + 1) : want < 0 && fold_beats_tiles(Lgu, 0, M, E, k, sms);
    r.fold_dn = want == 2 ? fold_fits(Ldn, E + 1) : want < 0 && fold_beats_tiles(Ldn, 1, M, E, k, sms);
    r.tiles_gu = !r.fold_gu;
    r.tiles_dn = !r.fold_dn;
    return r;
}

}  // namespace pgb
