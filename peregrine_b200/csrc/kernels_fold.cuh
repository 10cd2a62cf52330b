// int4 x int8 expert matmul on the fifth-generation tensor cores with the ordered fp32 fold as its
// bound: experts with several to thousands of activation rows.
//
// What bounds it.  Results are those of the reference's sequential fold (crates/peregrine-kernels/src/
// idot.rs:98-110, matmul.rs:75-106): per weight row and activation row one rounded multiply and one
// rounded add per scale group, in ascending order.  At group 32 that is two fp32 operations per 64
// integer operations: 128 fp32 lanes per SM make it 4096 integer operations per cycle and SM, half of
// what the tensor cores do.  So everything else is taken off the fp32 lanes:
//
//   * the dots come from tcgen05.mma kind::f16.  int4 weights and int8 activations are exact in fp16,
//     a product has at most 11 bits, a group's sum stays below 2^19 and is exact in the fp32
//     accumulator: the accumulator IS (float)dot, with no conversion, no magic number and no -8*sum(q)
//     correction (the nibbles are expanded to their signed values).  kind::i8 is twice as fast on the
//     tensor pipe but costs the fold a third operation per group.
//   * weight rows are the M dimension: a fold thread owns one weight row (TMEM lane), so a group's scale
//     is one register; the columns are activation rows.
//   * the expanded weights go straight into tensor memory (A operand of the MMA), not through shared
//     memory, whose bandwidth the B operand and the copies need.
//
// Tile of a CTA: 2 halves of 128 weight rows (mode 0: 128 gate + the same 128 up rows, so a thread holds
// both values of its SwiGLU; mode 1: 256 down rows) x 64 activation rows of one expert.  Roles:
//
//   warps 0-7    fold and epilogue: warp w owns TMEM lanes 32 (w % 4).. and the 16-column groups
//                w/4, w/4 + 2, ..; accumulators in registers
//   warps 8-11   expand: 32 rows of both halves per warp, one 32-element block at a time, into a ring of
//                four blocks in tensor memory
//   warp 12      one lane issues the MMAs: four per block (two halves, K = 16 each); dots of a group go to
//                one of six accumulators of 64 columns
//   warps 13, 14 bulk copies of the packed weight chunks (8 tiles each), a chunk of 256 elements per stage; warp 13 also
//                takes work items from a device counter and publishes them to the other roles
//   warp 15      TMA tiles of the activations: fp16 rows, 64 elements x 32 rows, 128-byte swizzle
//
// Measured (B200): about 880 cycles per 32-element block of the 256 x 64 tile, epilogue included, against 256 of fold
// arithmetic and 128 of MMA: a fold warp waits for a barrier, loads from tensor memory (60-80 cycles), waits and
// folds, twice per block, and only two fold warps share a scheduler.  Issue slots 62 % busy, tensor pipe 16 %, DRAM
// 4 % (1024 tokens, 16 experts of 6144 x 2048, group 32).  Layer of 256 such experts, 4096 tokens: 10.9 ms with the
// mma.sync tiles, 10.0 ms here; 6144 x 32000 at 100 rows 199 us with the small-batch kernel, 169 us here.  Which
// launches come here: expert_route.h.
//
// Persistent: one CTA per SM; the copies and MMAs of the next item run during an item's epilogue.  Items
// are handed out heaviest first.  Every wait is bounded; one that runs out sets the device error word and
// a flag that all roles poll; every path reaches the tail that lets copies and MMAs in flight end and
// frees the tensor memory.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "expert_route.h"
#include "kernels_tcgen05.cuh"

namespace pgb {

constexpr int kFoThreads = 512;
constexpr int kFoXGroup = 64;       // elements of K per activation copy (one 128-byte swizzle row of fp16)
constexpr int kFoXStages = 8;
constexpr int kFoXBoxRows = 32;
constexpr int kFoWStageBytes = 16 * kChunkMaxBytes;
constexpr int kFoAStages = 4;       // 32-element blocks of expanded weights in tensor memory
constexpr int kFoACol = 384;        // their first column: 4 blocks x 2 halves x 16 columns
constexpr int kFoQueue = 4;

constexpr int kFoWStages = 3;        // chunks of the item's 16 tiles
constexpr int kFoNBuf = 6;           // accumulators of kFoTok columns in tensor memory
constexpr int kFoWOff = kFoXStages * kFoTok * 128;
constexpr int kFoTabOff = kFoWOff + kFoWStages * kFoWStageBytes;
constexpr int kFoTabBytes = (3 * kFoMaxSlots + 4) * 4;
constexpr int kFoBarOff = kFoTabOff + kFoTabBytes;
// 1024 bytes of slack: the swizzled tiles need a 1024-byte boundary
constexpr int kFoSmemBytes = kFoBarOff + 512 + 1024;

// Work counter of the launches (next item, CTAs that have finished; the last one clears both): launches
// on a device are ordered by the context's stream.  Zero when the module is loaded.
__device__ unsigned g_fold_dyn[2];

// Position of activation elements inside a 32-element block: word j of a packed segment holds elements
// 4j..4j+3 and 16+4j..16+4j+3 in nibbles that unpack two at a time as (4j, 4j+2), (4j+1, 4j+3) and the
// same of the upper half.  The fp16 activation rows are stored in that order (the dot of a block does
// not depend on it): eight values from two int8 words.
__device__ __forceinline__ uint4 fold_pack8(uint32_t lo, uint32_t hi) {
    // int8 -> fp16: biased byte as the low mantissa bits of 1024, minus 1024 + 128
    auto two = [](uint32_t w, uint32_t sel) {
        const uint32_t h = __byte_perm(w ^ 0x80808080u, 0x64646464u, sel);
        const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&h), __half2half2(__ushort_as_half(0x6480)));
        return *reinterpret_cast<const uint32_t *>(&v);
    };
    return make_uint4(two(lo, 0x4240), two(lo, 0x4341), two(hi, 0x4240), two(hi, 0x4341));
}

// fp32 rows -> fp16 rows of their int8 values (crates/peregrine-kernels/src/quant.rs:14-33), kp elements each.
// One CTA per row; a thread makes eight neighbouring outputs from two aligned quads of the row (16-byte
// loads and stores).  amax_bits as in qrow_i8_kernel.
__global__ void __launch_bounds__(256) qrow_f16_kernel(const float *__restrict__ x, long long ldx, int K, int kp,
                                                       __half *__restrict__ xh, float *__restrict__ sx,
                                                       const int *__restrict__ n_rows_dev, int n_rows,
                                                       const unsigned *__restrict__ amax_bits, int vec) {
    const int row = blockIdx.x;
    if (row >= (n_rows_dev ? *n_rows_dev : n_rows)) return;
    const float *xr = x + (long long)row * ldx;
    __shared__ float red[8];
    float m = 0.0f;
    if (amax_bits) {
        m = __uint_as_float(amax_bits[row]);
    } else {
        for (int i = threadIdx.x; i < K; i += 256) {
            const float a = fabsf(xr[i]);
            if (a > m) m = a;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float a = __shfl_xor_sync(0xffffffffu, m, o);
            if (a > m) m = a;
        }
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        m = red[0];
        for (int w = 1; w < 8; ++w)
            if (red[w] > m) m = red[w];
    }
    float s = __fdiv_rn(m, 127.0f);
    if (s < 1e-12f) s = 1e-12f;
    const float inv = __fdiv_rn(1.0f, s);
    if (threadIdx.x == 0) sx[row] = s;
    for (int u = threadIdx.x; u < (kp >> 3); u += 256) {
        const int i0 = (u >> 2) * 32 + (u & 3) * 4;
        uint32_t w[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = i0 + 16 * h;
            float v[4];
            if (vec && i + 4 <= K) {
                const float4 f = *reinterpret_cast<const float4 *>(xr + i);
                v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = i + e < K ? xr[i + e] : 0.0f;
            }
            w[h] = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int q = max(-128, min(127, __float2int_rn(__fmul_rn(v[e], inv))));
                w[h] |= (uint32_t)(q & 255) << (8 * e);
            }
        }
        reinterpret_cast<uint4 *>(xh + (long long)row * kp)[u] = fold_pack8(w[0], w[1]);
    }
}

// Pair-ordered fp16 copy of the int8 token rows the routing launch left: output row p is token
// pair_token[p].  One CTA per pair row, 16-byte stores.
__global__ void __launch_bounds__(256) gather_pair_f16_kernel(const int8_t *__restrict__ xq_tok,
                                                              const float *__restrict__ sx_tok, int kp,
                                                              const int *__restrict__ pair_token,
                                                              const int *__restrict__ n_pairs_dev,
                                                              __half *__restrict__ xh, float *__restrict__ sxp) {
    const int p = blockIdx.x;
    if (p >= *n_pairs_dev) return;
    const int tok = pair_token[p];
    const uint32_t *src = reinterpret_cast<const uint32_t *>(xq_tok + (long long)tok * kp);
    for (int u = threadIdx.x; u < (kp >> 3); u += 256) {
        const int j = (u >> 2) * 8 + (u & 3);
        reinterpret_cast<uint4 *>(xh + (long long)p * kp)[u] = fold_pack8(__ldg(src + j), __ldg(src + j + 4));
    }
    if (threadIdx.x == 0) sxp[p] = sx_tok[tok];
}

// The 32 nibbles of one packed segment as 16 fp16 pairs (signed values, in the order of fold_pack8).
__device__ __forceinline__ void fold_expand(const uint4 &w, uint32_t (&o)[16]) {
    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
    const __half2 b1 = __half2half2(__ushort_as_half(0xE408));   // -1032
    const __half2 b16 = __half2half2(__ushort_as_half(0xD480));  // -72
    const __half2 r16 = __half2half2(__ushort_as_half(0x2C00));  // 1/16
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t a = ws[j], c = ws[j] >> 8;
        const uint32_t t[4] = {(a & 0x000F000Fu) | 0x64006400u, (c & 0x000F000Fu) | 0x64006400u,
                               (a & 0x00F000F0u) | 0x64006400u, (c & 0x00F000F0u) | 0x64006400u};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const __half2 v = *reinterpret_cast<const __half2 *>(&t[e]);
            const __half2 r = e < 2 ? __hadd2(v, b1) : __hfma2(v, r16, b16);  // 1024 + n - 1032; (1024 + 16 n)/16 - 72
            o[4 * j + e] = *reinterpret_cast<const uint32_t *>(&r);
        }
    }
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(taddr)
        : "memory");
}
// the wait names the registers of the load it covers: nothing that reads them may move above it
__device__ __forceinline__ void tmem_wait_ld16(float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                   "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
// a += s * v on pairs (two neighbouring columns), product and sum rounded on their own (see fold_pair in
// kernels_mma.cuh for the form); pairs are kept packed so that they stay in aligned registers
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fold_mul(uint64_t v, uint64_t s, uint64_t nz) {
    uint64_t p;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(v), "l"(s), "l"(nz));
    return p;
}
__device__ __forceinline__ void fold_add(uint64_t &a, uint64_t p) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(p)); }
// 16 columns of one lane: all products before the sums, so that no sum waits for its own product
__device__ __forceinline__ void fold16(uint64_t (&a)[8], const float (&b)[16], uint64_t s, uint64_t nz) {
    uint64_t p[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) p[c] = fold_mul(pack2(b[2 * c], b[2 * c + 1]), s, nz);
#pragma unroll
    for (int c = 0; c < 8; ++c) fold_add(a[c], p[c]);
}

// A ring position: index and the parity of its current pass
template <int N>
struct RingPos {
    int i = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void next() {
        if (++i == N) {
            i = 0;
            ph ^= 1u;
        }
    }
};

// Grid: one CTA per SM.  Activations: fp16 rows through `xmap` (qrow_f16_kernel / gather_pair_f16_kernel),
// P.sx per row; P.xq / P.csum are not used.
template <bool GROUPED, int BPG>
__global__ void __launch_bounds__(kFoThreads, 1)
    ffn_w4a8_fold_kernel(const __grid_constant__ CUtensorMap xmap, const GemvParams P) {
    constexpr int GPC = kChunkBlocks / BPG;
    constexpr int CHUNK_BYTES = kChunkSlabBytes + (GROUPED ? GPC * 64 : 0);
    constexpr int TOK = kFoTok, WST = kFoWStages, NBUF = kFoNBuf;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ int s_fail, s_total;
    __shared__ uint32_t s_tmem;
    __shared__ __align__(16) int4 s_queue[kFoQueue];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t smem_u = smem_u32(smem);
    const uint32_t bar0 = smem_u + kFoBarOff;
    const uint32_t xfull = bar0, xempty = xfull + 8 * kFoXStages, wfull = xempty + 8 * kFoXStages,
                   wempty = wfull + 8 * 4, afull = wempty + 8 * 4, aempty = afull + 8 * kFoAStages,
                   dfull = aempty + 8 * kFoAStages, dempty = dfull + 8 * 8, qfull = dempty + 8 * 8,
                   qempty = qfull + 8 * kFoQueue, drain = qempty + 8 * kFoQueue;
    int *t_key = reinterpret_cast<int *>(smem + kFoTabOff);  // rows per block of a slot
    int *t_slot = t_key + kFoMaxSlots;                              // slot of rank r
    int *t_cum = t_slot + kFoMaxSlots;                              // first row block of rank r
    volatile int *fail = &s_fail;
    const int n_slots = min(*P.n_slots, kFoMaxSlots);
    const int n_ob = P.mode == 0 ? (P.ntile + 7) / 8 : (P.ntile + 15) / 16;

    if (tid == 0) {
        s_fail = 0;
        for (int s = 0; s < kFoXStages; ++s) {
            mbar_init(xfull + 8 * s, 1);
            mbar_init(xempty + 8 * s, 1);
        }
        for (int s = 0; s < WST; ++s) {
            mbar_init(wfull + 8 * s, 2);
            mbar_init(wempty + 8 * s, GROUPED ? 4 + 8 : 4);
        }
        for (int s = 0; s < kFoAStages; ++s) {
            mbar_init(afull + 8 * s, 4);
            mbar_init(aempty + 8 * s, 1);
        }
        for (int s = 0; s < NBUF; ++s) {
            mbar_init(dfull + 8 * s, 1);
            mbar_init(dempty + 8 * s, 8);
        }
        for (int s = 0; s < kFoQueue; ++s) {
            mbar_init(qfull + 8 * s, 1);
            mbar_init(qempty + 8 * s, 15);
        }
        mbar_init(drain, 1);
        fence_mbar_init();
        fence_proxy_async();
    }
    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // ---- row blocks: a slot's rows are dealt evenly to ceil(rows / TOK) blocks, slots ranked by block size
    for (int s = tid; s < n_slots; s += kFoThreads) {
        const int nr = max(P.slots[s].nrows, 0), nb = (nr + TOK - 1) / TOK;
        t_key[s] = nb ? 8 * (((nr + 7) / 8 + nb - 1) / nb) : 0;
    }
    __syncthreads();
    for (int s = tid; s < n_slots; s += kFoThreads) {
        const int key = t_key[s];
        int rank = 0;
        for (int o = 0; o < n_slots; ++o) rank += (t_key[o] > key || (t_key[o] == key && o < s)) ? 1 : 0;
        t_slot[rank] = s;
    }
    __syncthreads();
    if (warp == 0) {
        int base = 0;
        for (int r0 = 0; r0 < n_slots; r0 += 32) {
            const int r = r0 + lane;
            int nb = 0;
            if (r < n_slots) {
                const int key = t_key[t_slot[r]];
                nb = key ? (P.slots[t_slot[r]].nrows + key - 1) / key : 0;
            }
            int inc = nb;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (r < n_slots) t_cum[r] = base + inc - nb;
            base += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) {
            t_cum[n_slots] = base;
            s_total = base * n_ob;
        }
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = s_tmem;

    RingPos<kFoQueue> qp;
    // the next work item {slot, first pair row, rows, block of weight rows}; slot < 0: the end
    auto next_item = [&](int4 &it) -> bool {
        if (!__all_sync(0xffffffffu, um_wait(qfull + 8 * qp.i, qp.ph, fail))) return false;
        it = *const_cast<const int4 *>(&s_queue[qp.i]);
        __syncwarp();
        if (lane == 0) mbar_arrive(qempty + 8 * qp.i);
        qp.next();
        return it.x >= 0;
    };

    if (warp < 8) {
        // ============================================================ fold and epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
        const int q = warp & 3, hf = warp >> 2;
        const uint32_t tlane = tmem + ((uint32_t)(32 * q) << 16) + 16 * hf;
        const int wtile = 2 * q + (lane >> 4), wrow = lane & 15;  // this lane's row inside a half
        const uint64_t nz = pack2(P.neg_zero, P.neg_zero);
        RingPos<WST> wp;
        RingPos<NBUF> dp;
        bool ok = true;
        int4 it;
        while (ok && next_item(it)) {
            const int nr = it.z;
            // 16-column groups of this warp: hf, hf + 2, ..; with an odd number both take the larger half (the
            // last group of one reads columns that nothing uses), so that all fold warps run the same code
            const int cnt = ((nr + 15) / 16 + 1) >> 1;
            // Fold and epilogue of the item.  The number of groups is a constant of the code: with a run-time count
            // every group was a branch, and the fold took twice as long.
            auto run_item = [&](auto cc) {
                constexpr int CNT = decltype(cc)::value;
                uint64_t acc[2][CNT][8];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < CNT; ++i)
#pragma unroll
                        for (int c = 0; c < 8; ++c) acc[h][i][c] = 0;
                // One accumulator buffer of half h: its dots are folded in (grouped) or are the values themselves.
                // Two groups are loaded before the first is used (a load takes 60-80 cycles).
                auto drain_buf = [&](int h, float sc) {
                    um_spin(dfull + 8 * dp.i, dp.ph, fail);
                    tmem_fence_after();
                    const uint32_t base = tlane + dp.i * TOK;
                    const uint64_t ss = pack2(sc, sc);
                    auto use = [&](int i, const float(&b)[16]) {
                        if (GROUPED) {
                            fold16(acc[h][i], b, ss, nz);
                        } else {
#pragma unroll
                            for (int c = 0; c < 8; ++c) acc[h][i][c] = pack2(b[2 * c], b[2 * c + 1]);
                        }
                    };
#pragma unroll
                    for (int i = 0; i < CNT; i += 2) {
                        float b0[16], b1[16];
                        tmem_ld16(base + 32 * i, b0);
                        if (i + 1 < CNT) tmem_ld16(base + 32 * (i + 1), b1);
                        tmem_wait_ld16(b0);
                        if (i + 1 < CNT) tmem_wait_ld16(b1);
                        if (i + 2 >= CNT) {
                            tmem_fence_before();
                            mbar_arrive_lane0(dempty + 8 * dp.i, lane);
                        }
                        use(i, b0);
                        if (i + 1 < CNT) use(i + 1, b1);
                    }
                    dp.next();
                };
                if (!GROUPED) {
                    drain_buf(0, 0.0f);
                    drain_buf(1, 0.0f);
                }
#pragma unroll 1
                for (int chunk = 0; GROUPED && chunk < P.nchunk; ++chunk) {
                    um_spin(wfull + 8 * wp.i, wp.ph, fail);
                    const uint8_t *st = smem + kFoWOff + wp.i * kFoWStageBytes;
                    constexpr int SB = GPC < 2 ? 1 : 2;  // groups whose scales are read at once
                    // (one or two groups per loop trip: the body has to stay inside the instruction cache)
#pragma unroll 1
                    for (int g0 = 0; g0 < GPC; g0 += SB) {
                        const float *sp =
                            reinterpret_cast<const float *>(st + wtile * kChunkMaxBytes + kChunkSlabBytes) + wrow * GPC + g0;
                        const float *sq = sp + 8 * kChunkMaxBytes / 4;
                        float2 s0, s1;
                        if (SB == 2) {
                            s0 = *reinterpret_cast<const float2 *>(sp);
                            s1 = *reinterpret_cast<const float2 *>(sq);
                        } else {
                            s0 = make_float2(sp[0], 0.0f);
                            s1 = make_float2(sq[0], 0.0f);
                        }
#pragma unroll 1
                        for (int g = 0; g < SB; ++g) {
                            drain_buf(0, s0.x);
                            drain_buf(1, s1.x);
                            s0.x = s0.y;
                            s1.x = s1.y;
                        }
                    }
                    __syncwarp();
                    mbar_arrive_lane0(wempty + 8 * wp.i, lane);
                    wp.next();
                }
                if (__any_sync(0xffffffffu, *fail)) return;
                // ---- epilogue: lane = weight row, so the stores of a column are 128 consecutive bytes.  The
                // column loops are rolled (registers are rotated under them): the body holds an fp64 exponential
                // and unrolled over 64 columns it would be fetched from memory for every item.
                const int l = 32 * q + lane;
                const int o0 = (P.mode == 0 ? it.w * 128 : it.w * 256) + l, o1 = P.mode == 0 ? o0 : o0 + 128;
                float rs0 = 0.0f, rs1 = 0.0f;
                if (!GROUPED) {
                    const GemvSlot *sl = P.slots + it.x;
                    if (o0 < P.O) rs0 = sl->a_rs[o0];
                    if (o1 < P.O) rs1 = (P.mode == 0 ? sl->b_rs : sl->a_rs)[o1];
                }
                const float *sxp = P.sx + it.y;
                float *outp = P.out + (long long)it.y * P.out_stride;
#pragma unroll 1
                for (int i = 0; i < CNT; ++i) {
                    const int col0 = (2 * i + hf) * 16;
#pragma unroll 1
                    for (int c = 0; c < 16; c += 2) {
                        float a0[2], a1[2];
                        unpack2(acc[0][0][0], a0[0], a0[1]);
                        unpack2(acc[1][0][0], a1[0], a1[1]);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int col = col0 + c + e;
                            const bool valid = col < nr;
                            const float sxa = sxp[valid ? col : 0];
                            float v0 = a0[e], v1 = a1[e];
                            if (!GROUPED) v0 = __fmul_rn(v0, rs0), v1 = __fmul_rn(v1, rs1);
                            v0 = __fmul_rn(v0, sxa);
                            v1 = __fmul_rn(v1, sxa);
                            float *op = outp + (long long)col * P.out_stride;
                            if (P.mode == 0) {
                                const float hval = __fmul_rn(silu32(v0), v1);
                                const bool st = valid && o0 < P.O;
                                if (st) op[o0] = hval;
                                if (P.amax_out != nullptr) {
                                    const float a = fabsf(hval);
                                    const unsigned m =
                                        __reduce_max_sync(0xffffffffu, st && a == a ? __float_as_uint(a) : 0u);
                                    if (lane == 0 && m > 0u) atomicMax(P.amax_out + it.y + col, m);
                                }
                            } else {
                                if (valid && o0 < P.O) op[o0] = v0;
                                if (valid && o1 < P.O) op[o1] = v1;
                            }
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
#pragma unroll
                            for (int k = 0; k < 7; ++k) acc[h][0][k] = acc[h][0][k + 1];
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int k = 0; k + 1 < CNT; ++k)
#pragma unroll
                            for (int c = 0; c < 8; ++c) acc[h][k][c] = acc[h][k + 1][c];
                }
            };
            if (cnt == 2)
                run_item(std::integral_constant<int, 2>{});
            else
                run_item(std::integral_constant<int, 1>{});
            ok = __all_sync(0xffffffffu, !*fail);
        }
    } else if (warp < 12) {
        // ============================================================ expand
        asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
        const int q = warp & 3;
        const uint32_t tlane = tmem + ((uint32_t)(32 * q) << 16) + kFoACol;
        const int off = (2 * q + (lane >> 4)) * kChunkMaxBytes + (lane & 15) * 16;
        RingPos<WST> wp;
        RingPos<kFoAStages> ap;
        bool ok = true;
        int4 it;
        while (ok && next_item(it)) {
            for (int chunk = 0; chunk < P.nchunk && ok; ++chunk) {
                ok = __all_sync(0xffffffffu, um_wait(wfull + 8 * wp.i, wp.ph, fail));
                if (!ok) break;
                const uint8_t *st = smem + kFoWOff + wp.i * kFoWStageBytes + off;
                uint4 w0 = *reinterpret_cast<const uint4 *>(st);
                uint4 w1 = *reinterpret_cast<const uint4 *>(st + 8 * kChunkMaxBytes);
#pragma unroll 1
                for (int b = 0; b < kChunkBlocks; ++b) {
                    uint32_t e0[16], e1[16];
                    fold_expand(w0, e0);
                    fold_expand(w1, e1);
                    if (b + 1 < kChunkBlocks) {
                        w0 = *reinterpret_cast<const uint4 *>(st + (b + 1) * kSlabBytes);
                        w1 = *reinterpret_cast<const uint4 *>(st + 8 * kChunkMaxBytes + (b + 1) * kSlabBytes);
                    } else {
                        __syncwarp();
                        mbar_arrive_lane0(wempty + 8 * wp.i, lane);
                    }
                    um_spin(aempty + 8 * ap.i, ap.ph ^ 1u, fail);
                    tmem_fence_after();
                    tmem_st16(tlane + ap.i * 32, e0);
                    tmem_st16(tlane + ap.i * 32 + 16, e1);
                    tmem_wait_st();
                    tmem_fence_before();
                    __syncwarp();
                    mbar_arrive_lane0(afull + 8 * ap.i, lane);
                    ap.next();
                }
                wp.next();
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        // one elected thread per role (see elect_one)
        auto next_item_1 = [&](int4 &it) -> bool {
            if (!um_wait(qfull + 8 * qp.i, qp.ph, fail)) return false;
            it = *const_cast<const int4 *>(&s_queue[qp.i]);
            mbar_arrive(qempty + 8 * qp.i);
            qp.next();
            return it.x >= 0;
        };
        if (elect_one()) {
            bool ok = true;
            int issued = 0;
            int4 it;
            if (warp == 12) {
                // ==================================================== MMA issue
                RingPos<kFoXStages> xp;
                RingPos<kFoAStages> ap;
                RingPos<NBUF> d0, d1;
                d1.next();
                while (ok && next_item_1(it)) {
                    const uint32_t n = (uint32_t)((it.z + 15) / 16) * 16;
                    // D = f32, A = B = f16, both K-major, M = 128
                    const uint32_t idesc = (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
                    for (int chunk = 0; chunk < P.nchunk && ok; ++chunk)
#pragma unroll 2
                        for (int b = 0; b < kChunkBlocks; ++b) {
                            if ((b & 1) == 0) ok = um_wait(xfull + 8 * xp.i, xp.ph, fail);
                            ok = ok && um_wait(afull + 8 * ap.i, ap.ph, fail);
                            if (!ok) break;
                            const bool first = GROUPED ? (b % BPG == 0) : (chunk == 0 && b == 0);
                            const bool last = GROUPED ? (b % BPG == BPG - 1)
                                                      : (chunk == P.nchunk - 1 && b == kChunkBlocks - 1);
                            // 128-byte swizzle, 8-row groups 1024 bytes apart
                            const uint64_t bd = (uint64_t)(((smem_u + xp.i * (TOK * 128) + (b & 1) * 64) & 0x3FFFFu) >> 4) |
                                                (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
                            const uint32_t a = tmem + kFoACol + ap.i * 32;
                            if (first) ok = um_wait(dempty + 8 * d0.i, d0.ph ^ 1u, fail);
                            if (!ok) break;
                            tmem_fence_after();
                            umma_f16_ts(tmem + d0.i * TOK, a, bd, idesc, first ? 0u : 1u);
                            umma_f16_ts(tmem + d0.i * TOK, a + 8, bd + 2, idesc, 1u);
                            if (last) umma_commit(dfull + 8 * d0.i);
                            if (first) {
                                ok = um_wait(dempty + 8 * d1.i, d1.ph ^ 1u, fail);
                                if (!ok) break;
                                tmem_fence_after();
                            }
                            umma_f16_ts(tmem + d1.i * TOK, a + 16, bd, idesc, first ? 0u : 1u);
                            umma_f16_ts(tmem + d1.i * TOK, a + 24, bd + 2, idesc, 1u);
                            if (last) umma_commit(dfull + 8 * d1.i);
                            umma_commit(aempty + 8 * ap.i);
                            ap.next();
                            if (b & 1) {
                                umma_commit(xempty + 8 * xp.i);
                                xp.next();
                            }
                            if (last) {
                                d0.next();
                                d0.next();
                                d1.next();
                                d1.next();
                            }
                        }
                }
                // the last commits may still be under way (after a failure, MMAs too): one on a barrier of its
                // own arrives behind them
                umma_commit(drain);
                const long long t0 = clock64();
                while (!mbar_try_wait(drain, 0u))
                    if (clock64() - t0 > 2000000000LL) {
                        *fail = 1;
                        break;
                    }
            } else if (warp < 15) {
                // ==================================================== weight chunks (and the work queue)
                const int h = warp - 13;
                RingPos<WST> wp;
                RingPos<kFoQueue> fp;  // (warp 13) queue position to fill
                while (ok) {
                    if (h == 0) {
                        it = make_int4(-1, 0, 0, 0);
                        ok = um_wait(qempty + 8 * fp.i, fp.ph ^ 1u, fail);
                        if (!ok) break;
                        const int i = (int)atomicAdd(&g_fold_dyn[0], 1u);
                        if (i < s_total) {
                            const int u = i / n_ob;
                            int lo = 0, hi = n_slots;  // last rank whose first block is at most u
                            while (hi - lo > 1) {
                                const int mid = (lo + hi) >> 1;
                                if (t_cum[mid] <= u)
                                    lo = mid;
                                else
                                    hi = mid;
                            }
                            const int slot = t_slot[lo], per = t_key[slot], r0 = (u - t_cum[lo]) * per;
                            it = make_int4(slot, P.slots[slot].row0 + r0, min(per, P.slots[slot].nrows - r0), i - u * n_ob);
                        }
                        s_queue[fp.i] = it;
                        mbar_arrive(qfull + 8 * fp.i);
                        fp.next();
                        if (it.x < 0) break;
                    } else if (!next_item_1(it)) {
                        break;
                    }
                    // this half's tiles
                    const int tile0 = P.mode == 0 ? it.w * 8 : it.w * 16 + h * 8;
                    const int n_wt = max(0, min(8, P.ntile - tile0));
                    const uint8_t *src = (P.mode == 0 && h ? P.slots[it.x].b : P.slots[it.x].a) +
                                         (unsigned long long)tile0 * P.tile_bytes;
                    for (int chunk = 0; chunk < P.nchunk; ++chunk, src += CHUNK_BYTES) {
                        ok = um_wait(wempty + 8 * wp.i, wp.ph ^ 1u, fail);
                        if (!ok) break;
                        const uint32_t bar = wfull + 8 * wp.i;
                        const uint32_t dst = smem_u + kFoWOff + wp.i * kFoWStageBytes + 8 * h * kChunkMaxBytes;
                        // (the phase needs both warps' arrivals, so no copy can complete it early)
                        mbar_expect_tx(bar, n_wt * CHUNK_BYTES);
                        if (n_wt == 8) {
#pragma unroll
                            for (int t = 0; t < 8; ++t)
                                bulk_g2s(dst + t * kChunkMaxBytes, src + t * P.tile_bytes, CHUNK_BYTES, bar);
                        } else {
                            for (int t = 0; t < n_wt; ++t)
                                bulk_g2s(dst + t * kChunkMaxBytes, src + t * P.tile_bytes, CHUNK_BYTES, bar);
                        }
                        ++issued;
                        wp.next();
                    }
                }
                if (!ok || *fail) {
                    // copies in flight land before the shared memory is given up (bounded)
                    for (int k = 0; k < WST && k < issued; ++k) {
                        const int c = issued - 1 - k;
                        const long long t0 = clock64();
                        while (!mbar_try_wait(wfull + 8 * (c % WST), (c / WST) & 1u))
                            if (clock64() - t0 > 200000000LL) break;
                    }
                }
            } else {
                // ==================================================== activation tiles
                RingPos<kFoXStages> xp;
                while (ok && next_item_1(it)) {
                    const int nbox = (it.z + kFoXBoxRows - 1) / kFoXBoxRows;
                    for (int kg = 0; kg < P.nchunk * (kChunkElems / kFoXGroup); ++kg) {
                        ok = um_wait(xempty + 8 * xp.i, xp.ph ^ 1u, fail);
                        if (!ok) break;
                        const uint32_t bar = xfull + 8 * xp.i;
                        mbar_expect_tx(bar, nbox * (kFoXBoxRows * 128));
                        for (int r = 0; r < nbox; ++r)
                            tma_load_2d(smem_u + xp.i * (TOK * 128) + r * (kFoXBoxRows * 128), &xmap, kg * kFoXGroup,
                                        it.y + r * kFoXBoxRows, bar);
                        ++issued;
                        xp.next();
                    }
                }
                if (!ok || *fail) {
                    for (int k = 0; k < kFoXStages && k < issued; ++k) {
                        const int c = issued - 1 - k;
                        const long long t0 = clock64();
                        while (!mbar_try_wait(xfull + 8 * (c % kFoXStages), (c / kFoXStages) & 1u))
                            if (clock64() - t0 > 200000000LL) break;
                    }
                }
            }
        }
        __syncwarp();
    }
    // ---- common tail
    __syncwarp();
    tmem_fence_before();
    __syncthreads();
    // (behind the barrier: by now every role has noted its failure)
    if (tid == 0 && *fail) report_error(P.err, kErrBarrierTimeout);
    if (warp == 12) {
        tmem_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
    // the last CTA re-arms the work counter
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&g_fold_dyn[1], 1u) == gridDim.x - 1) {
            g_fold_dyn[0] = 0u;
            g_fold_dyn[1] = 0u;
            __threadfence();
        }
    }
}

}  // namespace pgb
