// Residue form of the split-precision GEMMs: residue planes of FP64 rows, the persistent
// tcgen05 GEMM of one modulus per work item, and the reconstruction (see residue.h).
#include "residue.h"

#include <algorithm>
#include <atomic>
#include <cmath>

#include <cuda_bf16.h>

#include "follow.cuh"
#include "gain_internal.h"
#include "tcgen05.cuh"

namespace gain {
namespace split {
namespace {

// ------------------------------------------------------------------- constants
// An integer |X| < 2^58 is split into four balanced 15-bit digits, X = sum_k d_k 2^(15 k),
// |d_k| <= 2^14, so that sum_k d_k c_k with balanced constants |c_k| <= 207 is an exact FP32
// integer below 2^24 congruent to X.
constexpr int kDigitBits = 15;

constexpr int mod_pow2(int e, int m) {
    int r = 1;
    for (int i = 0; i < e; ++i) r = r * 2 % m;
    return r;
}
constexpr int mod_inverse(int a, int m) {   // m < 416: the inverse by trial
    a %= m;
    for (int x = 1; x < m; ++x)
        if (a * x % m == 1) return x;
    return 0;
}
constexpr int balanced(int r, int m) { return 2 * r > m ? r - m : r; }

// digit[t][i][k]: the constant of digit k modulo m_i.  t = 0: 2^(15 k) (the A operand);
// t = n: 2^(15 k) (M / m_i)^-1 mod m_i for the set of the first n moduli (the B operand, so
// that the GEMM's residues are the CRT's coefficients r_i of C / M = sum_i r_i / m_i mod 1).
struct ModTables {
    float digit[kMaxMod + 1][kMaxMod][4];
    float inv[kMaxMod], m[kMaxMod];
    unsigned int frac[kMaxMod][3];   // floor(2^80 / m_i): the low 16 bits, then two 32-bit words
};
constexpr ModTables make_tables() {
    ModTables t{};
    for (int i = 0; i < kMaxMod; ++i) {
        const int m = kModuli[i];
        t.m[i] = (float)m;
        t.inv[i] = 1.0f / (float)m;
        unsigned long long rem = 1;   // long division of 2^80 by m, word by word
        for (int w = 2; w >= 0; --w) {
            const unsigned long long cur = rem << (w ? 32 : 16);
            t.frac[i][w] = (unsigned int)(cur / (unsigned)m);
            rem = cur % (unsigned)m;
        }
        for (int n = 0; n <= kMaxMod; ++n) {
            int f = 1;
            if (n > i) {
                int others = 1;
                for (int j = 0; j < n; ++j)
                    if (j != i) others = others * (kModuli[j] % m) % m;
                f = mod_inverse(others, m);
            }
            for (int k = 0; k < 4; ++k)
                t.digit[n][i][k] = (float)balanced(mod_pow2(kDigitBits * k, m) * f % m, m);
        }
    }
    return t;
}
__constant__ ModTables c_tab = make_tables();

constexpr float kRoundMagic = 12582912.0f;   // 1.5 2^23: adding it rounds to an integer

// v mod m, balanced: |v| < 2^24 an integer; |result| <= m (1/2 + 0.003), below 208 for every modulus.
__device__ __forceinline__ float mod_balanced(float v, float inv, float neg_m) {
    const float q = __fadd_rn(__fmaf_rn(v, inv, kRoundMagic), -kRoundMagic);
    return __fmaf_rn(neg_m, q, v);
}

// Packed FP32 pairs: half the issue slots of the scalar operations, the same roundings.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, uint32_t& x, uint32_t& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=r"(x), "=r"(y) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mod_balanced2(f32x2 v, f32x2 inv, f32x2 neg_m) {
    const f32x2 q = add2(fma2(v, inv, pack2(kRoundMagic, kRoundMagic)), pack2(-kRoundMagic, -kRoundMagic));
    return fma2(neg_m, q, v);
}

// ------------------------------------------------------------------- the GEMM
constexpr int KS = 2, NST = 3;                   // k-blocks per stage (8 MMAs per barrier wait), stages
static_assert(kChunkBlocks % KS == 0, "a stage lies inside one chunk");
constexpr uint32_t BOX_A = BM * BK * 2;          // 16 KB: 128 rows of A
constexpr uint32_t BOX_B = 64 * BK * 2;          // 8 KB: 64 rows of B
constexpr uint32_t STA = KS * BOX_A, STB = KS * 2 * BOX_B;
constexpr int EPI_WARPS = 8;
constexpr int NTHREADS = 64 + 32 * EPI_WARPS;
constexpr uint32_t ACC_COLS = 256;               // TMEM columns of one accumulator; two fill TMEM
// after the stage ring and the barriers: 32 rows x 128 bytes per epilogue warp, in which the
// residues are turned from a row per thread to whole lines per store
constexpr uint32_t TURN_OFF = NST * (STA + STB) + 256;
constexpr uint32_t kSmemBytes = TURN_OFF + EPI_WARPS * 4096 + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

__device__ __forceinline__ uint32_t idesc_of(bool pair, int ncols) {   // BF16 x BF16 -> F32, K-major
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(ncols >> 3) << 17) |
           ((uint32_t)((pair ? 2 * BM : BM) >> 4) << 24);
}

// Persistent kernel over (tile, modulus) items.  Warp 0 issues TMA, warp 1 the MMAs, warps
// 2-9 are the epilogue: two per TMEM lane quadrant, each half of the tile's columns.
//
// An item is one output tile for one modulus.  Its inner dimension runs in chunks of kChunkK,
// exact in FP32; after each chunk the epilogue reduces the accumulator modulo m_i in place
// (TMEM load, three packed FP32 operations per two outputs, TMEM store) and the next chunk's
// MMAs accumulate onto the residues.  A unit runs two items at a time, one per accumulator,
// chunk by chunk in turn: the MMAs of one run while the other is reduced.  (One item over both
// accumulators, with the running residues in 128 registers a thread, left no registers to
// overlap the TMEM loads: a drain took longer than a chunk's MMAs and paced the kernel.)
// Nothing is kept per output but its accumulator, so that may be 256 columns wide: a CTA pair
// computes 256 x 256 tiles, at which the shared-memory port (6 KB read and 6 KB written per 128
// x 128 x 16 MMA at 128 columns, 4 + 4 at 256) no longer paces the tensor pipe.  Items of one
// tile are independent: small problems spread their tiles' moduli over the chip instead of
// running them one after another.  Order: modulus by modulus over all tiles, so a modulus's A
// plane stays in L2 while the tiles run through B.
//
// Measured (GB300, 2000 x 12 000 outputs, inner length 12 288, 13 moduli): 4.18 ms, 1885
// TFLOP/s, where the 21 products of 8-bit digits took 9.0 ms at 1340; the chip's power limit
// bounds it (SM clock 1.9 GHz instead of 2.07, tensor pipe above 80 % of its cycles).  Band
// GEMM of the same run (12 288 columns, up to 3072 deep): 1.10 ms, with 28 digit products 3.0.
// 550 x 1200 outputs, inner length 1408: 47 us, with digits (30 tiles on 76 pairs) 167.
template <bool PAIR, bool GROUPED>
__global__ void __launch_bounds__(NTHREADS, 1)
k_residue_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const ResGemmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = smem;
    uint8_t* sB = smem + NST * STA;
    uint64_t* bars = (uint64_t*)(sB + NST * STB);
    uint64_t* full = bars;
    uint64_t* empty = bars + NST;
    uint64_t* accfull = bars + 2 * NST;
    uint64_t* accempty = bars + 2 * NST + 2;
    uint64_t* drain = bars + 2 * NST + 4;
    uint32_t* tmem_holder = (uint32_t*)(bars + 2 * NST + 5);
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_rank() : 0u;
    const int unit = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int nunits = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int nitems = GROUPED ? a.ntiles : a.ntiles * a.nmod;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&accfull[b]), 1);
            mbar_init(smem_u32(&accempty[b]), (PAIR ? 2 : 1) * EPI_WARPS);   // one arrival per epilogue warp
        }
        mbar_init(smem_u32(drain), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (!GROUPED && warp == 0 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&tmA) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&tmB) : "memory");
    }
    if (warp == 1) {
        if (PAIR) {
            tmem_alloc_pair(smem_u32(tmem_holder), 2 * ACC_COLS);   // both CTAs, same columns
        } else {
            tmem_alloc(smem_u32(tmem_holder), 2 * ACC_COLS);
            tmem_relinquish();
        }
    }
    tc_fence_before();
    if (PAIR) cluster_sync_all();   // the peer's barriers are initialised before any remote use
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_holder;
    follow_next();
    follow_wait();
    if (a.span && threadIdx.x == 0) atomicMax(&a.span[0], ~globaltimer());

    // The unit's items (unit, unit + nunits, ...) alternate between two streams, one per
    // accumulator; every role walks both in the same order.
    struct Stream {
        ResTile tl;
        int it;    // the item (>= nitems: none left)
        int kb;    // its next k-block
        int w;     // the accumulator
        uint32_t chunks;   // the stream's chunks so far
    };
    auto load_item = [&](Stream& x) {   // the first filled slot from x.it on
        for (; x.it < nitems; x.it += 2 * nunits) {
            if (GROUPED) {
                x.tl = a.tiles[x.it];
                if (x.tl.group < 0) continue;
            } else {
                const int mod = x.it / a.ntiles;
                x.tl = a.tiles[x.it - mod * a.ntiles];
                x.tl.mod = mod;
            }
            break;
        }
        x.kb = 0;
    };
    // ... with inner range (an item without one has no chunks: its residues are zero)
    auto load_work = [&](Stream& x) {
        for (load_item(x); x.it < nitems && x.tl.nkb <= 0; load_item(x)) x.it += 2 * nunits;
    };
    // x runs next, y after it: the roles swap the two instead of indexing or unrolling over them,
    // so that their code exists once (a short launch fetches it cold)
    Stream x, y;
    x.it = unit;
    x.w = 0;
    y.it = unit + nunits;
    y.w = 1;
    x.chunks = y.chunks = 0;
    auto swap_streams = [&]() {
        const Stream t = x;
        x = y;
        y = t;
    };

    if (warp == 0) {
        // ---------------- TMA producer
        if (lane == 0) {
            uint32_t stage = 0, phase = 0, issued_mask = 0, last_par = 0;
            bool ok = true;
            load_work(x);
            load_work(y);
            for (; ok && (x.it < nitems || y.it < nitems); swap_streams()) {
                if (x.it < nitems) {
                    const ResTile& tl = x.tl;
                    const CUtensorMap* mapA = GROUPED ? &a.groups[tl.group].tmA : &tmA;
                    const CUtensorMap* mapB = GROUPED ? &a.groups[tl.group].tmB : &tmB;
                    if (GROUPED && x.kb == 0) {   // the tile's tensor maps live in global memory: fetch them early
                        asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)mapA) : "memory");
                        asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)mapB) : "memory");
                    }
                    const int nbx = PAIR ? tl.ncols / 128 : tl.ncols / 64;   // 64-row boxes of B per CTA
                    const int arow = a.m_base + tl.m0 + (int)rank * BM;
                    const int brow = tl.n0 + (PAIR ? (int)rank * (tl.ncols / 2) : 0);
                    const int end = x.kb + kChunkBlocks < tl.nkb ? x.kb + kChunkBlocks : tl.nkb;
                    for (int kb = x.kb; kb < end; kb += KS) {
                        const int nk = end - kb < KS ? end - kb : KS;
                        if (!mbar_wait(smem_u32(&empty[stage]), phase ^ 1, abort_flag, a.err, 1)) {
                            ok = false;
                            break;
                        }
                        const uint32_t bytes = (uint32_t)nk * (BOX_A + (uint32_t)nbx * BOX_B);
                        // both CTAs of a pair complete on the first one's barrier, which expects the bytes of both
                        const uint32_t fb = PAIR ? cluster_map(smem_u32(&full[stage]), 0) : smem_u32(&full[stage]);
                        if (!PAIR || rank == 0) mbar_expect_tx(smem_u32(&full[stage]), PAIR ? 2u * bytes : bytes);
                        for (int h = 0; h < nk; ++h) {
                            const uint32_t da = smem_u32(sA + stage * STA + h * BOX_A);
                            const uint32_t db = smem_u32(sB + stage * STB + h * 2 * BOX_B);
                            const int ka = tl.a_k0 + (kb + h) * BK, kbb = (kb + h) * BK;
                            if (PAIR) tma_load_3d_pair(da, mapA, fb, ka, arow, tl.mod);
                            else tma_load_3d(da, mapA, fb, ka, arow, tl.mod);
                            for (int y = 0; y < nbx; ++y) {
                                if (PAIR) tma_load_3d_pair(db + y * BOX_B, mapB, fb, kbb, brow + 64 * y, tl.mod);
                                else tma_load_3d(db + y * BOX_B, mapB, fb, kbb, brow + 64 * y, tl.mod);
                            }
                        }
                        issued_mask |= 1u << stage;
                        last_par = (last_par & ~(1u << stage)) | (phase << stage);
                        if (++stage == NST) { stage = 0; phase ^= 1; }
                    }
                    x.kb = end;
                    if (end >= tl.nkb) {
                        x.it += 2 * nunits;
                        load_work(x);
                    }
                }
            }
            if (!ok) {
                // let the copies already issued land before the CTA leaves (the second CTA of a
                // pair cannot observe the first's barrier: it allows them 100 us)
                if (!PAIR || rank == 0) {
                    for (int s = 0; s < NST; ++s)
                        if (issued_mask & (1u << s))
                            mbar_wait(smem_u32(&full[s]), (last_par >> s) & 1, abort_flag, a.err, 1, true);
                } else {
                    const unsigned long long t0 = globaltimer();
                    while (globaltimer() - t0 < 100000ull) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (one thread; of the first CTA of a pair)
        if (lane == 0 && rank == 0) {
            uint32_t stage = 0, phase = 0;
            bool ok = true, any = false;
            load_work(x);
            load_work(y);
            for (; ok && (x.it < nitems || y.it < nitems); swap_streams()) {
                if (x.it < nitems) {
                    // the accumulator's last chunk has been reduced (or its residues stored)
                    if (!mbar_wait(smem_u32(&accempty[x.w]), (x.chunks & 1) ^ 1, abort_flag, a.err, 2)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t idesc = idesc_of(PAIR, x.tl.ncols);
                    const uint32_t d = tmem + x.w * ACC_COLS;
                    const int end = x.kb + kChunkBlocks < x.tl.nkb ? x.kb + kChunkBlocks : x.tl.nkb;
                    for (int kb = x.kb; kb < end; kb += KS) {
                        const int nk = end - kb < KS ? end - kb : KS;
                        if (!mbar_wait(smem_u32(&full[stage]), phase, abort_flag, a.err, 3)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint64_t ad = smem_desc(smem_u32(sA + stage * STA));
                        const uint64_t bd = smem_desc(smem_u32(sB + stage * STB));
#pragma unroll
                        for (int h = 0; h < KS; ++h) {
                            if (h < nk) {
#pragma unroll
                                for (int kk = 0; kk < BK / 16; ++kk) {
                                    const uint32_t acc = (kb > 0 || h > 0 || kk > 0) ? 1u : 0u;
                                    const uint64_t a2 = ad + h * (BOX_A >> 4) + 2 * kk;
                                    const uint64_t b2 = bd + h * (2 * BOX_B >> 4) + 2 * kk;
                                    if (PAIR) mma_bf16_pair(d, a2, b2, idesc, acc);
                                    else mma_bf16(d, a2, b2, idesc, acc);
                                }
                            }
                        }
                        any = true;
                        if (PAIR) mma_commit_pair(smem_u32(&empty[stage]), (uint16_t)3);
                        else mma_commit(smem_u32(&empty[stage]));
                        if (++stage == NST) { stage = 0; phase ^= 1; }
                    }
                    if (!ok) break;
                    if (PAIR) mma_commit_pair(smem_u32(&accfull[x.w]), (uint16_t)3);
                    else mma_commit(smem_u32(&accfull[x.w]));
                    ++x.chunks;
                    x.kb = end;
                    if (end >= x.tl.nkb) {
                        x.it += 2 * nunits;
                        load_work(x);
                    }
                }
            }
            if (any) {   // all MMAs of this CTA (pair) complete before TMEM is released
                if (PAIR) mma_commit_pair(smem_u32(drain), (uint16_t)1);
                else mma_commit(smem_u32(drain));
                mbar_wait(smem_u32(drain), 0, abort_flag, a.err, 4, true);
            }
        }
    } else {
        // ---------------- epilogue: one TMEM lane (output row) per thread
        const int q = warp & 3;
        const int half = (warp - 2) >> 2;   // which half of the tile's columns
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        // balanced residues of 32 columns to [0, m) and 16 bits (a float's low half over 2^23)
        auto pack = [&](const uint32_t (&v)[32], float m, uint32_t* o) {
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const float x = __uint_as_float(v[j]), y = __uint_as_float(v[j + 1]);
                o[j / 2] = __byte_perm(__float_as_uint(__fadd_rn(x < 0.0f ? __fadd_rn(x, m) : x, 8388608.0f)),
                                       __float_as_uint(__fadd_rn(y < 0.0f ? __fadd_rn(y, m) : y, 8388608.0f)), 0x5410);
            }
        };
        // the warp's packed residues (32 rows, ncols / 2 columns each) of an item, 64 columns at a
        // time through shared memory: eight threads then store one row's 128 bytes.  (A row per
        // thread took 32 lines per store instruction: about 5 us an item, as long as the MMAs of
        // an inner length of 1200.)
        char* turn = reinterpret_cast<char*>(smem) + TURN_OFF + (warp - 2) * 4096;
        auto ld_of = [&](const ResTile& tl) { return GROUPED ? a.groups[tl.group].ldr : a.ldr; };
        auto rows_of = [&](const ResTile& tl) {   // the warp's first row, its half of the columns
            return (GROUPED ? a.groups[tl.group].res : a.res) +
                   (long)tl.mod * (GROUPED ? a.groups[tl.group].plane : a.plane) +
                   (long)(tl.m0 + (int)rank * BM + q * 32) * ld_of(tl) + tl.n0 + half * (tl.ncols / 2);
        };
        auto store = [&](const ResTile& tl, const uint32_t (&o)[64]) {
            uint16_t* dst = rows_of(tl);
            const long ldr = ld_of(tl);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (h < tl.ncols / 128) {
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        *reinterpret_cast<uint4*>(turn + lane * 128 + ((c ^ (lane & 7)) * 16)) =
                            make_uint4(o[32 * h + 4 * c], o[32 * h + 4 * c + 1], o[32 * h + 4 * c + 2], o[32 * h + 4 * c + 3]);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = 4 * i + (lane >> 3), c = lane & 7;
                        *reinterpret_cast<uint4*>(dst + (long)r * ldr + 64 * h + 8 * c) =
                            *reinterpret_cast<const uint4*>(turn + r * 128 + ((c ^ (r & 7)) * 16));
                    }
                }
            }
        };
        auto load_chunks = [&](Stream& x) {   // items without an inner range: zeros
            for (load_item(x); x.it < nitems && x.tl.nkb <= 0; load_item(x)) {
                uint4* d = reinterpret_cast<uint4*>(rows_of(x.tl) + (long)lane * ld_of(x.tl));
                for (int g = 0; g < x.tl.ncols / 16; ++g) d[g] = make_uint4(0u, 0u, 0u, 0u);
                x.it += 2 * nunits;
            }
        };
        bool ok = true;
        load_chunks(x);
        load_chunks(y);
        for (; ok && (x.it < nitems || y.it < nitems); swap_streams()) {
            if (x.it < nitems) {
                const float m = c_tab.m[x.tl.mod], inv = c_tab.inv[x.tl.mod];
                const int npc = x.tl.ncols / 64;   // 32-column pieces of this warp (2 or 4)
                if (!mbar_wait(smem_u32(&accfull[x.w]), x.chunks & 1, abort_flag, a.err, 5)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t0 = tmem + lane_off + x.w * ACC_COLS + (uint32_t)(half * (x.tl.ncols / 2));
                x.kb += kChunkBlocks;
                const bool last = x.kb >= x.tl.nkb;
                auto reduce = [&](int p, uint32_t (&v)[32]) {   // 32 columns at a time
                    tmem_ld32(t0 + p * 32, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; j += 2)
                        unpack2(mod_balanced2(pack2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), pack2(inv, inv),
                                              pack2(-m, -m)),
                                v[j], v[j + 1]);
                };
                uint32_t o[64];   // (last chunk) packed residues: stored after the accumulator is released
                if (last) {
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        if (p < npc) {
                            uint32_t v[32];
                            reduce(p, v);
                            pack(v, m, o + 16 * p);
                        }
                    }
                } else {
#pragma unroll 1
                    for (int p = 0; p < npc; ++p) {
                        uint32_t v[32];
                        reduce(p, v);
                        tmem_st32(t0 + p * 32, v);
                    }
                    tmem_wait_st();
                }
                tc_fence_before();
                __syncwarp();
                // The warp's accesses to the accumulator are complete.  (The arrival is relaxed: the
                // fences order the TMEM accesses, and nothing else is handed over.  A release at
                // cluster scope waited for this warp's global stores: 1800 clocks a chunk.)
                if (lane == 0) mbar_arrive_relaxed(PAIR ? cluster_map(smem_u32(&accempty[x.w]), 0) : smem_u32(&accempty[x.w]));
                if (last) store(x.tl, o);
                ++x.chunks;
                if (last) {
                    x.it += 2 * nunits;
                    load_chunks(x);
                }
            }
        }
    }
    tc_fence_before();
    // a pair stays together until the first CTA's MMAs (which read the second's shared memory
    // and write its TMEM) have drained
    if (PAIR) cluster_sync_all();
    else __syncthreads();
    if (a.span && threadIdx.x == 0) atomicMax(&a.span[1], globaltimer());
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tmem_dealloc_pair(tmem, 2 * ACC_COLS);
        else tmem_dealloc(tmem, 2 * ACC_COLS);
    }
}

// ------------------------------------------------------------------- residue planes
// One row per block iteration: the scale exponent from the largest |x| (integer compares on
// the IEEE bits), then COLS destination columns per thread: X = round(x 2^(bits - e)) in
// integer arithmetic, its four digits as floats, and per modulus the residue (seven packed FP32
// operations per two columns), stored as BF16 (a residue's float is exact in BF16: its upper
// half).  Row statistics: e, non-zero count, ||x^||_2 rounded up.
template <bool G, int NT, int COLS>
__device__ __forceinline__ void residue_rows(const SliceArgs& a0, const SliceGroups& gs) {
    const int tid = threadIdx.x;
    __shared__ unsigned long long red_u[NT / 32];
    __shared__ float red_f[NT / 32];
    __shared__ int red_i[NT / 32];
    __shared__ SliceArgs sa;
    const int nflat = G ? gs.rows : a0.nrows;
    for (int flat = blockIdx.x; flat < nflat; flat += gridDim.x) {
        int row = flat;
        if (G) {   // the row's slicing: its arguments to shared memory
            int lo = 0, hi = gs.n - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (gs.offs[mid] <= flat) lo = mid;
                else hi = mid - 1;
            }
            const uint32_t* src = reinterpret_cast<const uint32_t*>(gs.args + lo);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&sa);
            for (int w = tid; w < (int)(sizeof(SliceArgs) / 4); w += NT) dst[w] = src[w];
            __syncthreads();
            row = flat - gs.offs[lo];
        }
        const SliceArgs& a = G ? sa : a0;
        const long srow = a.src_rows ? (long)a.src_rows[row] : (long)row;
        const unsigned long long* src = (const unsigned long long*)(a.src + srow * a.ld_src);
        const int* map = a.col_inv;   // source column of each destination column, -1: padding
        unsigned long long mx = 0;
        auto top = [&](unsigned long long b) {
            b &= 0x7FFFFFFFFFFFFFFFull;
            mx = b > mx ? b : mx;
        };
        if (((uintptr_t)src & 15) == 0) {   // 16-byte loads
            const ulonglong2* s2 = reinterpret_cast<const ulonglong2*>(src);
            const int n2 = a.ncols >> 1;
            int c = tid;
            for (; c + 7 * NT < n2; c += 8 * NT) {
                ulonglong2 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = __ldg(s2 + c + u * NT);
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    top(v[u].x);
                    top(v[u].y);
                }
            }
            {   // the rest (a short row: all of it), loads first as well
                ulonglong2 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = c + u * NT < n2 ? __ldg(s2 + c + u * NT) : make_ulonglong2(0ull, 0ull);
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    top(v[u].x);
                    top(v[u].y);
                }
            }
            if ((a.ncols & 1) && tid == 0) top(src[a.ncols - 1]);
        } else {
#pragma unroll 8
            for (int c = tid; c < a.ncols; c += NT) top(__ldg(src + c));
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = __shfl_xor_sync(0xffffffffu, mx, o);
            mx = y > mx ? y : mx;
        }
        if ((tid & 31) == 0) red_u[tid >> 5] = mx;
        __syncthreads();
        mx = 0;
        for (int w = 0; w < NT / 32; ++w) mx = red_u[w] > mx ? red_u[w] : mx;
        if (mx >= 0x7FF0000000000000ull) mx = 0x7FEFFFFFFFFFFFFFull;   // non-finite input: clamp scale
        const int Emax = (int)(mx >> 52);
        const bool zero_row = (mx == 0);
        const int e = zero_row ? 0 : (Emax > 0 ? Emax - 1022 : -1022);
        const int nmod = a.slices, tab = a.tab;
        const int r0 = 1085 - a.bits + e;   // a column's shift is r0 - max(E, 1)
        const float scale = pow2f(-a.bits);
        const long sstride = a.slice_stride;
        __nv_bfloat16* drow = a.digits + (long)row * a.kpad;
        int nnz = 0;
        float l2sq = 0.0f;
        for (int dc = COLS * tid; dc < a.kpad; dc += COLS * NT) {
            f32x2 d[COLS / 2][4];
            unsigned long long cur[COLS];
            int sc[COLS];
            if (map) {
#pragma unroll
                for (int u = 0; u < COLS; u += 4) {
                    const int4 q = __ldg(reinterpret_cast<const int4*>(map + dc + u));
                    sc[u] = q.x;
                    sc[u + 1] = q.y;
                    sc[u + 2] = q.z;
                    sc[u + 3] = q.w;
                }
            } else {
#pragma unroll
                for (int u = 0; u < COLS; ++u) sc[u] = dc + u < a.ncols ? dc + u : -1;
            }
#pragma unroll
            for (int u = 0; u < COLS; ++u) cur[u] = sc[u] >= 0 ? __ldg(src + sc[u]) : 0ull;
#pragma unroll
            for (int u = 0; u < COLS; u += 2) {
                float dd[2][4];
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const unsigned long long bits = cur[u + w];
                    const uint32_t blo = (uint32_t)bits, bhi = (uint32_t)(bits >> 32);
                    const uint32_t E = (bhi >> 20) & 0x7FFu;
                    // |x| = mant 2^(max(E, 1) - 1075); mant 2^10 shifted down by r >= 7 (bits <= 56), to
                    // nearest, ties up
                    uint32_t mhi = (bhi & 0xFFFFFu) | (E ? 0x100000u : 0u);
                    const bool some = ((mhi | blo) != 0u) && E != 0x7FFu;   // not zero and finite
                    nnz += some;
                    const int r = min(r0 - max((int)E, 1), 64);
                    unsigned long long m = ((unsigned long long)mhi << 32 | blo) << 10;
                    m = some ? ((m >> (r - 1)) + 1ull) >> 1 : 0ull;
                    const long long sgn = (long long)(int)bhi >> 31;
                    const long long I = ((long long)m ^ sgn) - sgn;
                    // digits of I offset to be non-negative: 15-bit fields of I + 2^14 (1 + 2^15 + 2^30 + 2^45)
                    const unsigned long long f =
                        (unsigned long long)(I + ((1ll << 14) + (1ll << 29) + (1ll << 44) + (1ll << 59)));
                    const uint32_t flo = (uint32_t)f, fhi = (uint32_t)(f >> 32);
                    const float off = 8388608.0f + 16384.0f;
                    dd[w][0] = __uint_as_float(0x4B000000u | (flo & 0x7FFFu)) - off;
                    dd[w][1] = __uint_as_float(0x4B000000u | ((flo >> 15) & 0x7FFFu)) - off;
                    dd[w][2] = __uint_as_float(0x4B000000u | (__funnelshift_r(flo, fhi, 30) & 0x7FFFu)) - off;
                    dd[w][3] = __uint_as_float(0x4B000000u | (fhi >> 13)) - off;
                    // x^ to a few FP32 roundings (the row norm's slack covers them)
                    const float xv = __fmaf_rn(__fmaf_rn(__fmaf_rn(dd[w][3], 32768.0f, dd[w][2]), 32768.0f, dd[w][1]),
                                               32768.0f, dd[w][0]) * scale;
                    l2sq = __fmaf_ru(xv, xv, l2sq);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) d[u / 2][k] = pack2(dd[0][k], dd[1][k]);
            }
#pragma unroll 1
            for (int i = 0; i < nmod; ++i) {
                const float k0 = c_tab.digit[tab][i][0], k1 = c_tab.digit[tab][i][1], k2 = c_tab.digit[tab][i][2],
                            k3 = c_tab.digit[tab][i][3], inv = c_tab.inv[i], neg_m = -c_tab.m[i];
                const f32x2 q0 = pack2(k0, k0), q1 = pack2(k1, k1), q2 = pack2(k2, k2), q3 = pack2(k3, k3),
                            inv2 = pack2(inv, inv), neg_m2 = pack2(neg_m, neg_m);
                uint32_t o[COLS / 2];
#pragma unroll
                for (int u = 0; u < COLS / 2; ++u) {
                    uint32_t x, y;
                    const f32x2 t = fma2(d[u][3], q3, fma2(d[u][2], q2, fma2(d[u][1], q1, mul2(d[u][0], q0))));
                    unpack2(mod_balanced2(t, inv2, neg_m2), x, y);
                    o[u] = __byte_perm(x, y, 0x7632);
                }
                __nv_bfloat16* dst = drow + i * sstride + dc;
                if constexpr (COLS == 8) *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
                else *reinterpret_cast<uint2*>(dst) = make_uint2(o[0], o[1]);
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            l2sq = __fadd_ru(l2sq, __shfl_xor_sync(0xffffffffu, l2sq, o));
            nnz += __shfl_xor_sync(0xffffffffu, nnz, o);
        }
        if ((tid & 31) == 0) {
            red_f[tid >> 5] = l2sq;
            red_i[tid >> 5] = nnz;
        }
        __syncthreads();
        if (tid == 0) {
            float L2 = 0.0f;
            int N = 0;
            for (int w = 0; w < NT / 32; ++w) { L2 = __fadd_ru(L2, red_f[w]); N += red_i[w]; }
            // rounding of x^ to `bits` fractional bits: |delta| <= 2^{-bits-1} per non-zero entry
            const float dq = __fmul_ru(__fsqrt_ru((float)N), pow2f(-a.bits - 1));
            a.st.e[row] = e;
            a.st.nnz[row] = N;
            a.st.l2[row] = __fadd_ru(__fmul_ru(__fsqrt_ru(L2), 1.0f + 2.0e-6f), dq);
            a.st.dn[row] = dq;
            if (a.st.inerr) {
                float v = 0.0f;
                if (a.inerr2_prev && !zero_row) {
                    const int de = a.e_prev[row] - e;
                    v = __fmul_ru(__fmul_ru(__fsqrt_ru(a.inerr2_prev[row]), 1.0001f), pow2f(max(-126, min(127, de))));
                    if (de > 127) v = __int_as_float(0x7f800000);   // cannot certify: infinite bound
                }
                a.st.inerr[row] = v;
            }
        }
        __syncthreads();   // the shared buffers are reused by the next row
    }
}

// Four blocks of 256 threads (eight of 128) to an SM.  Measured, 12 000 rows of 12 288 columns and 13
// moduli (1.15 GB read, 3.8 GB written): 0.96 ms, 5.1 TB/s, where scalar loads and scalar FP32 took
// 1.04.  Neither the stores (one plane stored instead of 13: 0.95), the residues' arithmetic (none:
// 0.91) nor the search for the maximum (none: 0.88) bounds it alone; more loads in flight per
// thread cost resident blocks and gained nothing (0.96 to 1.03 over 2 to 5 blocks).
template <int NT, int COLS>
__global__ void __launch_bounds__(NT, 1024 / NT) k_residue_slice(const SliceArgs a) {
    follow_wait();
    residue_rows<false, NT, COLS>(a, SliceGroups{});
}
template <int NT, int COLS>
__global__ void __launch_bounds__(NT, 1024 / NT) k_residue_slice_grouped(const SliceGroups gs) {
    residue_rows<true, NT, COLS>(SliceArgs{}, gs);
}

// ------------------------------------------------------------------- reconstruction
constexpr int kCrtThreads = 128, kCrtCols = 4 * kCrtThreads;
// Threads of a block that share a row (four columns each): rows of few columns leave room for two
// or four rows side by side.
__host__ __device__ __forceinline__ int crt_width(int cols) { return cols <= 128 ? 32 : cols <= 256 ? 64 : kCrtThreads; }
__host__ __device__ __forceinline__ int crt_col_blocks(int cols) { return (cols + kCrtCols - 1) / kCrtCols; }

// Bits of the double nearest (ties up) to F 2^-80 M 2^E0: F a signed 80-bit integer in three words
// (w2, w1, 16 bits w0), M = m_mant 2^(m_exp - 63), E = m_exp - 126 + E0; *mag = |value| 2^-es as a
// float, truncated.  Integer operations: the FP64 units are slow on this part.
__device__ __forceinline__ unsigned long long crt_bits(uint32_t w0, uint32_t w1, uint32_t w2, unsigned long long m_mant,
                                                       int E, int es, float* mag) {
    const uint32_t sgn = (uint32_t)((int)w2 >> 31);
    unsigned long long hi = ((unsigned long long)w2 << 32) | w1;
    uint32_t lo = w0 << 16;       // the word below hi
    if (sgn) {                    // |F|
        lo = 0u - lo;
        hi = ~hi + (lo == 0u ? 1ull : 0ull);
    }
    *mag = 0.0f;
    if (hi == 0ull) {             // |F| below 2^16: one step down
        hi = (unsigned long long)lo << 16;
        lo = 0u;
        E -= 48;
        if (hi == 0ull) return 0ull;
    }
    // leading 64 bits
    int z = __clzll((long long)hi);
    E -= z;
    uint32_t a2 = (uint32_t)(hi >> 32), a1 = (uint32_t)hi, a0 = lo;
    if (z >= 32) {
        a2 = a1;
        a1 = a0;
        a0 = 0u;
        z -= 32;
    }
    const unsigned long long f = ((unsigned long long)__funnelshift_l(a1, a2, z) << 32) | __funnelshift_l(a0, a1, z);
    const unsigned long long P = __umul64hi(f, m_mant);   // 63 or 64 bits; value = P 2^(E + 63)
    const int top = (int)(P >> 63);
    const int ex = E + 62 + 63 + top;                     // exponent of the leading bit
    const int fe = ex - es;
    if (fe >= -126 && fe <= 127)
        *mag = __uint_as_float(((unsigned)(fe + 127) << 23) | ((unsigned)(P >> (39 + top)) & 0x7FFFFFu));
    const unsigned long long q = ((P >> (9 + top)) + 1ull) >> 1;   // 53 bits, or 2^53
    const int be = ex + 1023;
    const unsigned long long sign = (unsigned long long)(sgn & 0x80000000u) << 32;
    if (be <= 0 || be >= 2046)    // outside the normal range: the FP64 route
        return sign | (unsigned long long)__double_as_longlong(ldexp((double)P, E + 63));
    return sign | (((unsigned long long)(be - 1) << 52) + q);   // q's leading bit, or its carry, adds to the exponent
}

// Four columns per thread, a.nrow rows per block.  Per output: C / M = sum_i r_i / m_i mod 1 as
// an 80-bit fixed-point sum (three multiply-adds per modulus, carries combined at the end), then value, certified bound and flag.  Reads the residues once
// (2 bytes per modulus) and writes 8 (12 with bounds) bytes per output.  NM: the number of
// moduli, 0 for any; all of a row's residues are loaded before the first is used.
// Measured: 24.6 M outputs 185 us (0.14 ms at the copy bandwidth; the rest is integer issue), 330
// with rolled loads, 96-bit sums, 64-bit finalisation and block-wide row sums; 50 x 600 outputs 6 us,
// with four rows to a block there 20; the 16 M outputs of a 52-pair plan 140 us, one row to a block 172.
template <bool G, int NM>
__global__ void __launch_bounds__(kCrtThreads) k_crt(const CrtArgs a0, const CrtGroups gs) {
    __shared__ CrtArgs sa;
    __shared__ unsigned long long red_m[kCrtThreads / 32];
    const int tid = threadIdx.x;
    int blk = (int)blockIdx.x;
    follow_next();
    follow_wait();
    if (G) {
        int lo = 0, hi = gs.n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (gs.offs[mid] <= blk) lo = mid;
            else hi = mid - 1;
        }
        const uint32_t* src = reinterpret_cast<const uint32_t*>(gs.args + lo);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&sa);
        for (int w = tid; w < (int)(sizeof(CrtArgs) / 4); w += kCrtThreads) dst[w] = src[w];
        blk -= gs.offs[lo];
    }
    if (G) __syncthreads();
    const CrtArgs& a = G ? sa : a0;
    const int ncb = crt_col_blocks(a.cols), width = crt_width(a.cols);
    const int rb = blk / ncb, cb = blk - rb * ncb;
    const int lane = tid & 31, warp = tid >> 5;
    const int c = cb * kCrtCols + 4 * (tid & (width - 1));   // a warp lies in one row
    const int nmod = NM ? NM : a.nmod;
    const int lr1 = min((rb + 1) * a.nrow, a.rows);
    unsigned long long vmax = 0ull;
    if (c < a.cols) {
        const int4 eB4 = *reinterpret_cast<const int4*>(a.B.e + c);
        const float4 lB4 = *reinterpret_cast<const float4*>(a.B.l2 + c), dB4 = *reinterpret_cast<const float4*>(a.B.dn + c);
        const int eB[4] = {eB4.x, eB4.y, eB4.z, eB4.w};
        const float l2B[4] = {lB4.x, lB4.y, lB4.z, lB4.w}, dqB[4] = {dB4.x, dB4.y, dB4.z, dB4.w};
#pragma unroll 1
        for (int lr = rb * a.nrow + tid / width; lr < lr1; lr += kCrtThreads / width) {
            const int r = a.row0 + lr;
            const uint2* src = reinterpret_cast<const uint2*>(a.res + (long)lr * a.ldr + c);
            uint32_t s0[4] = {0, 0, 0, 0}, s2[4] = {0, 0, 0, 0};   // s0: 16 x 25 bits; s2 wraps (mod 1)
            unsigned long long s1[4] = {0, 0, 0, 0};
            auto add = [&](int i, uint2 v) {
                const uint32_t f0 = c_tab.frac[i][0], f1 = c_tab.frac[i][1], f2 = c_tab.frac[i][2];
                const uint32_t x[4] = {v.x & 0xFFFFu, v.x >> 16, v.y & 0xFFFFu, v.y >> 16};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s0[j] += x[j] * f0;
                    s1[j] += (unsigned long long)x[j] * f1;
                    s2[j] += x[j] * f2;
                }
            };
            if (NM) {
                uint2 v[NM ? NM : 1];
#pragma unroll
                for (int i = 0; i < NM; ++i) v[i] = __ldcs(src + (long)i * (a.plane >> 2));
#pragma unroll
                for (int i = 0; i < NM; ++i) add(i, v[i]);
            } else {
                for (int i = 0; i < nmod; ++i) add(i, __ldcs(src + (long)i * (a.plane >> 2)));
            }
            const int eA = a.A.e[r];
            const float l2A = a.A.l2[r], dqA = a.A.dn[r], inA = a.A.inerr ? a.A.inerr[r] : 0.0f;
            const float cf64A = __fmul_ru(a.c_f64, l2A);
            double vout[4];
            float bout[4];
            float rowerr2 = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned long long t1 = s1[j] + (s0[j] >> 16);
                const int es = eA + eB[j];
                float av;
                bout[j] = 0.0f;
                vout[j] = 0.0;
                if (l2A == 0.0f || l2B[j] == 0.0f) continue;   // an exact zero
                const unsigned long long vb = crt_bits(s0[j] & 0xFFFFu, (uint32_t)t1, s2[j] + (uint32_t)(t1 >> 32),
                                                       a.m_mant, a.m_exp - 126 + es - 2 * a.bits, es, &av);
                vout[j] = __longlong_as_double((long long)vb);
                const float f64b = __fmul_ru(cf64A, l2B[j]);
                const float limit = a.flag_mode == 1 ? fmaxf(a.tol * av, f64b) : f64b;
                // |x^ y^ - X Y| <= ||x^ - X|| ||y^|| + ||X|| ||y^ - Y||
                float bound = __fadd_ru(__fmaf_ru(dqA, l2B[j], __fmul_ru(l2A, dqB[j])), a.c_fix);
                bound = __fmaf_ru(inA, l2B[j], bound);
                if (a.bnd) bout[j] = es > 127 ? __int_as_float(0x7f800000) : __fmul_ru(bound, pow2f(max(es, -126)));
                if (a.rowerr2) {
                    const float bb = __fmul_ru(bound, pow2f(max(-126, min(127, eB[j]))));
                    rowerr2 = __fmaf_ru(bb, bb, rowerr2);
                }
                if (c + j < a.cols_valid) {
                    if (a.absmax) {
                        const unsigned long long ab = vb & 0x7FFFFFFFFFFFFFFFull;
                        vmax = ab > vmax ? ab : vmax;
                    }
                    if (a.flag_mode && bound > limit) {
                        const unsigned int idx = atomicAdd(a.nflags, 1u);
                        if ((int)idx < a.max_flags) a.flags[idx] = make_int2(r, c + j);
                    }
                }
            }
            double2* o = reinterpret_cast<double2*>(a.out + (long)r * a.ldo + c);
            o[0] = make_double2(vout[0], vout[1]);
            o[1] = make_double2(vout[2], vout[3]);
            if (a.bnd) *reinterpret_cast<float4*>(a.bnd + (long)r * a.ldb + c) = make_float4(bout[0], bout[1], bout[2], bout[3]);
            if (a.rowerr2) {   // (columns is a multiple of 128: whole warps are here together)
                for (int o = 16; o > 0; o >>= 1) rowerr2 = __fadd_ru(rowerr2, __shfl_xor_sync(0xffffffffu, rowerr2, o));
                if (lane == 0 && rowerr2 > 0.0f) atomicAdd(&a.rowerr2[r], rowerr2 * 1.0001f);   // (the atomics round to nearest)
            }
        }
    }
    // the largest value: warp maxima, one atomic per block that raises it
    if (a.absmax) {
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = __shfl_xor_sync(0xffffffffu, vmax, o);
            vmax = y > vmax ? y : vmax;
        }
        if (lane == 0) red_m[warp] = vmax;
    }
    __syncthreads();
    if (a.absmax && tid == 0) {
        for (int w = 1; w < kCrtThreads / 32; ++w) vmax = red_m[w] > vmax ? red_m[w] : vmax;
        if (vmax > *(volatile unsigned long long*)a.absmax) atomicMax(a.absmax, vmax);
    }
}

// Function attributes are per device: set them once on each device that launches.
cudaError_t set_attributes_once() {
    static std::atomic<unsigned long long> done{0};   // bit per device ordinal (< 64)
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load() & bit) return cudaSuccess;
    const void* gemms[] = {(const void*)k_residue_gemm<false, false>, (const void*)k_residue_gemm<true, false>,
                           (const void*)k_residue_gemm<false, true>, (const void*)k_residue_gemm<true, true>};
    for (const void* k : gemms) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }
    if (e != cudaSuccess) return e;
    done.fetch_or(bit);
    return cudaSuccess;
}

}  // namespace

double residue_log2m(int n) {
    double s = 0.0;
    for (int i = 0; i < n; ++i) s += std::log2((double)kModuli[i]);
    return s * (1.0 - 1e-12);
}

int residue_moduli(int bits, int K) {
    const double need = 2.0 * bits + std::log2((double)std::max(K, 1)) + 1.0 + 1e-9;
    for (int n = 1; n <= kMaxMod; ++n)
        if (residue_log2m(n) > need) return n;
    return 0;
}

void crt_constants(CrtArgs* a) {
    // M exactly, as 32-bit limbs (16 moduli: 138 bits)
    uint32_t w[6] = {1, 0, 0, 0, 0, 0};
    double msum = 0.0;
    for (int i = 0; i < a->nmod; ++i) {
        unsigned long long carry = 0;
        for (int k = 0; k < 6; ++k) {
            const unsigned long long t = (unsigned long long)w[k] * (unsigned)kModuli[i] + carry;
            w[k] = (uint32_t)t;
            carry = t >> 32;
        }
        msum += kModuli[i];
    }
    int top = 191;
    while (top > 0 && !((w[top >> 5] >> (top & 31)) & 1u)) --top;
    unsigned long long mant = 0;
    for (int k = 0; k < 64; ++k) {
        const int b = top - k;
        mant = (mant << 1) | (b >= 0 ? (w[b >> 5] >> (b & 31)) & 1u : 0u);
    }
    a->m_mant = mant;
    a->m_exp = top;
    // each floor(2^80 / m_i) is short of 2^80 / m_i by less than one unit, times r_i < m_i;
    // units of 2^{eA+eB}: M 2^-80 2^(-2 bits) (2^-51 for 13 moduli at 48 bits).  The final
    // rounding is a relative 2^-53.
    a->c_fix = (float)(std::ldexp(msum, top + 1 - 80 - 2 * a->bits) * 1.01);
}

int crt_blocks(const CrtArgs& a) {
    return crt_col_blocks(a.cols) * ((a.rows + a.nrow - 1) / a.nrow);
}

// Blocks go over several rows (sharing the column statistics, and a grouped launch's look-up of the
// block's arguments) once that leaves every SM plenty of blocks.
void crt_set_rows(CrtArgs* a, int n) {
    long base = 0;
    for (int q = 0; q < n; ++q) {
        a[q].nrow = kCrtThreads / crt_width(a[q].cols);
        base += crt_blocks(a[q]);
    }
    const int k = (int)std::max(1l, std::min(8l, base / 4864));
    for (int q = 0; q < n; ++q) a[q].nrow *= k;
}

cudaError_t launch_residue_gemm(const CUtensorMap& tmA, const CUtensorMap& tmB, const ResGemmArgs& a, int num_sms,
                                cudaStream_t st, bool pair) {
    cudaError_t e = set_attributes_once();
    if (e != cudaSuccess) return e;
    if (a.ntiles <= 0) return cudaSuccess;
    if (a.nmod < 1 || a.nmod > kMaxMod) return cudaErrorInvalidValue;
    const long items = (long)a.ntiles * a.nmod;
    if (items > (1l << 30)) return cudaErrorInvalidValue;
    const int units = (int)std::min<long>(items, pair ? num_sms / 2 : num_sms);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(pair ? 2 * units : units));
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pair ? 2 : 1;
    return pair ? cudaLaunchKernelEx(&cfg, k_residue_gemm<true, false>, tmA, tmB, a)
                : cudaLaunchKernelEx(&cfg, k_residue_gemm<false, false>, tmA, tmB, a);
}

cudaError_t launch_residue_gemm_grouped(const ResGemmArgs& a, int units, cudaStream_t st, bool pair) {
    cudaError_t e = set_attributes_once();
    if (e != cudaSuccess) return e;
    if (a.ntiles <= 0 || units <= 0) return cudaSuccess;
    if (!a.groups || a.ntiles % units) return cudaErrorInvalidValue;
    const CUtensorMap unused = {};   // every item's maps come from its group
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(pair ? 2 * units : units));
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pair ? 1 : 0;
    return pair ? cudaLaunchKernelEx(&cfg, k_residue_gemm<true, true>, unused, unused, a)
                : cudaLaunchKernelEx(&cfg, k_residue_gemm<false, true>, unused, unused, a);
}

cudaError_t launch_crt(const CrtArgs& a0, cudaStream_t st) {
    if (a0.cols % 128) return cudaErrorInvalidValue;   // (the kernel's warps lie whole in a row)
    CrtArgs a = a0;
    crt_set_rows(&a, 1);
    const int nb = crt_blocks(a);
    if (nb <= 0) return cudaSuccess;
    const auto k = a.nmod == 13   ? k_crt<false, 13>
                   : a.nmod == 14 ? k_crt<false, 14>
                   : a.nmod == 15 ? k_crt<false, 15>
                                  : k_crt<false, 0>;
    return launch_following(k, (unsigned)nb, kCrtThreads, st, a, CrtGroups{});
}

cudaError_t launch_crt_grouped(const CrtGroups& g, cudaStream_t st) {
    if (g.blocks <= 0 || g.n <= 0) return cudaSuccess;
    const auto k = g.nmod == 13   ? k_crt<true, 13>
                   : g.nmod == 14 ? k_crt<true, 14>
                   : g.nmod == 15 ? k_crt<true, 15>
                                  : k_crt<true, 0>;
    k<<<g.blocks, kCrtThreads, 0, st>>>(CrtArgs{}, g);
    return cudaGetLastError();
}

// Rows of at most 4096 destination columns take 128 threads of four columns, longer ones 256 of eight
// (as the digit slicing: twice the rows in flight for the same threads).  Where such rows are too
// few to fill the chip with 128 threads each, a row is a chain of passes on a few warps of a
// nearly idle SM: 256 or 512 threads then share it.
constexpr long kFullThreads = 152 * 1024 * 3 / 4;
cudaError_t launch_residue_slice(const SliceArgs& a, cudaStream_t st) {
    if (a.nrows <= 0) return cudaSuccess;
    const unsigned rows = (unsigned)a.nrows;
    if (a.kpad > kShortRow) return launch_following(k_residue_slice<256, 8>, rows, 256, st, a);
    int nt = 128;
    while (nt < 512 && (long)rows * nt < kFullThreads && 4 * nt < a.kpad) nt *= 2;
    return nt == 128   ? launch_following(k_residue_slice<128, 4>, rows, 128, st, a)
           : nt == 256 ? launch_following(k_residue_slice<256, 4>, rows, 256, st, a)
                       : launch_following(k_residue_slice<512, 4>, rows, 512, st, a);
}

cudaError_t launch_residue_slice_grouped(const SliceGroups& g, bool short_rows, cudaStream_t st) {
    if (g.rows <= 0 || g.n <= 0) return cudaSuccess;
    if (short_rows) k_residue_slice_grouped<128, 4><<<g.rows, 128, 0, st>>>(g);
    else k_residue_slice_grouped<256, 8><<<g.rows, 256, 0, st>>>(g);
    return cudaGetLastError();
}

cudaError_t prepare_residue() { return set_attributes_once(); }

}  // namespace split
}  // namespace gain
