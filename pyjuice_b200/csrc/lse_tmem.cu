// Log-sum-exp contractions with the samples along the tensor-memory lanes, for tiles of any
// number of terms (same result as pcb_lse_contract in its BF16 forms):
//   acc[r, b] = sum_k W(k, r) * exp(src[krow[k], b] - m_b)
// with mode 0 writing log(acc) + m (sum forward) and modes 1/2 writing acc * exp(aux + m)
// (element flows; mode 2 first turns node flows into log f - log m).
//
// D[128 samples x n rows] = E[128 samples x k] W[k x n rows]: a thread owns one sample. It
// reads its sample's values of the source rows (a warp reads whole 128-byte lines whatever the
// alignment of the rows), keeps the maximum in a register, exponentiates, rounds to bf16 (hi
// and, in the split form, the remainder's lo) and writes the A operand to tensor memory; the
// packed weights are the B operand in shared memory, and the epilogue writes rows of 32
// consecutive samples. So no operand passes through shared memory on its way to the tensor
// cores, tiles of few rows cost only the columns they have, and the kernel is bound by the
// rows it reads and writes and by the exponentials and logarithms (16 per SM and cycle).
//
// A CTA takes one tile and 128 samples: 8 warps (two per lane quarter, each with half of a
// chunk's 128 terms) load, exponentiate and finish; warp 8 copies weights and row numbers
// ahead and issues the MMAs. Two CTAs share an SM (256 tensor-memory columns each: 128
// accumulators, 2 x 64 of A), so that one loads while the other computes.
//
// Tiles of more than 128 terms: the chunks are split over a cluster of up to 8 CTAs, which
// exchange their accumulators through distributed shared memory and add them in rank order
// (deterministic), each scaled from its CTA's maximum to the common one. A CTA with several
// chunks starts D afresh for each and adds it to FP32 sums in shared memory: the tensor cores
// truncate when they accumulate (about 3e-8 of the sum per instruction, always downwards), so
// that 16 chunks accumulated in D would be 1.3e-5 too small, against 3e-7 this way.
//
// Measured (forward, split form, weights packed, graph-timed): 119 tiles of 128 x 128, batch 512
// (70 MB): 18.3 us, 3.8 TB/s, against 33.9 us for the best of the forms that keep the samples in
// shared memory (lse_tc05.cu); 200 regions of 256 x 256 (262 MB): 83.4 us, 3.1 TB/s, on the
// persistent form below, against 305 us in 128-term chunks; element flows of the same layer
// (367 MB): 105.6 us (139 us without the element values' prefetch and with the next rows'
// loads after the conversion), against 444 us. What is left of a chunk there, about 6,000 cycles:
// 1,800 until its rows are requested (a SM takes about 37 bytes per cycle), 1,200 of
// exponentials, up to 1,500 of sums or results, 900 of maxima and waits.
//
// Every wait is bounded; a CTA whose wait runs out writes NaN rows and reports
// PCB_STATUS_WAIT_TIMEOUT.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "tc05.cuh"

namespace cg = cooperative_groups;

namespace {

using namespace pcb::tc05;

constexpr int KT = 128;                        // terms per chunk
constexpr int NS = 128;                        // samples per CTA (the MMA's M)
constexpr int kComputeThreads = 256;
constexpr int kThreads = kComputeThreads + 32;
constexpr int HT = KT / 2;                     // terms per thread and chunk
constexpr uint32_t kHalfBytes = 128 * KT * 2;  // one bf16 copy of a packed 128 x 128 tile
constexpr uint32_t kTileBytes = 2 * kHalfBytes;
constexpr uint32_t kLBO = 128;                 // bytes between core matrices along K
constexpr uint32_t kSBO = (KT / 8) * 128;      // bytes between 8-row groups
constexpr uint32_t kColsD = 128, kColsA = KT / 2, kCols = 256;
constexpr int kMaxCluster = 8;
constexpr uint32_t kShared = 77 * 1024;        // least shared memory of a CTA

struct Smem {
    // the weights come first (n_pad x 128 x (hi + lo) bf16), and in their place, once the MMAs
    // are done, what the cluster's other CTAs send: per CTA the column blocks owned here
    uint32_t sum, part, max, rows, bar, slot, total;
    __host__ __device__ Smem(int n_pad, bool several, int ks) {
        const uint32_t w = (uint32_t)n_pad * KT * 4;
        const int blocks = n_pad / 16, owned = (blocks + ks - 1) / ks;
        const uint32_t recv = (uint32_t)((ks - 1) * owned) * 16 * NS * 4;
        sum = w > recv ? w : recv;
        part = sum + (several ? w : 0);  // [n_pad][NS] FP32 sums of a CTA with several chunks
        max = part + 2 * 2 * NS * 4;       // [2 buffers][2 halves][NS] chunk maxima; [CTA][NS] final ones
        rows = max + kMaxCluster * NS * 4; // [2 buffers][KT] source rows of a chunk
        bar = rows + 2 * KT * 4;
        slot = bar + 6 * 8;
        total = slot + 16;
    }
};

// D (tensor memory) += A (tensor memory, K-major) B (shared memory)
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d),
        "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 16 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::
            "r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint64_t* m) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(m)) : "memory");
}

// Packed FP32 pairs (one instruction for two values)
__device__ __forceinline__ uint64_t pair(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpair(uint64_t x) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float lg2(float x) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f, kFloatMin = 1.17549435e-38f;

// bf16 roundings of a pair (hi) and of what they leave (lo), packed
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// x[j] = log(x[j]) + m[j]: one logarithm and one multiply-add each while every x is a normal
// number and every m finite (voted by the warp), else the careful form. SIGN -1 subtracts m.
template <int N, int SIGN>
__device__ __forceinline__ void log_add(float (&x)[N], const float (&m)[N]) {
    float lo = x[0], ml = m[0];
#pragma unroll
    for (int j = 1; j < N; ++j) lo = fminf(lo, x[j]), ml = fminf(ml, m[j]);
    if (__all_sync(0xffffffffu, lo >= kFloatMin && ml > -INFINITY)) {
#pragma unroll
        for (int j = 0; j < N; ++j) x[j] = fmaf(lg2(x[j]), kLn2, SIGN * m[j]);
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) x[j] = m[j] == -INFINITY ? -INFINITY : pcb::fast_log(x[j]) + SIGN * m[j];
    }
}

// 16 values down a column: to rows 0 .. rows - 1 of it, ld apart
__device__ __forceinline__ void store16(float* __restrict__ dst, int64_t ld, const float (&x)[16], bool in, int rows) {
    if (in && rows >= 16) {
#pragma unroll
        for (int j = 0; j < 16; ++j) dst[(int64_t)j * ld] = x[j];
    } else if (in) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (j < rows) dst[(int64_t)j * ld] = x[j];
    }
}

// Barrier of the 256 compute threads
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, 256;\n" ::: "memory"); }

// Instruction descriptor: D f32, A and B bf16, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t idesc_n(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// The MMAs of one chunk into a fresh accumulator d (a: A's parts, kColsA columns apart; w: the
// weights' parts, wp bytes apart). Tiles of several chunks, and the FP32 form, take the small
// products first: what additions to an already large accumulator truncate is then left by the
// hi * hi steps alone. Split tiles of one chunk take them step by step, like the other tcgen05
// kernels, whose results theirs equal. The FP32 form halves what truncation is left with a
// second accumulator.
template <int NP>
__device__ __forceinline__ void issue_mmas(uint32_t d, uint32_t a, uint32_t w, uint32_t wp, int steps, uint32_t idesc,
                                           bool small_first) {
    auto mma = [&](int s, int pa, int pw, uint32_t acc, uint32_t dd) {
        mma_ts(dd, a + pa * kColsA + s * 8, desc(w + pw * wp + (uint32_t)s * 2 * kLBO, kLBO, kSBO), idesc, acc);
    };
    if (NP == 3) {
        // half of the hi * hi steps to the accumulator behind d, alone
        const uint32_t d2 = d + kColsD;
        const int h = (steps + 1) / 2;
        for (int s = 0; s < steps; ++s) {
            mma(s, 0, 2, s > 0 ? 1u : 0u, d);
            mma(s, 2, 0, 1u, d);
            mma(s, 1, 1, 1u, d);
        }
        for (int s = 0; s < steps; ++s) {
            mma(s, 0, 1, 1u, d);
            mma(s, 1, 0, 1u, d);
        }
        for (int s = 0; s < h; ++s) mma(s, 0, 0, s > 0 ? 1u : 0u, d2);
        for (int s = h; s < steps; ++s) mma(s, 0, 0, 1u, d);
    } else if (NP == 1 || !small_first) {
        for (int s = 0; s < steps; ++s) {
            mma(s, 0, 0, s > 0 ? 1u : 0u, d);
            if (NP == 2) {
                mma(s, 0, 1, 1u, d);
                mma(s, 1, 0, 1u, d);
            }
        }
    } else {
        for (int s = 0; s < steps; ++s) {
            mma(s, 0, 1, s > 0 ? 1u : 0u, d);
            mma(s, 1, 0, 1u, d);
        }
        for (int s = 0; s < steps; ++s) mma(s, 0, 0, 1u, d);
    }
}

template <int MODE, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 2)
lse_tmem_kernel(const float* __restrict__ src, const float* __restrict__ src2, const float* __restrict__ aux,
                float* __restrict__ out, int64_t ld, int B, const uint8_t* __restrict__ packed,
                const PcbLseTile* __restrict__ tiles, const int* __restrict__ krow,
                const int* __restrict__ chunk_index, int chunk_ld, int n_max, bool several,
                int num_slices, int32_t* __restrict__ status) {
    pcb::pdl_trigger();
    extern __shared__ __align__(1024) uint8_t sm[];
    cg::cluster_group cluster = cg::this_cluster();
    const int ks = (int)cluster.num_blocks();
    const int rank = (int)cluster.block_rank();
    const Smem S(n_max, several, ks);
    float* sSum = reinterpret_cast<float*>(sm + S.sum);  // [rows][samples]
    float* sPart = reinterpret_cast<float*>(sm + S.part);
    float* sMax = reinterpret_cast<float*>(sm + S.max);
    int* sRows = reinterpret_cast<int*>(sm + S.rows);
    uint64_t* barW = reinterpret_cast<uint64_t*>(sm + S.bar);  // weights of a chunk arrived
    uint64_t* barM = barW + 1;                                 // MMAs of a chunk completed
    uint64_t* barA = barW + 2;                                 // A operand of a chunk written
    uint64_t* barR = barW + 3;                                 // [2] row numbers of a chunk written
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + S.slot);

    const int unit = blockIdx.x / ks;
    const int tile_id = unit / num_slices;
    const int b0 = (unit - tile_id * num_slices) * NS;
    const PcbLseTile t = tiles[tile_id];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_pad = (t.n_rows + 15) & ~15;
    const int nch_tile = (t.k_cnt + KT - 1) / KT;
    const int nch = rank < nch_tile ? (nch_tile - rank + ks - 1) / ks : 0;  // chunks rank, rank + ks, ...
    auto chunk_of = [&](int i) { return rank + i * ks; };
    auto terms_of = [&](int i) { return min(KT, t.k_cnt - chunk_of(i) * KT); };

    if (warp == 8) {
        tmem_alloc(slot, kCols);
        fence_before_sync();
    }
    // the first chunk's source rows (compiled tables), the tile's first one beyond its terms
    if (tid < KT && nch > 0) sRows[tid] = __ldg(krow + t.k_off + (tid < terms_of(0) ? chunk_of(0) * KT + tid : 0));
    if (tid == 0) {
        mbar_init(barW, 1);
        mbar_init(barM, 1);
        mbar_init(barA, kComputeThreads / 32);
        mbar_init(barR, 1);
        mbar_init(barR + 1, 1);
        slot[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    fence_after_sync();
    const uint32_t taddr = slot[0];
    bool fail = false;
    float own[2][16];  // this thread's sums of the column blocks that its CTA owns

    if (warp == 8) {
        auto put_rows = [&](int i) {  // source rows of a later chunk
            const int nk = terms_of(i);
            int* dst = sRows + (i & 1) * KT;
#pragma unroll
            for (int j = 0; j < KT / 32; ++j) {
                const int k = lane + 32 * j;
                dst[k] = __ldg(krow + t.k_off + (k < nk ? chunk_of(i) * KT + k : 0));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(barR + (i & 1));
        };
        if (nch > 1) put_rows(1);
        pcb::pdl_wait();
        auto copy_weights = [&](int i) {
            if (lane != 0) return;
            const int c = chunk_index ? __ldg(chunk_index + (int64_t)tile_id * chunk_ld + chunk_of(i)) : tile_id;
            const uint8_t* w = packed + (size_t)c * kTileBytes;
            const uint32_t half = (uint32_t)n_pad * KT * 2;
            mbar_expect_tx(barW, SPLIT ? 2 * half : half);
            bulk_copy_g2s(sm, w, half, barW);
            if (SPLIT) bulk_copy_g2s(sm + half, w + kHalfBytes, half, barW);
        };
        if (nch > 0) copy_weights(0);
        for (int i = 0; i < nch; ++i) {
            bool ok = mbar_wait_bounded(barA, (uint32_t)(i & 1));
            ok = mbar_wait_bounded(barW, (uint32_t)(i & 1)) && ok;
            fence_after_sync();
            if (lane == 0) {
                if (ok) {
                    const uint32_t idesc = idesc_n(n_pad);
                    const uint32_t w = smem_u32(sm), wp = (uint32_t)n_pad * KT * 2;
                    const uint32_t a = taddr + kColsD;
                    const int steps = (terms_of(i) + 15) / 16;
                    issue_mmas<SPLIT ? 2 : 1>(taddr, a, w, wp, steps, idesc, nch_tile > 1);
                } else {
                    slot[1] = 1;
                }
                commit(barM);
            }
            __syncwarp();
            if (i + 2 < nch) put_rows(i + 2);  // the compute warps have read the rows of chunk i
            if (i + 1 < nch) {
                if (!mbar_wait_bounded(barM, (uint32_t)(i & 1)) && lane == 0) slot[1] = 1;
                copy_weights(i + 1);
            }
        }
        if (ks > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        }
    } else {
        const int half = warp >> 2;
        const int s = (warp & 3) * 32 + lane;  // this thread's sample (tensor-memory lane)
        const uint32_t tlane = taddr + ((uint32_t)((warp & 3) * 32) << 16);
        const bool active = b0 + (warp & 3) * 32 < B;  // any sample of this warp in the batch
        const int b = min(b0 + s, B - 1);
        const float* psrc = src + b;
        const float* psrc2 = MODE == 2 ? src2 + b : nullptr;
        float mref = -INFINITY, scale = 1.f;
        pcb::pdl_wait();
        const uint32_t traw = tlane + half * HT;                   // raw values, in D's columns
        const uint32_t ta = tlane + kColsD + half * (HT / 2);      // hi, then lo
        const uint64_t log2e = pair(kLog2e, kLog2e), minus1 = pair(-1.f, -1.f);
        for (int i = 0; i < nch; ++i) {
            // row numbers: buffer i & 1 is written for chunks 1, 3, .. and 2, 4, ..
            if (i > 0 && !mbar_wait_bounded(barR + (i & 1), (uint32_t)(((i - 1) >> 1) & 1))) fail = true;
            const int4* rows = reinterpret_cast<const int4*>(sRows + (i & 1) * KT + half * HT);
            const int nk = terms_of(i) - half * HT;  // terms of this half
            if (i > 0) {
                // the MMAs of the last chunk are done: A is free, and D goes to the sums
                if (!mbar_wait_bounded(barM, (uint32_t)((i - 1) & 1))) fail = true;
                fence_after_sync();
#pragma unroll 1
                for (int c = half * 16; c < n_pad; c += 32) {
                    float d[16];
                    tmem_ld16(tlane + c, d);
                    wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float* p = sSum + (c + j) * NS + s;
                        *p = (i > 1 ? *p * scale : 0.f) + d[j];
                    }
                }
                fence_before_sync();
                compute_sync();  // both halves have read D before either writes raw values to it
                fence_after_sync();
            }
            // values of the source rows: their maximum, and themselves to tensor memory
            float m = -INFINITY;
            constexpr int G = MODE == 2 ? 32 : 64;  // rows whose loads are in flight together
#pragma unroll 1
            for (int g = 0; g < HT; g += G) {
                float v[G];
                if (active && g < nk) {
                    float m2[MODE == 2 ? G : 1];
#pragma unroll
                    for (int j = 0; j < G; j += 4) {
                        const int4 r4 = rows[(g + j) / 4];
                        const int rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int64_t o = (int64_t)rr[q] * ld;
                            v[j + q] = __ldg(psrc + o);
                            if (MODE == 2) m2[j + q] = __ldg(psrc2 + o);
                        }
                    }
                    if constexpr (MODE == 2) log_add<G, -1>(v, m2);
                    if (g + G > nk) {  // places beyond the chunk's terms count as -inf
#pragma unroll
                        for (int j = 0; j < G; ++j)
                            if (g + j >= nk) v[j] = -INFINITY;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < G; ++j) v[j] = -INFINITY;
                }
#pragma unroll
                for (int j = 0; j < G; j += 2) m = fmaxf(m, fmaxf(v[j], v[j + 1]));
#pragma unroll
                for (int j = 0; j < G; j += 16) {
                    uint32_t w[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) w[q] = __float_as_uint(v[j + q]);
                    tmem_st16(traw + g + j, w);
                }
            }
            wait_st();
            float* part = sPart + (i & 1) * 2 * NS;
            part[half * NS + s] = m;
            compute_sync();
            m = fmaxf(fmaxf(m, part[(half ^ 1) * NS + s]), mref);
            scale = m == mref ? 1.f : pcb::fast_exp(mref - m);  // of the sums so far
            mref = m;
            const float mu = mref == -INFINITY ? 0.f : mref;
            const uint64_t nmu = pair(-mu, -mu);
#pragma unroll 1
            for (int g = 0; g < HT; g += 16) {
                float v[16];
                tmem_ld16(traw + g, v);
                wait_ld();
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint64_t x = mul2(add2(pair(v[2 * j], v[2 * j + 1]), nmu), log2e);
                    const float2 x2 = unpair(x);
                    const float e0 = ex2(x2.x), e1 = ex2(x2.y);
                    hi[j] = bf16x2(e0, e1);
                    if (SPLIT) {
                        const uint64_t h = pair(__uint_as_float(hi[j] << 16), __uint_as_float(hi[j] & 0xffff0000u));
                        const float2 l = unpair(fma2(h, minus1, pair(e0, e1)));
                        lo[j] = bf16x2(l.x, l.y);
                    }
                }
                tmem_st8(ta + g / 2, hi);
                if (SPLIT) tmem_st8(ta + kColsA + g / 2, lo);
            }
            wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(barA);
        }
        const bool in = b0 + s < B;
        const int nb16 = n_pad / 16;  // column blocks, alternating between the halves
        const bool none = mref == -INFINITY;  // no term above -inf: log 0 / no flow
        const bool solo = ks == 1;
        // element values of a column block, one block ahead of their use
        float a[MODE == 0 ? 1 : 16];
        auto load_aux = [&](int blk) {
            if constexpr (MODE != 0) {
                if (!active || blk >= nb16) return;
                const float* ax = aux + ((int64_t)t.aux_row + blk * 16) * ld + b;
#pragma unroll
                for (int j = 0; j < 16; ++j) a[j] = __ldg(ax + (int64_t)min(j, t.n_rows - 1 - blk * 16) * ld);
            }
        };
        if (solo) load_aux(half);
        if (nch > 0 && !mbar_wait_bounded(barM, (uint32_t)((nch - 1) & 1))) fail = true;
        fence_after_sync();
        fail = fail || slot[1] != 0;
        if (solo) {
#pragma unroll 1
            for (int blk = half; blk < nb16; blk += 2) {
                float d[16];
                tmem_ld16(tlane + blk * 16, d);
                wait_ld();
                if (nch > 1) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) d[j] += sSum[(blk * 16 + j) * NS + s] * scale;
                }
                // all values first, then all stores: 16 independent chains
                if (MODE == 0) {
                    float m[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) m[j] = mref;
                    log_add<16, 1>(d, m);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) d[j] = none ? 0.f : d[j] * ex2((a[MODE == 0 ? 0 : j] + mref) * kLog2e);
                    load_aux(blk + 2);
                }
                if (fail) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) d[j] = __int_as_float(0x7fc00000);
                }
                store16(out + ((int64_t)t.out_row + blk * 16) * ld + b0 + s, ld, d, in, t.n_rows - blk * 16);
            }
        } else {
            // Column block c belongs to CTA c % ks. This thread's own blocks (its half takes every
            // other one, two at most) to registers, the others to their owners once every CTA
            // of the cluster is done with its weights.
            asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
            auto sums = [&](int blk, float (&d)[16]) {
                if (nch > 0) {
                    tmem_ld16(tlane + blk * 16, d);
                    wait_ld();
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (nch == 0) d[j] = 0.f;
                    if (nch > 1) d[j] += sSum[(blk * 16 + j) * NS + s] * scale;
                    if (fail) d[j] = __int_as_float(0x7fc00000);
                }
            };
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int blk = rank + ks * (half + 2 * o);
                if (blk < nb16) sums(blk, own[o]);
            }
            asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
            const int owned_max = (nb16 + ks - 1) / ks;
            for (int blk = half; blk < nb16; blk += 2) {
                const int to = blk % ks;
                if (to == rank) continue;
                float d[16];
                sums(blk, d);
                const int from = rank < to ? rank : rank - 1;  // place among the owner's senders
                float* dst = cluster.map_shared_rank(reinterpret_cast<float*>(sm), to) +
                             (size_t)((from * owned_max + blk / ks) * 16) * NS + s;
#pragma unroll
                for (int j = 0; j < 16; ++j) dst[j * NS] = d[j];
            }
            if (half == 0) {
                for (int r = 0; r < ks; ++r) cluster.map_shared_rank(sMax, r)[rank * NS + s] = mref;
            }
        }
        fence_before_sync();
    }
    if (fail) pcb::report_status(status, PCB_STATUS_WAIT_TIMEOUT);
    __syncthreads();
    if (warp == 8) {
        fence_after_sync();
        tmem_dealloc(taddr, kCols);
    }
    if (ks == 1) return;
    cluster.sync();
    if (warp == 8) return;
    const int half = warp >> 2;
    const int s = (warp & 3) * 32 + lane;
    const bool in = b0 + s < B;
    // own sums + what the others sent, in rank order, each scaled to the common maximum
    float f[kMaxCluster];
    float mm = -INFINITY;
#pragma unroll
    for (int r = 0; r < kMaxCluster; ++r) {
        f[r] = r < ks ? sMax[r * NS + s] : -INFINITY;
        mm = fmaxf(mm, f[r]);
    }
#pragma unroll
    for (int r = 0; r < kMaxCluster; ++r) f[r] = f[r] == -INFINITY ? 0.f : pcb::fast_exp(f[r] - mm);
    const int nb16 = n_pad / 16;
    const int owned_max = (nb16 + ks - 1) / ks;
#pragma unroll
    for (int o = 0; o < 2; ++o) {
        const int blk = rank + ks * (half + 2 * o);
        if (blk >= nb16) break;
        float a[16], x[16];
        if (MODE != 0) {
            const float* ax = aux + ((int64_t)t.aux_row + blk * 16) * ld + b0 + s;
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = in ? __ldg(ax + (int64_t)min(j, t.n_rows - 1 - blk * 16) * ld) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = 0.f;
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) {
            if (r >= ks) break;
            if (r == rank) {
#pragma unroll
                for (int j = 0; j < 16; ++j) x[j] += own[o][j] * f[r];
            } else {
                const float* p = reinterpret_cast<const float*>(sm) +
                                 (size_t)(((r < rank ? r : r - 1) * owned_max + half + 2 * o) * 16) * NS + s;
#pragma unroll
                for (int j = 0; j < 16; ++j) x[j] += p[j * NS] * f[r];
            }
        }
        if (MODE == 0) {
            float m[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) m[j] = mm;
            log_add<16, 1>(x, m);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = mm == -INFINITY ? 0.f : x[j] * ex2((a[j] + mm) * kLog2e);
        }
        store16(out + ((int64_t)t.out_row + blk * 16) * ld + b0 + s, ld, x, in, t.n_rows - blk * 16);
    }
}

// ---------------------------------------------------------------------------------------
// Persistent form, for layers with a (tile, 128-sample slice) unit per SM or more: one CTA per
// SM walks a contiguous run of units, chunk by chunk (q = 0, 1, ... over all of them). 16
// compute warps (four per lane quarter, 32 terms of a chunk each) hold a chunk's values in
// registers; warp 16 issues the MMAs and copies weights and row numbers ahead. A, D and the
// weights are double buffered (slot q & 1): while chunk q's MMAs run, the compute warps have
// the rows of chunk q + 1 in flight, and finish the unit that ended at q - 1. A unit of two
// chunks keeps both accumulators apart until its end; of more, the older one goes to FP32 sums
// in shared memory (for the same reason as above). Consecutive slices of a tile reuse its
// weights.
//
// A SM takes a 128-byte load of 32 lanes every 4.5 cycles: 2,300 of a chunk's cycles. Values
// (mode 0) therefore come as 16-byte asynchronous copies through shared memory (COPY), one
// instruction per row: 200 regions of 256 x 256 86.8 -> 83.4 us, 1 of 2048 x 2048 57.5 -> 51.8, FP32
// 119 of 128 x 128 with the pack 46.8 -> 41.6. Element flows keep the loads (copied: 119 tiles 32.4
// against 31.2, 200 regions 105.0 against 105.2): their registers spill. Bulk copies of a row (512
// bytes) take 100 cycles each (156 us); three loader warps have too few copies in flight (88 us).
//
// NP parts per operand: 1 single bf16, 2 split (hi, lo), 3 (hi, mid, lo: 24 bits; the six products
// down to 2^-18, smallest first, then hi * hi alone truncates). Three parts are not FP32 arithmetic:
// the truncation leaves a mean error of -1.6e-7 in the log values (FFMA with rounding: -2e-8), and
// of an exponential below e^-75 the low part falls under bf16's subnormals (2^-18 of the value
// left at e^-80, 2^-13 at e^-84, nothing below e^-87). So callers choose this form, it is no default. With
// three parts A has one slot, D's two hold one chunk, whose sums go to shared memory when another
// follows, and the weights then have one slot too. 119 tiles of 128 x
// 128, batch 512: 40 us with the pack against 102 us for FFMA; norm of the element flows' error
// 3.04e-7 against 3.06e-7.
constexpr int kPWarps = 16;
constexpr int kPThreads = 32 * kPWarps + 32;
constexpr int PT = KT / 4;  // terms per thread and chunk
constexpr int EB = 8;       // accumulator columns per epilogue step
constexpr int kRowRing = 4;
constexpr uint32_t kPShared = 152 * 1024;  // least shared memory of a CTA
constexpr uint32_t kPSlots = 216 * 1024;  // shared memory for weights, sums and values

struct PSmem {
    uint32_t wslot, sum, vals, part, rows, bar, slot, total;  // the weight slots come first
    int nw;
    __host__ __device__ PSmem(int n_pad, int np, bool sums, bool copied) {
        wslot = (uint32_t)n_pad * KT * 2 * (np < 2 ? 2 : np);
        const uint32_t rest = (sums ? (uint32_t)n_pad * NS * 4 : 0) + (copied ? KT * NS * 4 : 0);
        nw = (np == 3 && sums) || 2 * wslot + rest > kPSlots ? 1 : 2;
        sum = nw * wslot;
        vals = sum + (sums ? (uint32_t)n_pad * NS * 4 : 0);  // [KT][NS] values of a chunk (copied rows)
        part = vals + (copied ? KT * NS * 4 : 0);              // [2 buffers][4 parts][NS] chunk maxima
        rows = part + 2 * 4 * NS * 4;       // [kRowRing][KT]
        bar = rows + kRowRing * KT * 4;
        slot = bar + 16 * 8;
        total = slot + 16;
    }
    __host__ __device__ bool fits() const { return part <= kPSlots; }
};

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// exp(m - to) for a scale between maxima; equal ones (also both -inf) give 1
__device__ __forceinline__ float rescale(float m, float to) { return m == to ? 1.f : pcb::fast_exp(m - to); }

template <int MODE, int NP, bool COPY>
__global__ void __launch_bounds__(kPThreads, 1)
lse_tmem_persistent_kernel(const float* __restrict__ src, const float* __restrict__ src2,
                           const float* __restrict__ aux, float* __restrict__ out, int64_t ld, int B,
                           const uint8_t* __restrict__ packed, const PcbLseTile* __restrict__ tiles,
                           const int* __restrict__ krow, const int* __restrict__ chunk_index, int chunk_ld, int n_max,
                           bool sums, int num_slices, int num_units, int32_t* __restrict__ status) {
    pcb::pdl_trigger();
    extern __shared__ __align__(1024) uint8_t sm[];
    constexpr int AS = NP == 3 ? 1 : 2;  // slots of A
    static_assert(NP < 3 || MODE < 2, "the FP32 form takes rewritten flows");
    const PSmem S(n_max, NP, sums, COPY);
    float* sSum = reinterpret_cast<float*>(sm + S.sum);  // [rows][samples]
    float* sVals = reinterpret_cast<float*>(sm + S.vals);
    float* sPart = reinterpret_cast<float*>(sm + S.part);
    int* sRows = reinterpret_cast<int*>(sm + S.rows);
    uint64_t* barW = reinterpret_cast<uint64_t*>(sm + S.bar);  // [2] weights arrived
    uint64_t* barM = barW + 2;                                 // [2] MMAs completed
    uint64_t* barA = barW + 4;                                 // [2] A written, D read
    uint64_t* barR = barW + 6;                                 // [kRowRing] row numbers written
    uint64_t* barV = barW + 10;                                // values of a chunk arrived
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + S.slot);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int u0 = (int)((int64_t)num_units * blockIdx.x / gridDim.x);
    const int u1 = (int)((int64_t)num_units * (blockIdx.x + 1) / gridDim.x);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(barW + i, 1);
            mbar_init(barM + i, 1);
            mbar_init(barA + i, kPWarps);
        }
        for (int i = 0; i < kRowRing; ++i) mbar_init(barR + i, 1);
        mbar_init(barV, 32 * kPWarps);
        slot[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    uint32_t taddr = 0;
    auto columns = [slot]() {  // all warps, once warp 16 has allocated
        asm volatile("bar.sync 2, %0;\n" ::"n"(kPThreads) : "memory");
        fence_after_sync();
        return *slot;
    };
    // columns: D of slots 0 and 1, then A (its parts side by side) of slots 0 and 1
    auto d_cols = [&](int q) { return taddr + (NP == 3 ? 0 : (q & 1) * kColsD); };
    auto a_cols = [&](int q) { return taddr + 2 * kColsD + (AS == 1 ? 0 : (q & 1) * 2 * kColsA); };
    auto chunks_of = [&](const PcbLseTile& t) { return max(1, (t.k_cnt + KT - 1) / KT); };
    bool fail = false;

    if (warp == kPWarps) {
        // position of the next chunk whose row numbers, and whose weights, are fetched
        int ru = u0, ri = 0, rq = 0, wu = u0, wi = 0, wq = 0;
        int held[2] = {-1, -1}, loads[2] = {0, 0};
        auto put_rows = [&]() {
            if (ru >= u1) return;
            const PcbLseTile t = tiles[ru / num_slices];
            int* dst = sRows + (rq % kRowRing) * KT;
#pragma unroll
            for (int j = 0; j < KT / 32; ++j) {
                const int k = ri * KT + lane + 32 * j;
                dst[lane + 32 * j] = t.k_cnt > 0 ? __ldg(krow + t.k_off + (k < t.k_cnt ? k : 0)) : 0;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(barR + rq % kRowRing);
            ++rq;
            if (++ri == chunks_of(t)) ri = 0, ++ru;
        };
        auto copy_weights = [&]() {
            if (wu >= u1) return;
            const int tile_id = wu / num_slices;
            const PcbLseTile t = tiles[tile_id];
            const int c = chunk_index ? __ldg(chunk_index + (int64_t)tile_id * chunk_ld + wi) : tile_id;
            const int sl = S.nw == 1 ? 0 : wq & 1;
            if (held[sl] != c) {
                held[sl] = c;
                ++loads[sl];
                if (lane == 0) {
                    const uint8_t* w = packed + (size_t)c * (NP == 3 ? 3 * kHalfBytes : kTileBytes);
                    const uint32_t bytes = (uint32_t)((t.n_rows + 15) & ~15) * KT * 2;
                    mbar_expect_tx(barW + sl, NP * bytes);
                    for (int p = 0; p < NP; ++p)
                        bulk_copy_g2s(sm + sl * S.wslot + p * bytes, w + p * kHalfBytes, bytes, barW + sl);
                }
            }
            ++wq;
            if (++wi == chunks_of(t)) wi = 0, ++wu;
        };
        put_rows();
        put_rows();
        put_rows();
        pcb::pdl_wait();
        if (S.nw == 2) copy_weights();
        __syncwarp();
        tmem_alloc(slot, 512);
        fence_before_sync();
        taddr = columns();
        int q = 0;
        for (int u = u0; u < u1; ++u) {
            const PcbLseTile t = tiles[u / num_slices];
            const int nch = chunks_of(t);
            const int n_pad = (t.n_rows + 15) & ~15;
            for (int i = 0; i < nch; ++i, ++q) {
                const int sl = q & 1;
                // chunk q + 1's weights (with one slot chunk q's) once the MMAs of chunk q - 1 have
                // left their slot
                if (q > 0 && !mbar_wait_bounded(barM + (sl ^ 1), (uint32_t)(((q - 1) >> 1) & 1)) && lane == 0) slot[1] = 1;
                copy_weights();
                bool ok = mbar_wait_bounded(barA + sl, (uint32_t)((q >> 1) & 1));
                const int ws = S.nw == 1 ? 0 : sl;
                ok = mbar_wait_bounded(barW + ws, (uint32_t)((loads[ws] - 1) & 1)) && ok;
                fence_after_sync();
                if (lane == 0) {
                    if (ok) {
                        const uint32_t idesc = idesc_n(n_pad);
                        const uint32_t w = smem_u32(sm + ws * S.wslot), wp = (uint32_t)n_pad * KT * 2;
                        const uint32_t a = a_cols(q), d = d_cols(q);
                        const int steps = max(1, (min(KT, t.k_cnt - i * KT) + 15) / 16);
                        issue_mmas<NP>(d, a, w, wp, steps, idesc, nch > 1);
                    } else {
                        slot[1] = 1;
                    }
                    commit(barM + sl);
                }
                __syncwarp();
                put_rows();  // chunk q + 3: the rows of chunk q - 1 have been read
            }
        }
        // the copies in flight (at most one beyond the last MMA's) have all been waited for above
    } else {
        const int part = warp >> 2;
        const int s = (warp & 3) * 32 + lane;  // this thread's tensor-memory lane
        const uint32_t tlane = (uint32_t)((warp & 3) * 32) << 16;
        const uint64_t log2e = pair(kLog2e, kLog2e), minus1 = pair(-1.f, -1.f);
        pcb::pdl_wait();

        constexpr int NL = MODE == 2 ? PT / 2 : PT;  // terms loaded ahead
        float v[PT], w[MODE == 2 ? NL : 1];
        // rows [j0, j0 + NL) of chunk q of a unit with first sample b0 into v (and w)
        auto load = [&](int q, int b0, int k_cnt, auto first) {
            constexpr int j0 = decltype(first)::value;
            if (b0 + (warp & 3) * 32 >= B || k_cnt <= 0) return;
            const int64_t b = min(b0 + s, B - 1);
            const int4* rows = reinterpret_cast<const int4*>(sRows + (q % kRowRing) * KT + part * PT + j0);
#pragma unroll
            for (int j = 0; j < NL; j += 4) {
                const int4 r4 = rows[j / 4];
                const int rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    const int64_t o = (int64_t)rr[z] * ld + b;
                    v[j0 + j + z] = __ldg(src + o);
                    if (MODE == 2) w[MODE == 2 ? j + z : 0] = __ldg(src2 + o);
                }
            }
        };
        auto wait_rows = [&](int q) {
            if (!mbar_wait_bounded(barR + q % kRowRing, (uint32_t)((q / kRowRing) & 1))) fail = true;
        };
        // COPY: this warp's eight rows of chunk q to shared memory, 16 bytes per lane; barV follows
        auto copy = [&](int q, int b0, int nk) {
            constexpr int n = KT / kPWarps;
            const int* rows = sRows + (q % kRowRing) * KT + warp * n;
            float* to = sVals + warp * n * NS + 4 * lane;
            if (b0 + 4 * lane < B) {  // ld is a multiple of 4
#pragma unroll
                for (int j = 0; j < n; ++j)
                    if (warp * n + j < nk) pcb::cp_async16(to + j * NS, src + (int64_t)rows[j] * ld + b0 + 4 * lane);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(barV)) : "memory");
        };
        // log f - log m of the terms loaded last (mode 2)
        auto to_log = [&](auto first) {
            if constexpr (MODE == 2) {
                constexpr int j0 = decltype(first)::value;
                float f[NL];
#pragma unroll
                for (int j = 0; j < NL; ++j) f[j] = v[j0 + j];
                log_add<NL, -1>(f, w);
#pragma unroll
                for (int j = 0; j < NL; ++j) v[j0 + j] = f[j];
            }
        };
        // maxima that the accumulators of the unit's last two chunks, and its sums, are relative to
        float m0 = -INFINITY, m1 = -INFINITY, ms = -INFINITY;
        // the unit that ended at chunk q: n chunks, all in D (the last two) and the sums
        auto finish = [&](int q, const PcbLseTile& t, int nch, int b0) {
            if (!mbar_wait_bounded(barM + (q & 1), (uint32_t)((q >> 1) & 1))) fail = true;
            fence_after_sync();
            fail = fail || slot[1] != 0;
            const bool in = b0 + s < B, active = b0 + (warp & 3) * 32 < B;
            const int blocks = ((t.n_rows + 15) & ~15) / EB;
            const float f1 = nch > 1 ? rescale(m1, m0) : 0.f, fs = nch > (NP == 3 ? 1 : 2) ? rescale(ms, m0) : 0.f;
            const float* ax = MODE != 0 ? aux + (int64_t)t.aux_row * ld + min(b0 + s, B - 1) : nullptr;
            float* o = out + (int64_t)t.out_row * ld + b0 + s;
            float a[MODE == 0 ? 1 : EB];
            auto load_aux = [&](int blk) {
                if constexpr (MODE != 0) {
                    if (!active || blk >= blocks) return;
#pragma unroll
                    for (int j = 0; j < EB; ++j) a[j] = __ldg(ax + (int64_t)min(blk * EB + j, t.n_rows - 1) * ld);
                }
            };
            load_aux(part);
#pragma unroll 1
            for (int blk = part; blk < blocks; blk += 4) {
                float d[EB];
                tmem_ld8(d_cols(q) + tlane + blk * EB, d);
                if (NP == 3) {
                    float e[EB];
                    tmem_ld8(d_cols(q) + kColsD + tlane + blk * EB, e);
                    wait_ld();
#pragma unroll
                    for (int j = 0; j < EB; ++j) d[j] += e[j];
                    if (nch > 1) {
#pragma unroll
                        for (int j = 0; j < EB; ++j) d[j] = fmaf(sSum[(blk * EB + j) * NS + s], fs, d[j]);
                    }
                } else if (nch > 1) {
                    float e[EB];
                    tmem_ld8(d_cols(q - 1) + tlane + blk * EB, e);
                    wait_ld();
#pragma unroll
                    for (int j = 0; j < EB; ++j) d[j] = fmaf(e[j], f1, d[j]);
                    if (nch > 2) {
#pragma unroll
                        for (int j = 0; j < EB; ++j) d[j] = fmaf(sSum[(blk * EB + j) * NS + s], fs, d[j]);
                    }
                } else {
                    wait_ld();
                }
                if (MODE == 0 && NP == 3) {
#pragma unroll
                    for (int j = 0; j < EB; ++j) d[j] = m0 == -INFINITY ? -INFINITY : logf(d[j]) + m0;
                } else if (MODE == 0) {
                    float m[EB];
#pragma unroll
                    for (int j = 0; j < EB; ++j) m[j] = m0;
                    log_add<EB, 1>(d, m);
                } else {
#pragma unroll
                    for (int j = 0; j < EB; ++j)
                        d[j] = m0 == -INFINITY ? 0.f : d[j] * ex2((a[MODE == 0 ? 0 : j] + m0) * kLog2e);
                    load_aux(blk + 4);
                }
                if (fail) {
#pragma unroll
                    for (int j = 0; j < EB; ++j) d[j] = __int_as_float(0x7fc00000);
                }
                float* dst = o + (int64_t)(blk * EB) * ld;
                if (in && blk * EB + EB <= t.n_rows) {
#pragma unroll
                    for (int j = 0; j < EB; ++j) dst[(int64_t)j * ld] = d[j];
                } else if (in) {
#pragma unroll
                    for (int j = 0; j < EB; ++j)
                        if (blk * EB + j < t.n_rows) dst[(int64_t)j * ld] = d[j];
                }
            }
        };

        // this warp's 128-byte lines of a unit's element values into L2, one line per lane, well
        // ahead of finish()'s loads
        auto prefetch_aux = [&](const PcbLseTile& t, int b0) {
            const int r = (part + 4 * (lane / EB)) * EB + lane % EB;
            const int b = b0 + (warp & 3) * 32;
            if (r < t.n_rows && b < B)
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(aux + ((int64_t)t.aux_row + r) * ld + b));
        };

        using Z = std::integral_constant<int, 0>;
        using H = std::integral_constant<int, PT / 2>;
        PcbLseTile t = {}, tp = {};  // tiles of this unit and of the one before
        int q = 0, nchp = 0, b0p = 0;
        if (u0 < u1) {
            wait_rows(0);
            const int b0 = (u0 % num_slices) * NS, nk = tiles[u0 / num_slices].k_cnt;
            if constexpr (COPY) {
                copy(0, b0, nk);
            } else {
                load(0, b0, nk, Z{});
            }
        }
        taddr = columns();  // the first rows are already requested
        for (int u = u0; u < u1; ++u) {
            t = tiles[u / num_slices];
            const int nch = chunks_of(t);
            const int b0 = (u % num_slices) * NS;
            const bool active = b0 + (warp & 3) * 32 < B;
            float mrun = -INFINITY;
            for (int i = 0; i < nch; ++i, ++q) {
                if constexpr (COPY) {
                    if (!mbar_wait_bounded(barV, (uint32_t)(q & 1))) fail = true;
                    const float* p = sVals + part * PT * NS + s;
#pragma unroll
                    for (int j = 0; j < PT; ++j) v[j] = p[j * NS];
                }
                if (MODE == 2) {
                    to_log(Z{});
                    load(q, b0, t.k_cnt, H{});
                    to_log(H{});
                }
                const int nk = t.k_cnt - i * KT - part * PT;  // terms of this part
                if (!active || nk < PT) {                     // places beyond them count as -inf
#pragma unroll
                    for (int j = 0; j < PT; ++j)
                        if (!active || j >= nk) v[j] = -INFINITY;
                }
                float m = v[0];
#pragma unroll
                for (int j = 1; j < PT; ++j) m = fmaxf(m, v[j]);
                float* pm = sPart + (q & 1) * 4 * NS + s;
                pm[part * NS] = m;
                // A's slot: the MMAs of chunk q - AS have read it
                if (q >= AS && !mbar_wait_bounded(barM + ((q - AS) & 1), (uint32_t)(((q - AS) >> 1) & 1))) fail = true;
                fence_after_sync();
                const uint32_t ta = a_cols(q) + tlane + part * (PT / 2);
                const bool last = i + 1 == nch;
                if constexpr (!COPY) {
                    // The values wait for the maximum in the columns that their first two parts will
                    // take, and the next chunk's rows are on their way while they are converted.
#pragma unroll
                    for (int g = 0; g < PT; g += 16) {
                        uint32_t raw[2][8];
#pragma unroll
                        for (int j = 0; j < 16; ++j) raw[j / 8][j % 8] = __float_as_uint(v[g + j]);
                        tmem_st8(ta + g / 2, raw[0]);
                        tmem_st8(ta + kColsA + g / 2, raw[1]);
                    }
                    if (!last || u + 1 < u1) {
                        wait_rows(q + 1);
                        load(q + 1, last ? ((u + 1) % num_slices) * NS : b0, last ? tiles[(u + 1) / num_slices].k_cnt : t.k_cnt, Z{});
                    }
                    wait_st();
                }
                asm volatile("bar.sync 1, 512;\n" ::: "memory");
                if (COPY && (!last || u + 1 < u1)) {  // every warp has read chunk q's values
                    wait_rows(q + 1);
                    if (last) copy(q + 1, ((u + 1) % num_slices) * NS, tiles[(u + 1) / num_slices].k_cnt);
                    else copy(q + 1, b0, t.k_cnt - (i + 1) * KT);
                }
                m = fmaxf(fmaxf(fmaxf(pm[0], pm[NS]), fmaxf(pm[2 * NS], pm[3 * NS])), mrun);
                mrun = m;
                const float mu = m == -INFINITY ? 0.f : m;
                const uint64_t nmu = pair(-mu, -mu);
#pragma unroll
                for (int g = 0; g < PT; g += 16) {
                    float raw[2][8];
                    if constexpr (COPY) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) raw[j / 8][j % 8] = v[g + j];
                    } else {
                        tmem_ld8(ta + g / 2, raw[0]);
                        tmem_ld8(ta + kColsA + g / 2, raw[1]);
                        wait_ld();
                    }
                    uint32_t parts[NP][8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint64_t x = mul2(add2(pair(raw[j / 4][2 * j % 8], raw[j / 4][2 * j % 8 + 1]), nmu), log2e);
                        const float2 x2 = unpair(x);
                        uint64_t e = pair(ex2(x2.x), ex2(x2.y));
#pragma unroll
                        for (int p = 0; p < NP; ++p) {
                            const float2 f = unpair(e);
                            const uint32_t h = parts[p][j] = bf16x2(f.x, f.y);
                            if (p + 1 < NP)
                                e = fma2(pair(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), minus1, e);
                        }
                    }
#pragma unroll
                    for (int p = 0; p < NP; ++p) tmem_st8(ta + p * kColsA + g / 2, parts[p]);
                }
                if (MODE != 0 && last) prefetch_aux(t, b0);
                // D's slot: what chunk q - 2 left there
                if (i == 0) {
                    if (u > u0) finish(q - 1, tp, nchp, b0p);
                } else if (i >= (NP == 3 ? 1 : 2)) {
                    const float mo = NP == 3 ? m0 : m1;  // what that accumulator is relative to
                    const bool more = i > (NP == 3 ? 1 : 2);
                    const float f = more ? rescale(ms, mo) : 0.f;
                    const int blocks = ((t.n_rows + 15) & ~15) / EB;
#pragma unroll 1
                    for (int blk = part; blk < blocks; blk += 4) {
                        float d[EB], e[EB];
                        tmem_ld8(d_cols(q) + tlane + blk * EB, d);
                        if (NP == 3) tmem_ld8(d_cols(q) + kColsD + tlane + blk * EB, e);
                        wait_ld();
#pragma unroll
                        for (int j = 0; j < EB; ++j) {
                            float* p = sSum + (blk * EB + j) * NS + s;
                            const float x = NP == 3 ? d[j] + e[j] : d[j];
                            *p = more ? fmaf(*p, f, x) : x;
                        }
                    }
                    ms = mo;
                }
                m1 = m0;
                m0 = m;
                wait_st();
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(barA + (q & 1));
            }
            tp = t;
            nchp = nch;
            b0p = b0;
        }
        if (u0 < u1) finish(q - 1, tp, nchp, b0p);
        fence_before_sync();
    }
    if (fail) pcb::report_status(status, PCB_STATUS_WAIT_TIMEOUT);
    __syncthreads();
    if (warp == kPWarps) {
        fence_after_sync();
        tmem_dealloc(taddr, 512);
    }
}

template <int MODE, int NP, bool COPY>
int launch_persistent(const float* src, const float* src2, const float* aux, float* out, int64_t ld, int B,
                      const uint8_t* packed, const PcbLseTile* tiles, int num_tiles, int n_max, const int* krow,
                      const int* chunk_index, int chunk_ld, cudaStream_t s) {
    const bool sums = chunk_index && chunk_ld > (NP == 3 ? 1 : 2);
    const PSmem S(n_max, NP, sums, COPY);
    if constexpr (COPY) {
        // Rows that 16-byte copies can read, a full slice of samples (below that the copies' lanes
        // idle), and room for a chunk of values.
        if (!pcb::vec_ok(src, ld) || B < NS || !S.fits())
            return launch_persistent<MODE, NP, false>(src, src2, aux, out, ld, B, packed, tiles, num_tiles, n_max, krow,
                                                      chunk_index, chunk_ld, s);
    }
    // no CTA of the other form, which allocates early, beside this one (tc05.cuh)
    const size_t smem = std::max<size_t>(S.total, kPShared);
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    dev = dev < 0 ? 0 : (dev > 63 ? 63 : dev);
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(lse_tmem_persistent_kernel<MODE, NP, COPY>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return pcb::set_error(PCB_E_CUDA, "pcb_lse_contract_tmem: %s", cudaGetErrorString(e));
        configured[dev] = true;
    }
    const int slices = (int)pcb::cdiv(B, NS);
    const int64_t units = (int64_t)num_tiles * slices;
    if (units > INT32_MAX) return pcb::set_error(PCB_E_ARG, "pcb_lse_contract_tmem: too many tiles");
    return pcb::launch_status(
        pcb::launch_k(lse_tmem_persistent_kernel<MODE, NP, COPY>, dim3((unsigned)std::min<int64_t>(units, pcb::num_sms())),
                      dim3(kPThreads), smem, s, 1u, src, src2, aux, out, ld, B, packed, tiles, krow, chunk_index,
                      chunk_ld, n_max, sums, slices, (int)units, pcb::status_word()),
        "pcb_lse_contract_tmem");
}

template <int MODE, bool SPLIT>
int launch(const float* src, const float* src2, const float* aux, float* out, int64_t ld, int B, const uint8_t* packed,
           const PcbLseTile* tiles, int num_tiles, int n_max, const int* krow, const int* chunk_index, int chunk_ld,
           int ksplit, cudaStream_t s) {
    const bool several = chunk_index && chunk_ld > ksplit;
    // CTAs wait with their tensor memory allocated (for the grid before, for the cluster's others), so
    // never more of them than it serves, two, may be on an SM (tc05.cuh).
    const size_t smem = std::max<size_t>(Smem(n_max, several, ksplit).total, kShared);
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    dev = dev < 0 ? 0 : (dev > 63 ? 63 : dev);
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(lse_tmem_kernel<MODE, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             227 * 1024);
        if (e != cudaSuccess) return pcb::set_error(PCB_E_CUDA, "pcb_lse_contract_tmem: %s", cudaGetErrorString(e));
        configured[dev] = true;
    }
    const int slices = (int)pcb::cdiv(B, NS);
    const int64_t grid = (int64_t)num_tiles * slices * ksplit;
    if (grid > INT32_MAX) return pcb::set_error(PCB_E_ARG, "pcb_lse_contract_tmem: too many tiles");
    return pcb::launch_status(
        pcb::launch_k(lse_tmem_kernel<MODE, SPLIT>, dim3((unsigned)grid), dim3(kThreads), smem, s, (unsigned)ksplit,
                      src, src2, aux, out, ld, B, packed, tiles, krow, chunk_index, chunk_ld, n_max, several, slices,
                      pcb::status_word()),
        "pcb_lse_contract_tmem");
}

}  // namespace

extern "C" int pcb_lse_contract_tmem(const float* src, const float* src2, const float* aux, float* out, int64_t ld,
                                     int32_t B, const uint8_t* packed, const PcbLseTile* tiles, int32_t num_tiles,
                                     int32_t tile_rows, const int32_t* krow, const int32_t* chunk_index,
                                     int32_t chunk_ld, int32_t mode, int32_t prec, int32_t ksplit, void* stream) {
    if (!src || !out || !packed || !tiles || !krow || B <= 0 || ld < B || num_tiles < 0 || tile_rows < 1 ||
        tile_rows > 128 || mode < 0 || mode > 2 || (mode == 2 && !src2) || (mode >= 1 && !aux) || prec < 0 || prec > 2 ||
        (prec == 0 && (ksplit != 0 || mode == 2)) ||
        ksplit < 0 || ksplit > kMaxCluster || (chunk_index && chunk_ld < 1) ||
        (reinterpret_cast<uintptr_t>(packed) & 15) != 0)
        return pcb::set_error(PCB_E_ARG, "pcb_lse_contract_tmem: bad arguments");
    if (num_tiles == 0) return PCB_OK;
    const int n_max = (tile_rows + 15) & ~15;
    cudaStream_t s = pcb::as_stream(stream);
    if (ksplit == 0) {
#define PCB_TP(M, P) \
    launch_persistent<M, P, M == 0>(src, src2, aux, out, ld, B, packed, tiles, num_tiles, n_max, krow, chunk_index, chunk_ld, s)
        if (prec == 0) return mode == 0 ? PCB_TP(0, 3) : PCB_TP(1, 3);
        if (prec == 1) return mode == 0 ? PCB_TP(0, 1) : (mode == 1 ? PCB_TP(1, 1) : PCB_TP(2, 1));
        return mode == 0 ? PCB_TP(0, 2) : (mode == 1 ? PCB_TP(1, 2) : PCB_TP(2, 2));
#undef PCB_TP
    }
#define PCB_TM(M) \
    (prec == 2 ? launch<M, true>(src, src2, aux, out, ld, B, packed, tiles, num_tiles, n_max, krow, chunk_index, \
                                 chunk_ld, ksplit, s) \
               : launch<M, false>(src, src2, aux, out, ld, B, packed, tiles, num_tiles, n_max, krow, chunk_index, \
                                  chunk_ld, ksplit, s))
    return mode == 0 ? PCB_TM(0) : (mode == 1 ? PCB_TM(1) : PCB_TM(2));
#undef PCB_TM
}
