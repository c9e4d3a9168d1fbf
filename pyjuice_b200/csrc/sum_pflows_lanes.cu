// Sum-layer parameter flows of large layers on the tcgen05 tensor cores: the contraction of
// sum_pflows_tc05.cu,
//   pf(r, k) += params(r, k) * sum_b A[r, b] * C[k, b],
//   A[r, b] = exp(lf[nid + r, b] - M_b),  C[k, b] = exp(em[cids[k], b] + M_b),
// with one sample per lane instead of rows staged in shared memory.
//
// Both operands are contracted over samples, and a thread that owns a sample holds, row by
// row, what one K index of an MN-major operand needs: 8 consecutive rows are one 16-byte entry
// of a core matrix, so a warp writes 512 contiguous bytes and nothing is transposed. The
// rows are read as whole 128-byte lines at any alignment, the maximum over the nodes stays in
// registers but for one exchange between the four warps of a sample group, and only bf16
// operands pass through shared memory. A CTA of 8 warps takes a tile of 128 nodes x 64 or 128
// children over the whole batch, in chunks of 64 samples; two CTAs share an SM, one computing
// while the other's rows arrive. D's lanes are nodes, so the epilogue updates the flow slots
// (nodes fastest) as whole lines. The small products (lo * hi, hi * lo) have an accumulator of
// their own: additions to a large one are truncated, about 3e-8 each, and so only a third of
// them counts (error against FP64 at batch 512: 3.2e-6, 4.1e-6 with one accumulator).
//
// Bound by the rows' way from L2 and the exponentials: 200 regions of 256 x 256, batch 512:
// 117 us against 245 us (rewritten flows); 119 of 128 x 128: 29.6 us against 46.5 us. Layers of
// fewer than about one tile per SM keep the kernels that split the batch over a cluster.
#include "tc05.cuh"

namespace {

using namespace pcb::tc05;

constexpr int kThreads = 256;
constexpr int TMN = 128;   // nodes per tile (the MMA's M)
constexpr int KB = 64;     // samples per chunk
constexpr int PR = 32;     // nodes per thread and chunk
constexpr float kLog2e = 1.4426950408889634f;
constexpr uint32_t kLBO = 128;             // core matrices adjacent along K (samples)
constexpr uint32_t kSBO = (KB / 8) * 128;  // groups of 8 rows
constexpr uint32_t kA = TMN * KB * 2;      // one bf16 copy of A

template <int TKC>
struct Plan {
    static constexpr uint32_t kC = TKC * KB * 2;
    static constexpr uint32_t oA = 0, oC = 2 * kA;               // hi, lo each
    static constexpr uint32_t oPart = oC + 2 * kC;               // [2][4][KB] chunk maxima
    static constexpr uint32_t oIdx = oPart + 2 * 4 * KB * 4;     // cids, pids, pfids
    static constexpr uint32_t oBar = oIdx + 3 * TKC * 4;
    static constexpr uint32_t oSlot = oBar + 8;
    static constexpr size_t bytes() { return oSlot + 16; }
};

// D f32, A and B bf16, both MN-major, M = 128, N
template <int N>
__device__ __forceinline__ constexpr uint32_t idesc_mn() {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(128 >> 4) << 24);
}

// exp(v + m) of N rows (multiples of 8, from row r0 of the operand) of sample k, as bf16 hi
// [and lo] entries of an MN-major operand
template <int N, bool SPLIT>
__device__ __forceinline__ void put_rows(uint8_t* hi, uint32_t lo_off, int r0, int k, const float (&v)[N], float m) {
    uint8_t* dst = hi + (uint32_t)(r0 >> 3) * kSBO + (uint32_t)(k >> 3) * kLBO + (uint32_t)(k & 7) * 16;
#pragma unroll
    for (int g = 0; g < N; g += 8) {
        uint32_t h[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float e0 = ex2((v[g + 2 * j] + m) * kLog2e), e1 = ex2((v[g + 2 * j + 1] + m) * kLog2e);
            const __nv_bfloat162 b = __floats2bfloat162_rn(e0, e1);
            h[j] = *reinterpret_cast<const uint32_t*>(&b);
            if (SPLIT) {
                const __nv_bfloat162 c = __floats2bfloat162_rn(e0 - __uint_as_float(h[j] << 16),
                                                               e1 - __uint_as_float(h[j] & 0xffff0000u));
                l[j] = *reinterpret_cast<const uint32_t*>(&c);
            }
        }
        *reinterpret_cast<uint4*>(dst + (g / 8) * kSBO) = make_uint4(h[0], h[1], h[2], h[3]);
        if (SPLIT) *reinterpret_cast<uint4*>(dst + lo_off + (g / 8) * kSBO) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

template <int TKC, bool MODIFIED, bool ATOMIC, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 2)
sum_pflows_lanes_kernel(const float* __restrict__ nf, const float* __restrict__ nm, const float* __restrict__ em,
                        int64_t ld, int B, const float* __restrict__ params, float* __restrict__ pf,
                        const PcbPflowTile* __restrict__ tiles, int rpb_log2, const int* __restrict__ cids,
                        const int* __restrict__ pids, const int* __restrict__ pfids, int32_t* __restrict__ status) {
    using P = Plan<TKC>;
    constexpr int CP = TKC / 4;  // children per warp part
    extern __shared__ __align__(1024) uint8_t sm[];
    float* sPart = reinterpret_cast<float*>(sm + P::oPart);
    int* sCid = reinterpret_cast<int*>(sm + P::oIdx);
    int* sPid = sCid + TKC;
    int* sPfid = sPid + TKC;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + P::oBar);
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + P::oSlot);
    constexpr uint32_t kCols = SPLIT ? 2 * TKC : TKC;  // D, then the small products' D
    const PcbPflowTile t = tiles[blockIdx.x];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    for (int i = tid; i < TKC; i += kThreads) {  // places beyond the children read the first one's row
        const int k = t.k_off + (i < t.k_cnt ? i : 0);
        sCid[i] = __ldg(cids + k);
        sPid[i] = __ldg(pids + k);
        sPfid[i] = __ldg(pfids + k);
    }
    if (warp == 0) {
        pcb::pdl_wait();
        tmem_alloc(slot, kCols);
        pcb::pdl_trigger();  // not before: tc05.cuh
        fence_before_sync();
    }
    if (tid == 32) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    fence_after_sync();
    const uint32_t taddr = slot[0];
    pcb::pdl_wait();

    const int part = warp >> 1;                     // 32 nodes, TKC / 4 children
    const int kk = (warp & 1) * 32 + lane;          // this thread's sample of a chunk
    const int r0 = part * PR, c0 = part * CP;
    const int nrow = min(PR, t.n_rows - r0);        // may be <= 0
    const int ncol = t.k_cnt - c0;
    const int nch = (B + KB - 1) / KB;
    bool fail = false;

    auto load_children = [&](int64_t b, bool in, float (&w)[CP]) {
        const int4* rows = reinterpret_cast<const int4*>(sCid + c0);
#pragma unroll
        for (int j = 0; j < CP; j += 4) {
            const int4 q = rows[j / 4];
            w[j] = __ldg(em + (int64_t)q.x * ld + b);
            w[j + 1] = __ldg(em + (int64_t)q.y * ld + b);
            w[j + 2] = __ldg(em + (int64_t)q.z * ld + b);
            w[j + 3] = __ldg(em + (int64_t)q.w * ld + b);
        }
        if (!in || CP > ncol) {
#pragma unroll
            for (int j = 0; j < CP; ++j)
                if (!in || j >= ncol) w[j] = -INFINITY;
        }
    };

    for (int c = 0; c < nch; ++c) {
        const bool in = c * KB + kk < B;
        const int64_t b = in ? c * KB + kk : B - 1;
        // log f - log m of this part's nodes
        float v[PR];
        const float* pa = nf + ((int64_t)t.nid + r0) * ld + b;
        if (MODIFIED) {
            if (in && nrow == PR) {
#pragma unroll
                for (int j = 0; j < PR; ++j) v[j] = __ldg(pa + (int64_t)j * ld);
            } else {
#pragma unroll
                for (int j = 0; j < PR; ++j) v[j] = in && j < nrow ? __ldg(pa + (int64_t)j * ld) : -INFINITY;
            }
        } else {
            const float* pm = nm + ((int64_t)t.nid + r0) * ld + b;
#pragma unroll
            for (int g = 0; g < PR; g += 16) {
                float f[16], m2[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const bool ok = in && g + j < nrow;
                    f[j] = ok ? __ldg(pa + (int64_t)(g + j) * ld) : 0.f;
                    m2[j] = ok ? __ldg(pm + (int64_t)(g + j) * ld) : -INFINITY;
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) v[g + j] = m2[j] == -INFINITY ? -INFINITY : logf(f[j]) - m2[j];
            }
        }
        float w[CP];
        load_children(b, in, w);
        float m = v[0];
#pragma unroll
        for (int j = 1; j < PR; ++j) m = fmaxf(m, v[j]);
        float* pm = sPart + (c & 1) * 4 * KB + kk;
        pm[part * KB] = m;
        // the operands are free once the last chunk's MMAs are done
        if (c > 0 && !mbar_wait_bounded(bar, (uint32_t)((c - 1) & 1))) fail = true;
        __syncthreads();
        m = fmaxf(fmaxf(pm[0], pm[KB]), fmaxf(pm[2 * KB], pm[3 * KB]));
        put_rows<PR, SPLIT>(sm + P::oA, kA, r0, kk, v, m == -INFINITY ? -INFINITY : -m);
        put_rows<CP, SPLIT>(sm + P::oC, P::kC, c0, kk, w, m);
        fence_smem_async();
        __syncthreads();
        fence_after_sync();
        if (tid == 0) {
            constexpr uint32_t idesc = idesc_mn<TKC>();
            const uint32_t ah = smem_u32(sm + P::oA), ch = smem_u32(sm + P::oC);
#pragma unroll
            for (int s = 0; s < KB / 16; ++s) {
                const uint32_t o = (uint32_t)s * 2 * kLBO;
                const uint32_t acc = (c > 0 || s > 0) ? 1u : 0u;
                mma_bf16(taddr, desc(ah + o, kLBO, kSBO), desc(ch + o, kLBO, kSBO), idesc, acc);
                if (SPLIT) {
                    mma_bf16(taddr + TKC, desc(ah + kA + o, kLBO, kSBO), desc(ch + o, kLBO, kSBO), idesc, acc);
                    mma_bf16(taddr + TKC, desc(ah + o, kLBO, kSBO), desc(ch + P::kC + o, kLBO, kSBO), idesc, 1u);
                }
            }
            commit(bar);
        }
    }

    // ---- flow slots: lane quarter q (nodes 32 q ..), every other block of 16 children per warp ----
    {
        const int r = (warp & 3) * 32 + lane;
        const bool ok = r < t.n_rows;
        const int64_t node = (int64_t)t.p_add + (r & ((1 << rpb_log2) - 1));
        const float* pp = params + node + (int64_t)(r >> rpb_log2) * t.gs_p;
        float* pq = pf + node + (int64_t)(r >> rpb_log2) * t.gs_pf;
        bool waited = false;
#pragma unroll 1
        for (int k0 = (warp >> 2) * 16; k0 < t.k_cnt; k0 += 32) {
            float wv[16], old[16], d[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const bool use = ok && k0 + j < t.k_cnt;
                wv[j] = use ? __ldg(pp + sPid[k0 + j]) : 0.f;
                old[j] = use && !ATOMIC ? pq[sPfid[k0 + j]] : 0.f;
            }
            if (!waited) {
                if (nch > 0 && !mbar_wait_bounded(bar, (uint32_t)((nch - 1) & 1))) fail = true;
                fence_after_sync();
                waited = true;
            }
            const uint32_t td = taddr + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)k0;
            tmem_ld16(td, d);
            if (SPLIT) {
                float e[16];
                tmem_ld16(td + TKC, e);
                wait_ld();
#pragma unroll
                for (int j = 0; j < 16; ++j) d[j] += e[j];
            } else {
                wait_ld();
            }
            if (fail) {
#pragma unroll
                for (int j = 0; j < 16; ++j) d[j] = __int_as_float(0x7fc00000);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (!(ok && k0 + j < t.k_cnt)) continue;
                float* p = pq + sPfid[k0 + j];
                if (ATOMIC) atomicAdd(p, d[j] * wv[j]);
                else *p = old[j] + d[j] * wv[j];
            }
        }
        if (!waited) {  // a warp without a block still waits for the MMAs that read the operands
            if (nch > 0 && !mbar_wait_bounded(bar, (uint32_t)((nch - 1) & 1))) fail = true;
        }
    }
    if (fail) pcb::report_status(status, PCB_STATUS_WAIT_TIMEOUT);
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        fence_after_sync();
        tmem_dealloc(taddr, kCols);
    }
}

template <int TKC, bool MODIFIED, bool ATOMIC, bool SPLIT>
int launch(const float* nf, const float* nm, const float* em, int64_t ld, int B, const float* params, float* pf,
           const PcbPflowTile* tiles, int num_tiles, int rpb_log2, const int* cids, const int* pids, const int* pfids,
           cudaStream_t s) {
    constexpr size_t smem = Plan<TKC>::bytes();
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    dev = dev < 0 ? 0 : (dev > 63 ? 63 : dev);
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(sum_pflows_lanes_kernel<TKC, MODIFIED, ATOMIC, SPLIT>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return pcb::set_error(PCB_E_CUDA, "pcb_sum_pflows_lanes: %s", cudaGetErrorString(e));
        configured[dev] = true;
    }
    return pcb::launch_status(
        pcb::launch_k(sum_pflows_lanes_kernel<TKC, MODIFIED, ATOMIC, SPLIT>, dim3((unsigned)num_tiles), dim3(kThreads),
                      smem, s, 1u, nf, nm, em, ld, B, params, pf, tiles, rpb_log2, cids, pids, pfids,
                      pcb::status_word()),
        "pcb_sum_pflows_lanes");
}

}  // namespace

extern "C" int pcb_sum_pflows_lanes(const float* node_flows, const float* node_mars, const float* element_mars,
                                    int64_t ld, int32_t B, const float* params, float* param_flows,
                                    const PcbPflowTile* tiles, int32_t num_tiles, int32_t rows_per_block,
                                    const int32_t* cids, const int32_t* pids, const int32_t* pfids, int32_t modified,
                                    int32_t atomic, int32_t tile_children, int32_t prec, void* stream) {
    if (!node_flows || !node_mars || !element_mars || !params || !param_flows || !tiles || !cids || !pids || !pfids ||
        B <= 0 || ld < B || num_tiles < 0 || rows_per_block <= 0 || (rows_per_block & (rows_per_block - 1)) ||
        (tile_children != 64 && tile_children != 128) || prec < 1 || prec > 2)
        return pcb::set_error(PCB_E_ARG, "pcb_sum_pflows_lanes: bad arguments");
    if (num_tiles == 0) return PCB_OK;
    int rpb_log2 = 0;
    while ((1 << rpb_log2) < rows_per_block) ++rpb_log2;
    auto go = [&](auto kernel) {
        return kernel(node_flows, node_mars, element_mars, ld, B, params, param_flows, tiles, num_tiles, rpb_log2, cids,
                      pids, pfids, pcb::as_stream(stream));
    };
#define PCB_PF(T, S) \
    (modified ? (atomic ? go(launch<T, true, true, S>) : go(launch<T, true, false, S>)) \
              : (atomic ? go(launch<T, false, true, S>) : go(launch<T, false, false, S>)))
    if (tile_children == 64) return prec == 2 ? PCB_PF(64, true) : PCB_PF(64, false);
    return prec == 2 ? PCB_PF(128, true) : PCB_PF(128, false);
#undef PCB_PF
}
