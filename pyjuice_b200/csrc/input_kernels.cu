// Categorical input layer: forward lookup and deterministic parameter-flow histogram.
#include <algorithm>

#include "common.cuh"

namespace {

// node_mars[node_offset + n, b] = log(params[s_pids[n] + x]) with x = data[vids[n], b], or
// 0 (log 1: the variable is summed out) where the missing mask is set,
// miss[b * m_sb + vids[n] * m_sv] != 0. A category outside [0, ncats) yields NaN (no
// out-of-range read).
constexpr int kFwdSlab = 256;
constexpr int kFwdThreads = 128;
constexpr int kFwdSamples = 4 * kFwdThreads;
constexpr int kRowNodes = 8;  // nodes per CTA, any vocabulary

// Any vocabulary: a CTA covers kRowNodes consecutive nodes over 512 samples (4 per thread), the logs
// of their parameter slabs (up to kFwdSlab categories) in shared memory; larger vocabularies gather
// their parameters, for which many CTAs of few nodes are best (8 variables x 1024 nodes x 33,279
// categories, 256 samples: 47 us, against 132 us with the 16 nodes per CTA of the form below).
__global__ void __launch_bounds__(kFwdThreads)
input_cat_fwd_kernel(const int64_t* __restrict__ data, int64_t data_ld, const float* __restrict__ params,
                     const int* __restrict__ vids, const int* __restrict__ s_pids, const int* __restrict__ ncats,
                     int num_nodes, int node_offset, float* __restrict__ nm, int64_t ld, int B, bool vec,
                     const uint8_t* __restrict__ miss, int64_t m_sb, int64_t m_sv, int32_t* __restrict__ status) {
    // The node tables and the parameter logs are read before the wait for the previous kernel
    // (the parameters' writers do not trigger early); the samples and outputs after it.
    pcb::pdl_trigger();
    __shared__ float slab[kRowNodes][kFwdSlab];
    __shared__ int sV[kRowNodes], sK[kRowNodes], sP[kRowNodes];
    const int n0 = blockIdx.x * kRowNodes;
    const int tid = threadIdx.x;
    if (tid < kRowNodes) {
        const int n = n0 + tid;
        sV[tid] = n < num_nodes ? __ldg(vids + n) : -1;
        sK[tid] = n < num_nodes ? __ldg(ncats + n) : 0;
        sP[tid] = n < num_nodes ? __ldg(s_pids + n) : 0;
    }
    __syncthreads();
    for (int i = tid; i < kRowNodes * kFwdSlab; i += blockDim.x) {
        const int j = i / kFwdSlab, k = i % kFwdSlab;
        if (k < sK[j] && sK[j] <= kFwdSlab) slab[j][k] = __logf(__ldcg(params + sP[j] + k));
    }
    __syncthreads();
    pcb::pdl_wait();
    const int b = blockIdx.y * kFwdSamples + tid * 4;
    if (b >= B) return;
    const int v0 = sV[0];
    int64_t x0[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) x0[q] = (b + q < B) ? __ldg(data + (int64_t)v0 * data_ld + b + q) : 0;
    for (int j = 0; j < kRowNodes && n0 + j < num_nodes; ++j) {
        const int v = sV[j], K = sK[j];
        float4 o;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float r = 0.f;
            if (b + q < B && miss && miss[(int64_t)(b + q) * m_sb + (int64_t)v * m_sv]) {
                r = 0.f;
            } else if (b + q < B) {
                const int64_t x = (v == v0) ? x0[q] : __ldg(data + (int64_t)v * data_ld + b + q);
                if (x >= 0 && x < K) r = (K <= kFwdSlab) ? slab[j][x] : __logf(__ldcg(params + sP[j] + x));
                else {
                    r = NAN;
                    pcb::report_status(status, PCB_STATUS_BAD_CATEGORY);
                }
            }
            pcb::set(o, q, r);
        }
        pcb::store4(nm, (int64_t)node_offset + n0 + j, ld, b, B, vec, o);
    }
}

// Vocabularies of up to kFwdSlab categories. Bound by HBM (the node rows written). A CTA covers kFwdNodes consecutive nodes over up to
// 512 samples, 4 per thread. The logs of the nodes' parameter slabs (up to kFwdSlab
// categories) are taken once into shared memory, four nodes side by side, with a NaN and a 0
// entry behind the categories: a sample's entry number (category, NaN or 0) is found once per
// variable, and one 16-byte shared load then gives four nodes' values of that sample, which a
// thread regroups into 16-byte stores of four rows. 784 variables x 256 nodes x 512 samples,
// 64 categories: 97 us (4.2 TB/s of rows), against 147 us with one scalar shared load
// per value and 8 nodes per CTA.
constexpr int kFwdNodes = 16;
constexpr int kFwdQuads = kFwdNodes / 4;

__global__ void __launch_bounds__(kFwdThreads)
input_cat_fwd_quads_kernel(const int64_t* __restrict__ data, int64_t data_ld, const float* __restrict__ params,
                     const int* __restrict__ vids, const int* __restrict__ s_pids, const int* __restrict__ ncats,
                     int num_nodes, int node_offset, float* __restrict__ nm, int64_t ld, int B, bool vec,
                     const uint8_t* __restrict__ miss, int64_t m_sb, int64_t m_sv, int32_t* __restrict__ status) {
    // The node tables and the parameter logs are read before the wait for the previous kernel
    // (the parameters' writers do not trigger early); the samples and outputs after it.
    pcb::pdl_trigger();
    __shared__ float4 slab[kFwdQuads][kFwdSlab + 2];
    __shared__ int sV[kFwdNodes], sK[kFwdNodes], sP[kFwdNodes];
    const int n0 = blockIdx.x * kFwdNodes;
    const int nn = min(kFwdNodes, num_nodes - n0);
    const int tid = threadIdx.x;
    if (tid < kFwdNodes) {
        const int n = n0 + tid;
        sV[tid] = n < num_nodes ? __ldg(vids + n) : -1;
        sK[tid] = n < num_nodes ? __ldg(ncats + n) : 0;
        sP[tid] = n < num_nodes ? __ldg(s_pids + n) : 0;
    }
    __syncthreads();
    // a quad: four nodes of one variable and category count that fits the slab
    auto quad_ok = [&](int qd) {
        const int j = 4 * qd;
        return j + 3 < nn && sK[j] <= kFwdSlab && sV[j] == sV[j + 1] && sV[j] == sV[j + 2] && sV[j] == sV[j + 3] &&
               sK[j] == sK[j + 1] && sK[j] == sK[j + 2] && sK[j] == sK[j + 3];
    };
#pragma unroll
    for (int qd = 0; qd < kFwdQuads; ++qd) {
        if (!quad_ok(qd)) continue;
        const int j = 4 * qd, K = sK[j];
        const float *p0 = params + sP[j], *p1 = params + sP[j + 1], *p2 = params + sP[j + 2], *p3 = params + sP[j + 3];
        for (int k = tid; k < K + 2; k += blockDim.x) {
            const float fill = k == K ? NAN : 0.f;
            slab[qd][k] = k >= K ? make_float4(fill, fill, fill, fill)
                                 : make_float4(__logf(__ldcg(p0 + k)), __logf(__ldcg(p1 + k)), __logf(__ldcg(p2 + k)),
                                               __logf(__ldcg(p3 + k)));
        }
    }
    __syncthreads();
    pcb::pdl_wait();
    // 4 consecutive samples per thread where rows take 16-byte stores, else 4 samples 32 apart
    // (a warp still writes whole lines)
    const int b = blockIdx.y * 4 * blockDim.x + (vec ? tid * 4 : (tid >> 5) * 128 + (tid & 31));
    const int bq = vec ? 1 : 32;
    if (b >= B) return;
    auto store = [&](int64_t row, float4 o) {
        float* p = nm + row * ld + b;
        if (vec && b + 3 < B) {
            *reinterpret_cast<float4*>(p) = o;
            return;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (b + q * bq < B) p[q * bq] = pcb::get(o, q);
    };
    int v0 = -1, K0 = -1;
    int x[4];  // entry of the thread's samples among variable v0's categories, K0 = NaN, K0 + 1 = 0
    auto load_entries = [&](int v, int K) {
        v0 = v;
        K0 = K;
        const int64_t* d = data + (int64_t)v * data_ld + b;
        int64_t c[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q] = (b + q * bq < B) ? __ldg(d + q * bq) : 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool in = b + q * bq < B;
            if (in && miss && miss[(int64_t)(b + q * bq) * m_sb + (int64_t)v * m_sv]) x[q] = K + 1;
            else if (c[q] >= 0 && c[q] < K) x[q] = (int)c[q];
            else {
                x[q] = K;
                if (in) pcb::report_status(status, PCB_STATUS_BAD_CATEGORY);
            }
        }
    };
#pragma unroll 1
    for (int qd = 0; qd < kFwdQuads; ++qd) {
        const int j = 4 * qd;
        if (j >= nn) break;
        if (quad_ok(qd)) {
            if (sV[j] != v0 || sK[j] != K0) load_entries(sV[j], sK[j]);
            const float4 a0 = slab[qd][x[0]], a1 = slab[qd][x[1]], a2 = slab[qd][x[2]], a3 = slab[qd][x[3]];
            const int64_t row = (int64_t)node_offset + n0 + j;
            store(row, make_float4(a0.x, a1.x, a2.x, a3.x));
            store(row + 1, make_float4(a0.y, a1.y, a2.y, a3.y));
            store(row + 2, make_float4(a0.z, a1.z, a2.z, a3.z));
            store(row + 3, make_float4(a0.w, a1.w, a2.w, a3.w));
            continue;
        }
        for (int jj = j; jj < min(j + 4, nn); ++jj) {
            const int K = sK[jj];
            if (sV[jj] != v0 || K != K0) load_entries(sV[jj], K);
            float4 o;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                pcb::set(o, q, x[q] < K ? __logf(__ldcg(params + sP[jj] + x[q])) : (x[q] == K ? NAN : 0.f));
            store((int64_t)node_offset + n0 + jj, o);
        }
    }
}

// Flow histogram of variables with few nodes.
// One CTA per variable group: stable counting sort of the batch by category (chunks of
// up to CB samples; warp-parallel prefix sum of the category counts), then one warp per
// node copies the node's flow row into shared memory with coalesced loads and sums it per
// category in sample order, adding the sums to the node's flow slots. Deterministic: no
// float atomics (unless flow slots are shared by tied nodes of different variables:
// atomic = 1 adds with atomics). Samples whose variable is missing (miss[b * m_sb + v * m_sv] != 0) form
// their own segment: their flow sum M is spread over the categories as M * params[k]
// (input_layer.py:537-571, categorical.py:102-134).
__global__ void __launch_bounds__(256)
input_cat_bwd_kernel(const int64_t* __restrict__ data, int64_t data_ld, const float* __restrict__ nf, int64_t ld,
                     int B, const int* __restrict__ grp_var, const int* __restrict__ grp_node0,
                     const int* __restrict__ grp_count, const int* __restrict__ grp_ncats,
                     const int* __restrict__ s_pfids, int node_offset, float* __restrict__ pf, bool logspace, int CB,
                     const uint8_t* __restrict__ miss, int64_t m_sb, int64_t m_sv, const int* __restrict__ s_pids,
                     const float* __restrict__ params, bool atomic) {
    pcb::pdl_begin();
    extern __shared__ int smem[];
    const int g = blockIdx.x;
    const int K = grp_ncats[g];
    const int64_t v = grp_var[g];
    const int node0 = grp_node0[g];
    const int cnt = grp_count[g];
    int* keys = smem;              // [CB]
    int* perm = keys + CB;         // [CB]
    float* rows = reinterpret_cast<float*>(perm + CB);  // [warps][CB]
    int* seg = perm + CB + (blockDim.x >> 5) * CB;      // [K + 3]: categories, dropped, missing
    int* ucat = seg + K + 3;                            // [CB]: the categories present in the chunk
    __shared__ int sU;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;

    for (int c0 = 0; c0 < B; c0 += CB) {
        const int nb = min(CB, B - c0);
        for (int i = tid; i < K + 3; i += blockDim.x) seg[i] = 0;
        __syncthreads();
        for (int i = tid; i < nb; i += blockDim.x) {
            int key;
            if (miss && miss[(int64_t)(c0 + i) * m_sb + v * m_sv]) {
                key = K + 1;  // missing: spread over the categories below
            } else {
                const int64_t x = data[v * data_ld + c0 + i];
                key = (x >= 0 && x < K) ? (int)x : K;  // out-of-range samples are dropped
            }
            keys[i] = key;
            atomicAdd(&seg[key + 1], 1);
        }
        __syncthreads();
        if (warp == 0) {
            int carry = 0;
            for (int base = 0; base < K + 3; base += 32) {
                const int i = base + lane;
                int v = (i < K + 3) ? seg[i] : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += t;
                }
                v += carry;
                if (i < K + 3) seg[i] = v;
                carry = __shfl_sync(0xffffffffu, v, 31);
            }
        }
        __syncthreads();
        // Stable scatter by warp 0: 32 samples at a time, ranks from lane matching.
        if (warp == 0) {
            for (int i0 = 0; i0 < nb; i0 += 32) {
                const int i = i0 + lane;
                const bool act = i < nb;
                const int key = act ? keys[i] : -1;
                const unsigned same = __match_any_sync(0xffffffffu, key);
                const int rank = __popc(same & ((1u << lane) - 1u));
                int pos = 0;
                if (act) pos = seg[key] + rank;
                __syncwarp();
                if (act) perm[pos] = i;
                // The highest lane of each key group advances the cursor.
                const bool leader = act && ((same >> lane) == 1u);
                __syncwarp();
                if (leader) seg[key] += __popc(same);
                __syncwarp();
            }
        }
        __syncthreads();
        // seg[k] now holds the end of category k; its start is the end of category k-1. The
        // categories that occur in this chunk, in order (at most one per sample): without
        // missing values only their slots change, so the nodes' loops run over them instead
        // of all K categories (a vocabulary of thousands against a batch of tens).
        if (warp == 0) {
            int nu = 0;
            for (int base = 0; base < K; base += 32) {
                const int k = base + lane;
                const bool present = k < K && seg[k] > (k == 0 ? 0 : seg[k - 1]);
                const unsigned bal = __ballot_sync(0xffffffffu, present);
                if (present) ucat[nu + __popc(bal & ((1u << lane) - 1u))] = k;
                nu += __popc(bal);
            }
            if (lane == 0) sU = nu;
        }
        __syncthreads();
        const bool dense = seg[K + 1] > seg[K];  // missing samples: every category gets flow
        const int L = dense ? K : sU;
        float* wrow = rows + warp * CB;
        const bool vec4 = ((ld & 3) == 0) && ((c0 & 3) == 0) && ((reinterpret_cast<uintptr_t>(nf) & 15) == 0);
        for (int n = warp; n < cnt; n += (blockDim.x >> 5)) {
            const int64_t row = (int64_t)node_offset + node0 + n;
            const float* frow = nf + row * ld + c0;
            const int64_t sf = s_pfids[node0 + n];
            if (vec4 && (nb & 3) == 0) {
                for (int i = lane; i < nb / 4; i += 32)
                    reinterpret_cast<float4*>(wrow)[i] = __ldg(reinterpret_cast<const float4*>(frow) + i);
            } else {
                for (int i = lane; i < nb; i += 32) wrow[i] = __ldg(frow + i);
            }
            __syncwarp();
            // flow of the samples with this variable missing (segment K + 1)
            float msum = 0.f;
            if (miss) {
                for (int p = seg[K] + lane; p < seg[K + 1]; p += 32) {
                    const float f = wrow[perm[p]];
                    msum += logspace ? __expf(f) : f;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) msum += __shfl_xor_sync(0xffffffffu, msum, o);
            }
            const int64_t sp = miss ? s_pids[node0 + n] : 0;
            // list entries lane, lane + 32, ... (all categories, or the present ones): the
            // slots' old values are loaded for a batch of kR entries at once (one round trip),
            // then summed and stored
            constexpr int kR = 8;
            for (int k0 = 0; k0 < L; k0 += 32 * kR) {
                float old[kR];
#pragma unroll
                for (int j = 0; j < kR; ++j) {
                    const int idx = k0 + lane + 32 * j;
                    old[j] = (idx < L && !atomic) ? pf[sf + (dense ? idx : ucat[idx])] : 0.f;
                }
#pragma unroll
                for (int j = 0; j < kR; ++j) {
                    const int idx = k0 + lane + 32 * j;
                    if (idx >= L) continue;
                    const int k = dense ? idx : ucat[idx];
                    const int s = (k == 0) ? 0 : seg[k - 1];
                    const int e = seg[k];
                    if (e == s && msum == 0.f) continue;
                    float acc = (msum != 0.f) ? msum * params[sp + k] : 0.f;
                    for (int p = s; p < e; ++p) {
                        const float f = wrow[perm[p]];
                        acc += logspace ? __expf(f) : f;
                    }
                    if (atomic) atomicAdd(pf + sf + k, acc);  // slot shared by tied nodes
                    else pf[sf + k] = old[j] + acc;
                }
            }
            __syncwarp();  // the next node overwrites this warp's row
        }
        __syncthreads();
    }
}

// The same for variables with many nodes. pf[s_pfids[n] + k] += sum over the samples of category k of nf[n, b], in
// sample order (deterministic: no float atomics, unless atomic = 1: slots shared by tied
// nodes). Samples whose variable is missing (miss[b * m_sb + v * m_sv] != 0) spread their sum
// M over the categories as M * params[k] (input_layer.py:537-571, categorical.py:102-134).
//
// Bound by HBM (the node flows read once). A CTA of 16 warps takes every gridDim.y-th tile of
// 32 nodes of one variable. It sorts the batch chunk by (category, sample) once, and copies
// tile after tile into shared memory (while the SM's other CTA sums its own) with rows of odd
// pitch, so that lane n reads node n: every lane then walks the same sorted samples, one conflict-free shared load and one addition each, with the category boundaries
// uniform over the warp. The warps share the sorted samples out between them at category
// boundaries, put the sums into a [32][categories] table, and add that to the slots row by row
// with coalesced accesses (the old values were loaded before the summing). 784 variables x 256
// nodes x 512 samples, 64 categories: 166 us, against 307 us with one node per warp and lanes
// over the categories, whose gathers from shared memory collide.
constexpr int kBwNodes = 32;
constexpr int kBwWarps = 16;
constexpr int kBwChunk = 512;      // samples ranked and staged at a time
constexpr int kBwOld = 4;          // slots per lane and node whose old values are loaded ahead
constexpr unsigned kBwLast = 1u;    // last sample of its category

struct BwdSmem {
    int pitch, epitch;
    uint32_t res, code, perm, ucat, start, total;  // byte offsets; the tile comes first
    __host__ __device__ BwdSmem(int CB, int max_ncats) {
        pitch = CB | 1;
        const int e = CB < max_ncats + 2 ? CB : max_ncats + 2;  // categories, dropped, missing
        epitch = e | 1;
        res = 4u * kBwNodes * pitch;
        code = (res + 4u * kBwNodes * epitch + 15u) & ~15u;
        perm = code + 4u * 2 * kBwChunk;
        ucat = perm + 4u * kBwChunk;
        start = ucat + 4u * (e + 1);
        total = start + 4u * (e + 1);
    }
};

template <bool LOG>
__global__ void __launch_bounds__(32 * kBwWarps, 2)
input_cat_bwd_tiles_kernel(const int64_t* __restrict__ data, int64_t data_ld, const float* __restrict__ nf, int64_t ld,
                     int B, const int* __restrict__ grp_var, const int* __restrict__ grp_node0,
                     const int* __restrict__ grp_count, const int* __restrict__ grp_ncats,
                     const int* __restrict__ s_pfids, int node_offset, float* __restrict__ pf, int CB,
                     int max_ncats, const uint8_t* __restrict__ miss, int64_t m_sb, int64_t m_sv,
                     const int* __restrict__ s_pids, const float* __restrict__ params, bool atomic) {
    pcb::pdl_trigger();
    extern __shared__ __align__(16) uint8_t bsm[];
    const BwdSmem S(CB, max_ncats);
    float* tile = reinterpret_cast<float*>(bsm);
    float* res = reinterpret_cast<float*>(bsm + S.res);
    uint32_t* code = reinterpret_cast<uint32_t*>(bsm + S.code);  // two buffers of the sort
    uint32_t* perm = reinterpret_cast<uint32_t*>(bsm + S.perm);  // byte offset in a tile row | kBwLast
    int* ucat = reinterpret_cast<int*>(bsm + S.ucat);    // categories present, in order
    int* start = reinterpret_cast<int*>(bsm + S.start);  // their first sorted sample
    __shared__ int sEntry[kBwWarps + 1];
    __shared__ int sU;
    const int g = blockIdx.x;
    const int K = __ldg(grp_ncats + g);
    const int64_t v = __ldg(grp_var + g);
    const int node0 = __ldg(grp_node0 + g);
    const int cnt = __ldg(grp_count + g);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int num_tiles = (cnt + kBwNodes - 1) / kBwNodes;
    pcb::pdl_wait();
    if ((int)blockIdx.y >= num_tiles) return;

    for (int c0 = 0; c0 < B; c0 += CB) {
        const int nb = min(CB, B - c0);
        auto load_tile = [&](int t) {
            float* dst = tile + lane;
            const float* src = nf + ((int64_t)node_offset + node0 + t * kBwNodes) * ld + c0 + lane;
            for (int n = warp; n < min(kBwNodes, cnt - t * kBwNodes); n += kBwWarps) {
                float* d = dst + n * S.pitch;
                const float* f = src + n * ld;
                if (nb == kBwChunk) {
#pragma unroll
                    for (int i = 0; i < kBwChunk; i += 32) pcb::cp_async4(d + i, f + i);
                } else {
                    for (int i = 0; i < nb - lane; i += 32) pcb::cp_async4(d + i, f + i);
                }
            }
            pcb::cp_async_commit();
        };
        load_tile(blockIdx.y);
        // One number per sample: (category, sample), categories outside [0, K) behind the others
        // (dropped), missing samples next, positions beyond the chunk last. Runs of 32 are
        // sorted in registers and merged pairwise, each number's place in the merged run found
        // by a binary search in the other run.
        uint32_t c = 0xfffffe00u | (uint32_t)tid;
        if (tid < nb) {
            int key;
            if (miss && miss[(int64_t)(c0 + tid) * m_sb + v * m_sv]) {
                key = K + 1;
            } else {
                const int64_t x = data[v * data_ld + c0 + tid];
                key = (x >= 0 && x < K) ? (int)x : K;
            }
            c = (uint32_t)key * kBwChunk + (uint32_t)tid;
        }
#pragma unroll
        for (int k = 2; k <= 32; k *= 2) {
#pragma unroll
            for (int j = k / 2; j > 0; j /= 2) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, c, j);
                c = (((lane & j) == 0) == ((lane & k) == 0)) ? min(c, o) : max(c, o);
            }
        }
        uint32_t* sorted = code;
        sorted[tid] = c;
        __syncthreads();
        for (int w = 32; w < nb; w *= 2) {
            const uint32_t x = sorted[tid];
            const uint32_t* other = sorted + ((tid / w) ^ 1) * w;
            int lo = 0;
            for (int h = w / 2; h > 0; h /= 2) lo += other[lo + h - 1] < x ? h : 0;
            lo += other[lo] < x ? 1 : 0;
            uint32_t* next = sorted == code ? code + kBwChunk : code;
            next[(tid & ~(2 * w - 1)) + (tid & (w - 1)) + lo] = x;
            sorted = next;
            __syncthreads();
        }
        if (tid < nb) {
            const uint32_t x = sorted[tid];
            const bool last = tid + 1 == nb || sorted[tid + 1] / kBwChunk != x / kBwChunk;
            perm[tid] = (x & (kBwChunk - 1)) * 4u | (last ? kBwLast : 0u);
        }
        if (warp == 0) {
            int nu = 0;
            for (int p0 = 0; p0 < nb; p0 += 32) {
                const int p = p0 + lane;
                const int key = p < nb ? (int)(sorted[p] / kBwChunk) : -1;
                const bool first = p < nb && (p == 0 || (int)(sorted[p - 1] / kBwChunk) != key);
                const unsigned bal = __ballot_sync(0xffffffffu, first);
                if (first) {
                    const int e = nu + __popc(bal & ((1u << lane) - 1u));
                    ucat[e] = key;
                    start[e] = p;
                }
                nu += __popc(bal);
            }
            if (lane == 0) {
                sU = nu;
                ucat[nu] = K + 2;
                start[nu] = nb;
            }
            __syncwarp();
            // warp w sums the categories whose first sample lies in its share of the positions
            if (lane <= kBwWarps) {
                const int at = (int)((int64_t)nb * lane / kBwWarps);
                int lo = 0, hi = nu;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (start[mid] < at) lo = mid + 1;
                    else hi = mid;
                }
                sEntry[lane] = lo;
            }
        }
        __syncthreads();
        const int U = sU;
        const int e0 = sEntry[warp], e1 = sEntry[warp + 1];
        const int p0 = start[e0], p1 = start[e1];
        const bool has_miss = U > 0 && ucat[U - 1] == K + 1;
        // entries that are categories
        int L = U - (has_miss ? 1 : 0);
        if (L > 0 && ucat[L - 1] == K) --L;
        for (int t = blockIdx.y; t < num_tiles; t += gridDim.y) {
            const int nn = min(kBwNodes, cnt - t * kBwNodes);
            // old values of this warp's nodes (warp, warp + 16), first 32 kBwOld entries
            float old[kBwNodes / kBwWarps][kBwOld];
            int64_t slot[kBwNodes / kBwWarps];
#pragma unroll
            for (int a = 0; a < kBwNodes / kBwWarps; ++a) {
                const int n = warp + a * kBwWarps;
                slot[a] = n < nn ? __ldg(s_pfids + node0 + t * kBwNodes + n) : 0;
            }
            if (!atomic && !has_miss) {
#pragma unroll
                for (int j = 0; j < kBwOld; ++j) {
                    if (32 * j >= L) break;
                    const int e = lane + 32 * j;
                    const int k = e < L ? ucat[e] : 0;
#pragma unroll
                    for (int a = 0; a < kBwNodes / kBwWarps; ++a)
                        old[a][j] = (e < L && warp + a * kBwWarps < nn) ? pf[slot[a] + k] : 0.f;
                }
            }
            pcb::cp_async_wait<0>();
            __syncthreads();  // the tile has arrived; the sums of the last one are written
            {
                const char* row =
                    reinterpret_cast<const char*>(tile + lane * S.pitch);
                float* out = res + lane * S.epitch + e0;
                float acc = 0.f;
                int p = p0;
                auto value = [&](uint32_t o) { return *reinterpret_cast<const float*>(row + (o & ~kBwLast)); };
                auto add = [&](uint32_t o, float f) {
                    acc += LOG ? __expf(f) : f;
                    const bool last = (o & kBwLast) != 0;
                    if (last) *out = acc;
                    out += last;
                    acc = last ? 0.f : acc;
                };
                for (; p < p1 && (p & 3); ++p) add(perm[p], value(perm[p]));
                for (; p + 3 < p1; p += 4) {
                    const uint4 o = *reinterpret_cast<const uint4*>(perm + p);
                    const float f0 = value(o.x), f1 = value(o.y), f2 = value(o.z), f3 = value(o.w);
                    add(o.x, f0);
                    add(o.y, f1);
                    add(o.z, f2);
                    add(o.w, f3);
                }
                for (; p < p1; ++p) add(perm[p], value(perm[p]));
            }
            __syncthreads();  // the tile is free, the sums are complete
            if (t + (int)gridDim.y < num_tiles) load_tile(t + gridDim.y);
#pragma unroll
            for (int a = 0; a < kBwNodes / kBwWarps; ++a) {
                const int n = warp + a * kBwWarps;
                if (n >= nn) continue;
                const float* r = res + n * S.epitch;
                float* dst = pf + slot[a];
                if (has_miss) {
                    const float msum = r[U - 1];
                    const float* th = params + __ldg(s_pids + node0 + t * kBwNodes + n);
                    for (int k = lane; k < K; k += 32) {
                        if (atomic) atomicAdd(dst + k, msum * th[k]);
                        else dst[k] += msum * th[k];
                    }
                    __syncwarp();
                }
                if (atomic || has_miss) {
                    for (int e = lane; e < L; e += 32) {
                        if (atomic) atomicAdd(dst + ucat[e], r[e]);
                        else dst[ucat[e]] += r[e];
                    }
                    continue;
                }
#pragma unroll
                for (int j = 0; j < kBwOld; ++j) {
                    if (32 * j >= L) break;
                    const int e = lane + 32 * j;
                    if (e < L) dst[ucat[e]] = old[a][j] + r[e];
                }
                for (int e = lane + 32 * kBwOld; e < L; e += 32) dst[ucat[e]] += r[e];
            }
        }
        __syncthreads();  // the next chunk reuses the tables and tiles
    }
}

}  // namespace

extern "C" int pcb_input_cat_fwd(const int64_t* data, int64_t data_ld, const float* params, const int32_t* vids,
                                 const int32_t* s_pids, const int32_t* ncats, int32_t num_nodes, int32_t node_offset,
                                 float* node_mars, int64_t ld, int32_t B, const uint8_t* missing, int64_t miss_sb,
                                 int64_t miss_sv, void* stream) {
    if (!data || !params || !vids || !s_pids || !ncats || !node_mars || B <= 0 || ld < B || data_ld < B || num_nodes < 0)
        return pcb::set_error(PCB_E_ARG, "pcb_input_cat_fwd: bad arguments");
    if (num_nodes == 0) return PCB_OK;
    const bool vec = pcb::vec_ok(node_mars, ld);
    const int64_t gy = pcb::cdiv(B, kFwdSamples);
    if (gy > 65535) return pcb::set_error(PCB_E_ARG, "pcb_input_cat_fwd: batch too large");
    return pcb::launch_status(pcb::launch_k(input_cat_fwd_kernel, dim3((unsigned)pcb::cdiv(num_nodes, kRowNodes),
                                                                       (unsigned)gy),
                                            dim3(kFwdThreads), 0, pcb::as_stream(stream), 1u, data, data_ld, params, vids,
                                            s_pids, ncats, num_nodes, node_offset, node_mars, ld, B, vec, missing,
                                            miss_sb, miss_sv, pcb::status_word()),
                              "pcb_input_cat_fwd");
}

extern "C" int pcb_input_cat_fwd_quads(const int64_t* data, int64_t data_ld, const float* params, const int32_t* vids,
                                 const int32_t* s_pids, const int32_t* ncats, int32_t num_nodes, int32_t node_offset,
                                 float* node_mars, int64_t ld, int32_t B, const uint8_t* missing, int64_t miss_sb,
                                 int64_t miss_sv, void* stream) {
    if (!data || !params || !vids || !s_pids || !ncats || !node_mars || B <= 0 || ld < B || data_ld < B || num_nodes < 0)
        return pcb::set_error(PCB_E_ARG, "pcb_input_cat_fwd_quads: bad arguments");
    if (num_nodes == 0) return PCB_OK;
    const bool vec = pcb::vec_ok(node_mars, ld);
    const int64_t gy = pcb::cdiv(B, kFwdSamples);
    if (gy > 65535) return pcb::set_error(PCB_E_ARG, "pcb_input_cat_fwd_quads: batch too large");
    return pcb::launch_status(pcb::launch_k(input_cat_fwd_quads_kernel, dim3((unsigned)pcb::cdiv(num_nodes, kFwdNodes),
                                                                       (unsigned)gy),
                                            dim3(kFwdThreads), 0, pcb::as_stream(stream), 1u, data, data_ld, params, vids,
                                            s_pids, ncats, num_nodes, node_offset, node_mars, ld, B, vec, missing,
                                            miss_sb, miss_sv, pcb::status_word()),
                              "pcb_input_cat_fwd_quads");
}

extern "C" int pcb_input_cat_bwd_tiles(const int64_t* data, int64_t data_ld, const float* node_flows, int64_t ld, int32_t B,
                                 const int32_t* grp_var, const int32_t* grp_node0, const int32_t* grp_count,
                                 const int32_t* grp_ncats, int32_t num_groups, int32_t max_ncats,
                                 const int32_t* s_pfids, int32_t node_offset, float* param_flows,
                                 int32_t logspace_flows, const uint8_t* missing, int64_t miss_sb, int64_t miss_sv,
                                 const int32_t* s_pids, const float* params, int32_t atomic, void* stream) {
    if (!data || !node_flows || !grp_var || !grp_node0 || !grp_count || !grp_ncats || !s_pfids || !param_flows ||
        B <= 0 || ld < B || data_ld < B || num_groups < 0 || max_ncats <= 0 || (missing && (!s_pids || !params)))
        return pcb::set_error(PCB_E_ARG, "pcb_input_cat_bwd_tiles: bad arguments");
    if (num_groups == 0) return PCB_OK;
    const int CB = B < kBwChunk ? B : kBwChunk;
    const size_t smem = BwdSmem(CB, max_ncats).total;
    // a sample's sort key is (category, sample) in 32 bits; the tables stop growing at 510 categories
    if (max_ncats > (int)(0xfffffe00u / kBwChunk) - 4)
        return pcb::set_error(PCB_E_ARG, "pcb_input_cat_bwd_tiles: too many categories (%d)", max_ncats);
    auto go = [&](auto kernel) {
        if (smem > 48 * 1024) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return pcb::set_error(PCB_E_CUDA, "pcb_input_cat_bwd_tiles: %s", cudaGetErrorString(e));
        }
        // CTAs per variable: one where the variables alone give three per SM (each sorts the
        // batch again), up to 16 for fewer; a CTA without a tile returns at once
        const int splits = (int)std::min<int64_t>(16, pcb::cdiv(3 * pcb::num_sms(), num_groups));
        return pcb::launch_status(pcb::launch_k(kernel, dim3(num_groups, splits), dim3(32 * kBwWarps), smem,
                                                pcb::as_stream(stream), 1u, data, data_ld, node_flows, ld, B, grp_var,
                                                grp_node0, grp_count, grp_ncats, s_pfids, node_offset, param_flows,
                                                CB, max_ncats, missing, miss_sb, miss_sv, s_pids, params, atomic != 0),
                                  "pcb_input_cat_bwd_tiles");
    };
    return logspace_flows ? go(input_cat_bwd_tiles_kernel<true>) : go(input_cat_bwd_tiles_kernel<false>);
}

extern "C" int pcb_input_cat_bwd(const int64_t* data, int64_t data_ld, const float* node_flows, int64_t ld, int32_t B,
                                 const int32_t* grp_var, const int32_t* grp_node0, const int32_t* grp_count,
                                 const int32_t* grp_ncats, int32_t num_groups, int32_t max_ncats,
                                 const int32_t* s_pfids, int32_t node_offset, float* param_flows,
                                 int32_t logspace_flows, const uint8_t* missing, int64_t miss_sb, int64_t miss_sv,
                                 const int32_t* s_pids, const float* params, int32_t atomic, void* stream) {
    if (!data || !node_flows || !grp_var || !grp_node0 || !grp_count || !grp_ncats || !s_pfids || !param_flows ||
        B <= 0 || ld < B || data_ld < B || num_groups < 0 || max_ncats <= 0 || (missing && (!s_pids || !params)))
        return pcb::set_error(PCB_E_ARG, "pcb_input_cat_bwd: bad arguments");
    if (num_groups == 0) return PCB_OK;
    const int CB = B < 1024 ? B : 1024;
    const size_t smem = (size_t)(2 * CB + 8 * CB + max_ncats + 3 + CB) * sizeof(int);
    if (smem > 200 * 1024) return pcb::set_error(PCB_E_ARG, "pcb_input_cat_bwd: too many categories (%d)", max_ncats);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(input_cat_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return pcb::set_error(PCB_E_CUDA, "pcb_input_cat_bwd: %s", cudaGetErrorString(e));
    }
    return pcb::launch_status(pcb::launch_k(input_cat_bwd_kernel, dim3(num_groups), dim3(256), smem,
                                            pcb::as_stream(stream), 1u, data, data_ld, node_flows, ld, B, grp_var,
                                            grp_node0, grp_count, grp_ncats, s_pfids, node_offset, param_flows,
                                            logspace_flows != 0, CB, missing, miss_sb, miss_sv, s_pids, params,
                                            atomic != 0),
                              "pcb_input_cat_bwd");
}
