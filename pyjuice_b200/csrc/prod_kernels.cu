// Product-layer gather-add (forward) and flow scatter (backward) plus the
// sum-layer "modify flows" pass. All are HBM-bound row gathers along the batch.
#include <type_traits>

#include "common.cuh"

namespace {

// A thread takes 4 consecutive samples of a row, B of which are ngrp = ceil(B / 4) positions. (Rows
// that do not allow 16-byte accesses: 4 scalar ones, whose lines the L1 keeps; 4 samples 32 or ngrp
// apart are slower, 51200 rows of 2 x 65 samples: 14.4 us against 10.8.)
//
// Row (or group of rows) and position of this thread: positions run on from row to row, so that a
// batch of any size leaves no lanes idle. 32-bit division where the numbers allow it.
struct Place {
    int64_t row;
    int t;
};
__device__ __forceinline__ Place place_of(int ngrp, bool narrow) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (narrow) {
        const uint32_t r = (uint32_t)i / (uint32_t)ngrp;
        return {(int64_t)r, (int)((uint32_t)i - r * (uint32_t)ngrp)};
    }
    return {(int64_t)(i / (uint64_t)ngrp), (int)(i % (uint64_t)ngrp)};
}

template <bool VEC>
__device__ __forceinline__ float4 load_row(const float* __restrict__ base, int64_t row, int64_t ld, int t, int B,
                                           float fill) {
    return pcb::load4(base, row, ld, 4 * t, B, VEC, fill);
}

template <bool VEC>
__device__ __forceinline__ void store_row(float* __restrict__ base, int64_t row, int64_t ld, int t, int B, float4 v) {
    pcb::store4(base, row, ld, 4 * t, B, VEC, v);
}

// Bound by HBM: arity reads and one write per output. A thread takes R consecutive rows of
// one block (their child rows are consecutive too, so the tables are read once) and 4
// samples, and has R x J row loads in flight. R = 4, J = 2 where the layer fills the GPU
// (200 vectors of 256 nodes, two children, 512 samples: 56 us, 5.6 TB/s, against 92 us
// with one row per thread and a 64-bit division per thread); R = 1, J = 8 for small layers,
// which are bound by latency and want the threads.
// MOD (overwrite, linear flows only): the rows of blocks g with mod_blk[g] != 0 are written as
// log(sum) - nm, the sum layer's "modified" node flows (log f - log m), instead of the sum.
template <int R, int J, bool VEC, bool ACCUM, bool LSE, bool MOD>
__global__ void __launch_bounds__(256)
prod_kernel(const float* __restrict__ in, float* __restrict__ out, int64_t ld, int B, const int* __restrict__ blk_row,
            const int* __restrict__ blk_off, const int* __restrict__ blk_cnt, const int* __restrict__ chs,
            int blk_size, int ngrp, int num_chunks, int chunks_per_blk, bool narrow, const float* __restrict__ nm,
            const int* __restrict__ mod_blk) {
    // The block tables (and the first J child indices) are read before the wait for the
    // previous kernel: they are compiled once and never written by a pass.
    pcb::pdl_trigger();
    const Place at = place_of(ngrp, narrow);
    if (at.row >= num_chunks) return;
    const int chunk = (int)at.row, t = at.t;
    const int g = chunk / chunks_per_blk;
    const int i0 = (chunk - g * chunks_per_blk) * R;
    const int nr = R == 1 ? 1 : min(R, blk_size - i0);
    const int off = __ldg(blk_off + g);
    const int cnt = __ldg(blk_cnt + g);
    const int64_t row = (int64_t)__ldg(blk_row + g) + i0;
    const bool rewrite = MOD && __ldg(mod_blk + g) != 0;
    int c[J];
#pragma unroll
    for (int j = 0; j < J; ++j) c[j] = (j < cnt) ? __ldg(chs + off + j) : -1;
    pcb::pdl_wait();
    float4 acc[R];
    if (!LSE) {
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        // J children at a time: all index loads, then all row loads, are independent
        for (int j0 = 0; j0 < cnt; j0 += J) {
            if (j0 > 0) {
#pragma unroll
                for (int j = 0; j < J; ++j) c[j] = (j0 + j < cnt) ? __ldg(chs + off + j0 + j) : -1;
            }
            float4 v[R][J];
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int j = 0; j < J; ++j)
                    v[r][j] = (c[j] >= 0 && r < nr) ? load_row<VEC>(in, (int64_t)c[j] + i0 + r, ld, t, B, 0.f)
                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    acc[r].x += v[r][j].x; acc[r].y += v[r][j].y; acc[r].z += v[r][j].z; acc[r].w += v[r][j].w;
                }
            }
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r >= nr) break;
            const int i = i0 + r;
            float4 m = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            for (int j = 0; j < cnt; ++j) {
                const float4 v = load_row<VEC>(in, (int64_t)__ldg(chs + off + j) + i, ld, t, B, -INFINITY);
                m.x = fmaxf(m.x, v.x); m.y = fmaxf(m.y, v.y); m.z = fmaxf(m.z, v.z); m.w = fmaxf(m.w, v.w);
            }
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int j = 0; j < cnt; ++j) {
                const float4 v = load_row<VEC>(in, (int64_t)__ldg(chs + off + j) + i, ld, t, B, -INFINITY);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float mq = pcb::get(m, q);
                    pcb::set(s, q, pcb::get(s, q) + (mq == -INFINITY ? 0.f : __expf(pcb::get(v, q) - mq)));
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float mq = pcb::get(m, q);
                pcb::set(acc[r], q, mq == -INFINITY ? -INFINITY : logf(pcb::get(s, q)) + mq);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (r >= nr) break;
        if (rewrite) {
            const float4 m = load_row<VEC>(nm, row + r, ld, t, B, 0.f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float mq = pcb::get(m, q);
                pcb::set(acc[r], q, mq == -INFINITY ? -INFINITY : logf(pcb::get(acc[r], q)) - mq);
            }
        }
        if (ACCUM) {
            const float4 old = load_row<VEC>(out, row + r, ld, t, B, 0.f);
            if (!LSE) {
                acc[r].x += old.x; acc[r].y += old.y; acc[r].z += old.z; acc[r].w += old.w;
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    pcb::set(acc[r], q, pcb::logaddexp(pcb::get(old, q), pcb::get(acc[r], q)));
            }
        }
        store_row<VEC>(out, row + r, ld, t, B, acc[r]);
    }
}

template <bool ACCUM, bool LSE, bool MOD>
int launch_prod(const char* name, const float* in, float* out, int64_t ld, int32_t B, const int32_t* blk_row,
                const int32_t* blk_off, const int32_t* blk_cnt, const int32_t* chs, int32_t num_blocks,
                int32_t blk_size, const float* nm, const int32_t* mod_blk, void* stream) {
    const bool vec = pcb::vec_ok(in, ld) && pcb::vec_ok(out, ld) && (!MOD || pcb::vec_ok(nm, ld));
    const int ngrp = (int)pcb::cdiv(B, 4);
    // Four rows per thread once that still leaves two full sets of threads per SM.
    const bool wide = !LSE && blk_size >= 4 && (int64_t)num_blocks * blk_size / 4 * ngrp >= 2LL * pcb::num_sms() * 2048;
    const int rows = wide ? 4 : 1;
    const int per_blk = (int)pcb::cdiv(blk_size, rows);
    const int64_t chunks = (int64_t)num_blocks * per_blk;
    const int64_t ctas = pcb::cdiv(chunks * ngrp, 256);
    if (chunks > INT32_MAX || ctas > INT32_MAX) return pcb::set_error(PCB_E_ARG, "%s: layer or batch too large", name);
    auto go = [&](auto kernel) {
        return pcb::launch_status(pcb::launch_k(kernel, dim3((unsigned)ctas), dim3(256), 0, pcb::as_stream(stream), 1u,
                                                in, out, ld, B, blk_row, blk_off, blk_cnt, chs, blk_size, ngrp,
                                                (int)chunks, per_blk, ctas * 256 <= UINT32_MAX, nm, mod_blk), name);
    };
    if (wide) {
        if constexpr (!LSE)
            return vec ? go(prod_kernel<4, 2, true, ACCUM, LSE, MOD>) : go(prod_kernel<4, 2, false, ACCUM, LSE, MOD>);
    }
    return vec ? go(prod_kernel<1, 8, true, ACCUM, LSE, MOD>) : go(prod_kernel<1, 8, false, ACCUM, LSE, MOD>);
}

// out = log f - log m (out may be the flows themselves). Bound by HBM: ROWS 16-byte accesses of each
// array in flight per thread. Four rows where that leaves three quarters of the threads an SM holds
// (51200 rows of 512 samples: 49 us, 6.4 TB/s; 16384 of 256: 7.7 us, 8.3 with one); one below, and where rows take scalar accesses, since four rows'
// logarithms in one thread are a chain of 1 us (64 rows of 64 samples: 2.7 us against 1.6; 16384 of
// 64: 4.7 against 3.1; 51200 of 209: 20.9 against 20.3).
constexpr int kModRows = 4;

template <int ROWS, bool VEC>
__global__ void __launch_bounds__(256)
modify_flows_kernel(const float* nf, const float* __restrict__ nm, float* out, int64_t ld, int B, int64_t row0,
                    int64_t out_row0, int64_t num_rows, int ngrp, bool narrow) {
    pcb::pdl_trigger();
    const Place at = place_of(ngrp, narrow);
    const int64_t r0 = at.row * ROWS;
    const int t = at.t;
    if (r0 >= num_rows) return;
    pcb::pdl_wait();
    float4 f[ROWS], m[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (r0 + r >= num_rows) break;
        if (VEC && 4 * t + 3 < B) {  // not the read-only path: out may be nf
            f[r] = *reinterpret_cast<const float4*>(nf + (row0 + r0 + r) * ld + 4 * t);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int b = 4 * t + q;
                pcb::set(f[r], q, b < B ? nf[(row0 + r0 + r) * ld + b] : 0.f);
            }
        }
        m[r] = load_row<VEC>(nm, row0 + r0 + r, ld, t, B, 0.f);
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (r0 + r >= num_rows) break;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float mq = pcb::get(m[r], q);
            pcb::set(f[r], q, mq == -INFINITY ? -INFINITY : logf(pcb::get(f[r], q)) - mq);
        }
        store_row<VEC>(out, out_row0 + r0 + r, ld, t, B, f[r]);
    }
}

int launch_modify(const char* name, const float* nf, const float* nm, float* out, int64_t ld, int32_t B, int64_t row0,
                  int64_t row1, int64_t out_row0, void* stream) {
    if (row1 == row0) return PCB_OK;
    const bool vec = pcb::vec_ok(nf, ld) && pcb::vec_ok(nm, ld) && pcb::vec_ok(out, ld);
    const int ngrp = (int)pcb::cdiv(B, 4);
    const bool wide = vec && (row1 - row0) / kModRows * ngrp >= pcb::num_sms() * 1536LL;
    const int64_t ctas = pcb::cdiv(pcb::cdiv(row1 - row0, wide ? kModRows : 1) * ngrp, 256);
    if (ctas > INT32_MAX) return pcb::set_error(PCB_E_ARG, "%s: too many rows", name);
    auto go = [&](auto kernel) {
        return pcb::launch_status(pcb::launch_k(kernel, dim3((unsigned)ctas), dim3(256), 0, pcb::as_stream(stream), 1u,
                                                nf, nm, out, ld, B, row0, out_row0, row1 - row0, ngrp,
                                                ctas * 256 <= UINT32_MAX), name);
    };
    if (wide) return go(modify_flows_kernel<kModRows, true>);
    return vec ? go(modify_flows_kernel<1, true>) : go(modify_flows_kernel<1, false>);
}

}  // namespace

extern "C" int pcb_prod_gather_sum(const float* in, float* out, int64_t ld, int32_t B, const int32_t* blk_row,
                                   const int32_t* blk_off, const int32_t* blk_cnt, const int32_t* chs,
                                   int32_t num_blocks, int32_t blk_size, int32_t accum, int32_t logsumexp,
                                   void* stream) {
    if (!in || !out || !blk_row || !blk_off || !blk_cnt || !chs || B <= 0 || ld < B || num_blocks < 0 || blk_size <= 0)
        return pcb::set_error(PCB_E_ARG, "pcb_prod_gather_sum: bad arguments");
    if (num_blocks == 0) return PCB_OK;
    auto go = [&](auto accumulate, auto lse) {
        return launch_prod<decltype(accumulate)::value, decltype(lse)::value, false>(
            "pcb_prod_gather_sum", in, out, ld, B, blk_row, blk_off, blk_cnt, chs, num_blocks, blk_size, nullptr,
            nullptr, stream);
    };
    using T = std::true_type;
    using F = std::false_type;
    if (logsumexp) return accum ? go(T{}, T{}) : go(F{}, T{});
    return accum ? go(T{}, F{}) : go(F{}, F{});
}

extern "C" int pcb_prod_gather_sum_modify(const float* in, float* out, int64_t ld, int32_t B, const int32_t* blk_row,
                                          const int32_t* blk_off, const int32_t* blk_cnt, const int32_t* chs,
                                          int32_t num_blocks, int32_t blk_size, const float* node_mars,
                                          const int32_t* block_rewrite, void* stream) {
    if (!in || !out || !blk_row || !blk_off || !blk_cnt || !chs || !node_mars || !block_rewrite || B <= 0 || ld < B ||
        num_blocks < 0 || blk_size <= 0)
        return pcb::set_error(PCB_E_ARG, "pcb_prod_gather_sum_modify: bad arguments");
    if (num_blocks == 0) return PCB_OK;
    return launch_prod<false, false, true>("pcb_prod_gather_sum_modify", in, out, ld, B, blk_row, blk_off, blk_cnt, chs,
                                           num_blocks, blk_size, node_mars, block_rewrite, stream);
}

extern "C" int pcb_modify_flows(float* node_flows, const float* node_mars, int64_t ld, int32_t B, int64_t row0,
                                int64_t row1, void* stream) {
    if (!node_flows || !node_mars || B <= 0 || ld < B || row0 < 0 || row1 < row0)
        return pcb::set_error(PCB_E_ARG, "pcb_modify_flows: bad arguments");
    return launch_modify("pcb_modify_flows", node_flows, node_mars, node_flows, ld, B, row0, row1, row0, stream);
}

extern "C" int pcb_flow_ratios(const float* node_flows, const float* node_mars, float* out, int64_t ld, int32_t B,
                               int64_t row0, int64_t row1, void* stream) {
    if (!node_flows || !node_mars || !out || B <= 0 || ld < B || row0 < 0 || row1 < row0)
        return pcb::set_error(PCB_E_ARG, "pcb_flow_ratios: bad arguments");
    return launch_modify("pcb_flow_ratios", node_flows, node_mars, out, ld, B, row0, row1, 0, stream);
}
