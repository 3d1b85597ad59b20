// Experts of a prefill chunk, grouped: every expert's weights meet only the rows that are routed to it.
//
//   moe_plan     : from the chunk's expert ids [T][S], the (row, slot) pairs sorted by expert (by row inside an expert) and
//                  the list of work items (expert, first pair, pairs)
//   moe_gather   : the pairs' quantised rows, one after the other ([pair][term][K]), and their block scales
//   tc_group     : a persistent tcgen05 GEMM over the items: 128 weight rows x up to NP pairs per item and row tile
//   moe_pair_act : h = silu(gate) * up * route weight of every pair, quantised
//
// With 64 rows x 10 routes over 512 experts an expert has about two rows, and the products' cost is the weights: 385 MB and
// 192 MB a layer at the 8-way shard, 59 and 29 us at the measured copy bandwidth.  Multiplying every expert by all rows of the
// chunk (three terms: 192 columns a weight tile, of which 2 x 3 are used) was bound by the read-back and scaling of those
// columns out of tensor memory, 230 and 109 us.  An item's MMA has 32 columns (NP = 10 pairs x 3 terms, 16 x 2 or 32 x 1), its
// terms are added as they leave tensor memory, and its row of the output is the pair's own.  One B200, 64 rows, 8-way shard:
// 67 and 38 us, 0.88 and 0.77 of the measured copy bandwidth.
#include <cuda.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include "api.h"
#include "common.cuh"
#include "mma_gemv.cuh"
#include "tc_common.cuh"

namespace {
using namespace nexrt;
using namespace nexrt::tc;

constexpr int kGroupCols = 32;                         // MMA N
constexpr int kGroupA = kBM * kSpan, kGroupB = kGroupCols * kSpan, kGroupStage = kGroupA + kGroupB;
constexpr int kGroupStages = 5;                        // 5 x 20 KB: two CTAs per SM
constexpr int kGroupBufs = 8;                          // accumulators: 8 x 32 columns x 2 CTAs = all of tensor memory
constexpr int kGroupItems = 256;                       // items of a CTA kept in shared memory (further ones are read from the list)
constexpr int kGroupSmem = 1024 + kGroupStages * kGroupStage + 1024;
constexpr int kMaxChunkRows = 128;

// Barrier of the four epilogue warps that also tells all of them whether any has given up.
__device__ __forceinline__ bool epilogue_any(bool gave_up) {
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(any)
        : "r"(static_cast<uint32_t>(gave_up))
        : "memory");
    return any != 0;
}

struct GroupArgs {
    const float* ws;        // weight block scales [expert][MT][KB]
    const float* xs;        // activation scales of term 0 [pair][KB] (term p: 16^-p of it)
    float* out;             // [row][ldo]
    const int* n_items;
    const int4* items;      // {expert, first pair, pairs, -}
    const int* out_row;     // row of `out` of every pair, or null: the pair's index
    int KB, MT, ldo;        // K blocks, row tiles per expert, floats between two rows of `out`
    int* status;
};

// P terms per pair, NP = 32 / P pairs per item.
template <int P>
__global__ void __launch_bounds__(kThreads, 2) tc_group_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, GroupArgs a) {
    constexpr int NP = kGroupCols / P, NS = kGroupStages, NAB = kGroupBufs, PER = (NAB * NP + 127) / 128;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int4 s_items[kGroupItems];
    __shared__ float s_sc[2][NAB * NP];                 // weight scale x activation scale of the pairs of eight K blocks
    __shared__ int s_row[2][NAB * NP];                  // and the output rows of those pairs
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base);
    uint8_t* smem = base + 1024;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * NS + 2 * NAB);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NS + 2 * NAB + 1);
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (NS + s); };
    auto tfull = [&](int b) { return bar0 + 8u * (2 * NS + b); };
    auto tempty = [&](int b) { return bar0 + 8u * (2 * NS + NAB + b); };
    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int b = 0; b < NAB; ++b) { mbar_init(tfull(b), 1); mbar_init(tempty(b), 4); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), NAB * kGroupCols);
    pdl_wait();
    // this CTA's tiles: blockIdx, blockIdx + grid, ... of the items x row tiles; the row tiles of an item are neighbours
    const int total = *a.n_items * a.MT, grid = static_cast<int>(gridDim.x), first = static_cast<int>(blockIdx.x);
    const int mine = first < total ? (total - first + grid - 1) / grid : 0;
    for (int j = threadIdx.x; j < min(mine, kGroupItems); j += blockDim.x) s_items[j] = a.items[(first + j * grid) / a.MT];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    auto item_of = [&](int j) { return j < kGroupItems ? s_items[j] : a.items[(first + j * grid) / a.MT]; };
    auto tile_of = [&](int j) { return (first + j * grid) % a.MT; };

    if (warp == 0) {
        if (lane == 0) {
            int q = 0;
            bool ok = true;
            for (int j = 0; j < mine && ok; ++j) {
                const int4 it = item_of(j);
                const int wrow = (it.x * a.MT + tile_of(j)) * kBM;
                for (int kb = 0; kb < a.KB; ++kb, ++q) {
                    const int s = q % NS;
                    ok = mbar_wait(empty(s), ((q / NS) & 1) ^ 1, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(full(s), kGroupA + kGroupB);
                    const uint32_t dst = smem_u32(smem + s * kGroupStage);
                    tma_load_2d(dst, &map_w, kb * kSpan, wrow, full(s));
                    tma_load_2d(dst + kGroupA, &map_x, kb * kSpan, it.y * P, full(s));
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = instr_desc<true>(kGroupCols);
            const int n = mine * a.KB;
            for (int q = 0; q < n; ++q) {
                const int s = q % NS, buf = q % NAB;
                if (!mbar_wait(tempty(buf), ((q / NAB) & 1) ^ 1, abort_flag)) break;
                if (!mbar_wait(full(s), (q / NS) & 1, abort_flag)) break;
                tc_fence_after();
                const uint32_t a0 = smem_u32(smem + s * kGroupStage);
                const uint64_t da = smem_desc(a0), db = smem_desc(a0 + kGroupA);
#pragma unroll
                for (int k = 0; k < 4; ++k) tc_mma<true>(tmem_base + buf * kGroupCols, da + 2u * k, db + 2u * k, idesc, k != 0);
                tc_commit(empty(s));
                tc_commit(tfull(buf));
            }
        }
    } else {
        const int wq = warp & 3, et = threadIdx.x - 64, n = mine * a.KB;
        // scales and output rows of K blocks 8 g .. 8 g + 7, one (K block, pair) per thread, requested a group ahead
        float nsc[PER];
        int nrow[PER];
        auto request = [&](int g) {
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int e = et + u * 128, q = g * NAB + e / NP, jp = e % NP;
                nsc[u] = 0.f;
                nrow[u] = 0;
                if (e < NAB * NP && q < n) {
                    const int j = q / a.KB, kb = q % a.KB;
                    const int4 it = item_of(j);
                    if (jp < it.z) {
                        nsc[u] = __ldg(a.ws + (static_cast<size_t>(it.x) * a.MT + tile_of(j)) * a.KB + kb) * __ldg(a.xs + static_cast<size_t>(it.y + jp) * a.KB + kb);
                        nrow[u] = a.out_row != nullptr ? __ldg(a.out_row + it.y + jp) : it.y + jp;
                    }
                }
            }
        };
        auto publish = [&](int g) {
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int e = et + u * 128;
                if (e < NAB * NP) { s_sc[g & 1][e] = nsc[u]; s_row[g & 1][e] = nrow[u]; }
            }
        };
        float acc[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) acc[i] = 0.f;
        request(0);
        publish(0);
        bool ok = !epilogue_any(false);
        int j = 0, kb = 0;
        for (int g = 0; g * NAB < n && ok; ++g) {
            request(g + 1);
            for (int k = 0; k < NAB && g * NAB + k < n; ++k) {
                ok = __all_sync(0xffffffffu, mbar_wait(tfull(k), g & 1, abort_flag));
                if (!ok) break;
                tc_fence_after();
                float p[kGroupCols];
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(32 * wq) << 16) + k * kGroupCols;
                tmem_ld16(taddr, p);
                tmem_ld16(taddr + 16, p + 16);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty(k));
                const float* sc = &s_sc[g & 1][k * NP];
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    float v = p[i * P + P - 1];
#pragma unroll
                    for (int t = P - 2; t >= 0; --t) v = fmaf(v, kTermInv, p[i * P + t]);
                    acc[i] = fmaf(v, sc[i], acc[i]);
                }
                if (++kb == a.KB) {
                    const int np = item_of(j).z;
                    float* o = a.out + tile_of(j) * kBM + 32 * wq + lane;
#pragma unroll
                    for (int i = 0; i < NP; ++i) {
                        if (i < np) o[static_cast<size_t>(s_row[g & 1][k * NP + i]) * a.ldo] = acc[i];
                        acc[i] = 0.f;
                    }
                    kb = 0;
                    ++j;
                }
            }
            publish(g + 1);                              // the other buffer: read by nobody since the last barrier
            ok = !epilogue_any(!ok);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 50000) {
        }
        if (threadIdx.x == 0 && a.status) atomicCAS(a.status, 0, static_cast<int>(kStatusPipeTimeout));
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_free(tmem_base, NAB * kGroupCols);
    }
}

// One CTA.  A row names an expert at most once, so an expert's rows are a set of at most 128 bits, and the place of a pair
// inside its expert is the number of set bits below its row: the order does not depend on timing.
__global__ void __launch_bounds__(1024) moe_plan_kernel(const int* __restrict__ ids, int4* __restrict__ items, int* __restrict__ n_items, int* __restrict__ pair_row,
                                                        int* __restrict__ out_row, int S, int T, int n_total, int NP) {
    constexpr int W = kMaxChunkRows / 32;
    extern __shared__ unsigned int s_mask[];            // [n_total][W], then [n_total] first pair
    __shared__ int s_warp[2][32];
    int* s_first = reinterpret_cast<int*>(s_mask + n_total * W);
    pdl_launch_dependents();
    for (int i = threadIdx.x; i < n_total * W; i += blockDim.x) s_mask[i] = 0u;
    __syncthreads();
    pdl_wait();
    const int pairs = T * S;
    auto expert = [&](int p) { return min(max(ids[p], 0), n_total - 1); };
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) atomicOr(&s_mask[expert(p) * W + (p / S) / 32], 1u << ((p / S) & 31));
    __syncthreads();
    // exclusive prefix sums over the experts of their pairs and of their items, 1024 experts at a time
    int pair0 = 0, item0 = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e0 = 0; e0 < n_total; e0 += blockDim.x) {
        const int e = e0 + static_cast<int>(threadIdx.x);
        int cnt = 0;
        if (e < n_total)
#pragma unroll
            for (int w = 0; w < W; ++w) cnt += __popc(s_mask[e * W + w]);
        const int tiles = (cnt + NP - 1) / NP;
        int a = cnt, b = tiles;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int ta = __shfl_up_sync(0xffffffffu, a, o), tb = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) { a += ta; b += tb; }
        }
        if (lane == 31) { s_warp[0][warp] = a; s_warp[1][warp] = b; }
        __syncthreads();
        int pa = pair0, pb = item0, ta = 0, tb = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) { pa += s_warp[0][w]; pb += s_warp[1][w]; }
            ta += s_warp[0][w]; tb += s_warp[1][w];
        }
        __syncthreads();
        if (e < n_total) {
            const int f = pa + a - cnt;
            s_first[e] = f;
            for (int i = 0; i < tiles; ++i) items[pb + b - tiles + i] = make_int4(e, f + i * NP, min(NP, cnt - i * NP), 0);
        }
        pair0 += ta;
        item0 += tb;
    }
    if (threadIdx.x == 0) *n_items = item0;
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int m = p / S, s = p % S, e = expert(p);
        int r = s_first[e];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const unsigned int bits = s_mask[e * W + w];
            r += w < m / 32 ? __popc(bits) : (w == m / 32 ? __popc(bits & ((1u << (m & 31)) - 1u)) : 0);
        }
        pair_row[r] = m;
        out_row[r] = s * T + m;
    }
}

// Pair i's terms: xp[(i * P + p)][K] = xq[(p * T + row)][K]; its scales sp[i][KB] are those of term 0.
__global__ void __launch_bounds__(256) moe_gather_kernel(const uint8_t* __restrict__ xq, const float* __restrict__ sx, const int* __restrict__ pair_row,
                                                         uint8_t* __restrict__ xp, float* __restrict__ sp, int T, int K, int P) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x, m = min(max(pair_row[i], 0), T - 1), n = K / 16;
    for (int c = threadIdx.x; c < P * n; c += blockDim.x) {
        const int p = c / n, k = c % n;
        reinterpret_cast<uint4*>(xp + (static_cast<size_t>(i) * P + p) * K)[k] = reinterpret_cast<const uint4*>(xq + (static_cast<size_t>(p) * T + m) * K)[k];
    }
    for (int b = threadIdx.x; b < K / 128; b += blockDim.x) sp[static_cast<size_t>(i) * (K / 128) + b] = sx[static_cast<size_t>(m) * (K / 128) + b];
}

// One warp per (pair, 128-wide block): h = silu(gate) * up * route weight as P terms hq[(i * P + p)][I], scales hs[i][I / 128].
template <int P>
__global__ void __launch_bounds__(256) moe_pair_act_kernel(const float* __restrict__ gu, const int* __restrict__ out_row, const float* __restrict__ wts,
                                                           uint8_t* __restrict__ hq, float* __restrict__ hs, int I, int S, int T) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, nb = I / 128, item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= T * S * nb) return;
    const int i = item / nb, b = item % nb, o = min(max(out_row[i], 0), T * S - 1);
    const float wt = wts[(o % T) * S + o / T];
    const float* g = gu + static_cast<size_t>(i) * 2 * I + b * 128 + lane * 4;
    const float4 gt = *reinterpret_cast<const float4*>(g), up = *reinterpret_cast<const float4*>(g + I);
    const float v[4] = {silu_f(gt.x) * up.x * wt, silu_f(gt.y) * up.y * wt, silu_f(gt.z) * up.z * wt, silu_f(gt.w) * up.w * wt};
    const float amax = warp_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
    const float scale = fmaxf(amax, 1e-12f) / 448.f, inv = 1.f / scale;
    float r[4] = {v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv};
    uint32_t out[P];
    split4<P>(r, out);
#pragma unroll
    for (int p = 0; p < P; ++p) reinterpret_cast<uint32_t*>(hq + (static_cast<size_t>(i) * P + p) * I + b * 128)[lane] = out[p];
    if (lane == 0) hs[static_cast<size_t>(i) * nb + b] = scale;
}

template <int P>
int launch_group(const CUtensorMap& mw, const CUtensorMap& mx, const GroupArgs& a, cudaStream_t st) {
    if (const cudaError_t e = pipe_budget_install()) return static_cast<int>(e);
    return launch(tc_group_kernel<P>, dim3(2 * sm_count()), dim3(kThreads), static_cast<size_t>(kGroupSmem), st, mw, mx, a);
}

}  // namespace

extern "C" {

// Sorts the chunk's (row, slot) pairs by expert.  ids [T][S], each row's experts distinct; items: int32 [T * S][4], n_items: 1 word,
// pair_row / out_row: [T * S] (row of the pair, and slot * T + row).  terms: as in nexrt_moe_group_gemm.
int nexrt_moe_plan(const void* ids, void* items, void* n_items, void* pair_row, void* out_row, int S, int T, int n_total, int terms, void* stream) {
    if (T < 1 || T > kMaxChunkRows || S < 1 || n_total < 1 || n_total > 8192 || terms < 1 || terms > 3) return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>(n_total) * (kMaxChunkRows / 32 + 1) * 4;
    return launch(moe_plan_kernel, dim3(1), dim3(1024), smem, static_cast<cudaStream_t>(stream), static_cast<const int*>(ids), static_cast<int4*>(items),
                  static_cast<int*>(n_items), static_cast<int*>(pair_row), static_cast<int*>(out_row), S, T, n_total, kGroupCols / terms);
}

// Rows of the pairs in sorted order: xq [terms * T][K], sx [terms * T][K / 128] -> xp [pairs * terms][K], sp [pairs][K / 128].
int nexrt_moe_gather(const void* xq, const void* sx, const void* pair_row, void* xp, void* sp, int pairs, int T, int K, int terms, void* stream) {
    if (pairs < 1 || T < 1 || K % 128 || terms < 1 || terms > 3) return cudaErrorInvalidValue;
    return launch(moe_gather_kernel, dim3(pairs), dim3(256), 0, static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(xq), static_cast<const float*>(sx),
                  static_cast<const int*>(pair_row), static_cast<uint8_t*>(xp), static_cast<float*>(sp), T, K, terms);
}

// out[row(i)][r] = sum_k W[expert(i)][r][k] * x_i[k] for every pair i of the plan: W e4m3 [n_total][R][K] with block scales, xp / sp
// as written by nexrt_moe_gather or nexrt_moe_pair_act, row(i) = out_row[i], or i where out_row is null.
int nexrt_moe_group_gemm(const void* w, const void* w_s, const void* xp, const void* sp, void* out, const void* items, const void* n_items, const void* out_row,
                         int pairs, int n_total, int R, int K, int terms, int* status, void* stream) {
    if (pairs < 1 || n_total < 1 || R % kBM || R < kBM || K % 128 || K < 128 || terms < 1 || terms > 3) return cudaErrorInvalidValue;
    CUtensorMap mw, mx;
    if (!tensor_map(&mw, w, static_cast<uint64_t>(n_total) * R, K, K, kBM, false) ||
        !tensor_map(&mx, xp, static_cast<uint64_t>(pairs) * terms, K, K, kGroupCols, false))
        return cudaErrorInvalidValue;
    GroupArgs a{static_cast<const float*>(w_s), static_cast<const float*>(sp), static_cast<float*>(out), static_cast<const int*>(n_items),
                static_cast<const int4*>(items), static_cast<const int*>(out_row), K / 128, R / kBM, R, status};
    auto st = static_cast<cudaStream_t>(stream);
    return terms == 1 ? launch_group<1>(mw, mx, a, st) : terms == 2 ? launch_group<2>(mw, mx, a, st) : launch_group<3>(mw, mx, a, st);
}

int nexrt_moe_pair_act(const void* gu, const void* out_row, const void* wts, void* hq, void* hs, int I, int S, int T, int terms, void* stream) {
    if (T < 1 || S < 1 || I % 128 || terms < 1 || terms > 3) return cudaErrorInvalidValue;
    const int items = T * S * (I / 128);
    auto go = [&](auto kern) {
        return launch(kern, dim3((items + 7) / 8), dim3(256), 0, static_cast<cudaStream_t>(stream), static_cast<const float*>(gu), static_cast<const int*>(out_row),
                      static_cast<const float*>(wts), static_cast<uint8_t*>(hq), static_cast<float*>(hs), I, S, T);
    };
    return terms == 1 ? go(moe_pair_act_kernel<1>) : terms == 2 ? go(moe_pair_act_kernel<2>) : go(moe_pair_act_kernel<3>);
}

}  // extern "C"
