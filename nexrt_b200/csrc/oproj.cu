// Mixer output projection fused with the tensor-parallel all-reduce and the residual add.
//
//   x[m] += all_reduce_sum_over_ranks( W_out[:, local] @ f(in[m]) )
//
// One kernel does: the input transform f (identity for attention, per-head gated RMSNorm *
// silu(z) for the gated delta net, or the context-parallel LSE merge * sigmoid(gate)), the
// block-scaled FP8 GEMV of this rank's column slice, the in-kernel all-reduce over NVSwitch
// (one 8-byte self-tagged packet per value, published with `multimem.st` or peer stores, summed
// in rank order), and the bf16 residual update.  Every rank ends with a bitwise identical
// residual stream, which is also the "all-gather" that feeds the next projection.
//
// Replaces the reference's LinearFinalOProjFusedPushKernel (nex_n2_5_pro/kernels/linear_attn/
// nex_n2_5_pro_linear_final_o_proj_ctypes.cu:51-259), OProjFusedPushKernel and
// WholeVectorReduceKernel (…full_attn/nex_n2_5_pro_o_proj_reduce_ctypes.cu:51-289), the CP tail
// (…cp_tail_ctypes.cu:117-211) and the M=4/M=8 o_proj kernels (…m4_attn_oproj_fused_ctypes.cu,
// …m8_attn_oproj_ctypes.cu, …m4_gdn_oproj_fused_ctypes.cu, …m8_gdn_oproj_ctypes.cu).
#include "api.h"
#include "epilogue.cuh"
#include "gemv.cuh"
#include "gemv_cta.cuh"
#include "mma_gemv.cuh"
#include "ll.cuh"

namespace nexrt {

struct OProjArgs {
    const float* in;        // [M][K]
    const float* z;         // mode 1: [M][K]; mode 2: gate [M][K]
    const float* gnorm_w;   // mode 1: [hd]
    const uint8_t* w;       // [H][K] fp8
    const float* s;         // [H/128][K/128]
    __nv_bfloat16* x;       // [M][H] residual stream (read-modify-write)
    int H, K, M, mode, hd;
    int overwrite;          // 1: x = reduced projection (no residual add)
    float eps;
    float* partial_out;     // library-baseline arm: fp32 partial sums go here, no exchange, no residual
    LLChannel ch;
    unsigned int site;
    LLChannel cp;           // mode 2: partial inbox of the context-parallel group
    unsigned int cp_site;
    const uint8_t* planes;  // staged form: e4m3 terms [3 M][K] and the row scales [M]
    const float* descale;
};

template <int MB>
__global__ void __launch_bounds__(512, 1) oproj_allreduce_kernel(OProjArgs a) {
    constexpr int U = MB == 1 ? 8 : 4;
    extern __shared__ __align__(16) float smem[];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int row0, row1;
    cta_range(a.H, blockIdx.x, gridDim.x, &row0, &row1);
    const int nrows = row1 - row0, max_rows = (a.H + gridDim.x - 1) / gridDim.x;
    if (nrows) prefetch_l2_range(a.w + static_cast<size_t>(row0) * a.K, static_cast<size_t>(nrows) * a.K);
    const GemvGeom gg = gemv_geom(a.K / 16, blockDim.x);
    float* xs = smem;                                        // [MB][K]
    float* part = xs + static_cast<size_t>(MB) * a.K;        // [max_rows][wpr][MB]
    float* res = part + gemv_part_floats(max_rows, MB, gg);  // [kMaxRows][nrows]
    GemvCta<MB, U, PlainFp8> gemv(PlainFp8{a.w, a.s, a.K}, row0, nrows, a.K);
    gemv.preload();
    pdl_wait();
    LLCall cpcall{0u, 0u};
    if (a.mode == 2) cpcall = ll_begin(a.cp, a.cp_site);
    for (int m0 = 0; m0 < a.M; m0 += MB) {
        const int mb = min(MB, a.M - m0);
        if (m0) __syncthreads();
        if (a.mode == 0) {
            for (int idx = threadIdx.x; idx < mb * a.K; idx += blockDim.x) xs[idx] = a.in[static_cast<size_t>(m0) * a.K + idx];
        } else if (a.mode == 1) {
            // gated RMSNorm per 128-wide head: gnorm_w * o * rsqrt(mean o^2 + eps) * silu(z)
            const int heads = a.K / 128;
            for (int v = warp; v < mb * heads; v += nwarps) {
                const int m = v / heads, h = v % heads;
                const size_t base = static_cast<size_t>(m0 + m) * a.K + h * 128 + lane * 4;
                const float4 o = *reinterpret_cast<const float4*>(a.in + base);
                const float4 zz = *reinterpret_cast<const float4*>(a.z + base);
                const float4 gw = *reinterpret_cast<const float4*>(a.gnorm_w + lane * 4);
                const float inv = rsqrtf(warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w) / 128.f + a.eps);
                float4 r;
                r.x = gw.x * o.x * inv * silu_f(zz.x);
                r.y = gw.y * o.y * inv * silu_f(zz.y);
                r.z = gw.z * o.z * inv * silu_f(zz.z);
                r.w = gw.w * o.w * inv * silu_f(zz.w);
                *reinterpret_cast<float4*>(xs + m * a.K + h * 128 + lane * 4) = r;
            }
        } else {
            // context-parallel merge: for every (row, local head, dim) combine the partial contexts
            // of the cp ranks with their log2-domain LSE weights, then gate.
            const int hd = a.hd, heads = a.K / hd;
            for (int idx = threadIdx.x; idx < mb * a.K; idx += blockDim.x) {
                const int m = idx / a.K, k = idx % a.K, lh = k / hd, d = k % hd;
                const unsigned int base = (static_cast<unsigned int>(m0 + m) * heads + lh) * (hd + 1);
                float lse[kMaxWorld], ctx[kMaxWorld], mx = -INFINITY;
                for (int sr = 0; sr < a.cp.world; ++sr) {
                    unsigned int pl, pc;
                    ll_wait(a.cp, cpcall, sr, base + hd, &pl, kStatusCpTimeout);
                    ll_wait(a.cp, cpcall, sr, base + d, &pc, kStatusCpTimeout);
                    lse[sr] = __uint_as_float(pl);
                    ctx[sr] = __uint_as_float(pc);
                    mx = fmaxf(mx, lse[sr]);
                }
                float num = 0.f, den = 0.f;
                for (int sr = 0; sr < a.cp.world; ++sr) {
                    const float wgt = lse[sr] == -INFINITY ? 0.f : exp2f(lse[sr] - mx);
                    num = fmaf(wgt, ctx[sr], num);
                    den += wgt;
                }
                const float gt = a.z[static_cast<size_t>(m0 + m) * a.K + k];
                xs[m * a.K + k] = (den > 0.f ? num / den : 0.f) * sigmoid_f(gt);
            }
        }
        __syncthreads();
        if (m0 == 0) gemv.run(xs, part);
        else gemv_cta<MB, U>(PlainFp8{a.w, a.s, a.K}, row0, nrows, xs, a.K, part);
        __syncthreads();
        for (int idx = threadIdx.x; idx < nrows * mb; idx += blockDim.x) {
            const int rl = idx / mb, m = idx % mb;
            res[(m0 + m) * nrows + rl] = gemv_result(part, rl, m, MB, gg.wpr);
        }
    }
    __syncthreads();
    allreduce_residual(a.ch, a.site, res, a.M, row0, nrows, a.H, a.x, a.overwrite == 0, a.partial_out);
}

// Four consecutive values k .. k + 3 of input row m (mode 0: plain; mode 1: gated RMSNorm of a 128-wide head, which one warp
// holds; mode 2: context-parallel merge of the group's partials).
template <int MODE>
__device__ __forceinline__ float4 oproj_input4(const OProjArgs& a, int m, int k, const float4& o, const float4& zz, const float4& gw, const LLCall& cpcall) {
    if (MODE == 0) return o;
    if (MODE == 1) {
        const float inv = rsqrtf(warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w) / 128.f + a.eps);
        return make_float4(gw.x * o.x * inv * silu_f(zz.x), gw.y * o.y * inv * silu_f(zz.y), gw.z * o.z * inv * silu_f(zz.z), gw.w * o.w * inv * silu_f(zz.w));
    }
    const int hd = a.hd, heads = a.K / hd;
    const float gate[4] = {zz.x, zz.y, zz.z, zz.w};
    float r[4];
    for (int i = 0; i < 4; ++i) {
        const int lh = (k + i) / hd, d = (k + i) % hd;
        const unsigned int base = (static_cast<unsigned int>(m) * heads + lh) * (hd + 1);
        float lse[kMaxWorld], ctx[kMaxWorld], mx = -INFINITY;
        for (int sr = 0; sr < a.cp.world; ++sr) {
            unsigned int pl, pc;
            ll_wait(a.cp, cpcall, sr, base + hd, &pl, kStatusCpTimeout);
            ll_wait(a.cp, cpcall, sr, base + d, &pc, kStatusCpTimeout);
            lse[sr] = __uint_as_float(pl);
            ctx[sr] = __uint_as_float(pc);
            mx = fmaxf(mx, lse[sr]);
        }
        float num = 0.f, den = 0.f;
        for (int sr = 0; sr < a.cp.world; ++sr) {
            const float wgt = lse[sr] == -INFINITY ? 0.f : exp2f(lse[sr] - mx);
            num = fmaf(wgt, ctx[sr], num);
            den += wgt;
        }
        r[i] = (den > 0.f ? num / den : 0.f) * sigmoid_f(gate[i]);
    }
    return make_float4(r[0], r[1], r[2], r[3]);
}

// Shared memory of the kernel below without and with the fp32 copy of the input rows.
template <int NT> constexpr size_t oproj_smem(int M, int K) {
    return static_cast<size_t>(M) * 3 * (K + kStreamPad) + sizeof(float) * 2 * kStreamWarps * 16 * MmaStream<NT, 8>::TILE_LD;
}

// Tensor-core form: the 8 warps of a CTA split K and walk the CTA's groups of 16 output rows (see MmaStream); the CTA that
// computed the rows reduces them across the ranks and updates the residual.  All rows of the step go through in one pass.
//
// What bounds it is the chain input -> split -> product -> store, not the weights (4 MB per rank at the 8-way shard).  One
// warp computes a whole 128-wide block of one row and the rows' largest magnitudes meet in shared memory, so however many
// rows there are the input takes two barriers (scale known, terms written); staged four rows at a time with a reduction of
// its own per row, eight rows took two passes over the weights and about twenty barriers.  The values wait for the scale in
// shared memory (`keep`), or are computed a second time where that memory would cost the SM its second CTA.
//
// MODE 3: the terms and row scales were made by a kernel in front (oproj_stage_split_kernel) and are only copied in.  Made
// here, they are made again by every CTA, and that - about 150 instructions per block and warp - is what several rows then
// cost.  One B200, 8-way shard (K = 1024), cost of the projection in the layer at 8 rows: 15.7 us staged four rows at a time,
// 12 us made here, 2.5 + 3.9 us with the kernel in front.
template <int NT, int MODE, int NB>
__global__ void __launch_bounds__(MODE == 3 ? 512 : 256, MODE == 3 ? 1 : 2) oproj_allreduce_mma_kernel(OProjArgs a, int keep) {
    using Stream = MmaStream<NT, NB>;
    constexpr int U = MODE == 2 ? 1 : 2;                                  // blocks of a warp in flight (next to the weight ring: 128 registers)
    extern __shared__ __align__(16) float smem[];
    __shared__ unsigned int s_max[kMaxRows];                             // bits of the largest magnitude of each row
    TraceCta tr;
    tr.begin(kTrOproj);
    pdl_launch_dependents();
    // MODE 3: one team of eight warps, or two that share the columns (and then have one tile buffer each)
    const int team = MODE == 3 ? threadIdx.x >> 8 : 0, teams = MODE == 3 ? blockDim.x >> 8 : 1, tid = threadIdx.x & 255;
    const int lane = threadIdx.x & 31, warp = tid >> 5;
    const int nb = a.K / 128, ldx = a.K + kStreamPad, items = a.M * nb;
    float* tiles = smem;                                                  // [2][8][16][TILE_LD]
    constexpr int kTiles = kStreamWarps * 16 * Stream::TILE_LD;
    uint8_t* xq = reinterpret_cast<uint8_t*>(tiles + 2 * kTiles);         // [3 M][ldx]
    float* xs = reinterpret_cast<float*>(xq + static_cast<size_t>(a.M) * 3 * ldx);   // [M][K] (keep)
    if (MODE != 3 && threadIdx.x < kMaxRows) s_max[threadIdx.x] = 0u;
    Stream mw(a.w, a.s, a.K, warp, kStreamWarps);
    int row0 = (static_cast<int>(blockIdx.x) * teams + team) * kRowsPerGroup;
    const int stride = static_cast<int>(gridDim.x) * teams * kRowsPerGroup;
    if (row0 < a.H) mw.preload(row0);
    __syncthreads();
    pdl_wait();
    tr.mark(1);
    LLCall call{0u, 0u}, cpcall{0u, 0u};
    if (a.ch.world > 1) call = ll_begin(a.ch, a.site);
    if (MODE == 2) cpcall = ll_begin(a.cp, a.cp_site);
    // thread (r, m) owns output row r of a group for token row m
    const int er = tid % kRowsPerGroup, em = tid / kRowsPerGroup;
    const bool owner = em < a.M;
    float descale = 0.f;
    if constexpr (MODE == 3) {
        if (owner) descale = a.descale[em];
        stage_columns(xq, ldx, a.planes, 3 * a.M, a.K);
    } else {
    float4 gw = make_float4(1.f, 1.f, 1.f, 1.f);
    if (MODE == 1) gw = *reinterpret_cast<const float4*>(a.gnorm_w + lane * 4);
    // input block v of this warp (row v / nb): what four values of it are made from
    auto request = [&](int v, float4& o, float4& zz) {
        const size_t at = static_cast<size_t>(v) * 128 + lane * 4;
        o = zz = make_float4(0.f, 0.f, 0.f, 0.f);
        if (v < items) {
            if (MODE != 2) o = *reinterpret_cast<const float4*>(a.in + at);
            if (MODE != 0) zz = *reinterpret_cast<const float4*>(a.z + at);
        }
    };
    for (int v0 = warp; v0 < items; v0 += U * kStreamWarps) {
        float4 o[U], zz[U];
#pragma unroll
        for (int u = 0; u < U; ++u) request(v0 + u * kStreamWarps, o[u], zz[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int v = v0 + u * kStreamWarps;
            if (v < items) {                                              // uniform across the warp
                const float4 x4 = oproj_input4<MODE>(a, v / nb, (v % nb) * 128 + lane * 4, o[u], zz[u], gw, cpcall);
                const float mx = warp_max(fmaxf(fmaxf(fabsf(x4.x), fabsf(x4.y)), fmaxf(fabsf(x4.z), fabsf(x4.w))));
                if (lane == 0) atomicMax(&s_max[v / nb], __float_as_uint(mx));
                if (keep) *reinterpret_cast<float4*>(xs + static_cast<size_t>(v) * 128 + lane * 4) = x4;
            }
        }
    }
    __syncthreads();
    // biased exponent of the power of two that brings the row's largest magnitude into [128, 256); 2^8 for a row without one,
    // as act_split has it; capped so that the factor and its inverse are normal numbers
    auto up_exp = [&](int m) {
        const float mx = __uint_as_float(s_max[m]);
        return mx > 0.f && mx < 3.0e38f ? min(261 - static_cast<int>(s_max[m] >> 23), 253) : 135;
    };
    for (int v = warp; v < items; v += kStreamWarps) {
        const int m = v / nb, b = v % nb;
        float4 x4;
        if (keep) {
            x4 = *reinterpret_cast<const float4*>(xs + static_cast<size_t>(v) * 128 + lane * 4);   // this thread's own values
        } else {
            float4 o, zz;
            request(v, o, zz);
            x4 = oproj_input4<MODE>(a, m, b * 128 + lane * 4, o, zz, gw, cpcall);
        }
        const float up = __uint_as_float(static_cast<unsigned int>(up_exp(m)) << 23);
        float r[4] = {x4.x * up, x4.y * up, x4.z * up, x4.w * up};
        uint32_t out[3];
        split4<3>(r, out);
#pragma unroll
        for (int term = 0; term < 3; ++term) *reinterpret_cast<uint32_t*>(xq + static_cast<size_t>(m * 3 + term) * ldx + b * 128 + lane * 4) = out[term];
    }
    if (owner) descale = __uint_as_float(static_cast<unsigned int>(254 - up_exp(em)) << 23);
    }
    __syncthreads();
    for (int buf = team; row0 < a.H; buf ^= teams == 1) {
        const int next = row0 + stride;
        const size_t o = static_cast<size_t>(em) * a.H + row0 + er;
        __nv_bfloat16 res = __ushort_as_bfloat16(0);        // requested before the product and kept as read: a conversion here would wait for it
        if (owner && !a.overwrite) res = a.x[o];
        float d[NT][4];
        mw.group(row0, next < a.H ? next : -1, xq, ldx, 3 * a.M, d);
        // one team: two tile buffers, and the barrier of the next group separates this group's readers from the writers after it
        float* tl = tiles + buf * kTiles;
        mw.store(tl, d);
        asm volatile("bar.sync %0, 256;" ::"r"(1 + team) : "memory");
        tr.mark(2);
        if (owner) {
            const float v = Stream::result(tl, kStreamWarps, er, em, descale);
            if (a.partial_out != nullptr) {
                a.partial_out[o] = v;
            } else {
                const float sum = ll_allreduce_f32(a.ch, call, static_cast<unsigned int>(o), v);
                a.x[o] = __float2bfloat16_rn(a.overwrite ? sum : __bfloat162float(res) + sum);
            }
        }
        if (teams == 2 && next < a.H) asm volatile("bar.sync %0, 256;" ::"r"(1 + team) : "memory");
        row0 = next;
    }
    tr.mark(3);
}

// Staging kernel of an out-projection: one CTA per token row builds the projection's input (mode 0 plain copy, 1 GDN gated
// RMSNorm with z, 2 context-parallel merge of the group's partials) and writes it as three e4m3 planes [3M][K] plus a
// power-of-two scale per row, for the kernel behind it that does the product, the all-reduce and the residual:
// oproj_allreduce_mma_kernel in mode 3, or where asked for the tcgen05 GEMM (nexrt_tc_oproj_allreduce in tc_moe.cu).
__global__ void __launch_bounds__(1024) oproj_stage_split_kernel(OProjArgs a, uint8_t* planes, float* descale_out) {
    extern __shared__ __align__(16) float xs[];          // [K]
    __shared__ float red[32];
    __shared__ float ds[1];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int m = blockIdx.x;
    pdl_wait();
    if (a.mode == 0) {
        for (int idx = threadIdx.x * 4; idx < a.K; idx += blockDim.x * 4)
            *reinterpret_cast<float4*>(xs + idx) = *reinterpret_cast<const float4*>(a.in + static_cast<size_t>(m) * a.K + idx);
    } else if (a.mode == 1) {
        const int heads = a.K / 128;
        const float4 gw = *reinterpret_cast<const float4*>(a.gnorm_w + lane * 4);
        for (int h = warp; h < heads; h += nwarps) {
            const size_t base = static_cast<size_t>(m) * a.K + h * 128 + lane * 4;
            const float4 o = *reinterpret_cast<const float4*>(a.in + base);
            const float4 zz = *reinterpret_cast<const float4*>(a.z + base);
            const float inv = rsqrtf(warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w) / 128.f + a.eps);
            *reinterpret_cast<float4*>(xs + h * 128 + lane * 4) =
                make_float4(gw.x * o.x * inv * silu_f(zz.x), gw.y * o.y * inv * silu_f(zz.y), gw.z * o.z * inv * silu_f(zz.z), gw.w * o.w * inv * silu_f(zz.w));
        }
    } else {
        const LLCall cpcall = ll_begin(a.cp, a.cp_site);
        const int hd = a.hd, heads = a.K / hd;
        for (int k = threadIdx.x; k < a.K; k += blockDim.x) {
            const int lh = k / hd, d = k % hd;
            const unsigned int base = (static_cast<unsigned int>(m) * heads + lh) * (hd + 1);
            float lse[kMaxWorld], ctx[kMaxWorld], mx = -INFINITY;
            for (int sr = 0; sr < a.cp.world; ++sr) {
                unsigned int pl, pc;
                ll_wait(a.cp, cpcall, sr, base + hd, &pl, kStatusCpTimeout);
                ll_wait(a.cp, cpcall, sr, base + d, &pc, kStatusCpTimeout);
                lse[sr] = __uint_as_float(pl);
                ctx[sr] = __uint_as_float(pc);
                mx = fmaxf(mx, lse[sr]);
            }
            float num = 0.f, den = 0.f;
            for (int sr = 0; sr < a.cp.world; ++sr) {
                const float wgt = lse[sr] == -INFINITY ? 0.f : exp2f(lse[sr] - mx);
                num = fmaf(wgt, ctx[sr], num);
                den += wgt;
            }
            xs[k] = (den > 0.f ? num / den : 0.f) * sigmoid_f(a.z[static_cast<size_t>(m) * a.K + k]);
        }
    }
    __syncthreads();
    act_split<3>(planes + static_cast<size_t>(m) * 3 * a.K, xs, 1, a.K, red, ds);
    if (threadIdx.x == 0) descale_out[m] = ds[0];
}

}  // namespace nexrt

using namespace nexrt;

extern "C" int nexrt_oproj_stage_split(const void* in, const void* z, const void* gnorm_w, void* planes, void* descale, int K, int M, int mode, float eps,
                                       int hd, const NexrtLLChannel* cp, unsigned int cp_site, void* stream) {
    mode &= 3;
    if (M < 1 || M > kMaxRows || K % 128 || mode < 0 || mode > 2) return cudaErrorInvalidValue;
    if (mode == 2 && (cp == nullptr || hd <= 0 || K % hd)) return cudaErrorInvalidValue;
    OProjArgs a{};
    a.in = static_cast<const float*>(in); a.z = static_cast<const float*>(z); a.gnorm_w = static_cast<const float*>(gnorm_w);
    a.K = K; a.M = M; a.mode = mode; a.hd = hd; a.eps = eps;
    if (cp) { a.cp = *cp; a.cp_site = cp_site; }
    return launch(oproj_stage_split_kernel, dim3(M), dim3(max(128, min(1024, K / 4))), sizeof(float) * K, static_cast<cudaStream_t>(stream), a, static_cast<uint8_t*>(planes),
                  static_cast<float*>(descale));
}

// Launches the tensor-core form (mode 3: staged terms); -1 when its shared memory does not fit.  The columns of all rows stay
// in shared memory: an unsharded K of 8192 with eight rows just fits, anything wider takes the CUDA-core kernel.
static int launch_oproj_mma(const OProjArgs& a, int mode, cudaStream_t st) {
    const int nt = (3 * a.M + 7) / 8, groups = a.H / kRowsPerGroup;
    const size_t base = nt == 1 ? oproj_smem<1>(a.M, a.K) : (nt == 2 ? oproj_smem<2>(a.M, a.K) : oproj_smem<3>(a.M, a.K)), half = 112 * 1024, all = 226 * 1024;
    if (base > all) return -1;
    const size_t kept = base + sizeof(float) * a.M * a.K;
    const int keep = mode != 3 && kept <= (base <= half ? half : all) ? 1 : 0;
    // what leaves room for two CTAs per SM runs as two; staged terms that do not are shared by the two teams of one CTA (in one
    // team, two groups follow each other there: an unsharded layer of four rows took 72 us, 59.5 with two)
    const int teams = mode == 3 && base > half ? 2 : 1, items = (groups + teams - 1) / teams;
    const int resident = sm_count() * (base <= half ? 2 : 1);
    const int rounds = (items + resident - 1) / resident;
    const dim3 g((items + rounds - 1) / rounds), b(256 * teams);         // as few CTAs as the rounds need: each stages the input once
    auto go = [&](auto kernel) { return launch(kernel, g, b, keep ? kept : base, st, a, keep); };
    // windows of one warp per group: the ring holds two, four or (wide K) eight of them, six beside 24 columns
    const int wpw = (a.K / kWin + kStreamWarps - 1) / kStreamWarps;
    if (nt == 1) {
        auto by_mode = [&](auto plain, auto gated, auto merge, auto staged) { return mode == 0 ? go(plain) : (mode == 1 ? go(gated) : (mode == 2 ? go(merge) : go(staged))); };
        if (wpw <= 2) return by_mode(oproj_allreduce_mma_kernel<1, 0, 2>, oproj_allreduce_mma_kernel<1, 1, 2>, oproj_allreduce_mma_kernel<1, 2, 2>, oproj_allreduce_mma_kernel<1, 3, 2>);
        if (wpw <= 4) return by_mode(oproj_allreduce_mma_kernel<1, 0, 4>, oproj_allreduce_mma_kernel<1, 1, 4>, oproj_allreduce_mma_kernel<1, 2, 4>, oproj_allreduce_mma_kernel<1, 3, 4>);
        return by_mode(oproj_allreduce_mma_kernel<1, 0, 8>, oproj_allreduce_mma_kernel<1, 1, 8>, oproj_allreduce_mma_kernel<1, 2, 8>, oproj_allreduce_mma_kernel<1, 3, 8>);
    }
    if (nt == 2) {
        if (mode != 3) return mode == 0 ? go(oproj_allreduce_mma_kernel<2, 0, 4>) : (mode == 1 ? go(oproj_allreduce_mma_kernel<2, 1, 4>) : go(oproj_allreduce_mma_kernel<2, 2, 4>));
        return wpw <= 2 ? go(oproj_allreduce_mma_kernel<2, 3, 2>) : (wpw <= 4 ? go(oproj_allreduce_mma_kernel<2, 3, 4>) : go(oproj_allreduce_mma_kernel<2, 3, 8>));
    }
    if (mode != 3) return mode == 0 ? go(oproj_allreduce_mma_kernel<3, 0, 4>) : (mode == 1 ? go(oproj_allreduce_mma_kernel<3, 1, 4>) : go(oproj_allreduce_mma_kernel<3, 2, 4>));
    return wpw <= 2 ? go(oproj_allreduce_mma_kernel<3, 3, 2>) : (wpw <= 4 ? go(oproj_allreduce_mma_kernel<3, 3, 4>) : go(oproj_allreduce_mma_kernel<3, 3, 6>));
}

extern "C" int nexrt_oproj_allreduce(const void* in, const void* z, const void* gnorm_w, const void* w, const void* s, void* x, int H, int K,
                                     int M, int mode, float eps, int hd, const NexrtLLChannel* ch, unsigned int site,
                                     const NexrtLLChannel* cp, unsigned int cp_site, int n_cta, void* stream) {
    const int overwrite = (mode & 4) ? 1 : 0;
    mode &= 3;
    if (M < 1 || M > kMaxRows || K % 128 || H % 2 || ch == nullptr || mode < 0 || mode > 2) return cudaErrorInvalidValue;
    if (mode == 2 && (cp == nullptr || hd <= 0 || K % hd)) return cudaErrorInvalidValue;
    if (ch->world > 1 && ch->slots < static_cast<unsigned int>(kMaxRows) * H) return cudaErrorInvalidValue;
    OProjArgs a{};
    a.in = static_cast<const float*>(in); a.z = static_cast<const float*>(z); a.gnorm_w = static_cast<const float*>(gnorm_w);
    a.w = static_cast<const uint8_t*>(w); a.s = static_cast<const float*>(s); a.x = static_cast<__nv_bfloat16*>(x);
    a.H = H; a.K = K; a.M = M; a.mode = mode; a.hd = hd; a.overwrite = overwrite; a.eps = eps; a.ch = *ch; a.site = site;
    a.partial_out = partial_out_buffer();
    if (cp) { a.cp = *cp; a.cp_site = cp_site; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if ((gemv_mode() & 2) && H % 16 == 0) {
        const int e = launch_oproj_mma(a, mode, st);
        if (e >= 0) return e;
    }
    const int mb = M == 1 ? 1 : 4;
    const int max_rows = (H + n_cta - 1) / n_cta;
    const size_t smem = sizeof(float) * (static_cast<size_t>(mb) * K + gemv_part_floats(max_rows, mb, gemv_geom(K / 16, gemv_threads())) +
                                         static_cast<size_t>(kMaxRows) * max_rows);
    dim3 g(n_cta), b(gemv_threads());
    if (mb == 1) return launch(oproj_allreduce_kernel<1>, g, b, smem, st, a);
    return launch(oproj_allreduce_kernel<4>, g, b, smem, st, a);
}

// The same with scratch for the input's terms (planes: e4m3 [3 M][K], descale: fp32 [M]): made once by a kernel of their own
// instead of by every CTA.  The line: several rows always gain (see above); one row gains where K is wide (one B200, a layer with its weights
// from memory, staged / not: K = 8192 41.8 / 44.0 us of attention and 42.7 / 46.5 of gated delta net, K = 4096 28.8 / 29.0 of gated delta
// net; of attention it depends on the kernel in front, see FullAttn).  At 2048 there is no difference, and at 1024 the second node costs
// more than the eight blocks that every CTA computes.
extern "C" int nexrt_oproj_rows_allreduce(const void* in, const void* z, const void* gnorm_w, const void* w, const void* s, void* x, void* planes, void* descale,
                                          int H, int K, int M, int mode, float eps, int hd, const NexrtLLChannel* ch, unsigned int site,
                                          const NexrtLLChannel* cp, unsigned int cp_site, int n_cta, void* stream) {
    const bool staged = M >= 1 && (M >= 2 || K >= 4096) && M <= kMaxRows && (gemv_mode() & 2) && H % 16 == 0 && K % 128 == 0 && ch != nullptr && planes != nullptr && descale != nullptr &&
                        (ch->world <= 1 || ch->slots >= static_cast<unsigned int>(kMaxRows) * H) && oproj_smem<3>(M, K) <= 226 * 1024;
    if (!staged) return nexrt_oproj_allreduce(in, z, gnorm_w, w, s, x, H, K, M, mode, eps, hd, ch, site, cp, cp_site, n_cta, stream);
    if (const int e = nexrt_oproj_stage_split(in, z, gnorm_w, planes, descale, K, M, mode, eps, hd, cp, cp_site, stream)) return e;
    OProjArgs a{};
    a.w = static_cast<const uint8_t*>(w); a.s = static_cast<const float*>(s); a.x = static_cast<__nv_bfloat16*>(x);
    a.H = H; a.K = K; a.M = M; a.mode = 3; a.hd = hd; a.overwrite = (mode & 4) ? 1 : 0; a.eps = eps; a.ch = *ch; a.site = site;
    a.partial_out = partial_out_buffer();
    a.planes = static_cast<const uint8_t*>(planes); a.descale = static_cast<const float*>(descale);
    return launch_oproj_mma(a, 3, static_cast<cudaStream_t>(stream));
}
