// Bayesian PCA group filter and aggregation weights for the active groups of
// one anchor frame (plain form, dual-PCA model).
//
// Reference semantics: transform_vnlb_coupled_samples / transform_vnlb_group,
// filter_vnlb_samples, compute_filter_coefficients,
// accumulate_aggregation_model, finalize_aggregation_weights and
// project_bayes_estimate (src/core/core.cpp:190-412, 578-871, 276-294) on top
// of compute_mean, center_rows, compute_gram_centered,
// topk_symmetric_eigen_jacobi and map_dual_eigenvectors_to_basis
// (src/linalg/linalg.cpp).
//
// Three kernels, each shaped to its parallelism:
//   prepare  a warp or a CTA per group: equality and flat-area tests, the
//            means of the first B rows, the centred model rows (shared memory)
//            and the B x B dual Gram, a 4 x 4 block of pairs per octet of lanes;
//   jacobi   the cyclic Jacobi of many groups per warp, a few lanes per group
//            (a latency-bound chain of dependent rotations, so throughput
//            comes from the number of groups in flight);
//   apply    a warp or a CTA per group: dual -> primal basis, Wiener
//            coefficients, precision and volume, then the retained rows in
//            tiles for their membership scores and shrunken reconstructions,
//            and finally the aggregation weights.
// Samples are addressed through a per-launch table of column offsets
// (channel, t, py, px) -> video offset, so a gather is one add and one load.
// All dot products use the pinned 8-lane order (per-lane fused accumulators,
// then the fixed fold), elementwise updates the CPU's fused/unfused split, and
// the elementary functions are correctly rounded, so results are
// bit-identical to the CPU core -- with one stated exception: the flat-area
// variance (double sums) is reduced in a fixed parallel order, which can move
// its float value by one ulp; that changes the flat decision only when the
// variance lies within one ulp of gamma*sigma^2.
#include <cfloat>

#include "vnlb_kernels.h"

namespace vnlbgpu {
namespace {

constexpr int kApplyThreads = 256;
constexpr int kApplyWarps = kApplyThreads / 32;
constexpr int kRecCols = 8;  // reconstruction columns held in registers per lane (blocks of 256)
constexpr int kPrepareWarps = 4;
constexpr float kEigenFloor = 128.0f * FLT_EPSILON;
constexpr int kTileRows = 4;       // rows of a tile of dot products
constexpr size_t kFilterSharedLimit = 227 * 1024;  // shared memory of one CTA on sm_100
// ... of which prepare_kernel's and the apply kernels' static arrays take this much at most
constexpr size_t kFilterStaticShared = 64;

// dot_contiguous_highway (the pinned 8-lane order) computed by an octet of
// lanes (j = lane & 7): lane j owns accumulator j; the fold follows reduce8.  All 8 lanes return the dot.
// Every lane of the warp must call it.
__device__ __forceinline__ float octet_dot8(const float* l, const float* r, int count, int j) {
    float v = 0.0f;
    int index = 0;
    if (count == kLanes || count == 2 * kLanes) {
        v = __fmul_rn(l[j], r[j]);
        if (count == 2 * kLanes) v = __fmaf_rn(l[kLanes + j], r[kLanes + j], v);
        index = count;
    } else {
        for (; index + kLanes <= count; index += kLanes) v = __fmaf_rn(l[index + j], r[index + j], v);
    }
    v = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, 4, 8));
    v = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, 2, 8));
    v = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, 1, 8));
    float total = __shfl_sync(0xffffffffu, v, 0, 8);
    for (; index < count; ++index) total = __fadd_rn(total, __fmul_rn(l[index], r[index]));
    return total;
}

__device__ __forceinline__ bool fused_column(int col, int count) {
    return count == kLanes || count == 2 * kLanes || col < (count / kLanes) * kLanes;
}

// add_scaled_contiguous_highway element `col` of a row of `count`.
__device__ __forceinline__ float add_scaled_elem(float out, float in, float scale, int col, int count) {
    return fused_column(col, count) ? __fmaf_rn(scale, in, out) : __fadd_rn(out, __fmul_rn(scale, in));
}

// Offset of column col = (channel, t, py, px) from a patch origin.
__device__ __forceinline__ int column_offset(const FilterLaunch& L, int col) {
    const int pd = L.patch_dim;
    const int c = col / pd;
    const int pos = col - c * pd;
    const int pp = L.P * L.P;
    const int t = pos / pp;
    const int rem = pos - t * pp;
    const int py = rem / L.P;
    const int px = rem - py * L.P;
    return ((t * L.channels + c) * L.height + py) * L.width + px;
}

__device__ __forceinline__ size_t row_base(const FilterLaunch& L, const MatchRow& m) {
    return (static_cast<size_t>(m.frame % L.ring) * L.channels * L.height + m.y) * static_cast<size_t>(L.width) + m.x;
}

__device__ __forceinline__ int bmax_of(const FilterLaunch& L) { return min(L.model_cap, L.max_rows); }

__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// One step of the halving fold: keeps `keep`, adds the partner's copy of it.
__device__ __forceinline__ float fold_half(float keep, float send, int mask) {
    return __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, mask));
}

// Folds the octet chains v[row][component]: lane j ends with row r =
// (j & 4) / 2 + (j & 2) / 2 and components 2 (j & 1), 2 (j & 1) + 1.
__device__ __forceinline__ float2 fold_tile(const float2 (&v)[kTileRows][2], int j) {
    float2 a[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const float2 lo = v[r][p], hi = v[r + 2][p];
            a[r][p].x = fold_half((j & 4) ? hi.x : lo.x, (j & 4) ? lo.x : hi.x, 4);
            a[r][p].y = fold_half((j & 4) ? hi.y : lo.y, (j & 4) ? lo.y : hi.y, 4);
        }
    float2 b[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        b[p].x = fold_half((j & 2) ? a[1][p].x : a[0][p].x, (j & 2) ? a[0][p].x : a[1][p].x, 2);
        b[p].y = fold_half((j & 2) ? a[1][p].y : a[0][p].y, (j & 2) ? a[0][p].y : a[1][p].y, 2);
    }
    float2 c;
    c.x = fold_half((j & 1) ? b[1].x : b[0].x, (j & 1) ? b[0].x : b[1].x, 1);
    c.y = fold_half((j & 1) ? b[1].y : b[0].y, (j & 1) ? b[0].y : b[1].y, 1);
    return c;
}

// One m16n8k8 TF32 tensor-core MMA with FP32 accumulation (row-major A,
// column-major B): d += a * b.
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// Dual Gram X X^T / B of up to 16 centred rows (row r, column k at X[r * rs + k *
// cs], D a multiple of 8) on the tensor cores, one warp: A = the rows (16 x 8 per step), B =
// their transpose in tiles of 8 columns; rows and columns past B are zero.
// Lane (g, q) = (lane / 4, lane % 4) holds A rows g, g + 8 at columns q, q + 4
// and the accumulators of rows g, g + 8 at columns 2q, 2q + 1.
__device__ __forceinline__ void gram_tf32(const float* X, int rs, int cs, int B, int D, float scale, float* gram,
                                          int lane) {
    const int g = lane >> 2, q = lane & 3;
    for (int n0 = 0; n0 < B; n0 += 8) {
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int k0 = 0; k0 < D; k0 += 8) {
            uint32_t a[4], b[2];
            a[0] = g < B ? to_tf32(X[g * rs + (k0 + q) * cs]) : 0u;
            a[1] = g + 8 < B ? to_tf32(X[(g + 8) * rs + (k0 + q) * cs]) : 0u;
            a[2] = g < B ? to_tf32(X[g * rs + (k0 + q + 4) * cs]) : 0u;
            a[3] = g + 8 < B ? to_tf32(X[(g + 8) * rs + (k0 + q + 4) * cs]) : 0u;
            const int n = n0 + g;  // B's column n is row n of X
            b[0] = n < B ? to_tf32(X[n * rs + (k0 + q) * cs]) : 0u;
            b[1] = n < B ? to_tf32(X[n * rs + (k0 + q + 4) * cs]) : 0u;
            mma_tf32(acc, a, b);
        }
        const int c0 = n0 + 2 * q;
        const int rows[2] = {g, g + 8};
        for (int h = 0; h < 2; ++h) {
            const int r = rows[h];
            if (r >= B) continue;
            if (c0 < B) gram[r * B + c0] = acc[2 * h] * scale;
            if (c0 + 1 < B) gram[r * B + c0 + 1] = acc[2 * h + 1] * scale;
        }
    }
}

// ---------------------------------------------------------------------------
// prepare: W warps per group.  W = 1 runs four groups per CTA, one per warp;
// W = 4 gives a CTA to one group, for model rows too large for four copies in
// shared memory to leave room for more than a few warps per SM (block 7,
// patch_time 2, YUV: 16 rows of 294 values).  The column sums and the centring
// are the thread's that owns the column and each Gram dot is one octet's chains
// and fold (blocks of 4 x 4 pairs per octet where the columns fit), in the same
// order either way; only the flat-area sums, doubles that the group's warps share
// by rows, differ between W = 1 and W = 4 in their last bits.
template <int W, int kHeld>
__global__ void __launch_bounds__(32 * kPrepareWarps) prepare_kernel(FilterLaunch L) {
    constexpr int kGroups = kPrepareWarps / W;  // groups per CTA
    constexpr int kT = 32 * W;                  // threads per group
    extern __shared__ __align__(16) float sm[];
    __shared__ double s_sums[2 * kPrepareWarps];  // flat-area sums per warp (W > 1)
    static_assert(sizeof(s_sums) <= kFilterStaticShared);
    const int D = L.dim;
    const int Bmax = bmax_of(L);
    int* coloff = reinterpret_cast<int*>(sm);
    size_t* bases_all = reinterpret_cast<size_t*>(sm + ((D + 3) & ~3));  // kGroups * max_rows
    // model row s, column col at X[s * rs + col * cs]: rows at a padded stride
    // (octets on different rows hit different banks), or, for the blocked dual
    // Gram, columns of ldc floats
    const int ldc = L.gram_columns;
    const int rs = ldc > 0 ? 1 : D + 8, cs = ldc > 0 ? ldc : 1;
    const int slot = threadIdx.x / kT;          // this group's slot in the CTA
    const int t = threadIdx.x - slot * kT;      // thread within the group
    float* X = reinterpret_cast<float*>(bases_all + kGroups * L.max_rows + (ldc > 0 ? kGroups * L.max_rows & 1 : 0)) +
               slot * (ldc > 0 ? D * ldc : Bmax * (D + 8));  // model rows; columns start on 16 bytes
    size_t* bases = bases_all + slot * L.max_rows;
    for (int col = threadIdx.x; col < D; col += blockDim.x) coloff[col] = column_offset(L, col);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int gwarp = t >> 5;  // warp within the group
    auto group_sync = [] {
        if constexpr (W == 1) __syncwarp();
        else __syncthreads();
    };
    auto group_any = [](bool p) -> bool {
        if constexpr (W == 1) return __any_sync(0xffffffffu, p);
        else return __syncthreads_or(p) != 0;
    };
    const StageConfig& P = L.cfg;
    const bool final_stage = L.stage == 1;
    const float* model_video = final_stage ? L.basic : L.noisy;
    const bool weights_enabled = P.weight_alpha != 0.0f || P.weight_beta != 0.0f || P.weight_gamma != 0.0f;
    const int active_count = L.counters->active;
    // model v = (active group a, model channel mc): one model per group when
    // the channels are coupled (or the clip has one plane), one per plane
    // otherwise (transform_vnlb_channel, core.cpp:795-808)
    const int models = L.models;
    const size_t hw = static_cast<size_t>(L.height) * L.width;
    const int RD = L.row_dim;
    for (int v = blockIdx.x * kGroups + slot; v < active_count * models; v += gridDim.x * kGroups) {
        group_sync();  // the previous group is done with bases and X
        const int a = v / models;
        const int mc = v - a * models;
        const size_t cb = mc * hw;  // plane offset of this model's channel
        const int g = L.active[a];
        const int S = L.row_counts[g];
        const MatchRow* rows = L.rows + static_cast<size_t>(g) * L.max_rows;
        const int r0 = L.row_offset[a];
        const int B = min(S, L.model_cap);
        for (int i = t; i < S; i += kT) {
            const MatchRow m = rows[i];
            if (mc == 0) {
                L.row_info[r0 + i] = m;
                L.row_group[r0 + i] = a;
            }
            bases[i] = row_base(L, m);
        }
        group_sync();
        // equal group (samples_are_equal / group_is_equal): the first two rows
        // differ in the first columns of nearly every group, which settles it
        bool differs = S <= 1 || (t < D && __ldg(L.noisy + bases[0] + coloff[t]) !=
                                               __ldg(L.noisy + bases[1] + coloff[t]));
        if (!group_any(differs)) {
            for (int col = t; col < D * models; col += kT) {
                const int cm = col / D;  // plane of an uncoupled group (group_is_equal, core.cpp:516-531)
                const float* src = L.noisy + cm * hw + coloff[col - cm * D];
                const float v0 = __ldg(src + bases[0]);
                int i = 1;
                for (; i + 4 <= S; i += 4) {
                    const float x0 = __ldg(src + bases[i]), x1 = __ldg(src + bases[i + 1]);
                    const float x2 = __ldg(src + bases[i + 2]), x3 = __ldg(src + bases[i + 3]);
                    differs |= (x0 != v0) | (x1 != v0) | (x2 != v0) | (x3 != v0);
                }
                for (; i < S; ++i) differs |= __ldg(src + bases[i]) != v0;
            }
        } else {
            differs = true;
        }
        if (!group_any(differs)) {
            // filtered = input, default aggregation model (core.cpp:253-274)
            for (int i = 0; i < S; ++i) {
                const size_t b = bases[i];
                float* out = L.filtered + static_cast<size_t>(r0 + i) * RD + mc * D;
                for (int col = t; col < D; col += kT) out[col] = __ldg(L.noisy + b + cb + coloff[col]);
            }
            const float tau = __fadd_rn(P.weight_epsilon, __fdiv_rn(static_cast<float>(D), static_cast<float>(B)));
            const float lgw = P.weight_alpha == 0.0f ? 0.0f : __fmul_rn(-P.weight_alpha, cr_logf(tau));
            float w = 1.0f;
            if (weights_enabled) {
                float lw = __fadd_rn(0.0f, lgw);
                lw = lw < -80.0f ? -80.0f : (80.0f < lw ? 80.0f : lw);
                w = cr_expf(lw);
            }
            if (mc == 0)
                for (int i = t; i < S; i += kT) L.weights[r0 + i] = w;
            if (t == 0) L.flags[v] = kGroupDone;
            continue;
        }
        // flat area (Final): mean channel variance of the noisy rows, in
        // double.  The warps of the group share a channel's rows; a lane sums
        // its columns of kFlatRows rows at a time (their loads in flight
        // together), then a fixed shuffle tree and the warps in order
        bool flat = false;
        if (final_stage && P.flat_areas) {
            constexpr int kFlatRows = 4;
            const int pd = L.patch_dim;
            const int channels = models > 1 ? models : D / pd;
            const int per_channel = pd * S;
            float variance = 0.0f;
            for (int c = 0; c < channels; ++c) {
                double sum = 0.0, sum2 = 0.0;
                for (int q = lane; q < pd; q += 32) {
                    const float* src = L.noisy + (models > 1 ? c * hw + coloff[q] : coloff[c * pd + q]);
                    for (int i0 = gwarp * kFlatRows; i0 < S; i0 += W * kFlatRows) {
                        float x[kFlatRows];
#pragma unroll
                        for (int k = 0; k < kFlatRows; ++k) x[k] = i0 + k < S ? __ldg(src + bases[i0 + k]) : 0.0f;
#pragma unroll
                        for (int k = 0; k < kFlatRows; ++k) {
                            sum += static_cast<double>(x[k]);
                            sum2 += static_cast<double>(x[k]) * static_cast<double>(x[k]);
                        }
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    sum2 += __shfl_xor_sync(0xffffffffu, sum2, o);
                }
                if constexpr (W > 1) {
                    if (lane == 0) {
                        s_sums[2 * gwarp] = sum;
                        s_sums[2 * gwarp + 1] = sum2;
                    }
                    group_sync();
                    sum = sum2 = 0.0;
                    for (int k = 0; k < W; ++k) {
                        sum += s_sums[2 * k];
                        sum2 += s_sums[2 * k + 1];
                    }
                    group_sync();
                }
                if (per_channel > 1) {
                    const double count = static_cast<double>(per_channel);
                    variance = __fadd_rn(variance, static_cast<float>((sum2 - (sum * sum / count)) / (count - 1.0)));
                }
            }
            if (per_channel > 1) variance = __fdiv_rn(variance, static_cast<float>(channels));
            flat = variance < __fmul_rn(__fmul_rn(P.sigma, P.sigma), P.gamma);
        }
        if (B < min(D, L.rank)) {
            if (t == 0) {
                atomicCAS(L.status, 0, kStatusRankNotCovered);
                L.flags[v] = kGroupSkip;
            }
            continue;
        }
        // model rows, means over the first B rows (compute_mean), centring: a
        // thread owns a column, whose rows' loads are in flight together
        const float inv_b = __fdiv_rn(1.0f, static_cast<float>(B));
        float* means = L.means + static_cast<size_t>(v) * 2 * D;
        if constexpr (kHeld > 0) {
            // up to kHeld rows stay in registers until they are centred
            for (int col = t; col < D; col += kT) {
                const float* src = model_video + cb + coloff[col];
                const float* noisy = L.noisy + cb + coloff[col];
                const bool own_center = final_stage && !flat;  // else the model rows' mean
                float x[kHeld], y[kHeld];
#pragma unroll
                for (int s2 = 0; s2 < kHeld; ++s2) x[s2] = s2 < B ? __ldg(src + bases[s2]) : 0.0f;
                if (own_center)
#pragma unroll
                    for (int s2 = 0; s2 < kHeld; ++s2) y[s2] = s2 < B ? __ldg(noisy + bases[s2]) : 0.0f;
                float mm = 0.0f, mn = 0.0f;
#pragma unroll
                for (int s2 = 0; s2 < kHeld; ++s2)
                    if (s2 < B) mm = __fadd_rn(mm, x[s2]);
                mm = __fmul_rn(mm, inv_b);
                if (own_center) {
#pragma unroll
                    for (int s2 = 0; s2 < kHeld; ++s2)
                        if (s2 < B) mn = __fadd_rn(mn, y[s2]);
                }
                means[col] = mm;
                means[D + col] = own_center ? __fmul_rn(mn, inv_b) : mm;
                float4* out = reinterpret_cast<float4*>(X + col * ldc);
#pragma unroll
                for (int q = 0; q < kHeld / 4; ++q)
                    if (4 * q < B)
                        out[q] = make_float4(__fsub_rn(x[4 * q], mm), __fsub_rn(x[4 * q + 1], mm),
                                             __fsub_rn(x[4 * q + 2], mm), __fsub_rn(x[4 * q + 3], mm));
            }
        } else {
            for (int col = t; col < D; col += kT) {
                const float* src = model_video + cb + coloff[col];
#pragma unroll 8
                for (int s2 = 0; s2 < B; ++s2) X[s2 * rs + col * cs] = __ldg(src + bases[s2]);
                float mm = 0.0f;
#pragma unroll 8
                for (int s2 = 0; s2 < B; ++s2) mm = __fadd_rn(mm, X[s2 * rs + col * cs]);
                mm = __fmul_rn(mm, inv_b);
                float center = mm;  // Basic: noisy mean; Final flat: basic mean
                if (final_stage && !flat) {
                    const float* noisy = L.noisy + cb + coloff[col];
                    float mn = 0.0f;
#pragma unroll 8
                    for (int s2 = 0; s2 < B; ++s2) mn = __fadd_rn(mn, __ldg(noisy + bases[s2]));
                    center = __fmul_rn(mn, inv_b);
                }
                means[col] = mm;
                means[D + col] = center;
#pragma unroll 8
                for (int s2 = 0; s2 < B; ++s2) X[s2 * rs + col * cs] = __fsub_rn(X[s2 * rs + col * cs], mm);
            }
        }
        group_sync();
        if (L.rank > 0) {
            const float scale = __fdiv_rn(1.0f, static_cast<float>(B));
            float* gram = L.gram + static_cast<size_t>(v) * L.nmax * L.nmax;
            if (D >= 64 && B < D && L.mixed && W == 1 && B <= 16 && D % 8 == 0) {
                // chosen forms: TF32 tensor-core Gram, FP32 accumulation
                gram_tf32(X, rs, cs, B, D, scale, gram, lane);
            } else if (ldc > 0) {
                // dual Gram (compute_gram_centered) in blocks of 4 x 4 pairs, an
                // octet per block: lane j runs the pinned chain j of the 16
                // pairs on two 16-byte loads per step, and the folds leave it
                // with row r and two columns of the block
                const int quads = (B + 3) / 4;
                const int blocks = quads * (quads + 1) / 2;
                const int j = lane & 7;
                const int full = D / kLanes;
                const int r = ((j >> 2) << 1) | ((j >> 1) & 1), c2 = 2 * (j & 1);
                for (int e0 = 0; e0 < blocks; e0 += kT / 8) {
                    const int e = min(e0 + (t >> 3), blocks - 1);
                    int qa = 0;
                    while ((qa + 1) * (qa + 2) / 2 <= e) ++qa;
                    const int qb = e - qa * (qa + 1) / 2;
                    float2 acc[4][2];
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = make_float2(0.0f, 0.0f);
                    const float* xa = X + j * ldc + 4 * qa;
                    const float* xb = X + j * ldc + 4 * qb;
#pragma unroll 4
                    for (int m = 0; m < full; ++m) {
                        const float4 a4 = *reinterpret_cast<const float4*>(xa + m * kLanes * ldc);
                        const float4 b4 = *reinterpret_cast<const float4*>(xb + m * kLanes * ldc);
                        const float2 b01 = make_float2(b4.x, b4.y), b23 = make_float2(b4.z, b4.w);
                        acc[0][0] = fma2_rn(dup2(a4.x), b01, acc[0][0]);
                        acc[0][1] = fma2_rn(dup2(a4.x), b23, acc[0][1]);
                        acc[1][0] = fma2_rn(dup2(a4.y), b01, acc[1][0]);
                        acc[1][1] = fma2_rn(dup2(a4.y), b23, acc[1][1]);
                        acc[2][0] = fma2_rn(dup2(a4.z), b01, acc[2][0]);
                        acc[2][1] = fma2_rn(dup2(a4.z), b23, acc[2][1]);
                        acc[3][0] = fma2_rn(dup2(a4.w), b01, acc[3][0]);
                        acc[3][1] = fma2_rn(dup2(a4.w), b23, acc[3][1]);
                    }
                    float2 dot = fold_tile(acc, j);
                    for (int idx = full * kLanes; idx < D; ++idx) {
                        const float x = X[idx * ldc + 4 * qa + r];
                        const float* y = X + idx * ldc + 4 * qb + c2;
                        dot.x = __fadd_rn(dot.x, __fmul_rn(x, y[0]));
                        dot.y = __fadd_rn(dot.y, __fmul_rn(x, y[1]));
                    }
                    const int row = 4 * qa + r;
                    const float vals[2] = {__fmul_rn(scale, dot.x), __fmul_rn(scale, dot.y)};
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int col = 4 * qb + c2 + q;
                        if (row < B && col <= row && e0 + (t >> 3) < blocks) {
                            gram[row * B + col] = vals[q];
                            gram[col * B + row] = vals[q];
                        }
                    }
                }
            } else if (D >= 64 && B < D) {
                // dual Gram (compute_gram_centered): octet k takes pair e0 + k;
                // lane j of the octet runs the pinned chain j (octet_dot8)
                const int pairs = B * (B + 1) / 2;
                const int oct = t >> 3;
                for (int e0 = 0; e0 < pairs; e0 += kT / 8) {
                    const int e = min(e0 + oct, pairs - 1);
                    int r = 0;
                    while ((r + 1) * (r + 2) / 2 <= e) ++r;
                    const int c = e - r * (r + 1) / 2;
                    const float val = __fmul_rn(scale, octet_dot8(X + r * rs, X + c * rs, D, lane & 7));
                    if ((lane & 7) == 0 && e0 + oct < pairs) {
                        gram[r * B + c] = val;
                        gram[c * B + r] = val;
                    }
                }
            } else {
                // covariance (compute_covariance_centered, linalg.cpp:378-412):
                // per sample, row r gets x[r] * x[r..] through
                // add_scaled_contiguous_highway, fused on the full 8-lane chunks of
                // the D - r columns it spans; then scaled, both triangles
                const int entries = D * (D + 1) / 2;
                for (int e = t; e < entries; e += kT) {
                    int r = 0, rem = e;
                    while (rem >= D - r) {
                        rem -= D - r;
                        ++r;
                    }
                    const int c = r + rem;
                    const bool fused = fused_column(rem, D - r);
                    float acc = 0.0f;
                    for (int s2 = 0; s2 < B; ++s2) {
                        const float left = X[s2 * rs + r];
                        const float x = X[s2 * rs + c];
                        acc = fused ? __fmaf_rn(left, x, acc) : __fadd_rn(acc, __fmul_rn(left, x));
                    }
                    const float val = __fmul_rn(acc, scale);
                    gram[r * D + c] = val;
                    gram[c * D + r] = val;
                }
            }
        }
        if (t == 0) L.flags[v] = 0;
    }
}

// The rotation (c, s) that zeroes apq (jacobi_rotate, linalg.cpp:152-196).
// kMixed (chosen forms): in FP64, so that near-degenerate pairs (aqq - app
// tiny against apq) keep their angle; kInline for short unrolled loops.
template <bool kMixed, bool kInline>
__device__ __forceinline__ void jacobi_angle(float app, float aqq, float apq, float& c, float& s) {
    if constexpr (kMixed) {
        const float2 r = kInline ? angle_fp64(app, aqq, apq) : angle_fp64_call(app, aqq, apq);
        c = r.x;
        s = r.y;
    } else {
        const float tau = __fdiv_rn(__fsub_rn(aqq, app), __fmul_rn(2.0f, apq));
        const float t_abs =
            __fdiv_rn(1.0f, __fadd_rn(fabsf(tau), __fsqrt_rn(__fadd_rn(1.0f, __fmul_rn(tau, tau)))));
        const float t = tau < 0.0f ? -t_abs : t_abs;
        c = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(1.0f, __fmul_rn(t, t))));
        s = __fmul_rn(t, c);
    }
}

// ---------------------------------------------------------------------------
// jacobi: topk_symmetric_eigen_jacobi (linalg.cpp:447-519) for matrices of more
// than 32 rows.  A group owns a segment of `seg` lanes (16 or 32, jacobi_shape);
// lane r of the segment owns matrix rows r, r + seg, ...
__global__ void __launch_bounds__(256) jacobi_kernel(FilterLaunch L, int seg, int ld, int gstride) {
    extern __shared__ __align__(16) float sm[];
    const int N = L.nmax;  // largest matrix dimension (model rows, or the dimension for covariance models)
    const int D = L.dim;
    const int R = L.rank;
    const int lane = threadIdx.x & 31;
    const int groups_per_warp = 32 / seg;
    const int slot = (threadIdx.x >> 5) * groups_per_warp + lane / seg;  // group slot in the CTA
    const int r0 = lane % seg;
    float* m = sm + static_cast<size_t>(slot) * gstride;
    float* v = m + N * ld;
    int* order = reinterpret_cast<int*>(v + N * ld);
    const int models_total = L.counters->active * L.models;
    const int slots_per_cta = (blockDim.x >> 5) * groups_per_warp;
    for (int base = blockIdx.x * slots_per_cta; base < models_total; base += gridDim.x * slots_per_cta) {
        const int a = base + slot;  // model index (group x model channel)
        bool valid = a < models_total && R > 0;
        int B = 0;  // matrix dimension: the dual Gram's B, or the covariance's D
        if (valid) {
            valid = L.flags[a] == 0;
            const int Bm = min(L.row_counts[L.active[a / L.models]], L.model_cap);
            B = (D >= 64 && Bm < D) ? Bm : D;  // use_dual_pca (core.cpp:656-658)
        }
        if (!valid) B = 0;
        const float* gram = L.gram + static_cast<size_t>(max(a, 0)) * N * N;
        float mx = 0.0f;
        for (int r = r0; r < B; r += seg) {
            for (int c = 0; c < B; ++c) {
                const float x = gram[r * B + c];
                m[r * ld + c] = x;
                v[r * ld + c] = r == c ? 1.0f : 0.0f;
                mx = std_max(mx, fabsf(x));
            }
        }
        for (int o = seg / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float threshold = std_max(0.0f, __fmul_rn(64.0f * FLT_EPSILON, std_max(1.0f, mx)));
        __syncwarp();
        if (__any_sync(0xffffffffu, B > 1)) {
            for (int sweep = 0; sweep < 64; ++sweep) {
                float off = 0.0f;
                for (int r = r0; r < B; r += seg)
                    for (int c = r + 1; c < B; ++c) off = std_max(off, fabsf(m[r * ld + c]));
                for (int o = seg / 2; o > 0; o >>= 1) off = fmaxf(off, __shfl_xor_sync(0xffffffffu, off, o));
                const bool busy = B > 1 && !(off <= threshold);
                if (!__any_sync(0xffffffffu, busy)) break;
                for (int p = 0; p + 1 < N; ++p) {
                    for (int q = p + 1; q < N; ++q) {
                        bool rot = false;
                        float app = 0.0f, aqq = 0.0f, apq = 0.0f;
                        if (busy && q < B) {
                            apq = m[p * ld + q];
                            rot = fabsf(apq) > threshold && apq != 0.0f;
                            if (rot) {
                                app = m[p * ld + p];
                                aqq = m[q * ld + q];
                            }
                        }
                        __syncwarp();
                        if (rot) {
                            float c, s;
                            if (L.mixed) jacobi_angle<true, true>(app, aqq, apq, c, s);
                            else jacobi_angle<false, true>(app, aqq, apq, c, s);
                            for (int r = r0; r < B; r += seg) {
                                if (r != p && r != q) {
                                    const float arp = m[r * ld + p];
                                    const float arq = m[r * ld + q];
                                    const float nrp = __fsub_rn(__fmul_rn(c, arp), __fmul_rn(s, arq));
                                    const float nrq = __fadd_rn(__fmul_rn(s, arp), __fmul_rn(c, arq));
                                    m[r * ld + p] = nrp;
                                    m[p * ld + r] = nrp;
                                    m[r * ld + q] = nrq;
                                    m[q * ld + r] = nrq;
                                }
                                const float vrp = v[r * ld + p];
                                const float vrq = v[r * ld + q];
                                v[r * ld + p] = __fsub_rn(__fmul_rn(c, vrp), __fmul_rn(s, vrq));
                                v[r * ld + q] = __fadd_rn(__fmul_rn(s, vrp), __fmul_rn(c, vrq));
                                const float cc = __fmul_rn(c, c), ss = __fmul_rn(s, s);
                                const float cs2 = __fmul_rn(2.0f, __fmul_rn(c, s));
                                if (r == p) {
                                    m[p * ld + p] = __fadd_rn(__fsub_rn(__fmul_rn(cc, app), __fmul_rn(cs2, apq)),
                                                                __fmul_rn(ss, aqq));
                                    m[p * ld + q] = 0.0f;
                                } else if (r == q) {
                                    m[q * ld + q] = __fadd_rn(__fadd_rn(__fmul_rn(ss, app), __fmul_rn(cs2, apq)),
                                                                __fmul_rn(cc, aqq));
                                    m[q * ld + p] = 0.0f;
                                }
                            }
                        }
                        __syncwarp();
                    }
                }
            }
        }
        // stable sort of the diagonal (descending), canonicalised top-rank
        // eigenvectors (canonicalize_vector_row, linalg.cpp:198-227).  NaN
        // beside numbers has no place in that order: positions coincide, and
        // the ones left over keep an index of their own
        for (int r = r0; r < B; r += seg) order[r] = r;
        __syncwarp();
        for (int r = r0; r < B; r += seg) {
            const float dr = m[r * ld + r];
            int pos = 0;
            for (int j = 0; j < B; ++j) {
                const float dj = m[j * ld + j];
                if (dj > dr || (j < r && !(dr > dj))) ++pos;
            }
            order[pos] = r;
        }
        __syncwarp();
        if (valid) {
            float* eig = L.eig + static_cast<size_t>(a) * R;
            float* dual = L.dual + static_cast<size_t>(a) * R * N;
            for (int out = r0; out < R; out += seg) {
                const int src = order[out];
                eig[out] = m[src * ld + src];
                float norm2 = 0.0f, best = 0.0f;
                int pivot = 0;
                for (int r = 0; r < B; ++r) {
                    const float x = v[r * ld + src];
                    norm2 = __fadd_rn(norm2, __fmul_rn(x, x));
                    const float ax = fabsf(x);
                    if (ax > best) {
                        best = ax;
                        pivot = r;
                    }
                }
                float sc = 1.0f;
                const bool scale = !(norm2 <= FLT_MIN);
                if (scale) {
                    sc = __fdiv_rn(1.0f, __fsqrt_rn(norm2));
                    if (v[pivot * ld + src] < 0.0f) sc = -sc;
                }
                for (int r = 0; r < B; ++r) {
                    const float x = v[r * ld + src];
                    dual[out * N + r] = scale ? __fmul_rn(x, sc) : x;
                }
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// jacobi, kSeg lanes per group, for matrices up to N x N (N = 8 to 32).  The
// rotations of a group are one chain of dependent divisions and square roots:
// latency bounds it (14k groups of 16 rows: issue slots 25% busy, 49% with FP64
// angles, whose pipe is 16% busy; a warp waits for its own last result), so as
// many groups as fit in shared memory are in flight, and few lanes repeat each
// angle.  Against jacobi_kernel (B200, one launch alone, the lanes per group that
// are launched): N = 8, 32k groups 155 -> 81 us; N = 16, 57k groups 1.08 -> 0.66
// ms, 0.6k groups 421 -> 218 us; with FP64 angles, 130k groups, 5.0 -> 2.4 ms.
// The strict upper triangle, the diagonal and the vectors lie in shared memory as
// [element][group].  Lane h owns rows i kSeg + h; its part of row p and of vector
// p stays in registers while q runs over an unrolled loop, and the samples a
// rotation will need are loaded before its angle is known.
// For row r = p the update works on the stale copy of (p, q); the write-back of
// row p replaces it.  Same rotations in the same order on the same values as
// jacobi_kernel, element by element.
constexpr size_t jacobi_small_bytes(int N, int seg) {
    return static_cast<size_t>(N * (N - 1) / 2 + N + N * N) * (32 / seg) * sizeof(float);
}

template <int N, int kSeg, bool kMixed>
__global__ void __launch_bounds__(32) jacobi_small_kernel(FilterLaunch L) {
    extern __shared__ __align__(16) float sm[];
    constexpr int kTri = N * (N - 1) / 2;
    constexpr int kG = 32 / kSeg;  // groups per warp: lane = h * kG + group
    constexpr int kRows = N / kSeg;
    const int lane = threadIdx.x;
    const int gi = lane % kG, h = lane / kG;
    float* tri = sm + gi;            // (r, c), r < c, at tri_at(r, c)
    float* diag = tri + kTri * kG;   // [N]
    float* vec = diag + N * kG;      // [vector][row]
    const auto tri_at = [](int r, int c) { return (r * (2 * N - r - 1) / 2 + c - r - 1) * kG; };
    const int total = L.counters->active * L.models;
    const int a = blockIdx.x * kG + gi;
    if (blockIdx.x * kG >= total) return;
    const int R = L.rank, D = L.dim, M = L.nmax;  // M: stride of the stored matrices and vectors
    const bool valid = a < total && L.flags[a] == 0;
    int B = 0;  // matrix dimension: the dual Gram's B, or the covariance's D
    if (valid) {
        const int Bm = min(L.row_counts[L.active[a / L.models]], L.model_cap);
        B = (D >= 64 && Bm < D) ? Bm : D;  // use_dual_pca (core.cpp:656-658)
    }
    const float* gram = L.gram + static_cast<size_t>(a) * M * M;
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int r = i * kSeg + h;
        if (B == N && M == N) {  // rows of whole 16-byte units
#pragma unroll
            for (int c0 = 0; c0 < N; c0 += 4) {
                if (c0 + 3 < i * kSeg) continue;
                const float4 q = __ldg(reinterpret_cast<const float4*>(gram + r * N + c0));
                const float x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (c0 + k < r) continue;
                    mx = std_max(mx, fabsf(x[k]));
                    *(c0 + k == r ? diag + r * kG : tri + tri_at(r, c0 + k)) = x[k];
                }
            }
        } else {
            for (int c = r; c < N; ++c) {
                const float x = r < B && c < B ? gram[r * B + c] : 0.0f;
                mx = std_max(mx, fabsf(x));
                *(c == r ? diag + r * kG : tri + tri_at(r, c)) = x;
            }
        }
#pragma unroll
        for (int c = 0; c < N; ++c) vec[(c * N + r) * kG] = r == c ? 1.0f : 0.0f;
    }
#pragma unroll
    for (int o = kG; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float threshold = std_max(0.0f, __fmul_rn(64.0f * FLT_EPSILON, std_max(1.0f, mx)));
    int row_of[kRows];  // (r, c) for r < c at row_of[i] + c * kG
#pragma unroll
    for (int i = 0; i < kRows; ++i) row_of[i] = tri_at(i * kSeg + h, 0);
    __syncwarp();
    for (int sweep = 0; sweep < 64; ++sweep) {
        float off = 0.0f;
#pragma unroll 8
        for (int e = h; e < kTri; e += kSeg) off = std_max(off, fabsf(tri[e * kG]));
#pragma unroll
        for (int o = kG; o < 32; o <<= 1) off = fmaxf(off, __shfl_xor_sync(0xffffffffu, off, o));
        const bool busy = B > 1 && !(off <= threshold);
        if (!__any_sync(0xffffffffu, busy)) break;
#pragma unroll 1
        for (int p = 0; p + 1 < N; ++p) {
            float ap[kRows], vp[kRows];
            const int row_p = tri_at(p, 0);
            float app = diag[p * kG];
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const int r = i * kSeg + h;
                ap[i] = r == p ? 0.0f : tri[r < p ? row_of[i] + p * kG : row_p + r * kG];
                vp[i] = vec[(p * N + r) * kG];
            }
#pragma unroll
            for (int q = 1; q < N; ++q) {
                if (q <= p) continue;
                const float apq = __shfl_sync(0xffffffffu, ap[q / kSeg], (q % kSeg) * kG + gi);
                const bool rot = busy && q < B && fabsf(apq) > threshold && apq != 0.0f;
                if (!__any_sync(0xffffffffu, rot)) continue;
                const float aqq = diag[q * kG];
                float* at[kRows];
                float arq[kRows], vrq[kRows];
#pragma unroll
                for (int i = 0; i < kRows; ++i) {
                    // row r against column q: above the diagonal, below it, or
                    // (in the block of q) either, by lane; r = q reads (and
                    // does not write) its own entry of vector q instead
                    const int r = i * kSeg + h;
                    at[i] = tri + (i * kSeg + kSeg <= q ? row_of[i] + q * kG
                                   : i * kSeg > q        ? tri_at(q, 0) + r * kG
                                   : r < q               ? row_of[i] + q * kG
                                   : r > q               ? tri_at(q, 0) + r * kG
                                                         : (kTri + N + q * N + r) * kG);
                    arq[i] = *at[i];
                    vrq[i] = vec[(q * N + r) * kG];
                }
                float dq = 0.0f;
                if (rot) {
                    float c, s;
                    jacobi_angle<kMixed, N <= 8>(app, aqq, apq, c, s);
#pragma unroll
                    for (int i = 0; i < kRows; ++i) {
                        const bool own = i == q / kSeg && i * kSeg + h == q;
                        const float arp = ap[i];
                        const float nrp = __fsub_rn(__fmul_rn(c, arp), __fmul_rn(s, arq[i]));
                        ap[i] = own ? 0.0f : nrp;
                        if (!own) *at[i] = __fadd_rn(__fmul_rn(s, arp), __fmul_rn(c, arq[i]));
                        const float vrp = vp[i];
                        vp[i] = __fsub_rn(__fmul_rn(c, vrp), __fmul_rn(s, vrq[i]));
                        vec[(q * N + i * kSeg + h) * kG] = __fadd_rn(__fmul_rn(s, vrp), __fmul_rn(c, vrq[i]));
                    }
                    const float cc = __fmul_rn(c, c), ss = __fmul_rn(s, s);
                    const float cs2 = __fmul_rn(2.0f, __fmul_rn(c, s));
                    dq = __fadd_rn(__fadd_rn(__fmul_rn(ss, app), __fmul_rn(cs2, apq)), __fmul_rn(cc, aqq));
                    app = __fadd_rn(__fsub_rn(__fmul_rn(cc, app), __fmul_rn(cs2, apq)), __fmul_rn(ss, aqq));
                }
                if constexpr (kSeg > 1) __syncwarp();
                if (rot && h == 0) diag[q * kG] = dq;  // every lane has read the old one; read again at the next p
            }
            if (h == 0) diag[p * kG] = app;
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const int r = i * kSeg + h;
                if (r != p) tri[r < p ? row_of[i] + p * kG : row_p + r * kG] = ap[i];
                vec[(p * N + r) * kG] = vp[i];
            }
            __syncwarp();
        }
    }
    // stable sort of the diagonal (descending), canonicalised top-rank
    // eigenvectors (canonicalize_vector_row, linalg.cpp:198-227); the sorted
    // order goes where the triangle was (positions that NaN leaves over keep an
    // index of their own)
    for (int r = h; r < B; r += kSeg) tri[r * kG] = __int_as_float(r);
    __syncwarp();
    for (int r = h; r < B; r += kSeg) {
        const float dr = diag[r * kG];
        int pos = 0;
        for (int j = 0; j < B; ++j) {
            const float dj = diag[j * kG];
            if (dj > dr || (j < r && !(dr > dj))) ++pos;
        }
        tri[pos * kG] = __int_as_float(r);
    }
    __syncwarp();
    if (!valid) return;
    float* eig = L.eig + static_cast<size_t>(a) * R;
    float* dual = L.dual + static_cast<size_t>(a) * R * M;
    for (int out = h; out < R; out += kSeg) {
        const int src = __float_as_int(tri[out * kG]);
        const float* v = vec + src * N * kG;
        eig[out] = diag[src * kG];
        float x[N];
        float norm2 = 0.0f, best = 0.0f, lead = 0.0f;
#pragma unroll
        for (int r = 0; r < N; ++r) {
            x[r] = 0.0f;
            if (r < B) {
                x[r] = v[r * kG];
                norm2 = __fadd_rn(norm2, __fmul_rn(x[r], x[r]));
                if (r == 0) lead = x[r];
                if (fabsf(x[r]) > best) {
                    best = fabsf(x[r]);
                    lead = x[r];
                }
            }
        }
        if (!(norm2 <= FLT_MIN)) {
            float sc = __fdiv_rn(1.0f, __fsqrt_rn(norm2));
            if (lead < 0.0f) sc = -sc;
#pragma unroll
            for (int r = 0; r < N; ++r) x[r] = __fmul_rn(x[r], sc);
        }
        if (B == N && M == N) {
#pragma unroll
            for (int r = 0; r < N; r += 4)
                *reinterpret_cast<float4*>(dual + out * N + r) = make_float4(x[r], x[r + 1], x[r + 2], x[r + 3]);
        } else {
#pragma unroll
            for (int r = 0; r < N; ++r)
                if (r < B) dual[out * M + r] = x[r];
        }
    }
}

// One model's term of a row's log weight (accumulate_aggregation_model,
// core.cpp:326-412): the group weight, minus beta times the membership.
__device__ __forceinline__ float model_log_weight(const StageConfig& P, bool membership_on, float lgw, float volume,
                                                  float score, float min_score) {
    if (P.weight_alpha == 0.0f && P.weight_beta == 0.0f) return 0.0f;
    if (!membership_on) return lgw;
    const float diff = __fsub_rn(score, min_score);
    const float membership = __fadd_rn(diff > 0.0f ? diff : 0.0f, volume);
    return __fsub_rn(lgw, __fmul_rn(P.weight_beta, membership));
}

// ---------------------------------------------------------------------------
// apply: one CTA per group.  Shared layout (floats unless noted):
//   coloff[D] (int), means[2D], X[B][ldx] centred model rows, basis[R][ldb],
//   dual[R*Bmax], per-component scalars (5R), scores[max_rows],
//   per-warp scratch (3 rows of ldb), row bases[max_rows] (size_t).
// Row strides are padded (ldx = D + 1, ldb = D + 8) so that lanes reading
// different rows at the same column hit different banks.
struct ApplyLayout {
    int D, Bmax, R, ldx, ldb, colpad;
    size_t means, X, basis, dual, scal, scores, scratch, bases, bytes;
};

__host__ __device__ inline ApplyLayout apply_layout(int D, int Bmax, int R, int max_rows, int warps) {
    ApplyLayout a{};
    a.D = D;
    a.Bmax = Bmax;
    a.R = R;
    a.ldx = D + 1;
    a.ldb = D + 8;
    a.colpad = (D + 3) & ~3;
    size_t off = static_cast<size_t>(a.colpad);
    a.means = off;   off += 2 * static_cast<size_t>(D);
    a.basis = off;   off += static_cast<size_t>(R) * a.ldb;
    a.dual = off;    off += static_cast<size_t>(R) * Bmax;
    a.scal = off;    off += 5 * static_cast<size_t>(R);
    a.scores = off;  off += static_cast<size_t>(max_rows);
    a.scratch = off;
    // the centred model rows are read only while the basis is built,
    // before any warp uses its row scratch: they share the space
    a.X = off;
    const size_t rows = static_cast<size_t>(warps) * (2 * a.ldb + R + 1);
    const size_t model = static_cast<size_t>(Bmax) * a.ldx;
    off += rows > model ? rows : model;
    off = (off + 1) & ~static_cast<size_t>(1);
    a.bases = off;   off += 2 * static_cast<size_t>(max_rows);
    a.bytes = off * sizeof(float);
    return a;
}

// The pinned 8-lane fold of an octet's chains as an xor butterfly: every lane
// of the octet ends with ((v0 + v4) + (v2 + v6)) + ((v1 + v5) + (v3 + v7)),
// the same additions as reduce8 (each one commutative).
__device__ __forceinline__ float octet_fold(float v) {
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
    return __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
}

// One row per warp with the components four at a time: any shape.
__global__ void __launch_bounds__(kApplyThreads, 3) apply_kernel(FilterLaunch L) {
    extern __shared__ __align__(16) float sm[];
    const int D = L.dim;
    const int Bmax = bmax_of(L);
    const int R = L.rank;
    const ApplyLayout lay = apply_layout(D, Bmax, R, L.max_rows, kApplyWarps);
    const int ldx = lay.ldx, ldb = lay.ldb;
    int* coloff = reinterpret_cast<int*>(sm);
    float* means = sm + lay.means;  // membership mean, reconstruction centre
    float* X = sm + lay.X;
    float* basis = sm + lay.basis;
    float* dual = sm + lay.dual;
    float* eig = sm + lay.scal;     // eigenvalues
    float* coef = eig + R;          // Wiener coefficients
    float* denom = coef + R;        // signal eigenvalue + membership noise
    float* inv_sqrt = denom + R;    // 1 / sqrt(eigenvalue)
    float* terms = inv_sqrt + R;    // log1p(signal / membership noise)
    float* scores = sm + lay.scores;
    float* scratch = sm + lay.scratch;
    size_t* bases = reinterpret_cast<size_t*>(sm + lay.bases);
    __shared__ float s_misc[4];
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    for (int col = tid; col < D; col += kApplyThreads) coloff[col] = column_offset(L, col);
    const StageConfig& P = L.cfg;
    const bool final_stage = L.stage == 1;
    const float* model_video = final_stage ? L.basic : L.noisy;
    const bool weights_enabled = P.weight_alpha != 0.0f || P.weight_beta != 0.0f || P.weight_gamma != 0.0f;
    const float sigma2 = __fmul_rn(__fmul_rn(P.beta, P.sigma), P.sigma);
    const float model_noise2 = final_stage ? __fmul_rn(__fmul_rn(P.beta, P.sigma_basic), P.sigma_basic) : sigma2;
    const float match_sigma = final_stage ? P.sigma_basic : P.sigma;
    const float mem2 = std_max(__fmul_rn(match_sigma, match_sigma),
                               __fmul_rn(__fmul_rn(P.membership_noise_floor, P.sigma), P.sigma));
    const bool membership_on = P.weight_beta != 0.0f;
    const int active_count = L.counters->active;
    const int models = L.models;  // models per group (planes when uncoupled)
    const size_t hw = static_cast<size_t>(L.height) * L.width;
    __syncthreads();
    for (int mi = blockIdx.x; mi < active_count * models; mi += gridDim.x) {
        if (L.flags[mi] != 0) continue;  // uniform: equal groups are done, skipped ones reported
        const int a = mi / models;
        const int mc = mi - a * models;
        const int g = L.active[a];
        const int S = L.row_counts[g];
        const MatchRow* rows = L.rows + static_cast<size_t>(g) * L.max_rows;
        const int r0 = L.row_offset[a];
        const int B = min(S, L.model_cap);
        const float* gm = L.means + static_cast<size_t>(mi) * 2 * D;
        for (int i = tid; i < 2 * D; i += kApplyThreads) means[i] = gm[i];
        const int N = L.nmax;  // row stride of the eigenvector rows
        const bool dual_model = D >= 64 && B < D;  // use_dual_pca (core.cpp:656-658)
        for (int i = tid; i < R * Bmax; i += kApplyThreads)
            dual[i] = L.dual[static_cast<size_t>(mi) * R * N + (i / Bmax) * N + i % Bmax];
        // row bases of this model's plane
        for (int i = tid; i < S; i += kApplyThreads) bases[i] = row_base(L, rows[i]) + mc * hw;
        // per-component scalars, computed once per group (same operations as
        // the CPU, which recomputes them where it uses them)
        for (int c = tid; c < R; c += kApplyThreads) {
            const float lambda = L.eig[static_cast<size_t>(mi) * R + c];
            eig[c] = lambda;
            const float diff = __fsub_rn(lambda, model_noise2);
            const float signal = diff > 0.0f ? diff : 0.0f;
            denom[c] = __fadd_rn(signal, mem2);
            inv_sqrt[c] = lambda > kEigenFloor ? __fdiv_rn(1.0f, __fsqrt_rn(lambda)) : 0.0f;
            terms[c] = (membership_on && signal > 0.0f) ? cr_log1pf(__fdiv_rn(signal, mem2)) : 0.0f;
            const float sigma_basic2 = final_stage ? model_noise2 : sigma2;
            const float threshold = __fmul_rn(P.variance_threshold, sigma2);
            float variance = lambda;
            if (sigma_basic2 > 0.0f) variance = __fsub_rn(variance, std_min(variance, sigma_basic2));
            coef[c] = variance > threshold ? __fdiv_rn(1.0f, __fadd_rn(1.0f, __fdiv_rn(sigma2, variance))) : 0.0f;
        }
        __syncthreads();
        const float* member_mean = means;
        const float* center_vec = means + D;
        if (R > 0 && !dual_model) {
            // covariance model: the canonicalised eigenvectors are the basis
            for (int b = warp; b < R; b += kApplyWarps)
                for (int col = lane; col < D; col += 32)
                    basis[b * ldb + col] = L.dual[static_cast<size_t>(mi) * R * N + static_cast<size_t>(b) * N + col];
            __syncthreads();
        }
        if (R > 0 && dual_model) {
            // centred model rows (compute_mean + center_rows of the first B rows)
            for (int s = warp; s < B; s += kApplyWarps) {
                const float* src = model_video + bases[s];
                for (int col = lane; col < D; col += 32)
                    X[s * ldx + col] = __fsub_rn(__ldg(src + coloff[col]), member_mean[col]);
            }
            __syncthreads();
            // dual -> primal basis (map_dual_eigenvectors_to_basis): one output
            // per lane, the samples accumulated in order
            for (int b = warp; b < R; b += kApplyWarps) {
                const bool live = eig[b] > kEigenFloor;
                for (int col = lane; col < D; col += 32) {
                    float acc = 0.0f;
                    if (live) {
                        const bool fused = fused_column(col, D);
                        for (int s = 0; s < B; ++s) {
                            const float x = X[s * ldx + col];
                            const float w = dual[b * Bmax + s];
                            acc = fused ? __fmaf_rn(w, x, acc) : __fadd_rn(acc, __fmul_rn(w, x));
                        }
                        acc = __fmul_rn(acc, inv_sqrt[b]);
                    }
                    basis[b * ldb + col] = acc;
                }
            }
            __syncthreads();
            for (int b = warp; b < R; b += kApplyWarps) {
                if (!(eig[b] > kEigenFloor)) continue;
                float* row = basis + b * ldb;
                const float norm2 = octet_dot8(row, row, D, lane & 7);
                __syncwarp();
                if (norm2 <= kEigenFloor) {
                    for (int col = lane; col < D; col += 32) row[col] = 0.0f;
                } else {
                    const float sc = __fdiv_rn(1.0f, __fsqrt_rn(norm2));
                    for (int col = lane; col < D; col += 32) row[col] = __fmul_rn(row[col], sc);
                }
            }
        }
        // group precision and volume (group_precision_tau, core.cpp:222-241,
        // 346-358): the terms are ready, the sums run in component order
        if (tid == 0) {
            float trace = 0.0f, volume = 0.0f;
            for (int c = 0; c < R; ++c) {
                const float diff = __fsub_rn(eig[c], model_noise2);
                const float lambda = diff > 0.0f ? diff : 0.0f;
                if (lambda > 0.0f) {
                    trace = __fadd_rn(trace, __fdiv_rn(lambda, __fadd_rn(lambda, sigma2)));
                    volume = __fadd_rn(volume, terms[c]);
                }
            }
            const float tau = __fadd_rn(
                __fadd_rn(P.weight_epsilon, __fdiv_rn(static_cast<float>(D), static_cast<float>(B))), trace);
            s_misc[0] = P.weight_alpha == 0.0f ? 0.0f : __fmul_rn(-P.weight_alpha, cr_logf(tau));
            s_misc[1] = __fdiv_rn(volume, static_cast<float>(D));
        }
        __syncthreads();
        const float lgw = s_misc[0];
        const float volume = s_misc[1];
        // per row: membership score and reconstruction.  In the Basic stage the
        // membership row and the reconstruction row are the same centred noisy
        // row, so its projections serve both.
        float* u = scratch + warp * (2 * ldb + R + 1);  // centred membership row
        float* v = u + ldb;                             // centred noisy row (Final)
        float* proj = v + ldb;                          // projections for the reconstruction
        const int j8 = lane & 7;
        const int oct = lane >> 3;
        const float score_scale = __fsqrt_rn(__fmul_rn(2.0f, static_cast<float>(D)));
        for (int i = warp; i < S; i += kApplyWarps) {
            const size_t b = bases[i];
            for (int col = lane; col < D; col += 32) {
                const float xn = __ldg(L.noisy + b + coloff[col]);
                if (final_stage) {
                    u[col] = __fsub_rn(__ldg(L.basic + b + coloff[col]), member_mean[col]);
                    v[col] = __fsub_rn(xn, center_vec[col]);
                } else {
                    u[col] = __fsub_rn(xn, member_mean[col]);
                }
            }
            __syncwarp();
            float distance = 0.0f, projected = 0.0f, norm2 = 0.0f;
            // pass over c0 = -1 (norm), 0, 4, ...: octet k computes component c0 + k
            for (int c0 = membership_on ? -1 : 0; c0 < R; c0 += 4) {
                const int c = min(c0 + oct, R - 1);
                const float dm = (membership_on || !final_stage) ? octet_dot8(u, c < 0 ? u : basis + c * ldb, D, j8)
                                                                 : 0.0f;
                const float dr = final_stage ? octet_dot8(v, basis + max(c, 0) * ldb, D, j8) : dm;
                for (int k = 0; k < 4; ++k) {
                    const int ck = c0 + k;
                    const float mk = __shfl_sync(0xffffffffu, dm, k * 8);
                    const float rk = __shfl_sync(0xffffffffu, dr, k * 8);
                    if (ck >= R) break;
                    if (ck < 0) {
                        norm2 = mk;
                        continue;
                    }
                    if (membership_on) {
                        const float proj2 = __fmul_rn(mk, mk);
                        distance = __fadd_rn(distance, __fdiv_rn(proj2, denom[ck]));
                        projected = __fadd_rn(projected, proj2);
                    }
                    if (lane == 0) proj[ck] = rk;
                }
            }
            if (membership_on) {
                const float res = __fsub_rn(norm2, projected);
                distance = __fadd_rn(distance, __fdiv_rn(res > 0.0f ? res : 0.0f, mem2));
                const float score = __fdiv_rn(__fsub_rn(distance, static_cast<float>(D)), score_scale);
                if (lane == 0) scores[i] = score;
            }
            __syncwarp();
            // reconstruction (project_bayes_estimate), components in order,
            // accumulated in registers over blocks of 32 * kRecCols columns
            float* out = L.filtered + static_cast<size_t>(r0 + i) * L.row_dim + mc * D;
            for (int base = 0; base < D; base += 32 * kRecCols) {
                float o[kRecCols];
#pragma unroll
                for (int j = 0; j < kRecCols; ++j) o[j] = 0.0f;
                for (int c = 0; c < R; ++c) {
                    if (coef[c] == 0.0f) continue;
                    const float scaled = __fmul_rn(coef[c], proj[c]);
                    const float* bc = basis + c * ldb;
#pragma unroll
                    for (int j = 0; j < kRecCols; ++j) {
                        const int col = base + lane + 32 * j;
                        if (col < D) o[j] = add_scaled_elem(o[j], bc[col], scaled, col, D);
                    }
                }
#pragma unroll
                for (int j = 0; j < kRecCols; ++j) {
                    const int col = base + lane + 32 * j;
                    if (col < D) out[col] = __fadd_rn(o[j], center_vec[col]);
                }
            }
            __syncwarp();
        }
        __syncthreads();
        // aggregation weights (accumulate_aggregation_model + finalize)
        if (tid == 0) {
            float mn = kInf;
            if (membership_on)
                for (int i = 0; i < S; ++i) mn = std_min(mn, scores[i]);
            s_misc[2] = mn;
        }
        __syncthreads();
        const float min_score = s_misc[2];
        for (int i = tid; i < S; i += kApplyThreads) {
            if (models > 1) {
                // this plane's term of the row's log weight; combine_weights
                // sums the planes in order and finalises
                L.logw[static_cast<size_t>(r0 + i) * models + mc] =
                    model_log_weight(P, membership_on, lgw, volume, scores[i], min_score);
                continue;
            }
            float w = 1.0f;
            if (weights_enabled) {
                float lw;
                if (P.weight_alpha == 0.0f && P.weight_beta == 0.0f) {
                    lw = 0.0f;
                } else if (membership_on) {
                    const float diff = __fsub_rn(scores[i], min_score);
                    const float membership = __fadd_rn(diff > 0.0f ? diff : 0.0f, volume);
                    lw = __fadd_rn(0.0f, __fsub_rn(lgw, __fmul_rn(P.weight_beta, membership)));
                } else {
                    lw = __fadd_rn(0.0f, lgw);
                }
                lw = lw < -80.0f ? -80.0f : (80.0f < lw ? 80.0f : lw);
                w = cr_expf(lw);
            }
            L.weights[r0 + i] = w;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// apply, row tiles: a CTA of up to kTileWarps warps per group, for the shapes
// with ranks up to 16 kQ that the warp-per-group kernel does not take (blocks
// of 7 over two frames and three planes, groups of 16 grown to 64 rows).
//
// Measured against one group per 8-warp CTA with two rows per warp and scalar
// shared loads (B200, one launch alone, 57k groups of dimension 294, rank 15):
// Basic 2.75 -> 1.19 ms, Final 3.72 -> 2.17 ms; 130k groups of dimension 128,
// rank 16: 6.7 -> 2.87 and 7.7 -> 3.34 ms.
// Now bound by latency: 16 (Basic) and 12 (Final) warps of an SM issue in 43 and
// 34% of its slots and wait for the samples, the shared loads and the barriers
// between a group's phases; the FMA pipe is 26 and 21% busy.  The layouts serve
// wide loads: the basis is [column][component], padded to 4 mod 8 quads so that the
// 8 columns of a quarter warp start on different banks, and a warp's tile of
// kTileRows rows is [column][row].  One 16-byte load then brings four
// components (or all four rows) of a column.  Lane (j, g) runs the pinned
// chain j (columns j + 8 m) of four rows against components 4 g .. 4 g + 3 of
// each block of 16; the chains are folded by halving exchanges (the additions
// of reduce8: xor 4, 2, 1), which leaves each lane with one row's dots of two
// components, and the unfused tail, the division by the component's
// variance and the shrinkage follow there.  The reconstruction takes blocks of
// 32 columns, one per lane and block, all components of a column in registers.
constexpr int kTileWarps = 4;

struct TileApplyLayout {
    int ldb, coloff, means, basis, dual, scal, scores, bases, tiles, tile_floats, bytes;
};

// kq: components in blocks of 16; per warp U [D][4], V [D][4] (Final), and per
// block of 16 the scaled projections [16][4], quotients [4][16] and squares
// [4][16], then the 4 norms.
__host__ __device__ inline TileApplyLayout tile_apply_layout(int D, int Bmax, int kq, int max_rows, int warps,
                                                             bool final_stage) {
    TileApplyLayout a{};
    const int comps = 16 * kq;
    a.ldb = comps + 4;
    int off = 0;
    a.coloff = off;  off += (D + 3) & ~3;
    a.means = off;   off += (2 * D + 3) & ~3;
    a.basis = off;   off += D * a.ldb;
    a.dual = off;    off += Bmax * comps;
    a.scal = off;    off += 6 * comps;
    a.scores = off;  off += (max_rows + 3) & ~3;
    a.bases = off;   off += 2 * ((max_rows + 1) & ~1);
    a.tiles = off;
    a.tile_floats = (final_stage ? 2 : 1) * kTileRows * D + 3 * kTileRows * comps + 4;
    off += warps * a.tile_floats;
    a.bytes = off * static_cast<int>(sizeof(float));
    return a;
}

// Dual -> primal basis of kCols columns (tid + 128-strided) of one thread:
// acc[c] += dual[c][s] * x_s[col], the samples in order, then the scale.
template <int kQ, int kCols>
__device__ __forceinline__ void tile_basis_columns(const FilterLaunch& L, const float* model_video, const size_t* bases,
                                                   const int* coloff, const float* mean, const float* dual,
                                                   const float* inv_sqrt, float* basis, int ldb, int D, int B, int col0,
                                                   int stride) {
    constexpr int kComps = 16 * kQ;
    const int full = (D / kLanes) * kLanes;
    int off[kCols];
    float mm[kCols];
    bool tail = false;
#pragma unroll
    for (int k = 0; k < kCols; ++k) {
        const int col = min(col0 + k * stride, D - 1);
        off[k] = coloff[col];
        mm[k] = mean[col];
        tail |= col >= full;
    }
#pragma unroll
    for (int c0 = 0; c0 < kComps; c0 += 16) {
        float2 acc[kCols][8];
#pragma unroll
        for (int k = 0; k < kCols; ++k)
#pragma unroll
            for (int p = 0; p < 8; ++p) acc[k][p] = make_float2(0.0f, 0.0f);
        if (!tail) {
#pragma unroll 4
            for (int s = 0; s < B; ++s) {
                const float* src = model_video + bases[s];
                float x[kCols];
#pragma unroll
                for (int k = 0; k < kCols; ++k) x[k] = __fsub_rn(__ldg(src + off[k]), mm[k]);
                const float4* w4 = reinterpret_cast<const float4*>(dual + s * kComps + c0);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 w = w4[q];
#pragma unroll
                    for (int k = 0; k < kCols; ++k) {
                        acc[k][2 * q] = fma2_rn(dup2(x[k]), make_float2(w.x, w.y), acc[k][2 * q]);
                        acc[k][2 * q + 1] = fma2_rn(dup2(x[k]), make_float2(w.z, w.w), acc[k][2 * q + 1]);
                    }
                }
            }
        } else {
            // a column past the last full chunk of 8 is among them: unfused there
            for (int s = 0; s < B; ++s) {
                const float* src = model_video + bases[s];
                const float* w = dual + s * kComps + c0;
#pragma unroll
                for (int k = 0; k < kCols; ++k) {
                    const float x = __fsub_rn(__ldg(src + off[k]), mm[k]);
                    const bool fused = col0 + k * stride < full;
#pragma unroll
                    for (int p = 0; p < 8; ++p) {
                        const float2 a = acc[k][p];
                        const float w0 = w[2 * p], w1 = w[2 * p + 1];
                        acc[k][p] = fused ? make_float2(__fmaf_rn(w0, x, a.x), __fmaf_rn(w1, x, a.y))
                                          : make_float2(__fadd_rn(a.x, __fmul_rn(w0, x)),
                                                        __fadd_rn(a.y, __fmul_rn(w1, x)));
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kCols; ++k) {
            const int col = col0 + k * stride;
            if (col >= D) continue;
            float4* out = reinterpret_cast<float4*>(basis + col * ldb + c0);
            const float* is = inv_sqrt + c0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                out[q] = make_float4(__fmul_rn(acc[k][2 * q].x, is[4 * q]), __fmul_rn(acc[k][2 * q].y, is[4 * q + 1]),
                                     __fmul_rn(acc[k][2 * q + 1].x, is[4 * q + 2]),
                                     __fmul_rn(acc[k][2 * q + 1].y, is[4 * q + 3]));
        }
    }
}

// Reconstruction (project_bayes_estimate) of a tile's rows over kBlocks blocks
// of 32 columns, components in order, and its store.
template <int kBlocks, bool kTail>
__device__ __forceinline__ void tile_reconstruct(const float* basis, int ldb, const float* coef, const float* sc,
                                                 const float* center, int R, int D, int base, int lane, float* out,
                                                 size_t row_stride, int nrows) {
    float2 o[kBlocks][2];  // rows (0, 1) and (2, 3)
    int col[kBlocks];
    const int full = (D / kLanes) * kLanes;
#pragma unroll
    for (int k = 0; k < kBlocks; ++k) {
        col[k] = min(base + 32 * k + lane, D - 1);
        o[k][0] = o[k][1] = make_float2(0.0f, 0.0f);
    }
    for (int c0 = 0; c0 < R; c0 += 4) {
        float b[kBlocks][4];
#pragma unroll
        for (int k = 0; k < kBlocks; ++k) {
            const float4 t = *reinterpret_cast<const float4*>(basis + col[k] * ldb + c0);
            b[k][0] = t.x;
            b[k][1] = t.y;
            b[k][2] = t.z;
            b[k][3] = t.w;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c0 + c >= R || coef[c0 + c] == 0.0f) continue;
            const float4 s = *reinterpret_cast<const float4*>(sc + (c0 + c) * kTileRows);
            const float2 s01 = make_float2(s.x, s.y), s23 = make_float2(s.z, s.w);
#pragma unroll
            for (int k = 0; k < kBlocks; ++k) {
                if (kTail && col[k] >= full) {
                    const float v = b[k][c];
                    o[k][0] = make_float2(__fadd_rn(o[k][0].x, __fmul_rn(s.x, v)),
                                          __fadd_rn(o[k][0].y, __fmul_rn(s.y, v)));
                    o[k][1] = make_float2(__fadd_rn(o[k][1].x, __fmul_rn(s.z, v)),
                                          __fadd_rn(o[k][1].y, __fmul_rn(s.w, v)));
                } else {
                    o[k][0] = fma2_rn(s01, dup2(b[k][c]), o[k][0]);
                    o[k][1] = fma2_rn(s23, dup2(b[k][c]), o[k][1]);
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kBlocks; ++k) {
        if (base + 32 * k + lane >= D) continue;
        const float mid = center[col[k]];
        float* at = out + col[k];
        at[0] = __fadd_rn(o[k][0].x, mid);
        if (nrows > 1) at[row_stride] = __fadd_rn(o[k][0].y, mid);
        if (nrows > 2) at[2 * row_stride] = __fadd_rn(o[k][1].x, mid);
        if (nrows > 3) at[3 * row_stride] = __fadd_rn(o[k][1].y, mid);
    }
}

template <int kQ, bool kFinal>
__global__ void __launch_bounds__(32 * kTileWarps, kQ == 1 ? 4 : 2) apply_tile_kernel(FilterLaunch L) {
    constexpr int kComps = 16 * kQ;
    extern __shared__ __align__(16) float sm[];
    __shared__ float s_misc[4];
    const int D = L.dim;
    const int Bmax = bmax_of(L);
    const int R = L.rank;
    const int threads = blockDim.x;
    const TileApplyLayout lay = tile_apply_layout(D, Bmax, kQ, L.max_rows, threads / 32, kFinal);
    const int ldb = lay.ldb;
    int* coloff = reinterpret_cast<int*>(sm);
    float* means = sm + lay.means;  // membership mean, reconstruction centre
    float* basis = sm + lay.basis;
    float* dual = sm + lay.dual;    // [sample][component]
    float* eig = sm + lay.scal;
    float* coef = eig + kComps;      // Wiener coefficients
    float* denom = coef + kComps;    // signal eigenvalue + membership noise
    float* inv_sqrt = denom + kComps;  // 1 / sqrt(eigenvalue), 0 below the floor
    float* terms = inv_sqrt + kComps;  // log1p(signal / membership noise)
    float* shares = terms + kComps;    // signal / (signal + noise)
    float* scores = sm + lay.scores;
    size_t* bases = reinterpret_cast<size_t*>(sm + lay.bases);
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int warps = threads >> 5;
    const int j = lane & 7;
    const int grp = lane >> 3;
    float* U = sm + lay.tiles + warp * lay.tile_floats;  // centred membership rows [D][4]
    float* V = U + kTileRows * D;                         // centred noisy rows (Final)
    float* sc = U + (kFinal ? 2 : 1) * kTileRows * D;     // scaled projections [component][row]
    float* quot = sc + kTileRows * kComps;                // projection^2 / variance [row][component]
    float* square = quot + kTileRows * kComps;            // projection^2 [row][component]
    float* norms = square + kTileRows * kComps;           // [row]
    for (int col = tid; col < D; col += threads) coloff[col] = column_offset(L, col);
    const StageConfig& P = L.cfg;
    const float* model_video = kFinal ? L.basic : L.noisy;
    const bool weights_enabled = P.weight_alpha != 0.0f || P.weight_beta != 0.0f || P.weight_gamma != 0.0f;
    const float sigma2 = __fmul_rn(__fmul_rn(P.beta, P.sigma), P.sigma);
    const float model_noise2 = kFinal ? __fmul_rn(__fmul_rn(P.beta, P.sigma_basic), P.sigma_basic) : sigma2;
    const float match_sigma = kFinal ? P.sigma_basic : P.sigma;
    const float mem2 = std_max(__fmul_rn(match_sigma, match_sigma),
                               __fmul_rn(__fmul_rn(P.membership_noise_floor, P.sigma), P.sigma));
    const bool membership_on = P.weight_beta != 0.0f;
    const int total = L.counters->active * L.models;
    const int models = L.models;  // models per group (planes when uncoupled)
    const size_t hw = static_cast<size_t>(L.height) * L.width;
    const int full = D / kLanes;
    const bool has_tail = full * kLanes < D;
    const float score_scale = __fsqrt_rn(__fmul_rn(2.0f, static_cast<float>(D)));
    // the next group's flag and anchor are loaded an iteration ahead
    int mi = blockIdx.x;
    int flag = 0, g = 0;
    if (mi < total) {
        flag = L.flags[mi];
        g = L.active[mi / models];
    }
    __syncthreads();
    for (; mi < total;) {
        const int a = mi / models;
        const int mc = mi - a * models;
        const int cur = mi, cur_flag = flag, cur_g = g;
        mi += gridDim.x;
        if (mi < total) {
            flag = L.flags[mi];
            g = L.active[mi / models];
        }
        if (cur_flag != 0) continue;  // uniform: equal groups are done, skipped ones reported
        const int S = L.row_counts[cur_g];
        const MatchRow* rows = L.rows + static_cast<size_t>(cur_g) * L.max_rows;
        const int r0 = L.row_offset[a];
        const int B = min(S, L.model_cap);
        const int N = L.nmax;  // row stride of the eigenvector rows
        const bool dual_model = D >= 64 && B < D;  // use_dual_pca (core.cpp:656-658)
        const float* gm = L.means + static_cast<size_t>(cur) * 2 * D;
        const float* gd = L.dual + static_cast<size_t>(cur) * R * N;
        for (int i = tid; i < S; i += threads) bases[i] = row_base(L, rows[i]) + mc * hw;  // this model's plane
        for (int i = tid; i < 2 * D; i += threads) means[i] = gm[i];
        if (dual_model)
            for (int i = tid; i < B * kComps; i += threads) {
                const int c = i / B, s = i - c * B;
                dual[s * kComps + c] = c < R ? gd[c * N + s] : 0.0f;
            }
        // per-component scalars, once per group
        if (tid < kComps) {
            const int c = tid;
            const float lambda = c < R ? L.eig[static_cast<size_t>(cur) * R + c] : 0.0f;
            eig[c] = lambda;
            const float diff = __fsub_rn(lambda, model_noise2);
            const float signal = diff > 0.0f ? diff : 0.0f;
            denom[c] = __fadd_rn(signal, mem2);
            inv_sqrt[c] = lambda > kEigenFloor ? __fdiv_rn(1.0f, __fsqrt_rn(lambda)) : 0.0f;
            terms[c] = (membership_on && signal > 0.0f) ? cr_log1pf(__fdiv_rn(signal, mem2)) : 0.0f;
            shares[c] = signal > 0.0f ? __fdiv_rn(signal, __fadd_rn(signal, sigma2)) : 0.0f;
            const float sigma_basic2 = kFinal ? model_noise2 : sigma2;
            const float threshold = __fmul_rn(P.variance_threshold, sigma2);
            float variance = lambda;
            if (sigma_basic2 > 0.0f) variance = __fsub_rn(variance, std_min(variance, sigma_basic2));
            coef[c] = c < R && variance > threshold ? __fdiv_rn(1.0f, __fadd_rn(1.0f, __fdiv_rn(sigma2, variance)))
                                                    : 0.0f;
        }
        __syncthreads();
        const float* member_mean = means;
        const float* center_vec = means + D;
        if (dual_model) {
            // dual -> primal basis (map_dual_eigenvectors_to_basis); components
            // at or below the floor are zero
            for (int col = tid; col < D; col += 2 * threads) {
                if (col - lane + threads < D)
                    tile_basis_columns<kQ, 2>(L, model_video, bases, coloff, member_mean, dual, inv_sqrt, basis, ldb, D,
                                              B, col, threads);
                else
                    tile_basis_columns<kQ, 1>(L, model_video, bases, coloff, member_mean, dual, inv_sqrt, basis, ldb, D,
                                              B, col, threads);
            }
            __syncthreads();
            for (int b0 = 4 * warp; b0 < R; b0 += 4 * warps) {
                const int b = min(b0 + grp, kComps - 1);  // an octet per component
                const float* col = basis + j * ldb + b;
                float v = 0.0f;
#pragma unroll 4
                for (int m = 0; m < full; ++m) {
                    const float x = col[m * kLanes * ldb];
                    v = __fmaf_rn(x, x, v);
                }
                float norm2 = octet_fold(v);
                for (int idx = full * kLanes; idx < D; ++idx) {
                    const float x = basis[idx * ldb + b];
                    norm2 = __fadd_rn(norm2, __fmul_rn(x, x));
                }
                __syncwarp();  // every lane has read its component's column
                const bool live = b < R && eig[b] > kEigenFloor;
                const bool none = !live || norm2 <= kEigenFloor;
                const float s = none ? 0.0f : __fdiv_rn(1.0f, __fsqrt_rn(norm2));
                for (int c = j; c < D; c += kLanes) {
                    float* at = basis + c * ldb + b;
                    *at = none ? 0.0f : __fmul_rn(*at, s);
                }
            }
        } else {
            // covariance model: the canonicalised eigenvectors are the basis
            for (int i = tid; i < kComps * D; i += threads) {
                const int c = i / D, col = i - c * D;
                basis[col * ldb + c] = c < R ? gd[static_cast<size_t>(c) * N + col] : 0.0f;
            }
        }
        // group precision and volume (group_precision_tau, core.cpp:222-241,
        // 346-358): the terms are ready, the sums run in component order
        if (tid == threads - 1) {
            float trace = 0.0f, volume = 0.0f;
            // (a component without signal adds zero to both)
#pragma unroll 4
            for (int c = 0; c < R; ++c) {
                trace = __fadd_rn(trace, shares[c]);
                volume = __fadd_rn(volume, terms[c]);
            }
            const float tau = __fadd_rn(
                __fadd_rn(P.weight_epsilon, __fdiv_rn(static_cast<float>(D), static_cast<float>(B))), trace);
            s_misc[0] = P.weight_alpha == 0.0f ? 0.0f : __fmul_rn(-P.weight_alpha, cr_logf(tau));
            s_misc[1] = __fdiv_rn(volume, static_cast<float>(D));
        }
        __syncthreads();
        for (int t0 = warp * kTileRows; t0 < S; t0 += warps * kTileRows) {
            const int nrows = min(kTileRows, S - t0);
            {
                // a missing row repeats the first
                const size_t b0 = bases[t0], b1 = bases[t0 + (nrows > 1 ? 1 : 0)];
                const size_t b2 = bases[t0 + (nrows > 2 ? 2 : 0)], b3 = bases[t0 + (nrows > 3 ? 3 : 0)];
#pragma unroll 2
                for (int col = lane; col < D; col += 32) {
                    const int off = coloff[col];
                    const float m = member_mean[col];
                    const float* nz = L.noisy + off;
                    const float x0 = __ldg(nz + b0), x1 = __ldg(nz + b1), x2 = __ldg(nz + b2), x3 = __ldg(nz + b3);
                    if constexpr (kFinal) {
                        const float* bs = L.basic + off;
                        const float y0 = __ldg(bs + b0), y1 = __ldg(bs + b1), y2 = __ldg(bs + b2), y3 = __ldg(bs + b3);
                        const float c = center_vec[col];
                        *reinterpret_cast<float4*>(U + 4 * col) = make_float4(__fsub_rn(y0, m), __fsub_rn(y1, m),
                                                                              __fsub_rn(y2, m), __fsub_rn(y3, m));
                        *reinterpret_cast<float4*>(V + 4 * col) = make_float4(__fsub_rn(x0, c), __fsub_rn(x1, c),
                                                                              __fsub_rn(x2, c), __fsub_rn(x3, c));
                    } else {
                        *reinterpret_cast<float4*>(U + 4 * col) = make_float4(__fsub_rn(x0, m), __fsub_rn(x1, m),
                                                                              __fsub_rn(x2, m), __fsub_rn(x3, m));
                    }
                }
            }
            __syncwarp();
            const int r = ((j >> 2) << 1) | ((j >> 1) & 1);  // this lane's row after the folds
#pragma unroll
            for (int q = 0; q < kQ; ++q) {
                float2 am[kTileRows][2], ar[kTileRows][2], an[2];
                an[0] = an[1] = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int i = 0; i < kTileRows; ++i)
#pragma unroll
                    for (int p = 0; p < 2; ++p) am[i][p] = ar[i][p] = make_float2(0.0f, 0.0f);
                const float* bp = basis + j * ldb + 16 * q + 4 * grp;
                const float* up = U + 4 * j;
                const float* vp = V + 4 * j;
#pragma unroll 2
                for (int m = 0; m < full; ++m) {
                    const float4 bv = *reinterpret_cast<const float4*>(bp + m * kLanes * ldb);
                    const float2 b01 = make_float2(bv.x, bv.y), b23 = make_float2(bv.z, bv.w);
                    const float4 u = *reinterpret_cast<const float4*>(up + m * 4 * kLanes);
                    am[0][0] = fma2_rn(dup2(u.x), b01, am[0][0]);
                    am[0][1] = fma2_rn(dup2(u.x), b23, am[0][1]);
                    am[1][0] = fma2_rn(dup2(u.y), b01, am[1][0]);
                    am[1][1] = fma2_rn(dup2(u.y), b23, am[1][1]);
                    am[2][0] = fma2_rn(dup2(u.z), b01, am[2][0]);
                    am[2][1] = fma2_rn(dup2(u.z), b23, am[2][1]);
                    am[3][0] = fma2_rn(dup2(u.w), b01, am[3][0]);
                    am[3][1] = fma2_rn(dup2(u.w), b23, am[3][1]);
                    if (q == 0) {
                        const float2 u01 = make_float2(u.x, u.y), u23 = make_float2(u.z, u.w);
                        an[0] = fma2_rn(u01, u01, an[0]);
                        an[1] = fma2_rn(u23, u23, an[1]);
                    }
                    if constexpr (kFinal) {
                        const float4 v = *reinterpret_cast<const float4*>(vp + m * 4 * kLanes);
                        ar[0][0] = fma2_rn(dup2(v.x), b01, ar[0][0]);
                        ar[0][1] = fma2_rn(dup2(v.x), b23, ar[0][1]);
                        ar[1][0] = fma2_rn(dup2(v.y), b01, ar[1][0]);
                        ar[1][1] = fma2_rn(dup2(v.y), b23, ar[1][1]);
                        ar[2][0] = fma2_rn(dup2(v.z), b01, ar[2][0]);
                        ar[2][1] = fma2_rn(dup2(v.z), b23, ar[2][1]);
                        ar[3][0] = fma2_rn(dup2(v.w), b01, ar[3][0]);
                        ar[3][1] = fma2_rn(dup2(v.w), b23, ar[3][1]);
                    }
                }
                float2 dm = fold_tile(am, j), dr = dm;
                if constexpr (kFinal) dr = fold_tile(ar, j);
                const int c = 16 * q + 4 * grp + 2 * (j & 1);  // this lane's components c, c + 1
                if (has_tail) {
                    // the unfused tail of each dot (dot_contiguous_highway)
                    for (int idx = full * kLanes; idx < D; ++idx) {
                        const float2 b = *reinterpret_cast<const float2*>(basis + idx * ldb + c);
                        const float u = U[4 * idx + r];
                        dm.x = __fadd_rn(dm.x, __fmul_rn(u, b.x));
                        dm.y = __fadd_rn(dm.y, __fmul_rn(u, b.y));
                        if constexpr (kFinal) {
                            const float v = V[4 * idx + r];
                            dr.x = __fadd_rn(dr.x, __fmul_rn(v, b.x));
                            dr.y = __fadd_rn(dr.y, __fmul_rn(v, b.y));
                        }
                    }
                    if constexpr (!kFinal) dr = dm;
                }
                sc[c * kTileRows + r] = __fmul_rn(coef[c], dr.x);
                sc[(c + 1) * kTileRows + r] = __fmul_rn(coef[c + 1], dr.y);
                if (membership_on) {
                    const float p0 = __fmul_rn(dm.x, dm.x), p1 = __fmul_rn(dm.y, dm.y);
                    *reinterpret_cast<float2*>(square + r * kComps + c) = make_float2(p0, p1);
                    *reinterpret_cast<float2*>(quot + r * kComps + c) =
                        make_float2(__fdiv_rn(p0, denom[c]), __fdiv_rn(p1, denom[c + 1]));
                    if (q == 0) {
                        // the rows' norms, folded like the dots
                        const float x = fold_half((j & 4) ? an[1].x : an[0].x, (j & 4) ? an[0].x : an[1].x, 4);
                        const float y = fold_half((j & 4) ? an[1].y : an[0].y, (j & 4) ? an[0].y : an[1].y, 4);
                        float n = fold_half((j & 2) ? y : x, (j & 2) ? x : y, 2);
                        n = __fadd_rn(n, __shfl_xor_sync(0xffffffffu, n, 1));
                        for (int idx = full * kLanes; idx < D; ++idx) {
                            const float u = U[4 * idx + r];
                            n = __fadd_rn(n, __fmul_rn(u, u));
                        }
                        if (grp == 0 && !(j & 1)) norms[r] = n;
                    }
                }
            }
            __syncwarp();
            // membership score of each row, components in order
            if (lane < nrows && membership_on) {
                const float* qr = quot + lane * kComps;
                const float* pr = square + lane * kComps;
                float distance = 0.0f, projected = 0.0f;
#pragma unroll
                for (int c0 = 0; c0 < kComps; c0 += 4) {
                    if (c0 >= R) break;
                    const float4 q4 = *reinterpret_cast<const float4*>(qr + c0);
                    const float4 p4 = *reinterpret_cast<const float4*>(pr + c0);
                    const float qs[4] = {q4.x, q4.y, q4.z, q4.w}, ps[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (c0 + c >= R) break;
                        distance = __fadd_rn(distance, qs[c]);
                        projected = __fadd_rn(projected, ps[c]);
                    }
                }
                const float resid = __fsub_rn(norms[lane], projected);
                distance = __fadd_rn(distance, __fdiv_rn(resid > 0.0f ? resid : 0.0f, mem2));
                scores[t0 + lane] = __fdiv_rn(__fsub_rn(distance, static_cast<float>(D)), score_scale);
            }
            float* out = L.filtered + static_cast<size_t>(r0 + t0) * L.row_dim + mc * D;
            int base = 0;
            for (; base + 128 <= full * kLanes; base += 128)
                tile_reconstruct<4, false>(basis, ldb, coef, sc, center_vec, R, D, base, lane, out, L.row_dim, nrows);
            for (; base + 64 <= D; base += 64)
                tile_reconstruct<2, true>(basis, ldb, coef, sc, center_vec, R, D, base, lane, out, L.row_dim, nrows);
            for (; base < D; base += 32)
                tile_reconstruct<1, true>(basis, ldb, coef, sc, center_vec, R, D, base, lane, out, L.row_dim, nrows);
            __syncwarp();
        }
        __syncthreads();
        // aggregation weights (accumulate_aggregation_model + finalize)
        const float lgw = s_misc[0];
        const float volume = s_misc[1];
        if (warp == 0) {
            float mn = kInf;
            if (membership_on)
                for (int i = lane; i < S; i += 32) mn = std_min(mn, scores[i]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mn = std_min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            if (lane == 0) s_misc[2] = mn;
        }
        __syncthreads();
        const float min_score = s_misc[2];
        for (int i = tid; i < S; i += threads) {
            const float lw0 = model_log_weight(P, membership_on, lgw, volume, scores[i], min_score);
            if (models > 1) {
                // this plane's term of the row's log weight; combine_weights
                // sums the planes in order and finalises
                L.logw[static_cast<size_t>(r0 + i) * models + mc] = lw0;
                continue;
            }
            float w = 1.0f;
            if (weights_enabled) {
                float lw = __fadd_rn(0.0f, lw0);
                lw = lw < -80.0f ? -80.0f : (80.0f < lw ? 80.0f : lw);
                w = cr_expf(lw);
            }
            L.weights[r0 + i] = w;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// apply, warp per group: the same arithmetic as apply_kernel, register-blocked
// for D % 32 == 0, rank <= 8 and at most 8 model rows (the shapes of the
// default parameter sets: 8x8 patches, one or three planes, rank 8, group 8).
//
// A lane owns columns lane + 32 jj for the elementwise work (the centred model
// rows and all components' basis values of a block of columns in registers, the
// reconstruction and its store).  The rows go in tiles of four, [column][row]
// beside a basis [column][component]: for the dot products lane (j, q, h) runs
// the pinned chain j (columns j + 8 m) of rows 2 h, 2 h + 1 against components
// 4 q .. 4 q + 3, so an 8-byte and a 16-byte load feed eight multiply-adds, and
// the halving folds leave every lane with one row's dot of one component.  (A
// row at a time with a component pair per octet, it took 490 / 548 us for 32k
// groups at D = 192, Basic / Final, now 255 / 407 us.)
// Per warp (floats): basis [D][12], U [D][4], V [D][4] (Final), dual [8][8],
// per-component scalars [5][8], projections [8][4], quotients and squares
// [4][8], norms [4], scores[max_rows], row bases[max_rows] (size_t).
constexpr int kWarpApplyWarps = 4;
constexpr int kWarpLdb = 12;  // floats per basis column: 8 columns start 3 bank quads apart

struct WarpApplyLayout {
    int basis, u, v, dual, scal, proj, quot, square, norms, scores, recon, rw, bases, per_warp;
};

// scatter: also the rows' scaled projections [max_rows][8] and weights
// [max_rows], kept for the second pass that adds the rows into the stack
__host__ __device__ inline WarpApplyLayout warp_apply_layout(int D, int max_rows, bool final_stage,
                                                             bool scatter) {
    WarpApplyLayout w{};
    int off = 0;
    w.basis = off;  off += kWarpLdb * D;
    w.u = off;      off += 4 * D;
    w.v = off;      off += final_stage ? 4 * D : 0;
    w.dual = off;   off += 64;
    w.scal = off;   off += 5 * 8;
    w.proj = off;   off += 32;
    w.quot = off;   off += 32;
    w.square = off; off += 32;
    w.norms = off;  off += 4;
    w.recon = off;  off += scatter ? 8 * ((max_rows + 3) & ~3) : 0;
    w.scores = off; off += max_rows;
    w.rw = off;     off += scatter ? max_rows : 0;
    off = (off + 1) & ~1;
    w.bases = off;  off += 2 * max_rows;
    off = (off + 3) & ~3;
    w.per_warp = off;
    return w;
}

// resident blocks per SM the warp-per-group apply is compiled for (a register
// budget); a build parameter for comparisons
#ifndef VNLB_APPLY_MIN_BLOCKS
#define VNLB_APPLY_MIN_BLOCKS 4
#endif

// Chosen forms: a lane's columns of one filtered row added into the anchor
// frame's stack, weight cw times the window at each pixel; the weight plane
// gets the same once per pixel (the columns of plane 0).  Slots outside the
// window are dropped, as the stack tiles drop them.  The additions' order is
// not fixed, so these forms are not bit-reproducible in the stacks' last
// bits.
//
// Pixel-interleaved stacks (L.scatter_pack = C+1): with C = 3 and 64
// columns per plane, a lane's columns jj, jj + kCols/3 and jj + 2 kCols/3
// are the same pixel of planes 0, 1 and 2, so the pixel's three values and
// its weight go in one 16-byte vector addition (C = 1: value and weight in
// one 8-byte one); a quarter (half) of the scalar atomics, and no shuffles.
// (Vector reductions of an octet's patch row in the planar layout, tried,
// were slower: the shuffles that gather a row cost more than they save.)
template <int kCols>
__device__ __forceinline__ void scatter_row(const FilterLaunch& L, const MatchRow& m, const float (&o)[kCols],
                                            float cw, int lane) {
    const size_t plane = static_cast<size_t>(L.height) * L.width;
    const int C = L.channels;
    const int P = L.P;
    const size_t base = static_cast<size_t>(m.y) * L.width + m.x;
    const int slot0 = m.frame + L.search_bwd - L.anchor_frame;
    if constexpr (kCols % 3 == 0) {
        if (L.scatter_pack == 4) {
            constexpr int kpp = kCols / 3;  // columns per plane and lane
#pragma unroll
            for (int jj = 0; jj < kpp; ++jj) {
                const int pos = lane + 32 * jj;  // (layer t, py, px) within the plane's patch
                const int t = pos / (P * P);
                const int rem = pos - t * P * P;
                const int py = rem / P;
                const int slot = slot0 + t;
                if (slot < 0 || slot >= L.slots) continue;
                const float w = L.windowed ? cw * __ldg(L.window + rem) : cw;
                const size_t at = base + static_cast<size_t>(py) * L.width + (rem - py * P);
                atomicAdd(reinterpret_cast<float4*>(L.scatter) + static_cast<size_t>(slot) * plane + at,
                          make_float4(w * o[jj], w * o[jj + kpp], w * o[jj + 2 * kpp], w));
            }
            return;
        }
    }
    if (L.scatter_pack == 2) {
#pragma unroll
        for (int jj = 0; jj < kCols; ++jj) {
            const int pos = lane + 32 * jj;
            const int t = pos / (P * P);
            const int rem = pos - t * P * P;
            const int py = rem / P;
            const int slot = slot0 + t;
            if (slot < 0 || slot >= L.slots) continue;
            const float w = L.windowed ? cw * __ldg(L.window + rem) : cw;
            const size_t at = base + static_cast<size_t>(py) * L.width + (rem - py * P);
            atomicAdd(reinterpret_cast<float2*>(L.scatter) + static_cast<size_t>(slot) * plane + at,
                      make_float2(w * o[jj], w));
        }
        return;
    }
#pragma unroll
    for (int jj = 0; jj < kCols; ++jj) {
        // column (plane c, layer t, py, px)
        const int col = lane + 32 * jj;
        const int c = col / L.patch_dim;
        const int pos = col - c * L.patch_dim;
        const int t = pos / (P * P);
        const int rem = pos - t * P * P;
        const int py = rem / P;
        const int slot = slot0 + t;
        if (slot < 0 || slot >= L.slots) continue;
        const float w = L.windowed ? cw * __ldg(L.window + rem) : cw;
        const size_t at = base + static_cast<size_t>(py) * L.width + (rem - py * P);
        atomicAdd(L.scatter + (static_cast<size_t>(slot) * (C + 1) + c) * plane + at, w * o[jj]);
        if (c == 0) atomicAdd(L.scatter + (static_cast<size_t>(slot) * (C + 1) + C) * plane + at, w);
    }
}

// A tile's reconstruction (project_bayes_estimate) of this lane's columns, the
// components in order: o[row][jj].
template <int kCols>
__device__ __forceinline__ void warp_reconstruct(const float* basis, const float* sc, const float* coef, int R, int lane,
                                                 const float (&cc)[kCols], float (&o)[4][kCols]) {
    float2 acc[kCols][2];
#pragma unroll
    for (int jj = 0; jj < kCols; ++jj) acc[jj][0] = acc[jj][1] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int c0 = 0; c0 < 8; c0 += 4) {
        if (c0 >= R) break;
        float b[kCols][4];
#pragma unroll
        for (int jj = 0; jj < kCols; ++jj) {
            const float4 t = *reinterpret_cast<const float4*>(basis + (lane + 32 * jj) * kWarpLdb + c0);
            b[jj][0] = t.x;
            b[jj][1] = t.y;
            b[jj][2] = t.z;
            b[jj][3] = t.w;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c0 + c >= R || coef[c0 + c] == 0.0f) continue;
            const float4 s = *reinterpret_cast<const float4*>(sc + 4 * (c0 + c));
            const float2 s01 = make_float2(s.x, s.y), s23 = make_float2(s.z, s.w);
#pragma unroll
            for (int jj = 0; jj < kCols; ++jj) {
                acc[jj][0] = fma2_rn(s01, dup2(b[jj][c]), acc[jj][0]);
                acc[jj][1] = fma2_rn(s23, dup2(b[jj][c]), acc[jj][1]);
            }
        }
    }
#pragma unroll
    for (int jj = 0; jj < kCols; ++jj) {
        o[0][jj] = __fadd_rn(acc[jj][0].x, cc[jj]);
        o[1][jj] = __fadd_rn(acc[jj][0].y, cc[jj]);
        o[2][jj] = __fadd_rn(acc[jj][1].x, cc[jj]);
        o[3][jj] = __fadd_rn(acc[jj][1].y, cc[jj]);
    }
}

template <int D, bool kFinal, bool kScatter>
__global__ void __launch_bounds__(32 * kWarpApplyWarps, VNLB_APPLY_MIN_BLOCKS) apply_warp_kernel(FilterLaunch L) {
    static_assert(D % 32 == 0, "columns are owned in blocks of 32");
    constexpr int kCols = D / 32;
    constexpr int kChain = D / 8;
    extern __shared__ __align__(16) float sm[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int j8 = lane & 7;
    const int oct = lane >> 3;
    const WarpApplyLayout lay = warp_apply_layout(D, L.max_rows, kFinal, kScatter);
    int* coloff = reinterpret_cast<int*>(sm);
    float* wr = sm + D + warp * lay.per_warp;
    float* basis = wr + lay.basis;  // component c, column col at col * kWarpLdb + c
    float* U = wr + lay.u;
    float* V = wr + lay.v;
    float* dual = wr + lay.dual;    // [sample][component]
    float* eig = wr + lay.scal;
    float* coef = eig + 8;
    float* denom = coef + 8;
    float* inv_sqrt = denom + 8;
    float* terms = inv_sqrt + 8;
    float* quot = wr + lay.quot;
    float* square = wr + lay.square;
    float* norms = wr + lay.norms;
    float* scores = wr + lay.scores;
    size_t* bases = reinterpret_cast<size_t*>(wr + lay.bases);
    for (int col = threadIdx.x; col < D; col += blockDim.x) coloff[col] = column_offset(L, col);

    const int Bmax = bmax_of(L);
    const int R = L.rank;
    const StageConfig& P = L.cfg;
    const float* model_video = kFinal ? L.basic : L.noisy;
    const bool weights_enabled = P.weight_alpha != 0.0f || P.weight_beta != 0.0f || P.weight_gamma != 0.0f;
    const float sigma2 = __fmul_rn(__fmul_rn(P.beta, P.sigma), P.sigma);
    const float model_noise2 = kFinal ? __fmul_rn(__fmul_rn(P.beta, P.sigma_basic), P.sigma_basic) : sigma2;
    const float match_sigma = kFinal ? P.sigma_basic : P.sigma;
    const float mem2 = std_max(__fmul_rn(match_sigma, match_sigma),
                               __fmul_rn(__fmul_rn(P.membership_noise_floor, P.sigma), P.sigma));
    const bool membership_on = P.weight_beta != 0.0f;
    const float score_scale = __fsqrt_rn(__fmul_rn(2.0f, static_cast<float>(D)));
    const int active_count = L.counters->active;
    const int models = L.models;  // models per group (planes when uncoupled)
    const size_t hw = static_cast<size_t>(L.height) * L.width;
    const int q4 = 4 * (oct & 1), h = oct >> 1;          // this lane's component quad and row pair
    const int row_l = 2 * h + (j8 >> 2);                 // ... and its row and component after the folds
    const int comp_l = q4 + (j8 & 3);
    __syncthreads();
    int off[kCols];
#pragma unroll
    for (int jj = 0; jj < kCols; ++jj) off[jj] = coloff[lane + 32 * jj];

    for (int mi = blockIdx.x * kWarpApplyWarps + warp; mi < active_count * models;
         mi += gridDim.x * kWarpApplyWarps) {
        if (L.flags[mi] != 0) {  // equal groups are done, skipped ones reported
            if constexpr (kScatter) {
                if (L.flags[mi] == kGroupDone) {
                    // the pass-through rows prepare wrote, with their weights
                    const int g0 = L.active[mi];
                    const int S0 = L.row_counts[g0];
                    const int q0 = L.row_offset[mi];
                    const MatchRow* rows0 = L.rows + static_cast<size_t>(g0) * L.max_rows;
                    for (int i = 0; i < S0; ++i) {
                        float o[kCols];
#pragma unroll
                        for (int jj = 0; jj < kCols; ++jj)
                            o[jj] = L.filtered[static_cast<size_t>(q0 + i) * L.row_dim + lane + 32 * jj];
                        scatter_row(L, rows0[i], o, L.weights[q0 + i], lane);
                    }
                }
            }
            continue;
        }
        const int a = mi / models;
        const int mc = mi - a * models;
        const int g = L.active[a];
        const int S = L.row_counts[g];
        const MatchRow* rows = L.rows + static_cast<size_t>(g) * L.max_rows;
        const int r0 = L.row_offset[a];
        const int B = min(S, L.model_cap);
        const float* gm = L.means + static_cast<size_t>(mi) * 2 * D;
        float mm[kCols], cc[kCols];
#pragma unroll
        for (int jj = 0; jj < kCols; ++jj) {
            mm[jj] = __ldg(gm + lane + 32 * jj);
            cc[jj] = __ldg(gm + D + lane + 32 * jj);
        }
        for (int i = lane; i < S; i += 32) bases[i] = row_base(L, rows[i]) + mc * hw;  // this model's plane
        for (int i = lane; i < 64; i += 32) {
            const int s = i >> 3, b = i & 7;
            dual[i] = s < B && b < R ? L.dual[static_cast<size_t>(mi) * R * Bmax + b * Bmax + s] : 0.0f;
        }
        if (lane < 8) {
            const int c = lane;
            const float lambda = c < R ? L.eig[static_cast<size_t>(mi) * R + c] : 0.0f;
            eig[c] = lambda;
            const float diff = __fsub_rn(lambda, model_noise2);
            const float signal = diff > 0.0f ? diff : 0.0f;
            denom[c] = __fadd_rn(signal, mem2);
            inv_sqrt[c] = lambda > kEigenFloor ? __fdiv_rn(1.0f, __fsqrt_rn(lambda)) : 0.0f;
            terms[c] = (membership_on && signal > 0.0f) ? cr_log1pf(__fdiv_rn(signal, mem2)) : 0.0f;
            const float sigma_basic2 = kFinal ? model_noise2 : sigma2;
            const float threshold = __fmul_rn(P.variance_threshold, sigma2);
            float variance = lambda;
            if (sigma_basic2 > 0.0f) variance = __fsub_rn(variance, std_min(variance, sigma_basic2));
            coef[c] = c < R && variance > threshold ? __fdiv_rn(1.0f, __fadd_rn(1.0f, __fdiv_rn(sigma2, variance)))
                                                    : 0.0f;
        }
        __syncwarp();

        // dual -> primal basis over blocks of this lane's columns: the centred
        // model rows of the block in registers, then every component's samples
        // accumulated in order (all columns fused); components at or below the
        // floor are zero
        {
            constexpr int kBlk = kCols % 3 == 0 ? 3 : (kCols % 2 == 0 ? 2 : 1);
#pragma unroll
            for (int j0 = 0; j0 < kCols; j0 += kBlk) {
                float2 acc[kBlk][4];
#pragma unroll
                for (int jj = 0; jj < kBlk; ++jj)
#pragma unroll
                    for (int p = 0; p < 4; ++p) acc[jj][p] = make_float2(0.0f, 0.0f);
                float x[8][kBlk];
#pragma unroll
                for (int s = 0; s < 8; ++s)
#pragma unroll
                    for (int jj = 0; jj < kBlk; ++jj)
                        x[s][jj] = s < B ? __ldg(model_video + bases[s] + off[j0 + jj]) : mm[j0 + jj];
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    if (s >= B) break;
                    const float4 w0 = *reinterpret_cast<const float4*>(dual + 8 * s);
                    const float4 w1 = *reinterpret_cast<const float4*>(dual + 8 * s + 4);
#pragma unroll
                    for (int jj = 0; jj < kBlk; ++jj) {
                        const float2 xx = dup2(__fsub_rn(x[s][jj], mm[j0 + jj]));
                        acc[jj][0] = fma2_rn(make_float2(w0.x, w0.y), xx, acc[jj][0]);
                        acc[jj][1] = fma2_rn(make_float2(w0.z, w0.w), xx, acc[jj][1]);
                        acc[jj][2] = fma2_rn(make_float2(w1.x, w1.y), xx, acc[jj][2]);
                        acc[jj][3] = fma2_rn(make_float2(w1.z, w1.w), xx, acc[jj][3]);
                    }
                }
#pragma unroll
                for (int jj = 0; jj < kBlk; ++jj) {
                    float4* out = reinterpret_cast<float4*>(basis + (lane + 32 * (j0 + jj)) * kWarpLdb);
#pragma unroll
                    for (int p = 0; p < 2; ++p)
                        out[p] = make_float4(__fmul_rn(acc[jj][2 * p].x, inv_sqrt[4 * p]),
                                             __fmul_rn(acc[jj][2 * p].y, inv_sqrt[4 * p + 1]),
                                             __fmul_rn(acc[jj][2 * p + 1].x, inv_sqrt[4 * p + 2]),
                                             __fmul_rn(acc[jj][2 * p + 1].y, inv_sqrt[4 * p + 3]));
                }
            }
        }
        __syncwarp();
        // unit norm: octet k normalises components k and k + 4
        {
            float2 nv = make_float2(0.0f, 0.0f);
            float* col = basis + j8 * kWarpLdb + oct;
#pragma unroll 8
            for (int m = 0; m < kChain; ++m) {
                const float2 x = make_float2(col[m * 8 * kWarpLdb], col[m * 8 * kWarpLdb + 4]);
                nv = fma2_rn(x, x, nv);
            }
            const float n0 = octet_fold(nv.x), n1 = octet_fold(nv.y);
            const bool none0 = !(oct < R && eig[oct] > kEigenFloor) || n0 <= kEigenFloor;
            const bool none1 = !(oct + 4 < R && eig[oct + 4] > kEigenFloor) || n1 <= kEigenFloor;
            const float s0 = none0 ? 0.0f : __fdiv_rn(1.0f, __fsqrt_rn(n0));
            const float s1 = none1 ? 0.0f : __fdiv_rn(1.0f, __fsqrt_rn(n1));
#pragma unroll 8
            for (int m = 0; m < kChain; ++m) {
                float* at = col + m * 8 * kWarpLdb;
                at[0] = none0 ? 0.0f : __fmul_rn(at[0], s0);
                at[4] = none1 ? 0.0f : __fmul_rn(at[4], s1);
            }
        }
        __syncwarp();
        // group precision and volume, component order (every lane, uniform)
        float lgw, volume;
        {
            float trace = 0.0f, vol = 0.0f;
            for (int c = 0; c < R; ++c) {
                const float diff = __fsub_rn(eig[c], model_noise2);
                const float lambda = diff > 0.0f ? diff : 0.0f;
                if (lambda > 0.0f) {
                    trace = __fadd_rn(trace, __fdiv_rn(lambda, __fadd_rn(lambda, sigma2)));
                    vol = __fadd_rn(vol, terms[c]);
                }
            }
            const float tau = __fadd_rn(
                __fadd_rn(P.weight_epsilon, __fdiv_rn(static_cast<float>(D), static_cast<float>(B))), trace);
            lgw = P.weight_alpha == 0.0f ? 0.0f : __fmul_rn(-P.weight_alpha, cr_logf(tau));
            volume = __fdiv_rn(vol, static_cast<float>(D));
        }

        // rows in tiles of four: membership scores and reconstruction
        float min_score = kInf;
        for (int t0 = 0; t0 < S; t0 += 4) {
            const int nrows = min(4, S - t0);
            {
                // a missing row repeats the first
                const size_t b0 = bases[t0], b1 = bases[t0 + (nrows > 1 ? 1 : 0)];
                const size_t b2 = bases[t0 + (nrows > 2 ? 2 : 0)], b3 = bases[t0 + (nrows > 3 ? 3 : 0)];
#pragma unroll
                for (int jj = 0; jj < kCols; ++jj) {
                    const float* nz = L.noisy + off[jj];
                    const float x0 = __ldg(nz + b0), x1 = __ldg(nz + b1), x2 = __ldg(nz + b2), x3 = __ldg(nz + b3);
                    float4* u4 = reinterpret_cast<float4*>(U) + lane + 32 * jj;
                    if constexpr (kFinal) {
                        const float* bs = L.basic + off[jj];
                        const float y0 = __ldg(bs + b0), y1 = __ldg(bs + b1), y2 = __ldg(bs + b2), y3 = __ldg(bs + b3);
                        *u4 = make_float4(__fsub_rn(y0, mm[jj]), __fsub_rn(y1, mm[jj]), __fsub_rn(y2, mm[jj]),
                                          __fsub_rn(y3, mm[jj]));
                        reinterpret_cast<float4*>(V)[lane + 32 * jj] =
                            make_float4(__fsub_rn(x0, cc[jj]), __fsub_rn(x1, cc[jj]), __fsub_rn(x2, cc[jj]),
                                        __fsub_rn(x3, cc[jj]));
                    } else {
                        *u4 = make_float4(__fsub_rn(x0, mm[jj]), __fsub_rn(x1, mm[jj]), __fsub_rn(x2, mm[jj]),
                                          __fsub_rn(x3, mm[jj]));
                    }
                }
            }
            __syncwarp();
            // chains of rows 2 h, 2 h + 1 against components q4 .. q4 + 3
            float2 am[2][2], ar[2][2], an = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int p = 0; p < 2; ++p) am[i][p] = ar[i][p] = make_float2(0.0f, 0.0f);
            const float* bp = basis + j8 * kWarpLdb + q4;
            const float* up = U + 4 * j8 + 2 * h;
            const float* vp = V + 4 * j8 + 2 * h;
#pragma unroll 8
            for (int m = 0; m < kChain; ++m) {
                const float4 b = *reinterpret_cast<const float4*>(bp + m * 8 * kWarpLdb);
                const float2 b01 = make_float2(b.x, b.y), b23 = make_float2(b.z, b.w);
                const float2 u = *reinterpret_cast<const float2*>(up + m * 32);
                am[0][0] = fma2_rn(dup2(u.x), b01, am[0][0]);
                am[0][1] = fma2_rn(dup2(u.x), b23, am[0][1]);
                am[1][0] = fma2_rn(dup2(u.y), b01, am[1][0]);
                am[1][1] = fma2_rn(dup2(u.y), b23, am[1][1]);
                an = fma2_rn(u, u, an);
                if constexpr (kFinal) {
                    const float2 v = *reinterpret_cast<const float2*>(vp + m * 32);
                    ar[0][0] = fma2_rn(dup2(v.x), b01, ar[0][0]);
                    ar[0][1] = fma2_rn(dup2(v.x), b23, ar[0][1]);
                    ar[1][0] = fma2_rn(dup2(v.y), b01, ar[1][0]);
                    ar[1][1] = fma2_rn(dup2(v.y), b23, ar[1][1]);
                }
            }
            // fold: row by bit 2 of j8, component by bits 1 and 0 (the
            // additions of reduce8: xor 4, then 2, then 1)
            const auto fold = [&](const float2 (&v)[2][2]) {
                const bool hi = j8 & 4;
                float2 r[2];
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    r[p].x = fold_half(hi ? v[1][p].x : v[0][p].x, hi ? v[0][p].x : v[1][p].x, 4);
                    r[p].y = fold_half(hi ? v[1][p].y : v[0][p].y, hi ? v[0][p].y : v[1][p].y, 4);
                }
                const bool second = j8 & 2;
                const float x = fold_half(second ? r[1].x : r[0].x, second ? r[0].x : r[1].x, 2);
                const float y = fold_half(second ? r[1].y : r[0].y, second ? r[0].y : r[1].y, 2);
                return fold_half((j8 & 1) ? y : x, (j8 & 1) ? x : y, 1);
            };
            const float mk = fold(am);
            float rk = mk;
            if constexpr (kFinal) rk = fold(ar);
            float* sc = kScatter ? wr + lay.recon + 8 * t0 : wr + lay.proj;  // [component][row]
            sc[comp_l * 4 + row_l] = __fmul_rn(coef[comp_l], rk);
            if (membership_on) {
                const float p2 = __fmul_rn(mk, mk);
                square[8 * row_l + comp_l] = p2;
                quot[8 * row_l + comp_l] = __fdiv_rn(p2, denom[comp_l]);
                float n = fold_half((j8 & 4) ? an.y : an.x, (j8 & 4) ? an.x : an.y, 4);
                n = __fadd_rn(n, __shfl_xor_sync(0xffffffffu, n, 2));
                n = __fadd_rn(n, __shfl_xor_sync(0xffffffffu, n, 1));
                if (q4 == 0 && (j8 & 3) == 0) norms[row_l] = n;
                __syncwarp();
                if (lane < nrows) {
                    float distance = 0.0f, projected = 0.0f;
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        if (c >= R) break;
                        distance = __fadd_rn(distance, quot[8 * lane + c]);
                        projected = __fadd_rn(projected, square[8 * lane + c]);
                    }
                    const float res = __fsub_rn(norms[lane], projected);
                    distance = __fadd_rn(distance, __fdiv_rn(res > 0.0f ? res : 0.0f, mem2));
                    const float score = __fdiv_rn(__fsub_rn(distance, static_cast<float>(D)), score_scale);
                    scores[t0 + lane] = score;
                    min_score = std_min(min_score, score);
                }
            }
            __syncwarp();
            if constexpr (!kScatter) {
                float o[4][kCols];
                warp_reconstruct<kCols>(basis, sc, coef, R, lane, cc, o);
                float* out = L.filtered + static_cast<size_t>(r0 + t0) * L.row_dim + mc * D + lane;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i >= nrows) break;
#pragma unroll
                    for (int jj = 0; jj < kCols; ++jj) out[static_cast<size_t>(i) * L.row_dim + 32 * jj] = o[i][jj];
                }
                __syncwarp();
            }
        }
        // each of lanes 0-3 holds the least score of its rows
        min_score = std_min(min_score, __shfl_xor_sync(0xffffffffu, min_score, 1));
        min_score = std_min(min_score, __shfl_xor_sync(0xffffffffu, min_score, 2));
        min_score = __shfl_sync(0xffffffffu, min_score, 0);
        // aggregation weights (accumulate_aggregation_model + finalize)
        for (int i = lane; i < S; i += 32) {
            const float lw0 = model_log_weight(P, membership_on, lgw, volume, scores[i], min_score);
            if (models > 1) {
                L.logw[static_cast<size_t>(r0 + i) * models + mc] = lw0;
                continue;
            }
            float w = 1.0f;
            if (weights_enabled) {
                float lw = __fadd_rn(0.0f, lw0);
                lw = lw < -80.0f ? -80.0f : (80.0f < lw ? 80.0f : lw);
                w = cr_expf(lw);
            }
            L.weights[r0 + i] = w;
            if constexpr (kScatter) wr[lay.rw + i] = w;
        }
        __syncwarp();
        if constexpr (kScatter) {
            // each row rebuilt from its scaled projections and added into the
            // stack with its weight
            for (int t0 = 0; t0 < S; t0 += 4) {
                float o[4][kCols];
                warp_reconstruct<kCols>(basis, wr + lay.recon + 8 * t0, coef, R, lane, cc, o);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (t0 + i >= S) break;
                    scatter_row(L, rows[t0 + i], o[i], wr[lay.rw + t0 + i], lane);
                }
            }
            __syncwarp();
        }
    }
}

// Weights of the rows of an uncoupled group: the log-weight terms of its
// plane models summed in plane order, times 1 / models, clamped and
// exponentiated (finalize_aggregation_weights, core.cpp:276-294).  Equal
// groups already hold their default-model weight.
__global__ void combine_weights_kernel(FilterLaunch L) {
    const StageConfig& P = L.cfg;
    const bool weights_enabled = P.weight_alpha != 0.0f || P.weight_beta != 0.0f || P.weight_gamma != 0.0f;
    const int models = L.models;
    const float inv_models = __fdiv_rn(1.0f, static_cast<float>(models));
    const int rows = L.counters->rows;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const int a = L.row_group[r];
        if (L.flags[static_cast<size_t>(a) * models] != 0) continue;
        float w = 1.0f;
        if (weights_enabled) {
            float acc = 0.0f;
            for (int c = 0; c < models; ++c) acc = __fadd_rn(acc, L.logw[static_cast<size_t>(r) * models + c]);
            float lw = __fmul_rn(acc, inv_models);
            lw = lw < -80.0f ? -80.0f : (80.0f < lw ? 80.0f : lw);
            w = cr_expf(lw);
        }
        L.weights[r] = w;
    }
}

// Segment width, row stride and per-group floats of jacobi_kernel for matrices of
// N > 32 rows: two groups per warp while both fit in shared memory (N up to 119),
// else one.  Rows are padded to N + 1.
struct JacobiShape {
    int seg, ld, gstride;
};
JacobiShape jacobi_shape(int N) {
    const int ld = N + 1;
    const int gstride = 2 * N * ld + N;
    const int seg = 2 * static_cast<size_t>(gstride) * sizeof(float) > kFilterSharedLimit ? 32 : 16;
    return JacobiShape{seg, ld, gstride};
}

template <int N, int kSeg>
cudaError_t launch_jacobi_small(const FilterLaunch& L, int max_groups, cudaStream_t stream) {
    auto kernel = L.mixed ? jacobi_small_kernel<N, kSeg, true> : jacobi_small_kernel<N, kSeg, false>;
    const size_t smem = jacobi_small_bytes(N, kSeg);
    const cudaError_t err = raise_smem_limit(reinterpret_cast<const void*>(kernel), smem);
    if (err != cudaSuccess) return err;
    constexpr int kGroups = 32 / kSeg;
    kernel<<<(max_groups + kGroups - 1) / kGroups, 32, smem, stream>>>(L);
    return cudaGetLastError();
}

template <int D>
cudaError_t launch_apply_warp(const FilterLaunch& L, int max_groups, cudaStream_t stream) {
    const bool scatter = L.scatter != nullptr;
    const bool final_stage = L.stage == 1;
    const WarpApplyLayout lay = warp_apply_layout(D, L.max_rows, final_stage, scatter);
    const size_t smem = (static_cast<size_t>(D) + static_cast<size_t>(kWarpApplyWarps) * lay.per_warp) * sizeof(float);
    auto kernel = final_stage ? (scatter ? apply_warp_kernel<D, true, true> : apply_warp_kernel<D, true, false>)
                              : (scatter ? apply_warp_kernel<D, false, true> : apply_warp_kernel<D, false, false>);
    cudaError_t err = raise_smem_limit(reinterpret_cast<const void*>(kernel), static_cast<int>(smem));
    if (err != cudaSuccess) return err;
    const int ctas = std::max(1, std::min((max_groups + kWarpApplyWarps - 1) / kWarpApplyWarps, 148 * 8));
    kernel<<<ctas, 32 * kWarpApplyWarps, smem, stream>>>(L);
    return cudaGetLastError();
}

// Warps per block of the row-tile apply for this shape, 0 where the
// row-per-warp kernel runs: no rank, ranks above 32, dimensions of 16 and less
// (their dots have an order of their own), and shapes whose block does not fit
// even with one warp.  Fewer warps than kTileWarps only where four do not fit, so
// that such shapes keep the kernel: with 64 rows from dimension 1456 (Basic) or
// 1033 (Final) at ranks up to 16, from 1003 or 777 above.
int tile_apply_warps(const FilterLaunch& L) {
    if (L.rank < 1 || L.rank > 32 || L.dim <= 16) return 0;
    const int Bmax = std::min(L.model_cap, L.max_rows);
    for (int warps = kTileWarps; warps >= 1; warps /= 2)
        if (static_cast<size_t>(tile_apply_layout(L.dim, Bmax, L.rank > 16 ? 2 : 1, L.max_rows, warps, L.stage == 1)
                                    .bytes) + kFilterStaticShared <= kFilterSharedLimit)
            return warps;
    return 0;
}

// The shapes of the warp-per-group apply, as far as its block's shared memory
// goes (thousands of rows per group do not fit).
bool warp_apply_shape(const FilterLaunch& L, bool scatter) {
    const int D = L.dim;
    const int Bmax = std::min(L.model_cap, L.max_rows);
    if (L.rank > 8 || Bmax > 8 || L.nmax != Bmax || (D != 64 && D != 128 && D != 192 && D != 256)) return false;
    const WarpApplyLayout lay = warp_apply_layout(D, L.max_rows, L.stage == 1, scatter);
    return (static_cast<size_t>(D) + static_cast<size_t>(kWarpApplyWarps) * lay.per_warp) * sizeof(float) <=
           kFilterSharedLimit;
}

}  // namespace

size_t filter_shared_bytes(const FilterLaunch& L) {
    const int D = L.dim;
    const int Bmax = std::min(L.model_cap, L.max_rows);
    const int R = L.rank;
    const size_t colpad = static_cast<size_t>((D + 3) & ~3);
    const size_t rows_bytes = static_cast<size_t>(Bmax) * (D + 8) * sizeof(float);
    const int groups_per_cta = rows_bytes > 8 * 1024 ? 1 : kPrepareWarps;
    size_t need = (colpad + static_cast<size_t>(groups_per_cta) * Bmax * (D + 8)) * sizeof(float) +
                  static_cast<size_t>(groups_per_cta) * L.max_rows * sizeof(size_t);
    if (R > 0 && L.nmax > 32) {  // the smaller ones' kernel takes 25 KB at most
        const JacobiShape js = jacobi_shape(L.nmax);
        need = std::max(need, static_cast<size_t>(32 / js.seg) * js.gstride * sizeof(float));
    }
    // the largest apply block.  The row tiles are sized to what is there
    // (tile_apply_warps), so this bound is the row-per-warp block's; ranks up
    // to 16 above dimension 16 keep the bound they have always been refused at
    // (eight warps of two-row tiles), which does not change with the kernels
    need = std::max(need, apply_layout(D, Bmax, R, L.max_rows, kApplyWarps).bytes);
    if (R >= 1 && R <= 16 && D > 16) {
        const size_t ldu = static_cast<size_t>((D + 23) & ~31) + 8;
        const size_t tiles = kApplyWarps * ((L.stage == 1 ? 2 : 1) * 2 * ldu + 66);
        const size_t model = static_cast<size_t>(Bmax) * (D + 1);
        const size_t fixed = colpad + 2 * static_cast<size_t>(D) + R * ldu + static_cast<size_t>(R) * Bmax +
                             5 * static_cast<size_t>(R) + L.max_rows;
        need = std::max(need, (((fixed + std::max(tiles, model) + 1) & ~static_cast<size_t>(1)) +
                               2 * static_cast<size_t>(L.max_rows)) * sizeof(float));
    }
    return need;
}

size_t filter_shared_limit() { return kFilterSharedLimit; }

bool filter_can_scatter(const FilterLaunch& L) { return L.models == 1 && warp_apply_shape(L, true); }

int filter_scatter_pack(const FilterLaunch& L) {
    if (!filter_can_scatter(L)) return 0;
    if (L.channels == 1 && L.dim == L.patch_dim) return 2;
    if (L.channels == 3 && L.dim == 192 && L.patch_dim == 64) return 4;
    return 0;
}

cudaError_t launch_filter(const FilterLaunch& L, int max_groups_in, cudaStream_t stream) {
    if (max_groups_in <= 0) return cudaSuccess;
    const int max_groups = max_groups_in * L.models;  // models to filter at most
    const int D = L.dim;
    const int Bmax = std::min(L.model_cap, L.max_rows);
    const int R = L.rank;
    const size_t colpad = static_cast<size_t>((D + 3) & ~3);
    // prepare: a warp per group while a group's model rows take at most
    // 8 KB of shared memory, else a CTA per group
    {
        const size_t rows_bytes = static_cast<size_t>(Bmax) * (D + 8) * sizeof(float);
        const bool wide = rows_bytes > 8 * 1024;
        const int groups_per_cta = wide ? 1 : kPrepareWarps;
        const size_t fixed = colpad * sizeof(float) +
                             static_cast<size_t>(groups_per_cta) * L.max_rows * sizeof(size_t);
        size_t smem = fixed + static_cast<size_t>(groups_per_cta) * Bmax * (D + 8) * sizeof(float);
        // the blocked Gram's columns: an odd number of 16-byte units each, so
        // that the 8 columns of a quarter warp start on different banks (without
        // the odd unit where a CTA holds four groups, whose number counts more,
        // or where it does not fit); rows where neither does
        FilterLaunch P = L;
        P.gram_columns = 0;
        if (D >= 64 && Bmax < D && (wide || (Bmax > 4 && Bmax <= 8))) {
            const int quads = (Bmax + 3) / 4;
            for (int ldc : {4 * (wide ? quads | 1 : quads), 4 * quads}) {
                const size_t bytes = fixed + (groups_per_cta * L.max_rows & 1) * sizeof(size_t) +
                                     static_cast<size_t>(groups_per_cta) * D * ldc * sizeof(float);
                if (bytes + kFilterStaticShared > kFilterSharedLimit) continue;
                P.gram_columns = ldc;
                smem = bytes;
                break;
            }
        }
        // rows held in registers: with several columns per thread their loads
        // overlap (57k groups of dimension 294 0.49 -> 0.35 and 0.91 -> 0.88 ms,
        // 32k warps of dimension 192 191 -> 124 us); with one, the registers cost
        // more blocks than that saves (130k groups of dimension 128, Final, 1.33
        // -> 1.61 ms)
        const bool held = P.gram_columns > 0 && Bmax <= 16 && D > 32 * kPrepareWarps;
        auto kernel = !wide ? (P.gram_columns > 0 ? prepare_kernel<1, 8> : prepare_kernel<1, 0>)
                            : (held ? prepare_kernel<kPrepareWarps, 16> : prepare_kernel<kPrepareWarps, 0>);
        cudaError_t err = raise_smem_limit(reinterpret_cast<const void*>(kernel),
                                               static_cast<int>(smem));
        if (err != cudaSuccess) return err;
        const int ctas = std::min((max_groups + groups_per_cta - 1) / groups_per_cta, 148 * 16);
        kernel<<<ctas, 32 * kPrepareWarps, smem, stream>>>(P);
        if ((err = cudaGetLastError()) != cudaSuccess) return err;
    }
    // jacobi
    if (R > 0) {
        const int N = L.nmax;  // largest matrix: model rows, or the dimension of covariance models
        if (N <= 32) {
            // lanes per group: more lanes repeat the angle on more lanes, but
            // leave fewer rows per lane and more warps to hide its latency
            // (1, 2 and 4 lanes: N = 8, 32k groups 77, 81, 86 us; N = 16, 57k
            // groups 0.95, 0.65, 0.66 ms, 0.6k groups 440, 290, 218 us, and
            // with FP64 angles, 130k groups, 4.1, 3.55, 2.85 ms, the angles then
            // without the test of their rounding)
            cudaError_t err;
            if (N <= 8) err = launch_jacobi_small<8, 2>(L, max_groups, stream);
            else if (N <= 16) err = launch_jacobi_small<16, 4>(L, max_groups, stream);
            else if (N <= 24) err = launch_jacobi_small<24, 4>(L, max_groups, stream);
            else err = launch_jacobi_small<32, 8>(L, max_groups, stream);
            if (err != cudaSuccess) return err;
        } else {
            const JacobiShape js = jacobi_shape(N);
            const int seg = js.seg, ld = js.ld, gstride = js.gstride;
            const size_t per_group = static_cast<size_t>(gstride) * sizeof(float);
            int warps = 8;
            while (warps > 1 && static_cast<size_t>(warps) * (32 / seg) * per_group > 160 * 1024) warps /= 2;
            const size_t smem = static_cast<size_t>(warps) * (32 / seg) * per_group;
            cudaError_t err = raise_smem_limit(reinterpret_cast<const void*>(jacobi_kernel),
                                                   static_cast<int>(smem));
            if (err != cudaSuccess) return err;
            const int per_cta = warps * (32 / seg);
            const int ctas = std::max(1, std::min((max_groups + per_cta - 1) / per_cta, 148 * 32));
            jacobi_kernel<<<ctas, 32 * warps, smem, stream>>>(L, seg, ld, gstride);
            if ((err = cudaGetLastError()) != cudaSuccess) return err;
        }
    }
    // apply
#ifndef VNLB_APPLY_WARP
#define VNLB_APPLY_WARP 1  // the warp-per-group apply for its shapes; a build parameter for comparisons
#endif
    const bool warp_shape = warp_apply_shape(L, L.scatter != nullptr);
    if (L.scatter && !(warp_shape && L.models == 1)) return cudaErrorInvalidValue;  // see filter_can_scatter
    if (L.scatter && L.scatter_pack != 0 &&
        (L.scatter_pack != filter_scatter_pack(L) ||
         reinterpret_cast<uintptr_t>(L.scatter) % (L.scatter_pack * sizeof(float)) != 0))
        return cudaErrorInvalidValue;
    if ((VNLB_APPLY_WARP || L.scatter) && warp_shape && (!L.apply_general || L.scatter)) {
        cudaError_t err = D == 64    ? launch_apply_warp<64>(L, max_groups, stream)
                          : D == 128 ? launch_apply_warp<128>(L, max_groups, stream)
                          : D == 192 ? launch_apply_warp<192>(L, max_groups, stream)
                                     : launch_apply_warp<256>(L, max_groups, stream);
        if (err != cudaSuccess) return err;
    } else {
        const int tile_warps = tile_apply_warps(L);
        cudaError_t err = cudaSuccess;
        if (tile_warps > 0) {
            const bool wide = R > 16, final_stage = L.stage == 1;
            auto kernel = wide ? (final_stage ? apply_tile_kernel<2, true> : apply_tile_kernel<2, false>)
                               : (final_stage ? apply_tile_kernel<1, true> : apply_tile_kernel<1, false>);
            const TileApplyLayout lay = tile_apply_layout(D, Bmax, wide ? 2 : 1, L.max_rows, tile_warps, final_stage);
            err = raise_smem_limit(reinterpret_cast<const void*>(kernel), lay.bytes);
            if (err != cudaSuccess) return err;
            const int ctas = std::min(max_groups, 148 * 8);
            kernel<<<ctas, 32 * tile_warps, lay.bytes, stream>>>(L);
        } else {
            const ApplyLayout lay = apply_layout(D, Bmax, R, L.max_rows, kApplyWarps);
            err = raise_smem_limit(reinterpret_cast<const void*>(apply_kernel), static_cast<int>(lay.bytes));
            if (err != cudaSuccess) return err;
            const int ctas = std::min(max_groups, 148 * 8);
            apply_kernel<<<ctas, kApplyThreads, lay.bytes, stream>>>(L);
        }
        if ((err = cudaGetLastError()) != cudaSuccess) return err;
    }
    if (L.models > 1) {
        const long long rows = static_cast<long long>(max_groups_in) * L.max_rows;
        const int ctas = static_cast<int>(std::max<long long>(1, std::min<long long>((rows + 255) / 256, 148 * 8)));
        combine_weights_kernel<<<ctas, 256, 0, stream>>>(L);
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

}  // namespace vnlbgpu
