// Contribution stacks and their normalisation (plain form).
//
// Reference semantics: write_sample_contributions_coupled_* and
// write_group_contributions (src/core/core.cpp:1587-1795) accumulate, pixel
// by pixel, the weighted filtered patches of the processed groups in raster
// group order and row order; render_aggregate_frame (src/vs/plugin.cpp:
// 966-1045) sums the stacks of the contributing anchor frames in anchor order
// and divides.
//
// Owner-computes tiles instead of atomics: a CTA owns one tile of up to four
// slots of the anchor frame's stack.  It finds the groups whose matches can
// reach the tile (anchors within the search reach, a contiguous range of the
// raster-ordered active list), collects the rows whose patch covers the tile
// in increasing global row order (= CPU order), and every thread applies them
// to its pixel in that order.  The result is bit-identical to the CPU's
// sequential accumulation, needs no clear, and writes every stack value
// exactly once.
#include "vnlb_kernels.h"

namespace vnlbgpu {
namespace {

constexpr int kTileThreads = kTile * kTile;
constexpr int kTileWarps = kTileThreads / 32;
constexpr int kMaxGridRows = 64;   // grid rows per collection round
constexpr int kTileSlots = 4;      // slots per CTA
constexpr int kTileEntries = 512;  // collected rows held before they are applied
constexpr int kTileBatch = 4;      // rows whose samples a warp has in flight

struct __align__(16) Entry {
    int r;     // global row
    int xy;    // x | y << 16
    float w;   // row weight
    int slot;  // slot of the row's first layer, relative to the CTA's first slot
};

// One CTA per (16x16 tile, four slots), one pixel per thread, 8 x 4 pixels
// per warp.  The rows that can cover the tile form one contiguous row range
// per grid row in reach (reach tables, built per grid); their concatenation is
// in increasing global row order.  All threads test 256 rows at a time, an
// ordered block compaction appends the covering ones to a list, and when the
// list could overflow (or the rows end) every warp applies it: per 32 entries
// and slot a ballot picks the rows whose patch touches the warp's 8 x 4 pixels
// (8 x 8 patches: a third of the tile's; visiting all of them on every thread
// left 7 of 8 lanes idle), and the samples of kTileBatch rows are loaded
// before the first is added.  The additions are the CPU's accumulation order.
// Bound by the latency of the scattered sample loads; one row at a time took
// 305 us at 1920x1080 YUV (8 rows per group), 1.15 ms at 960x540 YUV (groups
// of 16, patch_time 2); this takes 212 us and 0.67 ms.
template <int kChannels>
__global__ void __launch_bounds__(kTileThreads) tile_kernel(TileLaunch L) {
    __shared__ Entry entries[kTileEntries];
    __shared__ int s_rbeg[kMaxGridRows];
    __shared__ int s_rpre[kMaxGridRows + 1];
    __shared__ int s_warp[2][kTileWarps];
    extern __shared__ float window[];

    const int tx = blockIdx.x, ty = blockIdx.y;
    const int tx0 = tx * kTile, ty0 = ty * kTile;
    const int first_slot = blockIdx.z * kTileSlots;
    const int slots = min(kTileSlots, L.slots - first_slot);
    const int P = L.P;
    const int Pt = L.Pt;
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    for (int i = tid; i < P * P; i += blockDim.x) window[i] = L.window[i];

    const int wx = tx0 + 8 * (warp & 1), wy = ty0 + 4 * (warp >> 1);  // the warp's pixels
    const int px = wx + (lane & 7);
    const int py = wy + (lane >> 3);
    float num[kTileSlots][kChannels];
    float wt[kTileSlots];
#pragma unroll
    for (int s = 0; s < kTileSlots; ++s) {
        wt[s] = 0.0f;
#pragma unroll
        for (int c = 0; c < kChannels; ++c) num[s][c] = 0.0f;
    }
    const int fused_cols = (P == kLanes || P == 2 * kLanes) ? P : (P / kLanes) * kLanes;
    const bool unfused_window = !L.coupled || L.windowed;
    const int2 grid_rows = L.tile_grid_rows[ty];
    const int slot_base = L.search_bwd - L.anchor_frame - first_slot;  // slot = frame + slot_base

    const auto apply = [&](int count) {
        for (int e0 = 0; e0 < count; e0 += 32) {
            bool touches = false;
            int slot0 = 0;
            if (e0 + lane < count) {
                const Entry en = entries[e0 + lane];
                const int x = en.xy & 0xffff, y = en.xy >> 16;
                touches = x < wx + 8 && x + P > wx && y < wy + 4 && y + P > wy;
                slot0 = en.slot;
            }
            if (!__any_sync(0xffffffffu, touches)) continue;
#pragma unroll
            for (int s = 0; s < kTileSlots; ++s) {
                if (s >= slots) break;
                unsigned mask = __ballot_sync(0xffffffffu, touches && slot0 <= s && s < slot0 + Pt);
                while (mask) {
                    float val[kTileBatch][kChannels], w[kTileBatch];
                    bool fused[kTileBatch], inside[kTileBatch];
#pragma unroll
                    for (int k = 0; k < kTileBatch; ++k) {
                        inside[k] = false;
                        if (!mask) continue;
                        const Entry en = entries[e0 + __ffs(mask) - 1];
                        mask &= mask - 1;
                        const unsigned dx = static_cast<unsigned>(px - (en.xy & 0xffff));
                        const unsigned dy = static_cast<unsigned>(py - (en.xy >> 16));
                        inside[k] = dx < static_cast<unsigned>(P) && dy < static_cast<unsigned>(P);
                        if (!inside[k]) continue;
                        const int at = static_cast<int>(dy) * P + static_cast<int>(dx);
                        const float* f = L.filtered + static_cast<size_t>(en.r) * L.dim + (s - en.slot) * P * P + at;
#pragma unroll
                        for (int c = 0; c < kChannels; ++c) val[k][c] = __ldg(f + c * L.patch_dim);
                        fused[k] = !unfused_window && static_cast<int>(dx) < fused_cols;
                        w[k] = unfused_window ? __fmul_rn(en.w, window[at]) : en.w;
                    }
#pragma unroll
                    for (int k = 0; k < kTileBatch; ++k) {
                        if (!inside[k]) continue;
#pragma unroll
                        for (int c = 0; c < kChannels; ++c)
                            num[s][c] = fused[k] ? __fmaf_rn(w[k], val[k][c], num[s][c])
                                                 : __fadd_rn(num[s][c], __fmul_rn(w[k], val[k][c]));
                        wt[s] = __fadd_rn(wt[s], w[k]);
                    }
                }
            }
        }
    };

    int held = 0;  // entries collected and not applied (uniform)
    int parity = 0;
    for (int k0 = grid_rows.x; k0 < grid_rows.y; k0 += kMaxGridRows) {
        const int nk = min(kMaxGridRows, grid_rows.y - k0);
        __syncthreads();
        if (tid < nk) {
            const int2 anchors = L.tile_anchors[static_cast<size_t>(k0 + tid) * L.tiles_x + tx];
            const int rb = L.row_offset[L.active_prefix[anchors.x]];
            const int re = L.row_offset[L.active_prefix[anchors.y]];
            s_rbeg[tid] = rb;
            s_rpre[tid + 1] = re - rb;
        }
        __syncthreads();
        if (warp == 0) {
            // inclusive prefix of the two halves of the 64 row ranges
            int a = lane < nk ? s_rpre[lane + 1] : 0, b = lane + 32 < nk ? s_rpre[lane + 33] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int va = __shfl_up_sync(0xffffffffu, a, o), vb = __shfl_up_sync(0xffffffffu, b, o);
                if (lane >= o) {
                    a += va;
                    b += vb;
                }
            }
            b += __shfl_sync(0xffffffffu, a, 31);
            s_rpre[lane + 1] = a;
            s_rpre[lane + 33] = b;
            if (lane == 0) s_rpre[0] = 0;
        }
        __syncthreads();
        const int total = s_rpre[nk];
        for (int chunk = 0; chunk < total; chunk += kTileThreads) {
            // test one virtual row per thread
            const int vrow = chunk + tid;
            bool hit = false;
            Entry en{};
            if (vrow < total) {
                int lo = 0, hi = nk - 1;  // last k with s_rpre[k] <= vrow
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (s_rpre[mid] <= vrow) lo = mid;
                    else hi = mid - 1;
                }
                const int r = s_rbeg[lo] + (vrow - s_rpre[lo]);
                const MatchRow m = L.row_info[r];
                if (m.x <= tx0 + kTile - 1 && m.x + P - 1 >= tx0 && m.y <= ty0 + kTile - 1 && m.y + P - 1 >= ty0) {
                    // the temporal windows shift at the clip's ends: a row's
                    // first layers may lie before the slots while a later one
                    // lands in them
                    const int slot = m.frame + slot_base;
                    if (slot > -Pt && slot < slots) {
                        hit = true;
                        en.r = r;
                        en.xy = m.x | (m.y << 16);
                        en.w = L.weights[r];
                        en.slot = slot;
                    }
                }
            }
            // ordered append
            const unsigned ballot = __ballot_sync(0xffffffffu, hit);
            if (lane == 0) s_warp[parity][warp] = __popc(ballot);
            __syncthreads();
            int at = held;
#pragma unroll
            for (int w = 0; w < kTileWarps; ++w) {
                const int n = s_warp[parity][w];
                if (w < warp) at += n;
                held += n;
            }
            parity ^= 1;
            if (hit) entries[at + __popc(ballot & ((1u << lane) - 1u))] = en;
            if (held > kTileEntries - kTileThreads) {
                __syncthreads();
                apply(held);
                __syncthreads();
                held = 0;
            }
        }
    }
    __syncthreads();
    apply(held);
    // every pixel, so the stack needs no clearing
    if (px < L.width && py < L.height) {
        const size_t plane = static_cast<size_t>(L.width) * L.height;
#pragma unroll
        for (int s = 0; s < kTileSlots; ++s) {
            if (s >= slots) break;
            float* base = L.stack + static_cast<size_t>(first_slot + s) * (kChannels + 1) * plane +
                          static_cast<size_t>(py) * L.width + px;
#pragma unroll
            for (int c = 0; c < kChannels; ++c) base[c * plane] = num[s][c];
            base[kChannels * plane] = wt[s];
        }
    }
}

// A frame from the stacks of its contributing anchors: their slots summed in
// anchor order, divided by the summed weight, the source sample where no weight
// fell.  kPack: the stacks' layout, 0 planar or C+1 pixel-interleaved, one for
// all of them; a thread owns kPixels neighbouring pixels, so every load and
// store is 16 bytes, and the loads of two stacks are in flight at once.  Bound
// by HBM: count * (C+1) + 2 C planes of traffic at most.  (A pixel per thread
// with a scalar load per plane took 112 us for a 1920x1080 YUV frame of three
// planar stacks, 46 us of interleaved ones; now 21 and 22.)
template <int C, int kPack, int kPixels>
__global__ void __launch_bounds__(256) normalize_kernel(NormalizeLaunch L) {
    const size_t plane = static_cast<size_t>(L.width) * L.height;
    const size_t units = plane / kPixels;
    for (size_t u = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; u < units;
         u += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t i = u * kPixels;
        float num[C + 1][kPixels];
#pragma unroll
        for (int c = 0; c <= C; ++c)
#pragma unroll
            for (int q = 0; q < kPixels; ++q) num[c][q] = 0.0f;
#pragma unroll 2
        for (int k = 0; k < L.count; ++k) {
            const float* s = L.stacks[k] + static_cast<size_t>(L.slots[k]) * (C + 1) * plane;
            float v[C + 1][kPixels];
            if constexpr (kPack == 4) {
#pragma unroll
                for (int q = 0; q < kPixels; ++q) {
                    const float4 t = __ldg(reinterpret_cast<const float4*>(s) + i + q);
                    v[0][q] = t.x;
                    v[1][q] = t.y;
                    v[2][q] = t.z;
                    v[C][q] = t.w;
                }
            } else if constexpr (kPack == 2) {
#pragma unroll
                for (int q = 0; q < kPixels; ++q) {
                    const float2 t = __ldg(reinterpret_cast<const float2*>(s) + i + q);
                    v[0][q] = t.x;
                    v[C][q] = t.y;
                }
            } else {
#pragma unroll
                for (int c = 0; c <= C; ++c) {
                    if constexpr (kPixels == 4) {
                        const float4 t = __ldg(reinterpret_cast<const float4*>(s + c * plane + i));
                        v[c][0] = t.x;
                        v[c][1] = t.y;
                        v[c][2] = t.z;
                        v[c][3] = t.w;
                    } else {
                        v[c][0] = __ldg(s + c * plane + i);
                    }
                }
            }
#pragma unroll
            for (int c = 0; c <= C; ++c)
#pragma unroll
                for (int q = 0; q < kPixels; ++q) num[c][q] = __fadd_rn(num[c][q], v[c][q]);
        }
        bool empty = false;
#pragma unroll
        for (int q = 0; q < kPixels; ++q) empty |= !(num[C][q] > 0.0f);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float o[kPixels];
#pragma unroll
            for (int q = 0; q < kPixels; ++q) o[q] = __fdiv_rn(num[c][q], num[C][q]);
            if (empty)
#pragma unroll
                for (int q = 0; q < kPixels; ++q)
                    if (!(num[C][q] > 0.0f)) o[q] = L.source[c * plane + i + q];
            float* out = L.out + c * plane + i;
            if constexpr (kPixels == 4) *reinterpret_cast<float4*>(out) = make_float4(o[0], o[1], o[2], o[3]);
            else out[0] = o[0];
        }
    }
}

// Stacks of both layouts in one frame (a session whose forms changed between
// anchors): a pixel per thread.
__global__ void normalize_mixed_kernel(NormalizeLaunch L) {
    const size_t plane = static_cast<size_t>(L.width) * L.height;
    const int C = L.channels;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < plane;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float num[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        float w = 0.0f;
        for (int k = 0; k < L.count; ++k) {
            const float* s = L.stacks[k] + static_cast<size_t>(L.slots[k]) * (C + 1) * plane;
            if (L.packed[k] == 4) {  // [H][W][C+1] with C = 3: one 16-byte load
                const float4 v = __ldg(reinterpret_cast<const float4*>(s) + i);
                num[0] = __fadd_rn(num[0], v.x);
                num[1] = __fadd_rn(num[1], v.y);
                num[2] = __fadd_rn(num[2], v.z);
                w = __fadd_rn(w, v.w);
            } else if (L.packed[k] == 2) {  // C = 1
                const float2 v = __ldg(reinterpret_cast<const float2*>(s) + i);
                num[0] = __fadd_rn(num[0], v.x);
                w = __fadd_rn(w, v.y);
            } else {
                for (int c = 0; c < C; ++c) num[c] = __fadd_rn(num[c], s[c * plane + i]);
                w = __fadd_rn(w, s[C * plane + i]);
            }
        }
        for (int c = 0; c < C; ++c)
            L.out[c * plane + i] = w > 0.0f ? __fdiv_rn(num[c], w) : L.source[c * plane + i];
    }
}

__global__ void pack_kernel(const float* stack, int width, int height, int channels, int slots, float* out) {
    const size_t plane = static_cast<size_t>(width) * height;
    const size_t total = plane * channels * slots * 2;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t pix = i % plane;
        const size_t rest = i / plane;
        const int is_weight = static_cast<int>(rest % 2);
        const int slot = static_cast<int>((rest / 2) % slots);
        const int c = static_cast<int>(rest / (2 * slots));
        const float* s = stack + static_cast<size_t>(slot) * (channels + 1) * plane;
        out[i] = is_weight ? s[channels * plane + pix] : s[c * plane + pix];
    }
}

// The same packing from a pixel-interleaved stack [slots][H][W][kPack]
// (kPack = C+1 = 4 or 2): one thread per pixel and slot, one vector load,
// 2C coalesced stores.
template <int kPack>
__global__ void pack_interleaved_kernel(const float* stack, int width, int height, int slots, float* out) {
    constexpr int C = kPack - 1;
    const size_t plane = static_cast<size_t>(width) * height;
    const size_t total = plane * slots;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int slot = static_cast<int>(i / plane);
        const size_t pix = i - static_cast<size_t>(slot) * plane;
        const float* s = stack + (static_cast<size_t>(slot) * plane + pix) * kPack;
        float v[kPack];
        if constexpr (kPack == 4) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(s));
            v[0] = q.x;
            v[1] = q.y;
            v[2] = q.z;
            v[3] = q.w;
        } else {
            const float2 q = __ldg(reinterpret_cast<const float2*>(s));
            v[0] = q.x;
            v[1] = q.y;
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const size_t row = static_cast<size_t>(c * slots + slot) * 2;
            out[row * plane + pix] = v[c];
            out[(row + 1) * plane + pix] = v[C];
        }
    }
}

__global__ void aggregate_stacks_kernel(AggregateLaunch L) {
    const size_t plane = static_cast<size_t>(L.width) * L.height;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < plane * L.channels;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int c = static_cast<int>(i / plane);
        const size_t pix = i - static_cast<size_t>(c) * plane;
        const size_t y = pix / L.width;
        const size_t x = pix - y * L.width;
        float num = 0.0f, w = 0.0f;
        for (int k = 0; k < L.count; ++k) {
            const float* s = L.stacks[k] + static_cast<size_t>(c) * L.slots * 2 * plane;
            const size_t row = static_cast<size_t>(L.slots_of[k]) * 2 * L.height + y;
            num = __fadd_rn(num, s[row * L.width + x]);
            w = __fadd_rn(w, s[(row + L.height) * L.width + x]);
        }
        L.out[i] = w > 0.0f ? __fdiv_rn(num, w) : L.source[i];
    }
}

}  // namespace

cudaError_t launch_aggregate_stacks(const AggregateLaunch& L, cudaStream_t stream) {
    const size_t total = static_cast<size_t>(L.width) * L.height * L.channels;
    const int blocks = static_cast<int>(std::min<size_t>((total + 255) / 256, 148 * 16));
    aggregate_stacks_kernel<<<blocks, 256, 0, stream>>>(L);
    return cudaGetLastError();
}

cudaError_t launch_tiles(const TileLaunch& L, cudaStream_t stream) {
    if ((L.channels != 1 && L.channels != 3) || L.width >= (1 << 14) || L.height >= (1 << 14) || L.Pt > 7)
        return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>(L.P) * L.P * sizeof(float);
    const dim3 grid(L.tiles_x, L.tiles_y, (L.slots + kTileSlots - 1) / kTileSlots);
    if (L.channels == 1) tile_kernel<1><<<grid, kTileThreads, smem, stream>>>(L);
    else tile_kernel<3><<<grid, kTileThreads, smem, stream>>>(L);
    return cudaGetLastError();
}

cudaError_t launch_normalize(const NormalizeLaunch& L, cudaStream_t stream) {
    if (L.channels > 4 || L.count > kMaxContributors) return cudaErrorInvalidValue;
    for (int k = 0; k < L.count; ++k) {
        // the vector layouts hold C = 3 (16-byte pixels) or C = 1 (8-byte pixels)
        const int p = L.packed[k];
        if (p != 0 && !(p == L.channels + 1 && (p == 2 || p == 4) &&
                        reinterpret_cast<uintptr_t>(L.stacks[k]) % (p * sizeof(float)) == 0))
            return cudaErrorInvalidValue;
    }
    const size_t plane = static_cast<size_t>(L.width) * L.height;
    bool same = L.count > 0 && (L.channels == 1 || L.channels == 3);
    for (int k = 1; k < L.count; ++k) same &= L.packed[k] == L.packed[0];
    // four pixels per thread need whole 16-byte units in every plane
    bool wide = plane % 4 == 0 && reinterpret_cast<uintptr_t>(L.out) % 16 == 0;
    for (int k = 0; k < L.count; ++k) wide &= reinterpret_cast<uintptr_t>(L.stacks[k]) % 16 == 0;
    const auto run = [&](auto kernel, int pixels) {
        const int blocks = static_cast<int>(std::min<size_t>((plane / pixels + 255) / 256, 148 * 16));
        kernel<<<std::max(blocks, 1), 256, 0, stream>>>(L);
    };
    const int packed = L.count > 0 ? L.packed[0] : 0;
    if (!same) run(normalize_mixed_kernel, 1);
    else if (L.channels == 3 && packed) wide ? run(normalize_kernel<3, 4, 4>, 4) : run(normalize_kernel<3, 4, 1>, 1);
    else if (L.channels == 3) wide ? run(normalize_kernel<3, 0, 4>, 4) : run(normalize_kernel<3, 0, 1>, 1);
    else if (packed) wide ? run(normalize_kernel<1, 2, 4>, 4) : run(normalize_kernel<1, 2, 1>, 1);
    else wide ? run(normalize_kernel<1, 0, 4>, 4) : run(normalize_kernel<1, 0, 1>, 1);
    return cudaGetLastError();
}

cudaError_t launch_pack_stack(const float* stack, int packed, int width, int height, int channels, int slots,
                              float* out, cudaStream_t stream) {
    if (packed != 0 && !(packed == channels + 1 && (packed == 2 || packed == 4) &&
                         reinterpret_cast<uintptr_t>(stack) % (packed * sizeof(float)) == 0))
        return cudaErrorInvalidValue;
    if (packed != 0) {
        const size_t pixels = static_cast<size_t>(width) * height * slots;
        const int blocks = static_cast<int>(std::min<size_t>((pixels + 255) / 256, 148 * 16));
        if (packed == 4) pack_interleaved_kernel<4><<<blocks, 256, 0, stream>>>(stack, width, height, slots, out);
        else pack_interleaved_kernel<2><<<blocks, 256, 0, stream>>>(stack, width, height, slots, out);
        return cudaGetLastError();
    }
    const size_t total = static_cast<size_t>(width) * height * channels * slots * 2;
    const int blocks = static_cast<int>(std::min<size_t>((total + 255) / 256, 148 * 16));
    pack_kernel<<<blocks, 256, 0, stream>>>(stack, width, height, channels, slots, out);
    return cudaGetLastError();
}

}  // namespace vnlbgpu
