// Ordered paste mask and active-group compaction for one anchor frame.
//
// Reference semantics: process_anchor_impl visits the staggered grid in raster
// order and skips an anchor whose mask bit an earlier processed group cleared
// (src/core/core.cpp:1851-1903, apply_frame_paste_mask at :980-1008).  The
// match kernel has already turned every anchor's anchor-frame matches into the
// list of later grid anchors they clear (its "victims"), so the mask only
// needs one bit per grid anchor, in shared memory.
//
// The order only binds anchors that can reach each other: a match lies within
// reach_x columns of its anchor, so an anchor at x is decided once every
// earlier grid row is decided up to x + reach_x.  One block walks the grid as
// a wavefront: warp w takes grid rows w, w + 16, ... and goes along its row in
// batches of 32 anchors, each batch after the row above has passed the reach
// of the batch's last anchor (the rows further up are ahead of that row by the
// same rule, so the row above is all a warp waits for).  A batch is resolved
// in order among its own anchors (only those that name one another cost a
// step), then its living anchors clear their later victims' bits.  The chain
// is about two batches per grid row instead of every batch of the frame:
// one walker over all batches took 390 us at 1920x1080 with step 8 (33k
// anchors) and 1750 us at 960x540 with step 3 (57k anchors, more victims than
// it held on chip); the wavefront takes 265 us and 590 us.
//
// The compaction (active list, exclusive prefix of retained rows, active
// prefix per anchor) follows in two passes of the whole block over the bits.
#include "vnlb_kernels.h"

namespace vnlbgpu {
namespace {

constexpr int kHeld = 24;              // victims held in registers per anchor
constexpr int kPasteThreads = 512;
constexpr int kPasteWarps = kPasteThreads / 32;
constexpr int kPasteSpinLimit = 1 << 22;  // polls of the row above before the walk gives up

// The victims of one batch's anchors, one anchor per lane.  A batch's counts
// are loaded two batches ahead and the victims they name one batch ahead, so
// that the walk waits for neither.
struct PasteBatch {
    int x, count;
    int v[kHeld];
};

__device__ __forceinline__ void load_counts(const PasteLaunch& L, int j, int end, int& x, int& count) {
    x = j < end ? __ldg(&L.anchors[j].x) : 0;
    count = j < end ? __ldg(L.victim_counts + j) : 0;
}

__device__ __forceinline__ void load_victims(const PasteLaunch& L, PasteBatch& b, int j) {
    const int* list = L.victims + static_cast<size_t>(j) * L.victim_stride;
#pragma unroll
    for (int e = 0; e < kHeld; ++e) b.v[e] = e < b.count ? __ldg(list + e) : 0;
}

// Bits [j, j + 32) of the mask.
__device__ __forceinline__ unsigned bits_at(const volatile unsigned* alive, int j, int words) {
    const int w = j >> 5;
    return __funnelshift_r(alive[w], w + 1 < words ? alive[w + 1] : 0u, j & 31);
}

// How far a warp's row has come, in shared memory: the row in the high half,
// the column up to which all its anchors are decided in the low half.  The
// release and acquire order the mask's bits around it; a fence in the polling
// loop would also wait for the loads in flight.
__device__ __forceinline__ void publish(unsigned long long* slot, int row, int x) {
    const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(slot));
    const unsigned long long v = static_cast<unsigned long long>(static_cast<unsigned>(row)) << 32 |
                                 static_cast<unsigned>(x);
    asm volatile("st.release.cta.shared::cta.u64 [%0], %1;" ::"r"(at), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long progress(const unsigned long long* slot) {
    const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(slot));
    unsigned long long v;
    asm volatile("ld.acquire.cta.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(at) : "memory");
    return v;
}

__global__ void __launch_bounds__(kPasteThreads) paste_kernel(PasteLaunch L) {
    extern __shared__ __align__(16) unsigned paste_smem[];
    __shared__ unsigned long long passed[kPasteWarps];  // per row in flight
    __shared__ int active_sum[kPasteWarps + 1], rows_sum[kPasteWarps + 1];
    __shared__ volatile int gave_up;  // one warp's wait ran out: the others stop waiting too
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int words = (L.groups + 31) / 32;
    unsigned* alive = paste_smem;
    for (int w = tid; w < words; w += kPasteThreads) {
        const int rem = L.groups - w * 32;
        alive[w] = rem >= 32 ? 0xffffffffu : ((1u << rem) - 1u);
    }
    if (tid == 0) gave_up = 0;
    if (lane == 0) passed[warp] = static_cast<unsigned long long>(warp) << 32;  // its first row, nothing decided
    __syncthreads();
    const unsigned long long* above = passed + (warp + kPasteWarps - 1) % kPasteWarps;
    bool failed = false;
    for (int row = warp; row < L.grid_rows; row += kPasteWarps) {
        const int begin = L.row_first[row], end = L.row_first[row + 1];
        PasteBatch b, next;
        int x2, count2;
        load_counts(L, begin + lane, end, b.x, b.count);
        load_counts(L, begin + 32 + lane, end, next.x, next.count);
        load_victims(L, b, begin + lane);
        load_counts(L, begin + 64 + lane, end, x2, count2);
        load_victims(L, next, begin + 32 + lane);
        for (int j0 = begin; j0 < end; j0 += 32) {
            const int j = j0 + lane;
            const int n = min(32, end - j0);
            // victims inside the batch, and whether there are later ones
            unsigned mine = 0u;
            bool later = false;
            const int* list = L.victims + static_cast<size_t>(j) * L.victim_stride;
            const int filled = static_cast<int>(__reduce_max_sync(0xffffffffu, b.count));
#pragma unroll
            for (int e = 0; e < kHeld; ++e) {
                if (e >= filled) break;  // uniform
                if (e < b.count) {
                    if (b.v[e] < j0 + n) mine |= 1u << (b.v[e] - j0);
                    else later = true;
                }
            }
            for (int e = kHeld; e < b.count; ++e) {
                const int v = __ldg(list + e);
                if (v < j0 + n) mine |= 1u << (v - j0);
                else later = true;
            }
            const int most = min(kHeld, static_cast<int>(__reduce_max_sync(0xffffffffu, later ? b.count : 0)));
            const int last_x = __shfl_sync(0xffffffffu, b.x, n - 1);
            const int next_x = __shfl_sync(0xffffffffu, next.x, 0);
            // the row above has passed the reach of this batch's last anchor
            if (row > 0 && !failed) {
                int spins = 0;
                for (;;) {
                    const unsigned long long p = progress(above);
                    const int r = static_cast<int>(p >> 32), x = static_cast<int>(p & 0xffffffffu);
                    if (r > row - 1 || (r == row - 1 && x > last_x + L.reach_x)) break;
                    if (++spins >= kPasteSpinLimit || (spins % 256 == 0 && gave_up)) {
                        failed = true;
                        gave_up = 1;
                        break;
                    }
                }
                __syncwarp();
            }
            unsigned bits = bits_at(alive, j0, words);
            if (n < 32) bits &= (1u << n) - 1u;
            const unsigned before = bits;
            for (unsigned m = __ballot_sync(0xffffffffu, mine != 0u); m; m &= m - 1) {
                const int k = __ffs(m) - 1;
                const unsigned kills = __shfl_sync(0xffffffffu, mine, k);
                if ((bits >> k) & 1u) bits &= ~kills;
            }
            const unsigned dead = before & ~bits;
            if (dead && lane < 2) {
                const int sh = j0 & 31;
                const unsigned part = lane == 0 ? dead << sh : (sh ? dead >> (32 - sh) : 0u);
                if (part) atomicAnd(&alive[(j0 >> 5) + lane], ~part);
            }
            if (later && ((bits >> lane) & 1u)) {
#pragma unroll
                for (int e = 0; e < kHeld; ++e) {
                    if (e >= most) break;  // uniform
                    if (e < b.count && b.v[e] >= j0 + n) atomicAnd(&alive[b.v[e] >> 5], ~(1u << (b.v[e] & 31)));
                }
                for (int e = kHeld; e < b.count; ++e) {
                    const int v = __ldg(list + e);
                    if (v >= j0 + n) atomicAnd(&alive[v >> 5], ~(1u << (v & 31)));
                }
            }
            __syncwarp();
            if (lane == 0 && !L.stall) publish(passed + warp, row, j0 + 32 < end ? next_x : 0x7fffffff);
            // the batch after the next one
            b = next;
            next.x = x2;
            next.count = count2;
            load_victims(L, next, j + 64);
            load_counts(L, j + 96, end, x2, count2);
        }
        // this warp's next row: nothing of it is decided
        if (row + kPasteWarps < L.grid_rows && lane == 0 && !L.stall) publish(passed + warp, row + kPasteWarps, 0);
    }
    if (__syncthreads_or(failed)) {
        // the mask is not final: report it, and let no group through
        if (tid == 0) atomicCAS(L.status, 0, kStatusPasteTimeout);
        for (int w = tid; w < words; w += kPasteThreads) alive[w] = 0u;
        __syncthreads();
    }
    // compaction: a contiguous range of words per warp, first the sums ...
    const int per_warp = (words + kPasteWarps - 1) / kPasteWarps;
    const int w0 = warp * per_warp, w1 = min(words, w0 + per_warp);
    int active = 0, rows = 0;
#pragma unroll 4
    for (int w = w0; w < w1; ++w) {
        const unsigned bits = alive[w];
        active += __popc(bits);
        if ((bits >> lane) & 1u) rows += __ldg(L.row_counts + 32 * w + lane);
    }
    rows = __reduce_add_sync(0xffffffffu, rows);
    if (lane == 0) {
        active_sum[warp + 1] = active;
        rows_sum[warp + 1] = rows;
    }
    __syncthreads();
    if (tid == 0) {
        active_sum[0] = rows_sum[0] = 0;
        for (int w = 1; w <= kPasteWarps; ++w) {
            active_sum[w] += active_sum[w - 1];
            rows_sum[w] += rows_sum[w - 1];
        }
    }
    __syncthreads();
    // ... then the positions
    int running_active = active_sum[warp], running_rows = rows_sum[warp];
#pragma unroll 2
    for (int w = w0; w < w1; ++w) {
        const unsigned bits = alive[w];
        const int j = 32 * w + lane;
        const bool me = (bits >> lane) & 1u;
        const int s = me ? __ldg(L.row_counts + j) : 0;
        const int rank = __popc(bits & ((1u << lane) - 1u));
        int prefix = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, prefix, o);
            if (lane >= o) prefix += v;
        }
        if (j < L.groups) L.active_prefix[j] = running_active + rank;
        if (me) {
            const int a = running_active + rank;
            L.active[a] = j;
            L.active_xy[a] = __ldg(L.anchors + j);
            L.row_offset[a] = running_rows + prefix - s;
        }
        running_active += __popc(bits);
        running_rows += __shfl_sync(0xffffffffu, prefix, 31);
    }
    if (tid == 0) {
        const int total_active = active_sum[kPasteWarps], total_rows = rows_sum[kPasteWarps];
        L.row_offset[total_active] = total_rows;
        L.active_prefix[L.groups] = total_active;
        L.counters->active = total_active;
        L.counters->rows = total_rows;
        atomicAdd(L.totals, static_cast<unsigned long long>(total_active));
        atomicAdd(L.totals + 1, static_cast<unsigned long long>(total_rows));
    }
}

__global__ void anchor_map_kernel(const int2* anchors, int count, int width, int* map) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const int2 a = anchors[i];
        map[static_cast<size_t>(a.y) * width + a.x] = i;
    }
}

}  // namespace

cudaError_t launch_anchor_map(const int2* anchors, int count, int width, int* map, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    anchor_map_kernel<<<(count + 255) / 256, 256, 0, stream>>>(anchors, count, width, map);
    return cudaGetLastError();
}

cudaError_t launch_paste(const PasteLaunch& L, cudaStream_t stream) {
    const size_t smem = static_cast<size_t>((L.groups + 31) / 32) * sizeof(unsigned);
    if (smem > 175 * 1024) return cudaErrorInvalidValue;  // more grid anchors than the bitmask holds
    cudaError_t err = raise_smem_limit(reinterpret_cast<const void*>(paste_kernel),
                                           static_cast<int>(smem));
    if (err != cudaSuccess) return err;
    paste_kernel<<<1, kPasteThreads, smem, stream>>>(L);
    return cudaGetLastError();
}

}  // namespace vnlbgpu
