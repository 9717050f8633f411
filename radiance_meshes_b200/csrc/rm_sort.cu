// rm_sort.cu - stage (c): stable onesweep LSD radix sort of (int64 key, int32
// value) pairs on key bits [0, end_bit).
//
// Replaces sort_by_keys (sort_by_keys/sort_by_keys.cu:10-53), i.e.
// cub::DeviceRadixSort::SortPairs(keys, values, n, 0, 32 + msb) with
// msb = bit_length(grid_w * grid_h) (tile_shader_slang.py:57-59).
//
// Design: one histogram kernel computes the digit histograms of every pass in
// a single read of the keys; then one kernel per 8-bit digit pass.  Each CTA of
// a pass takes the next tile of 4096 or 6144 pairs (dynamic tile id, so
// predecessors are always running or done), ranks its keys per warp by the
// lanes of equal digit (warp-striped element order keeps the sort stable),
// publishes per-digit tile counts and obtains each digit's global offset by
// decoupled look-back over earlier tiles (bounded spin; a timeout sets
// RM_STATUS_SORT_TIMEOUT and the CTA proceeds), then scatters through shared
// memory so each digit run is written coalesced.
//
// The equal digits come from 8 ballots: match.any, whose cost grows with the
// distinct values in the warp, made a pass over random digits a seventh longer
// (100M pairs 6830 -> 5930 us).  The look-back has 8 words in flight: one at a
// time, the walk over the tiles that started together was a serial chain
// (30k pairs 72 -> 66 us, 100M 5930 -> 5520).
#include "rm_internal.cuh"

namespace rm {
namespace {

// Tile shape of a pass: kSortThreads threads with kSmallItems pairs each, from
// kLargeFrom pairs on kLargeItems (a digit's run in the output is then half as
// long again, which is what bounds a pass that fills the GPU; 100M pairs of 48
// key bits 5540 -> 4880 us, 4M 279 -> 263; but a tile's own chain is longer:
// 1M 116 -> 126, 30k 70 -> 82).
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSmallItems = 8;
constexpr int kLargeItems = 12;
constexpr int64_t kLargeFrom = 3 << 20;
static_assert(kSortThreads >= 256, "one thread per 8-bit digit");
constexpr int kRadix = 256;
constexpr int kMaxPasses = 8;
// Earlier tiles' words that a look-back has in flight at a time.
constexpr int kLookBack = 8;
constexpr uint32_t kLbAgg = 1u << 30;
constexpr uint32_t kLbInc = 2u << 30;
constexpr uint32_t kLbMask = (1u << 30) - 1;

struct SortHeader {
    uint32_t status;
    uint32_t hist_done;  // CTAs of hist_kernel that have added their counts
    uint32_t pad[2];
    uint32_t counters[kMaxPasses];
    uint32_t hist[kMaxPasses][kRadix];
};

__host__ __forceinline__ int64_t sort_tiles(int64_t n) {
    const int64_t tile = (int64_t)kSortThreads * (n < kLargeFrom ? kSmallItems : kLargeItems);
    return (n + tile - 1) / tile;
}

__host__ __forceinline__ size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct SortLayout {
    size_t lookback_off, alt_keys_off, alt_vals_off, total;
    size_t memset_bytes;  // header + lookback (zeroed every call, status excluded)
};

__host__ SortLayout sort_layout(int64_t n, int npasses) {
    SortLayout L;
    const int64_t tiles = sort_tiles(n) > 0 ? sort_tiles(n) : 1;
    L.lookback_off = align_up(sizeof(SortHeader), 256);
    // room for the small tiles at any n: the size grows with n, so that a
    // workspace for n pairs holds any fewer
    const int64_t room = (n + kSortThreads * kSmallItems - 1) / (kSortThreads * kSmallItems);
    const size_t lb = sizeof(uint32_t) * (size_t)npasses * (size_t)(room > 0 ? room : 1) * kRadix;
    L.alt_keys_off = align_up(L.lookback_off + lb, 256);
    L.alt_vals_off = align_up(L.alt_keys_off + sizeof(uint64_t) * (size_t)(n > 0 ? n : 1), 256);
    L.total = align_up(L.alt_vals_off + sizeof(uint32_t) * (size_t)(n > 0 ? n : 1), 256);
    L.memset_bytes = L.lookback_off + sizeof(uint32_t) * (size_t)npasses * (size_t)tiles * kRadix;
    return L;
}

// Look-back states: the flag and the count share one 32-bit word and nothing
// else is published through it, so relaxed GPU-scope accesses suffice (no
// release fence per store, no acquire per poll).
__device__ __forceinline__ void st_relaxed32(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Digit histograms of every pass in one read of the keys.  Each thread counts
// a contiguous run of kHistRun keys (16-byte vector loads when the run is
// whole and aligned; consecutive threads take consecutive runs) and adds to
// the block's shared histogram only where a pass's digit changes along the
// run, and once at its end: pairs emitted per tet or per tile repeat their
// digits, so most keys add nothing, and no warp vote is needed.
constexpr int kHistThreads = 256;
constexpr int kHistRun = 16;

__global__ void __launch_bounds__(kHistThreads) hist_kernel(const uint64_t* __restrict__ keys, int64_t cap,
                                                            const int64_t* __restrict__ n_dev, int npasses,
                                                            int begin_bit, int end_bit, SortHeader* hdr) {
    __shared__ uint32_t sh[kMaxPasses][kRadix];
    for (int j = threadIdx.x; j < kMaxPasses * kRadix; j += blockDim.x) (&sh[0][0])[j] = 0;
    __syncthreads();
    const int64_t n = n_dev ? min(*n_dev, cap) : cap;
    const uint64_t mask = end_bit >= 64 ? ~0ull : ((1ull << end_bit) - 1);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x * kHistRun;
    for (int64_t s0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * kHistRun; s0 < n; s0 += stride) {
        const int m = (int)min((int64_t)kHistRun, n - s0);  // >= 1
        uint64_t k[kHistRun];
        if (m == kHistRun && ((reinterpret_cast<uintptr_t>(keys + s0) & 15) == 0)) {
            const ulonglong2* v = reinterpret_cast<const ulonglong2*>(keys + s0);
#pragma unroll
            for (int i = 0; i < kHistRun / 2; ++i) {
                const ulonglong2 x = __ldg(v + i);
                k[2 * i] = x.x;
                k[2 * i + 1] = x.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < kHistRun; ++i) k[i] = i < m ? __ldg(keys + s0 + i) : 0ull;
        }
#pragma unroll
        for (int i = 0; i < kHistRun; ++i) k[i] = (k[i] & mask) >> begin_bit;
        for (int p = 0; p < npasses; ++p) {
            const int sh_p = 8 * p;
            uint32_t last = (uint32_t)(k[0] >> sh_p) & 255u, cnt = 1u;
#pragma unroll
            for (int i = 1; i < kHistRun; ++i) {
                const bool v = i < m;
                const uint32_t d = v ? ((uint32_t)(k[i] >> sh_p) & 255u) : last;
                if (d != last) {
                    atomicAdd(&sh[p][last], cnt);
                    last = d;
                    cnt = 0u;
                }
                cnt += v ? 1u : 0u;
            }
            atomicAdd(&sh[p][last], cnt);
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < npasses * kRadix; j += blockDim.x) {
        const uint32_t c = (&sh[0][0])[j];
        if (c) atomicAdd(&(&hdr->hist[0][0])[j], c);
    }
    // the last CTA to get here turns each pass's counts into exclusive offsets
    // (a kernel of its own for this was one launch more per sort)
    __shared__ bool last_cta;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_cta = atomicAdd(&hdr->hist_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last_cta) return;
    __threadfence();
    const int lane = threadIdx.x & 31;
    for (int p = threadIdx.x >> 5; p < npasses; p += kHistThreads / 32) {  // a warp a pass
        uint32_t v[kRadix / 32], sum = 0u;
#pragma unroll
        for (int i = 0; i < kRadix / 32; ++i) {
            v[i] = __ldcg(&hdr->hist[p][lane * (kRadix / 32) + i]);
            sum += v[i];
        }
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        uint32_t run = inc - sum;
#pragma unroll
        for (int i = 0; i < kRadix / 32; ++i) {
            hdr->hist[p][lane * (kRadix / 32) + i] = run;
            run += v[i];
        }
    }
}

template <int ITEMS>
struct PassSmem {
    uint32_t warp_hist[kSortWarps][kRadix];
    uint32_t tile_off[kRadix];
    uint32_t global_start[kRadix];
    uint32_t scan_tmp[kRadix / 32];
    uint32_t tile;
    uint64_t keys[kSortThreads * ITEMS];
    uint32_t vals[kSortThreads * ITEMS];
};

// A pass may be resident while the pass before it still writes kin and vin, so
// these are read past the read-only path (which asks for memory that nobody
// writes during the kernel's lifetime); every pair is read once.
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads, 1024 / kSortThreads) onesweep_kernel(
    const uint64_t* kin, const uint32_t* vin, uint64_t* kout, uint32_t* vout, int64_t cap, const int64_t* __restrict__ n_dev, int pass, int shift,
    uint32_t dmask, SortHeader* hdr, uint32_t* __restrict__ lookback, uint32_t* status, uint32_t spin_limit) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kSortTile = kSortThreads * ITEMS;
    PassSmem<ITEMS>& S = *reinterpret_cast<PassSmem<ITEMS>*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int d = lane; d < kRadix; d += 32) S.warp_hist[warp][d] = 0;
    // From here on memory that earlier kernels wrote (the launch may overlap
    // their end); the next pass may be set up once every CTA is here.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("" : "+l"(n_dev));  // its load, of a read-only parameter, must not move up past the wait
    const int64_t n = n_dev ? min(*n_dev, cap) : cap;
    if (threadIdx.x == 0) S.tile = atomicAdd(&hdr->counters[pass], 1u);
    __syncthreads();
    const uint32_t tile = S.tile;
    const int64_t tile_base = (int64_t)tile * kSortTile;
    if (tile_base >= n) return;
    const int64_t valid_in_tile = min((int64_t)kSortTile, n - tile_base);
    const uint32_t invalid = (uint32_t)(kSortTile - valid_in_tile);

    uint64_t key[ITEMS];
    uint32_t val[ITEMS];
    uint32_t dig[ITEMS];
    uint32_t rank[ITEMS];
    const int64_t wbase = tile_base + (int64_t)warp * (ITEMS * 32);
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int64_t idx = wbase + i * 32 + lane;
        const bool valid = idx < n;
        key[i] = valid ? __ldcg(kin + idx) : ~0ull;
        val[i] = valid ? __ldcg(vin + idx) : 0u;
        dig[i] = valid ? ((uint32_t)(key[i] >> shift) & dmask) : 255u;
    }
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t peers = warp_peers<8>(dig[i]);
        const uint32_t before = S.warp_hist[warp][dig[i]];
        __syncwarp();
        if ((peers & lt) == 0) S.warp_hist[warp][dig[i]] = before + __popc(peers);
        __syncwarp();
        rank[i] = before + __popc(peers & lt);
    }
    __syncthreads();
    // per digit: exclusive prefix over warps and the tile count, published at
    // once (the inclusive prefix for tile 0) so that successors can look back
    uint32_t count = 0, vcount = 0;
    if (threadIdx.x < kRadix) {
        const int d = threadIdx.x;
        uint32_t sum = 0;
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = S.warp_hist[w][d];
            S.warp_hist[w][d] = sum;
            sum += c;
        }
        count = sum;
        vcount = (d == 255) ? sum - invalid : sum;
        uint32_t* lb = lookback + (size_t)tile * kRadix + d;
        if (tile == 0) {
            const uint32_t excl = hdr->hist[pass][d];
            st_relaxed32(lb, kLbInc | ((excl + vcount) & kLbMask));
            S.global_start[d] = excl;
        } else {
            st_relaxed32(lb, kLbAgg | (vcount & kLbMask));
        }
    }
    // exclusive scan of the tile's digit counts -> start of each digit run in smem
    if (threadIdx.x < kRadix) {
        uint32_t inc = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) S.scan_tmp[warp] = inc;
        S.tile_off[threadIdx.x] = inc - count;  // warp-local for now
    }
    __syncthreads();
    if (threadIdx.x < kRadix) {
        uint32_t wpre = 0;
        for (int w = 0; w < warp; ++w) wpre += S.scan_tmp[w];
        S.tile_off[threadIdx.x] += wpre;
    }
    __syncthreads();
    // the local scatter needs no global offsets: it runs before the look-back,
    // so the other warps' scatter overlaps the digit threads' polling
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t lpos = S.tile_off[dig[i]] + S.warp_hist[warp][dig[i]] + rank[i];
        S.keys[lpos] = key[i];
        S.vals[lpos] = val[i];
    }
    if (threadIdx.x < kRadix && tile != 0) {
        const int d = threadIdx.x;
        uint32_t excl = 0;
        int64_t t = (int64_t)tile - 1;
        uint32_t budget = spin_limit;
        for (bool done = false; !done;) {
            uint32_t st[kLookBack];
#pragma unroll
            for (int k = 0; k < kLookBack; ++k)
                st[k] = t - k >= 0 ? ld_relaxed32(lookback + (size_t)(t - k) * kRadix + d) : kLbInc;
            int used = 0;  // words taken: up to the first that is not published or is inclusive
#pragma unroll
            for (int k = 0; k < kLookBack; ++k) {
                if (done || used < k || !(st[k] & ~kLbMask)) continue;
                excl += st[k] & kLbMask;
                done = (st[k] & kLbInc) != 0;
                used = k + 1;
            }
            t -= used;
            if (!done && used < kLookBack && !spin_budget(budget)) {
                atomicOr(status, RM_STATUS_SORT_TIMEOUT);
                break;
            }
        }
        st_relaxed32(lookback + (size_t)tile * kRadix + d, kLbInc | ((excl + vcount) & kLbMask));
        S.global_start[d] = excl;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int pos = i * kSortThreads + threadIdx.x;
        if (pos < valid_in_tile) {
            const uint64_t k = S.keys[pos];
            const uint32_t d = (uint32_t)(k >> shift) & dmask;
            const uint64_t dst = (uint64_t)S.global_start[d] + (uint64_t)(pos - S.tile_off[d]);
            if (dst < (uint64_t)n) {  // only a timed-out look-back can produce dst >= n
                kout[dst] = k;
                vout[dst] = S.vals[pos];
            }
        }
    }
}

}  // namespace
}  // namespace rm

extern "C" {

size_t rm_sort_workspace_size(int64_t n) {
    if (n < 0) return 0;
    return rm::sort_layout(n, rm::kMaxPasses).total;
}

int rm_sort_pairs_range(const int64_t* keys_in, const int32_t* values_in, int64_t n, const int64_t* n_dev,
                        int begin_bit, int end_bit, int64_t* keys_out, int32_t* values_out, void* workspace,
                        size_t workspace_bytes, uint32_t* status_dev, void* stream) {
    using namespace rm;
    if (n < 0) return rm_host::fail(RM_EINVAL, "rm_sort_pairs: negative size");
    if (end_bit < 1 || end_bit > 64 || begin_bit < 0 || begin_bit >= end_bit)
        return rm_host::fail(RM_EINVAL, "rm_sort_pairs: key bits [%d, %d) out of range", begin_bit, end_bit);
    if (n >= (int64_t)kLbMask) return rm_host::fail(RM_EINVAL, "rm_sort_pairs: at most 2^30-1 pairs");
    if (n == 0) return RM_OK;
    if (!keys_in || !values_in || !keys_out || !values_out || !workspace)
        return rm_host::fail(RM_EINVAL, "rm_sort_pairs: NULL pointer");
    const int npasses = (end_bit - begin_bit + 7) / 8;
    const SortLayout L = sort_layout(n, npasses);
    if (workspace_bytes < L.total)
        return rm_host::fail(RM_EINVAL, "rm_sort_pairs: workspace %zu < %zu bytes", workspace_bytes, L.total);
    if ((uintptr_t)workspace & 255) return rm_host::fail(RM_EINVAL, "rm_sort_pairs: workspace must be 256-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    char* ws = (char*)workspace;
    SortHeader* hdr = (SortHeader*)ws;
    uint32_t* lookback = (uint32_t*)(ws + L.lookback_off);
    uint64_t* alt_k = (uint64_t*)(ws + L.alt_keys_off);
    uint32_t* alt_v = (uint32_t*)(ws + L.alt_vals_off);
    cudaError_t e = cudaMemsetAsync(ws + 4, 0, L.memset_bytes - 4, s);
    if (e != cudaSuccess) return rm_host::fail(RM_ECUDA, "rm_sort_pairs: %s", cudaGetErrorString(e));
    const bool large = n >= kLargeFrom;
    const auto kernel = large ? onesweep_kernel<kLargeItems> : onesweep_kernel<kSmallItems>;
    const size_t smem = large ? sizeof(PassSmem<kLargeItems>) : sizeof(PassSmem<kSmallItems>);
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return rm_host::fail(RM_ECUDA, "rm_sort_pairs: %s", cudaGetErrorString(e));
    const int64_t tiles = sort_tiles(n);
    const int64_t runs = (n + kHistThreads * kHistRun - 1) / (kHistThreads * kHistRun);
    const int hist_blocks = (int)(runs < 148 * 4 ? runs : 148 * 4);
    hist_kernel<<<hist_blocks, kHistThreads, 0, s>>>((const uint64_t*)keys_in, n, n_dev, npasses, begin_bit, end_bit,
                                                     hdr);
    // Each pass's launch overlaps the end of the kernel before it: short passes
    // cost mostly their launches (30k pairs 70 -> 58 us, with the histogram's
    // scan inside its own kernel; 1M 116 -> 105).
    cudaLaunchAttribute overlap{};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3((unsigned)tiles);
    config.blockDim = dim3(kSortThreads);
    config.dynamicSmemBytes = smem;
    config.stream = s;
    config.attrs = &overlap;
    config.numAttrs = 1;
    const uint64_t* src_k = (const uint64_t*)keys_in;
    const uint32_t* src_v = (const uint32_t*)values_in;
    for (int p = 0; p < npasses; ++p) {
        // the last pass must land in the caller's output buffers
        const bool to_out = ((npasses - 1 - p) % 2) == 0;
        uint64_t* dk = to_out ? (uint64_t*)keys_out : alt_k;
        uint32_t* dv = to_out ? (uint32_t*)values_out : alt_v;
        const int shift = begin_bit + 8 * p;
        const int bits = (end_bit - shift) < 8 ? (end_bit - shift) : 8;
        const uint32_t dmask = (bits >= 8) ? 255u : ((1u << bits) - 1u);
        e = cudaLaunchKernelEx(&config, kernel, src_k, src_v, dk, dv, n, n_dev, p, shift, dmask, hdr,
                               lookback + (size_t)p * tiles * kRadix, status_dev ? status_dev : &hdr->status,
                               rm_host::wait_limit());
        if (e != cudaSuccess) return rm_host::fail(RM_ECUDA, "rm_sort_pairs: %s", cudaGetErrorString(e));
        src_k = dk;
        src_v = dv;
    }
    return rm_host::check_launch("rm_sort_pairs", 1 + npasses);
}

int rm_sort_pairs(const int64_t* keys_in, const int32_t* values_in, int64_t n, const int64_t* n_dev, int end_bit,
                  int64_t* keys_out, int32_t* values_out, void* workspace, size_t workspace_bytes,
                  uint32_t* status_dev, void* stream) {
    return rm_sort_pairs_range(keys_in, values_in, n, n_dev, 0, end_bit, keys_out, values_out, workspace,
                               workspace_bytes, status_dev, stream);
}

}  // extern "C"
