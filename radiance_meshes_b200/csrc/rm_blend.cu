// rm_blend.cu - stage (d): front-to-back tile blend and its back-to-front
// adjoint.
//
// Forward: splat_tiled / alpha_blend (alphablend_shader_interp.slang:194-271,
// 371-431) with evaluate_tetra_interp and integrate_tetra_segment
// (interp_version.slang:21-98) and ray_tetrahedron_intersect_fused
// (intersect.slang:394-624).  Backward: bwd_alpha_blend
// (alphablend_shader_interp.slang:273-369), with the per-tet derivatives that
// the reference obtains from Slang autodiff written out by hand.
//
// Work decomposition.  Per-tile list lengths are heavy-tailed (a few tiles
// hold 10-100x the mean), and a pixel whose ray sees through a dense region
// crosses thousands of tets.  Each pass is one persistent kernel fed by a
// heavy-first tile order computed on the device, whose work items differ by
// the length of the list:
//   * forward, warp items: half of a 64-pixel strip walked by one warp;
//   * forward, pair items: lists longer than a warp's share of the launch are
//     walked by a CTA that spreads the (entry, pixel) pairs over its threads,
//     the longest by quarters of a strip; the strictly ordered part of the
//     walk (log T, termination, distortion moments) is a few adds per entry
//     by one owner thread per pixel, in the same arithmetic, so results do
//     not depend on which kind of item ran a tile;
//   * backward: strips of 64 pixels, a warp per half, one pixel per lane, long
//     lists in stretches that start from states the forward left
//     (checkpoints).
// The backward's pair kernel (4 threads per pixel) and its staging by bulk
// copies run on request only.
// Per-tet records (128 B, packed once per frame by pack_kernel) are staged in
// shared memory per block of list entries.  Each backward warp adds up an
// entry's partials over its pixels; both warps' sums are turned into vertex and
// cell-value gradients once per (strip, stretch, entry) and added to global
// memory.
#include <mutex>

#include <cooperative_groups.h>

#include "rm_internal.cuh"
#include "rm_approx.cuh"

namespace rm {
namespace {

constexpr float kTermLogT = -5.5f;  // alphablend_shader_interp.slang:257
constexpr int kNGrad = 25;


// ------------------------------------------------------------------ packing --
// A tet with an index outside [0, n_verts) gets an all-zero record: zero
// normals and zero density, so no ray hits it, and its vertices are never read.
__global__ void __launch_bounds__(256) pack_kernel(const int4* __restrict__ indices, const float* __restrict__ verts,
                                                   int64_t n_verts, const float* __restrict__ cv, int64_t n_tets,
                                                   const int32_t* __restrict__ tiles, float4* __restrict__ recs) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n_tets) return;
    if (tiles && __ldg(tiles + g) <= 0) return;
    const int4 id = __ldg(indices + g);
    if (!tet_indices_ok(id, n_verts)) {
        float4* r = recs + (int64_t)kRecFloat4 * g;
#pragma unroll
        for (int k = 0; k < kRecFloat4; ++k) r[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const int ids[4] = {id.x, id.y, id.z, id.w};
    f3 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float* p = verts + 3 * (int64_t)ids[i];
        v[i] = {__ldg(p), __ldg(p + 1), __ldg(p + 2)};
    }
    // face normals of ray_tetrahedron_intersect_fused (intersect.slang:449-475)
    f3 n0 = cross3(v[1] - v[0], v[2] - v[0]);
    const bool f0 = dot3(n0, v[3] - v[0]) > 0.f;
    if (f0) n0 = neg3(n0);
    f3 n1 = cross3(v[1] - v[0], v[3] - v[0]);
    const bool f1 = dot3(n1, v[2] - v[0]) > 0.f;
    if (f1) n1 = neg3(n1);
    f3 n2 = cross3(v[2] - v[0], v[3] - v[0]);
    const bool f2 = dot3(n2, v[1] - v[0]) > 0.f;
    if (f2) n2 = neg3(n2);
    f3 n3 = cross3(v[2] - v[1], v[3] - v[1]);
    const bool f3b = dot3(n3, v[0] - v[1]) > 0.f;
    if (f3b) n3 = neg3(n3);
    const float* c = cv + 7 * g;
    const float density = fmaxf(__ldg(c), 0.f);
    const uint32_t flips = (f0 ? 1u : 0u) | (f1 ? 2u : 0u) | (f2 ? 4u : 0u) | (f3b ? 8u : 0u);
    float4* r = recs + (int64_t)kRecFloat4 * g;
    r[0] = make_float4(n0.x, n0.y, n0.z, density);
    r[1] = make_float4(n1.x, n1.y, n1.z, __ldg(c + 1));
    r[2] = make_float4(n2.x, n2.y, n2.z, __ldg(c + 2));
    r[3] = make_float4(n3.x, n3.y, n3.z, __ldg(c + 3));
    r[4] = make_float4(v[0].x, v[0].y, v[0].z, __ldg(c + 4));
    r[5] = make_float4(v[1].x, v[1].y, v[1].z, __ldg(c + 5));
    r[6] = make_float4(v[2].x, v[2].y, v[2].z, __ldg(c + 6));
    r[7] = make_float4(v[3].x, v[3].y, v[3].z, __uint_as_float(flips));
}

__device__ __forceinline__ f3 xyz(float4 q) { return {q.x, q.y, q.z}; }

// Ray / tet intersection (intersect.slang:394-624) on a staged record, with
// the clamps of evaluate_tetra_interp (interp_version.slang:88-89), written
// without branches: every plane is evaluated and the reference's sequential
// "if (tplane > t_enter)" / "if (tplane < t_exit)" updates become selects.
// The quotients are IEEE divisions, so t_enter / t_exit (and with them the
// hit decision, log T and n_contributors) are bit-identical to the reference
// rounding.  The backward also needs the selected planes and denominators.
struct Isect {
    float te, tx;        // raw entering / exiting distances
    float enter, exit;   // clamped
    float dene, denx;    // dot(n, d) of the selected planes
    int ie, ix;          // selected planes (-1: none)
    bool geo;            // geometric hit
};

template <bool PLANES>
__device__ __forceinline__ Isect intersect(const float4* __restrict__ q, f3 o, f3 d) {
    const f3 a0 = xyz(q[4]) - o;
    const f3 a1 = xyz(q[5]) - o;
    float te = -1e30f, tx = 1e30f, dene = 1.f, denx = 1.f;
    int ie = -1, ix = -1;
    bool miss = false;
    // With no plane nearly parallel to the ray (the common case) none is
    // skipped.  The other case computes its products again: kept, they cost
    // the common one registers (16 views: 32.1 against 31.6 ms).
    {
        float dist[4], den[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const f3 n = xyz(q[i]);
            dist[i] = -dot3(n, i == 3 ? a1 : a0);
            den[i] = dot3(n, d);
        }
        const float least = fminf(fminf(fabsf(den[0]), fabsf(den[1])), fminf(fabsf(den[2]), fabsf(den[3])));
        if (!(least < 1e-10f)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float tp = -dist[i] / den[i];
                const bool in = den[i] < 0.f;
                if (PLANES) {
                    const bool ue = in && tp > te, ux = !in && tp < tx;
                    te = ue ? tp : te;
                    tx = ux ? tp : tx;
                    ie = ue ? i : ie;
                    dene = ue ? den[i] : dene;
                    ix = ux ? i : ix;
                    denx = ux ? den[i] : denx;
                } else {
                    te = fmaxf(te, in ? tp : -1e30f);
                    tx = fminf(tx, in ? 1e30f : tp);
                }
            }
            Isect r;
            r.te = te;
            r.tx = tx;
            r.geo = !(te > tx) && !(tx <= 0.f);
            r.enter = fmaxf(te, 0.f);
            r.exit = fmaxf(tx, r.enter);
            r.dene = dene;
            r.denx = denx;
            r.ie = ie;
            r.ix = ix;
            return r;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const f3 n = xyz(q[i]);
        const float dist = -dot3(n, i == 3 ? a1 : a0);
        const float den = dot3(n, d);
        const bool par = fabsf(den) < 1e-10f;
        miss |= par && dist > 0.f;
        const float tp = -dist / den;
        const bool ue = !par && den < 0.f && tp > te;
        const bool ux = !par && !(den < 0.f) && tp < tx;
        te = ue ? tp : te;
        tx = ux ? tp : tx;
        if (PLANES) {
            ie = ue ? i : ie;
            dene = ue ? den : dene;
            ix = ux ? i : ix;
            denx = ux ? den : denx;
        }
    }
    Isect r;
    r.te = te;
    r.tx = tx;
    r.geo = !miss && !(te > tx) && !(tx <= 0.f);
    r.enter = fmaxf(te, 0.f);
    r.exit = fmaxf(tx, r.enter);
    r.dene = dene;
    r.denx = denx;
    r.ie = ie;
    r.ix = ix;
    return r;
}

// Weights of the closed-form segment integral (interp_version.slang:21-40)
// for optical depth x = density * dt >= 0:
//   alpha = exp(-x), phi = (1 - exp(-x)) / x, w0 = phi - alpha, w1 = 1 - phi.
// Below x = 0.25 w0 and w1 come from their Taylor series (8 terms, truncation
// < 4e-10 relative), which avoids the cancellation in phi - alpha and 1 - phi;
// above, phi = (1 - alpha) / x.  These feed only the colour channels, which
// are compared within a tolerance (log T uses x itself, never these weights).
struct Weights {
    float alpha, w0, w1;
};

// FUSED: the series with fused operations, for gradients.  The forward rounds
// each product and sum, as it always has: a last bit of the image decides the
// sign of an L1 loss where the two nearly meet.
template <bool FUSED = false>
__device__ __forceinline__ Weights seg_weights(float x) {
    Weights w;
    w.alpha = exp_approx(-x);
    if (x < 0.25f) {
        // w1 = x/2 - x^2/6 + x^3/24 - x^4/120 + x^5/720 - x^6/5040 + x^7/40320
        // w0 = x/2 - x^2/3 + x^3/8 - x^4/30 + x^5/144 - x^6/840 + x^7/5760
        const float c1[7] = {1.0f / 40320.0f, -1.0f / 5040.0f, 1.0f / 720.0f, -1.0f / 120.0f, 1.0f / 24.0f,
                             -1.0f / 6.0f, 0.5f};
        const float c0[7] = {1.0f / 5760.0f, -1.0f / 840.0f, 1.0f / 144.0f, -1.0f / 30.0f, 0.125f, -1.0f / 3.0f, 0.5f};
        w.w1 = c1[0];
        w.w0 = c0[0];
#pragma unroll
        for (int k = 1; k < 7; ++k) {
            w.w1 = FUSED ? fmaf(w.w1, x, c1[k]) : w.w1 * x + c1[k];
            w.w0 = FUSED ? fmaf(w.w0, x, c0[k]) : w.w0 * x + c0[k];
        }
        w.w1 = w.w1 * x;
        w.w0 = w.w0 * x;
    } else {
        const float phi = (1.0f - w.alpha) * rcp_approx(x);
        w.w0 = phi - w.alpha;
        w.w1 = 1.0f - phi;
    }
    return w;
}

// d phi / dx = -(d w1 / dx): series below 0.25, (alpha - phi) / x = -w0 / x above.
__device__ __forceinline__ float dphi_f(float x, const Weights& w) {
    if (x < 0.25f)
        return -fmaf(x, fmaf(x, fmaf(x, fmaf(x, fmaf(x, -1.0f / 840.0f, 1.0f / 144.0f), -1.0f / 30.0f), 0.125f),
                             -1.0f / 3.0f), 0.5f);
    return -w.w0 * rcp_approx(x);
}

struct Segment {
    float dt, a, x;
    f3 ve, vx;
    float ce, cx;
    Weights w;
    float rgb[3];
};

// integrate_tetra_segment + compute_integral (interp_version.slang:30-69):
// rgb = w0 * c_exit + w1 * c_enter with c = base + dot(grd, p - v0).
// The colours at the entry and exit points, given those points relative to
// v0 (s.ve, s.vx).
__device__ __forceinline__ void integrate_rel(const float4* __restrict__ q, Segment& s) {
    const float density = q[0].w;
    const f3 grd = {q[4].w, q[5].w, q[6].w};
    s.ce = dot3(grd, s.ve);
    s.cx = dot3(grd, s.vx);
    s.x = s.dt * density;
    s.w = seg_weights(s.x);
    const float base[3] = {q[1].w, q[2].w, q[3].w};
#pragma unroll
    for (int k = 0; k < 3; ++k) s.rgb[k] = fmaf(s.w.w1, s.ce + base[k], s.w.w0 * (s.cx + base[k]));
}

__device__ __forceinline__ void integrate(const float4* __restrict__ q, f3 o, f3 d, float enter, float exit,
                                          Segment& s) {
    const f3 v0 = xyz(q[4]);
    s.ve = {fmaf(enter, d.x, o.x) - v0.x, fmaf(enter, d.y, o.y) - v0.y, fmaf(enter, d.z, o.z) - v0.z};
    s.vx = {fmaf(exit, d.x, o.x) - v0.x, fmaf(exit, d.y, o.y) - v0.y, fmaf(exit, d.z, o.z) - v0.z};
    integrate_rel(q, s);
}


// Pixel (lx, ly) inside the tile of thread t of work item `sub`, for items of
// NT pixels: square blocks of 8x8 (NT = 64) or 4x4 (NT = 16) pixels, row-major
// over the tile, so that the pixels of one item see similar lists; tiles whose
// sides are not multiples of the block fall back to runs of whole rows.
template <int NT>
__device__ __forceinline__ void strip_pixel(const rm_camera& cam, int sub, int t, int& lx, int& ly) {
    constexpr int bw = NT >= 64 ? 8 : 4;
    constexpr int bh = NT / bw;
    if (cam.tile_width % bw == 0 && cam.tile_height % bh == 0) {
        const int nbx = cam.tile_width / bw;
        lx = (sub % nbx) * bw + t % bw;
        ly = (sub / nbx) * bh + t / bw;
    } else {
        const int tp = sub * NT + t;
        lx = tp % cam.tile_width;
        ly = tp / cam.tile_width;
    }
}

struct PixelState {
    float c[3];
    float logT;
    float D[5];
    float part[5];  // what the hits since the last checkpoint added to the colour, D2 and D3
};

// What a forward walk forms: the image; the image and what a backward needs
// (hit masks, checkpoints), whose five sums cost a frame 2 to 3% that has no
// use for them; or log T from 1 with masks and checkpoints (the statistics).
enum Walk { kImage, kImageAndMasks, kLogT };

// ------------------------------------------------------------------ forward --
template <int NT>
struct WarpShape {
    static constexpr unsigned kMask = NT >= 32 ? 0xffffffffu : ((1u << NT) - 1u);
    static constexpr int kTopOffset = NT >= 32 ? 16 : NT / 2;
};

// Hit masks written by the forward and read by the backward
// (RM_BLEND_HIT_MASKS; 64-pixel work items only).  A tile's list is cut into
// blocks of 32 entries counted from its start; pixel p of work item `sub`
// keeps, for block k of global tile t whose list starts at position x, one
// word at mask_word(t, x, k, sub, subs, p) whose bit i says whether entry
// x + 32k + i was a hit for that pixel before its termination.  Block ids
// floor(x / 32) + k + t are distinct over all tiles, so the words never
// overlap; a pixel's words of consecutive blocks are 64 words apart, and the
// 64 pixels of an item are contiguous (coalesced stores and loads).  Words at
// or beyond cap do not exist: the entries they would describe are tested.
__device__ __forceinline__ int64_t mask_word(int gtile, int x, int k, int sub, int subs, int p) {
    return (((int64_t)(x >> 5) + k + gtile) * subs + sub) * 64 + p;
}

struct HitMasks {
    uint32_t* words;  // nullptr: no masks
    int64_t cap;      // words
    const uint32_t* header;  // kMaskValid: this pass's forward wrote masks with 64-pixel items
    float* ck;        // checkpoints (nullptr: none); they lie after the mask words
    int64_t ck_cap;   // checkpoint ids below this exist
    int seg_shift;    // log2 of the list entries between two checkpoints
};

constexpr uint32_t kMaskValid = 0x6d61736bu;
constexpr uint32_t kMaskStats = 0x73746174u;  // written by the statistics' walk, of no use to a backward
constexpr int kNoSegments = 31;   // seg_shift of a pass without checkpoints
constexpr int kMinSegShift = 7;   // segments are whole batches (<= 64 entries) and whole mask blocks
constexpr int kCkFloats = 8;

// Checkpoints.  A pixel that is still active at list offset k << seg_shift
// (k >= 1) of a tile's list stores log T, D2 and D3 as they are there, and,
// once its walk has ended, the sums of what the entries from there on added to
// its colour, D2 and D3.  The backward pass then takes each stretch of
// 1 << seg_shift entries as a work item of its own, starting from the
// checkpoint at its end: the undo chains start from log T, D2 and D3 there, and
// what the later entries contribute to the adjoint state follows from the sums
// (seed_segment).  These are added up from the last stretch back, each
// stretch's own sum started at zero: a difference of the final and the earlier
// colour would hold the rounding of the whole colour, however little is left
// to come.  Without
// checkpoints the pixel with the longest walk bounds the launch: alone on the
// GPU the 14,506-entry tile of a 1.3M-tet frame takes 1.74 ms, of 2.57 ms in
// all.
// Ids floor(x / S) + k are distinct over the tiles because the lists do not
// overlap and offsets k * S lie inside them.
__device__ __forceinline__ int64_t ck_id(int x, int k, int shift) { return (int64_t)(x >> shift) + k; }
__device__ __forceinline__ float* ck_at(const HitMasks& hm, int64_t id, int sub, int subs, int p) {
    return hm.ck + ((id * subs + sub) * kCkFloats) * 64 + p;
}

// Entries between two checkpoints for lists of n_pairs entries in all: 128
// where the stretches are what fills the GPU, 512 above half a million entries
// and 4096 above 64M, where there are enough of them and each one's start (its
// rays, its state) and each pixel's state are what counts.  Backward, us, at 128
// and 512: 0.03M entries 87 and 211, 0.28M 188 and 332, 0.44M 284 and 285, 1.3M
// 514 and 507, 3.9M 1661 and 1614, 13.7M (2% hits) 1166 and 771; at 128, 512
// and 4096: 115M 8104, 4781 and 3943.
constexpr int64_t kShortLists = (int64_t)1 << 19, kLongLists = (int64_t)64 << 20;
__host__ __device__ inline int seg_shift_for(int64_t n_pairs) {
    return n_pairs <= kShortLists ? kMinSegShift : n_pairs <= kLongLists ? 9 : 12;
}
__host__ __device__ inline int64_t ck_count(int64_t n_pairs, int shift) { return (n_pairs >> shift) + 2; }
__host__ __device__ inline int64_t ck_words(int64_t n_pairs, int64_t subs, int shift) {
    return ck_count(n_pairs, shift) * subs * kCkFloats * 64;
}
__host__ __device__ inline int64_t mask_word_count(int64_t n_pairs, int64_t n_tiles, int64_t subs) {
    return (n_pairs / 32 + n_tiles + 2) * subs * 64;
}

// Where a pass with `words` words of room keeps its checkpoints: after the
// masks, at the end of the room.
struct MaskPlan {
    int shift;  // kNoSegments: nowhere
    int64_t ck_cap, ck_off;
};

// The shortest stretch that n_pairs entries (those of this pass's lists, not
// the most that the room was sized for) allow and whose checkpoints fit.
__host__ __device__ inline MaskPlan mask_plan(int64_t words, int64_t n_tiles, int64_t subs, int64_t n_pairs) {
    for (int shift = seg_shift_for(n_pairs); shift <= 12; shift += shift == kMinSegShift ? 2 : 3) {
        const int64_t ck = ck_words(n_pairs, subs, shift);
        if (mask_word_count(n_pairs, n_tiles, subs) + ck <= words) return {shift, ck_count(n_pairs, shift), words - ck};
    }
    return {kNoSegments, 0, words};
}

// The room of a forward with hit masks.  Its order kernel, which knows the
// lists' lengths, writes the header: [0] state, [1] shift, [2] checkpoint ids,
// [4..5] offset of the checkpoints in words after the mask words' start.
struct MaskRoom {
    uint32_t state;  // kMaskValid (kMaskStats in the statistics); 0: no masks
    int subs;
    int64_t words;
};

// The masks a kernel may use: none unless the header says that a walk of its
// own kind wrote them.  hm.cap is the room in words for masks and checkpoints
// together.
__device__ __forceinline__ HitMasks live_masks(HitMasks hm, int subs, uint32_t state = kMaskValid) {
    hm.ck = nullptr;
    hm.ck_cap = 0;
    hm.seg_shift = kNoSegments;
    if (!hm.words) return hm;
    if (!hm.header || __ldcg(hm.header) != state) {
        hm.words = nullptr;
        return hm;
    }
    const int shift = (int)__ldcg(hm.header + 1);
    const int64_t off = __ldcg((const int64_t*)(hm.header + 4));
    if (shift < kMinSegShift || shift >= kNoSegments || off <= 0 || off > hm.cap) return hm;
    const int64_t fit = (hm.cap - off) / ((int64_t)subs * kCkFloats * 64);
    hm.ck = (float*)(hm.words + off);
    hm.ck_cap = min((int64_t)__ldcg(hm.header + 2), fit);
    hm.cap = off;
    hm.seg_shift = shift;
    return hm;
}

// Work queue shared by the kernels of one pass.  order[] lists the tiles
// heaviest first; info[0] is the number of heavy tiles (the first entries of
// order[]), which go by pair items, the rest by warp items (forward) or to the
// kernels that take whole or cut lists (backward).
struct Queue {
    const int32_t* order;
    const int32_t* info;
    uint32_t* ticket;
    int G;
    int subs;  // strips per tile
    bool heavy;
    HitMasks hm;
    uint32_t* status;     // RM_STATUS_* bits of the pass (a staging copy whose wait gave up)
    uint32_t spin_limit;  // polls of a bounded wait
    int64_t n_recs;       // records (tets) the list ids may name
};

__device__ __forceinline__ int queue_items(const Queue& q) {
    const int nh = __ldg(q.info);
    return (q.heavy ? nh : q.G - nh) * q.subs;
}

__device__ __forceinline__ int queue_tile(const Queue& q, int item) {
    const int first = q.heavy ? 0 : __ldg(q.info);
    return __ldg(q.order + first + item / q.subs);
}

// The segment queue of the backward: item -> (tile, segment, strip), heaviest
// bucket first.  A tile of list-length bucket b (lengths [2^(b-1), 2^b)) owns
// 2^(b - seg_shift) segments (1 for shorter ones); those past the end of its
// list, or of all its pixels' walks, end at once.  seg_info is filled by
// order_kernel: entry 32 - b = first segment item of bucket b (without the
// strips), down to bucket seg_shift, where the one-segment tiles begin.
constexpr int kSegInfoOff = 33;  // of the workspace's info words (after the status word)

struct SegItem {
    int tile, seg, sub;
};

__device__ __forceinline__ int64_t segment_items(const int32_t* info, int G, int shift) {
    int64_t tiles = 0;
    for (int b = 32; b > shift; --b)
        tiles += (__ldg(info + kSegInfoOff + 33 - b) - __ldg(info + kSegInfoOff + 32 - b)) >> (b - shift);
    const int first = shift < 32 ? __ldg(info + kSegInfoOff + 32 - shift) : 0;
    return first + (G - tiles);
}

__device__ __forceinline__ SegItem segment_item(const Queue& q, int64_t item, int shift) {
    SegItem r;
    r.sub = (int)(item % q.subs);
    int s = (int)(item / q.subs);
    const int32_t* fi = q.info + kSegInfoOff;
    int tiles = 0;  // tiles of the buckets before
    for (int b = 32; b > shift; --b) {
        const int first = __ldg(fi + 32 - b), next = __ldg(fi + 33 - b);
        if (s < next) {
            r.seg = (s - first) & ((1 << (b - shift)) - 1);
            r.tile = __ldg(q.order + tiles + ((s - first) >> (b - shift)));
            return r;
        }
        tiles += (next - first) >> (b - shift);
    }
    s -= __ldg(fi + 32 - shift);
    r.seg = 0;
    r.tile = __ldg(q.order + tiles + s);
    return r;
}

__device__ __forceinline__ int next_item(const Queue& q, int* s_item) {
    if (threadIdx.x == 0) *s_item = (int)atomicAdd(q.ticket, 1u);
    __syncthreads();
    const int item = *s_item;
    __syncthreads();
    return item;
}

// A list entry's tet id, or -1 when it names no record.  Only lists left
// invalid by a scan or sort that gave up (or a caller's corrupt lists) hold
// such ids; the entry is then staged as a zero record, which no ray hits, and
// RM_STATUS_BAD_INDEX is set.
__device__ __forceinline__ int32_t list_id(const int32_t* __restrict__ ids, int64_t e, const Queue& lq) {
    const int32_t g = __ldg(ids + e);
    if (g >= 0 && (int64_t)g < lq.n_recs) return g;
    if (lq.status) atomicOr(lq.status, RM_STATUS_BAD_INDEX);
    return -1;
}

__device__ __forceinline__ float4 record_part(const float4* __restrict__ recs, int32_t g, int c) {
    return g >= 0 ? __ldg(recs + (int64_t)kRecFloat4 * g + c) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// Stores the checkpoint of pixel p (p of the strip's 64) at list position
// base, when one lies there, with the sums of the stretch before it.
template <bool LOGT>
__device__ __forceinline__ void write_checkpoint(const HitMasks& hm, PixelState& st, int x, int base, int sub,
                                                 int subs, int p) {
    const int off = base - x;
    if (off == 0 || (off & ((1 << kMinSegShift) - 1))) return;  // no segment length has one here
    if (!hm.ck || (off & ((1 << hm.seg_shift) - 1))) return;
    const int64_t id = ck_id(x, off >> hm.seg_shift, hm.seg_shift);
    if (id >= hm.ck_cap) return;
    float* c = ck_at(hm, id, sub, subs, p);
    c[0 * 64] = st.logT;
    if (LOGT) return;
    c[1 * 64] = st.D[2];
    c[2 * 64] = st.D[3];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        c[(3 + i) * 64] = st.part[i];
        st.part[i] = 0.f;
    }
}

// The sums of the stretches before the checkpoints of a pixel whose walk took
// nc entries turned into the sums over all of its later entries, from the last
// checkpoint (st.part: the sums after it) back.
__device__ __forceinline__ void finish_checkpoints(const HitMasks& hm, const PixelState& st, int x, int nc, int sub,
                                                   int subs, int p) {
    if (!hm.ck || nc <= (1 << hm.seg_shift)) return;
    int k = (nc - 1) >> hm.seg_shift;
    const int64_t first = ck_id(x, 0, hm.seg_shift);
    if (first + k >= hm.ck_cap) return;  // not all of them were stored: no pass starts from them
    const int64_t step = (int64_t)subs * kCkFloats * 64;
    float* c = ck_at(hm, first + k, sub, subs, p) + 3 * 64;
    float later[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) later[i] = st.part[i];
    constexpr int kAhead = 4;  // checkpoints read at a time
    for (; k > 0; k -= kAhead) {
        float before[kAhead][5];
#pragma unroll
        for (int j = 0; j < kAhead; ++j)
#pragma unroll
            for (int i = 0; i < 5; ++i) before[j][i] = j < k ? c[-j * step + i * 64] : 0.f;
#pragma unroll
        for (int j = 0; j < kAhead; ++j)
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                if (j < k) c[-j * step + i * 64] = later[i];
                later[i] = later[i] + before[j][i];
            }
        c -= kAhead * step;
    }
}

// One hit folded into the pixel state (update_alpha_out,
// alphablend_shader_interp.slang:84-183): colour += rgb * T, log T -= a, and
// the five distortion moments with m0 = density, m1 = density * (a + b) / 2.
template <bool PART>
__device__ __forceinline__ void fold_hit(PixelState& st, float a, float m0, float m1, float d4, const float* rgb) {
    const float T = exp_approx(st.logT);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        st.c[k] = fmaf(rgb[k], T, st.c[k]);
        if (PART) st.part[k] = fmaf(rgb[k], T, st.part[k]);
    }
    st.logT = st.logT - a;
    const float D2 = st.D[2], D3 = st.D[3];
    st.D[0] = fmaf(2.0f * m1, D2, st.D[0]);
    st.D[1] = fmaf(2.0f * m0, D3, st.D[1]);
    st.D[2] = D2 + m0;
    st.D[3] = D3 + m1;
    st.D[4] = st.D[4] + d4;
    if (PART) {
        st.part[3] = st.part[3] + m0;
        st.part[4] = st.part[4] + m1;
    }
}

// Result of testing one ray against one list entry, the same for every kind of
// item: a = density * dt (0 for a miss), m1, the D4 increment
// density^2 * dt / 3 and the segment colour.
struct EntryResult {
    float a, m1, d4;
    float rgb[3];
};

// LOGT: a only (the statistics' walk).
template <bool LOGT>
__device__ __forceinline__ EntryResult eval_entry(const float4* __restrict__ q, f3 o, f3 d) {
    EntryResult r;
    const Isect is = intersect<false>(q, o, d);
    Segment s;
    s.dt = fmaxf(is.exit - is.enter, 0.f);
    const float density = q[0].w;
    s.a = density * s.dt;
    r.a = 0.f;
    r.m1 = 0.f;
    r.d4 = 0.f;
    r.rgb[0] = r.rgb[1] = r.rgb[2] = 0.f;
    if (LOGT) {
        if (is.geo && s.a > 0.f) r.a = s.a;
    } else if (is.geo && s.a > 0.f) {
        r.a = s.a;
        integrate(q, o, d, is.enter, is.exit, s);
#pragma unroll
        for (int k = 0; k < 3; ++k) r.rgb[k] = s.rgb[k];
        r.m1 = density * (is.exit + is.enter) / 2.0f;
        r.d4 = third(density * density * s.dt);
    }
    return r;
}

// A bundle of rays from one point: every ray direction is a positive multiple
// of u * r0 + v * r1 + r2 for the camera axes r0, r1, r2, with (u, v) inside
// the box.
struct Bundle {
    float u0, u1, v0, v1;
};

// Whether a list entry can be hit by a ray of the bundle.  Seen from the
// camera position c, a hit ray d satisfies, for each face i that c lies
// outside of and each face j that c lies inside of (the silhouette),
//     g = dot(dist_j n_i - dist_i n_j, d) >= 0,  dist = dot(n, c - v):
// the quotients of eval_entry order as te <= tx exactly when every such g is
// not negative, and moving the ray's start along d leaves g alone.  g is
// linear in d, so its largest value over the box decides.  The margin covers
// the rounding of dist, n.d and of the ray origin in eval_entry (below 60
// units of 2^-24 of |n_i| |n_j| times the distance scale A), planes it skips
// as parallel (|n.d| < 1e-10) and axes orthonormal to 2e-6 only; faces whose
// side of c is within rounding take no part.  So an entry that is dropped is
// one for which eval_entry returns a miss for every ray of the bundle.
// r: the entry's record; inv_z: 1 / the least d.r2 of the unit directions.
__device__ __forceinline__ bool entry_reaches(const float4* __restrict__ r, const rm_camera& cam, const Bundle& bd,
                                              float inv_z) {
    const f3 c = {cam.cam_pos[0], cam.cam_pos[1], cam.cam_pos[2]};
    const float* M = cam.world_view;
    const f3 a0 = xyz(r[4]) - c, a1 = xyz(r[5]) - c;
    const float A = fmaxf(fabsf(a0.x) + fabsf(a0.y) + fabsf(a0.z), fabsf(a1.x) + fabsf(a1.y) + fabsf(a1.z)) +
                    (fabsf(c.x) + fabsf(c.y) + fabsf(c.z)) + cam.min_t;
    float dist[4], N[4];
    f3 m[4];
    uint32_t outside = 0, inside = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const f3 n = xyz(r[i]);
        dist[i] = -dot3(n, i == 3 ? a1 : a0);
        N[i] = fabsf(n.x) + fabsf(n.y) + fabsf(n.z);
        const float sure = fmaf(2e-6f * N[i], A, 1e-9f * (1.0f + cam.min_t));
        outside |= dist[i] > sure ? 1u << i : 0u;
        inside |= dist[i] < -sure ? 1u << i : 0u;
        m[i] = {dot3(mk3(M[0], M[1], M[2]), n), dot3(mk3(M[4], M[5], M[6]), n), dot3(mk3(M[8], M[9], M[10]), n)};
    }
    bool reach = true;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int j = i + 1; j < 4; ++j) {
            const bool ij = ((outside >> i) & (inside >> j) & 1u) != 0u, ji = ((outside >> j) & (inside >> i) & 1u) != 0u;
            if (!ij && !ji) continue;
            const float di = ij ? dist[i] : -dist[i], dj = ij ? dist[j] : -dist[j];
            const f3 e = {fmaf(dj, m[i].x, -(di * m[j].x)), fmaf(dj, m[i].y, -(di * m[j].y)),
                          fmaf(dj, m[i].z, -(di * m[j].z))};
            const float P = N[i] * N[j] * A;
            const float margin = fmaf(8e-6f, P, fmaf(1e-5f, fabsf(e.x) + fabsf(e.y) + fabsf(e.z),
                                                     2e-10f * A * (N[i] + N[j])));
            const float g = e.z + fmaxf(e.x * bd.u0, e.x * bd.u1) + fmaxf(e.y * bd.v0, e.y * bd.v1);
            if (P > 1e-25f && P < 1e30f && fmaf(margin, inv_z, g) < 0.f) reach = false;
        }
    }
    return reach;
}

// A ray's z (d.r2) as its bundle takes it: 0, for which entry_reaches does not
// apply, where the ray has no place in the box.  Such a ray (a jitter or a
// direction that is not a number) counts as a hit of every entry of positive
// density, which the other rays of the bundle must not drop.
__device__ __forceinline__ float bundle_z(float z, float u, float v) {
    return fabsf(u) < 1e30f && fabsf(v) < 1e30f ? z : 0.f;
}

// 1 / (least z) of a bundle, or 0 when entry_reaches does not apply (rays
// starting behind the camera position, axes that are no rotation, rays far
// off the axis).
__device__ __forceinline__ float bundle_inv_z(const rm_camera& cam, float z_min) {
    const float* M = cam.world_view;
    const f3 r0 = mk3(M[0], M[1], M[2]), r1 = mk3(M[4], M[5], M[6]), r2 = mk3(M[8], M[9], M[10]);
    const float skew = fmaxf(fmaxf(fmaxf(fabsf(dot3(r0, r1)), fabsf(dot3(r0, r2))), fabsf(dot3(r1, r2))),
                             fmaxf(fmaxf(fabsf(dot3(r0, r0) - 1.f), fabsf(dot3(r1, r1) - 1.f)),
                                   fabsf(dot3(r2, r2) - 1.f)));
    return cam.min_t >= 0.f && skew < 2e-6f && z_min > 0.05f ? 1.0f / z_min : 0.f;
}

// Pair forward item: a strip of PX pixels (PX / tile_width rows of one tile)
// handled by NT >= PX threads, or (quarter >= 0) one 4x4-pixel quarter of an
// 8x8 strip.  The first threads own one pixel each.
//
// The list is taken in blocks of RB entries.  A staging warp loads a block,
// one entry per lane, drops the entries that no ray of the strip can hit
// (entry_reaches, and those of zero density) and writes the records of the
// rest to shared memory, as many blocks per batch as fill the B records.  The
// still-active pixels are compacted into slots and all NT threads evaluate
// the (entry, slot) pairs -- a warp takes one entry at a time (its record is
// read as a broadcast) and its lanes take 32 slots, or groups of lanes take
// entries of their own where fewer are active -- writing each pair's a, m1,
// D4 increment and colour to shared memory (zeros for a miss).  Each owner
// then folds its pixel's results in list order while the other warps stage
// the next batch.  The fold is exactly the arithmetic of the
// one-thread-per-pixel walk (adding a miss's zeros changes no bit), so
// n_contributors, log T and the distortion moments are unchanged bit for bit.
//
// Bound: instruction issue in the evaluation (about 200 instructions for 32
// pairs); for the few lists of thousands of entries the chain of batches,
// hence the quarters and a fold whose only serial part is one add per entry.
template <int PX, int NT, int B>
struct PairShape {
    static constexpr int kOwnWarps = (PX + 31) / 32;
    static constexpr int kWarps = NT / 32;
    static constexpr int kStageWarps = kWarps - kOwnWarps;
    static constexpr int RB = B < 32 ? B : 32;
};

template <int PX, int B>
struct FwdPairSmem {
    static constexpr int kMaxStage = 6;
    float4 srec[B][kRecFloat4 + 1];  // padded: a warp writes whole records, one per lane
    float res[6][B][PX];   // a (0: miss), m1, d4, r, g, b per (entry, slot)
    float ray[6][PX];      // o, d of each slot (structure of arrays)
    float dens[2][B];      // densities of the batch being folded and of the one being staged
    uint8_t pos[2][B];     // list offset of each record inside its block
    uint32_t bal[kMaxStage];           // entries kept of the blocks a staging round looked at
    int32_t start[2][kMaxStage + 1];   // first record of each block of the batch; [n_blk]: their count
    int32_t n_blk[2];
    float bnd[2][(PX + 31) / 32][4];   // (min u, max u, min v, max v) of each owner warp's active pixels
    float z_min[(PX + 31) / 32];
    float uv[2][PX];       // each owner's (u, v), by owner thread
    int32_t warp_base[(PX + 31) / 32];
};

template <bool LOGT, int PX, int B>
__device__ __forceinline__ void store_result(FwdPairSmem<PX, B>& S, int j, int sl, const EntryResult& r) {
    S.res[0][j][sl] = r.a;
    if (LOGT) return;
    S.res[1][j][sl] = r.m1;
    S.res[2][j][sl] = r.d4;
    S.res[3][j][sl] = r.rgb[0];
    S.res[4][j][sl] = r.rgb[1];
    S.res[5][j][sl] = r.rgb[2];
}

// One record (a 128-byte line: four sectors, fetched one by one) into L1.
__device__ __forceinline__ void prefetch_record(const float4* r) {
#pragma unroll
    for (int k = 0; k < 4; ++k) asm volatile("prefetch.global.L1 [%0];" ::"l"(r + 2 * k));
}

// Stages a batch from block `blk` of the list [x, y) on with the staging
// warps (sw: this warp's number among them): looks at up to `tries` blocks,
// one per warp, and keeps as many as fit in B records (at least one).
template <int PX, int NT, int B>
__device__ __forceinline__ void stage_pair_batch(FwdPairSmem<PX, B>& S, int buf, int rd, int blk, int tries, int x, int y,
                                                 const int32_t* __restrict__ ids, const float4* __restrict__ recs,
                                                 const rm_camera& cam, float inv_z, const Queue& lq, int sw, int lane) {
    using Sh = PairShape<PX, NT, B>;
    tries = min(tries, (y - x - blk * Sh::RB + Sh::RB - 1) / Sh::RB);
    bool keep = false;
    uint32_t bal = 0;
    const float4* r = recs;
    if (sw < tries) {
        const int e = x + (blk + sw) * Sh::RB + lane;
        int32_t g = -1;
        if (lane < Sh::RB && e < y) g = list_id(ids, e, lq);
        if (g >= 0) {
            r = recs + (int64_t)kRecFloat4 * g;
            prefetch_record(r);  // the record's four sectors at once
            keep = __ldg(&r[0].w) > 0.f;  // a density of zero hits nothing
            if (keep && inv_z > 0.f) {
                Bundle bd = {S.bnd[rd][0][0], S.bnd[rd][0][1], S.bnd[rd][0][2], S.bnd[rd][0][3]};
#pragma unroll
                for (int w = 1; w < Sh::kOwnWarps; ++w)
                    bd = {fminf(bd.u0, S.bnd[rd][w][0]), fmaxf(bd.u1, S.bnd[rd][w][1]), fminf(bd.v0, S.bnd[rd][w][2]),
                          fmaxf(bd.v1, S.bnd[rd][w][3])};
                keep = entry_reaches(r, cam, bd, inv_z);
            }
        }
        bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) S.bal[sw] = bal;
    } else if (sw == tries) {
        // the block after: its records into L1, where the next staging finds
        // them (a batch of a long list is otherwise mostly load latency)
        const int e = x + (blk + sw) * Sh::RB + lane;
        if (lane < Sh::RB && e < y) {
            const int32_t g = __ldg(ids + e);
            if (g >= 0 && (int64_t)g < lq.n_recs) prefetch_record(recs + (int64_t)kRecFloat4 * g);
        }
    }
    if (Sh::kStageWarps > 1)
        asm volatile("bar.sync 1, %0;" ::"r"(Sh::kStageWarps * 32) : "memory");
    else
        __syncwarp();
    // how many blocks fit, and this warp's first record
    int m = 0, n = 0, mine = 0;
    for (; m < tries; ++m) {
        const int k = __popc(S.bal[m]);
        if (n + k > B) break;
        if (m == sw) mine = n;
        if (sw == 0 && lane == 0) S.start[buf][m] = n;
        n += k;
    }
    if (sw == 0 && lane == 0) {
        S.start[buf][m] = n;
        S.n_blk[buf] = m;
    }
    if (sw < m && keep) {
        const int j = mine + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
        for (int c = 0; c < kRecFloat4; ++c) S.srec[j][c] = __ldg(r + c);
        S.dens[buf][j] = __ldg(&r[0].w);
        S.pos[buf][j] = (uint8_t)lane;
    }
}

// One entry of the fold, hit or miss (a = 0, every increment zero).
template <bool PART>
__device__ __forceinline__ void fold_any(PixelState& st, float a, float m0, float m1, float d4, float r, float g,
                                         float b) {
    const float T = exp_approx(st.logT);
    st.c[0] = fmaf(r, T, st.c[0]);
    st.c[1] = fmaf(g, T, st.c[1]);
    st.c[2] = fmaf(b, T, st.c[2]);
    if (PART) {
        st.part[0] = fmaf(r, T, st.part[0]);
        st.part[1] = fmaf(g, T, st.part[1]);
        st.part[2] = fmaf(b, T, st.part[2]);
    }
    st.logT = st.logT - a;
    const float D2 = st.D[2], D3 = st.D[3];
    st.D[0] = fmaf(2.0f * m1, D2, st.D[0]);
    st.D[1] = fmaf(2.0f * m0, D3, st.D[1]);
    st.D[2] = D2 + m0;
    st.D[3] = D3 + m1;
    st.D[4] = st.D[4] + d4;
    if (PART) {
        st.part[3] = st.part[3] + m0;
        st.part[4] = st.part[4] + m1;
    }
}

template <int PX, int NT, int B, Walk WALK>
__device__ __forceinline__ void fwd_pair_item(int tile, int sub, int quarter, const int32_t* __restrict__ ids,
                                         const int2* __restrict__ ranges, const float4* __restrict__ recs,
                                         const float2* __restrict__ jitter, const rm_camera& cam,
                                         float4* __restrict__ out_img, float* __restrict__ out_dist,
                                         int32_t* __restrict__ out_nc, FwdPairSmem<PX, B>& S,
                                         const HitMasks& hm, int subs, int gtile, const Queue& lq) {
    using Sh = PairShape<PX, NT, B>;
    static_assert(PX <= 64 && NT >= 64, "two owner warps at most");
    static_assert(Sh::kStageWarps >= 1 && Sh::kStageWarps <= FwdPairSmem<PX, B>::kMaxStage, "staging warps");
    constexpr bool LOGT = WALK == kLogT, kMasks = PX == 64 && WALK != kImage;
    constexpr int RB = Sh::RB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool own_warp = warp < Sh::kOwnWarps;
    const bool owner = tid < (quarter >= 0 ? 16 : PX);
    const int2 rg = __ldg(ranges + tile);
    // the owner's pixel of the strip
    const int p = quarter < 0 ? tid : ((quarter >> 1) * 4 + (tid >> 2)) * 8 + (quarter & 1) * 4 + (tid & 3);
    const int tx = tile % cam.grid_width, ty = tile / cam.grid_width;
    int lx, ly;
    strip_pixel<PX>(cam, sub, p, lx, ly);
    const int px = tx * cam.tile_width + lx, py = ty * cam.tile_height + ly;
    const bool inside = owner && px < cam.image_width && py < cam.image_height;
    const int64_t pix = (int64_t)py * cam.image_width + px;
    PixelState st = {{0.f, 0.f, 0.f}, LOGT ? 1.0f : 0.f, {0.f, 0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f, 0.f}};
    int32_t nc = rg.y - rg.x;  // entries walked: all of them unless log T runs out
    bool active = inside && nc > 0;
    int rank = 0, slot = tid;  // rank among the warp's active pixels; where the pixel's ray and results lie
    const float* M = cam.world_view;
    // Box of the active pixels' (u, v), per owner warp.
    auto bounds = [&](int buf, bool in) {
        const float u = in ? S.uv[0][tid] : 0.f, v = in ? S.uv[1][tid] : 0.f;
        float u0 = in ? u : 3e38f, u1 = in ? u : -3e38f, v0 = in ? v : 3e38f, v1 = in ? v : -3e38f;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            u0 = fminf(u0, __shfl_xor_sync(0xffffffffu, u0, o));
            u1 = fmaxf(u1, __shfl_xor_sync(0xffffffffu, u1, o));
            v0 = fminf(v0, __shfl_xor_sync(0xffffffffu, v0, o));
            v1 = fmaxf(v1, __shfl_xor_sync(0xffffffffu, v1, o));
        }
        if (lane == 0) {
            S.bnd[buf][warp][0] = u0;
            S.bnd[buf][warp][1] = u1;
            S.bnd[buf][warp][2] = v0;
            S.bnd[buf][warp][3] = v1;
        }
    };
    auto rank_active = [&]() {
        const unsigned bal = __ballot_sync(0xffffffffu, active);
        if (lane == 0) S.warp_base[warp] = __popc(bal);
        return __popc(bal & ((1u << lane) - 1u));
    };
    if (own_warp) {
        f3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f};
        float z = 3e38f;
        rank = rank_active();
        if (active) {
            const float2 j = LOGT ? make_float2(0.5f, 0.5f) : __ldg(jitter + pix);
            make_ray(cam, px, py, j.x, j.y, o, d);
            z = dot3(mk3(M[8], M[9], M[10]), d);
            const float u = dot3(mk3(M[0], M[1], M[2]), d) / z, v = dot3(mk3(M[4], M[5], M[6]), d) / z;
            S.uv[0][tid] = u;
            S.uv[1][tid] = v;
            z = bundle_z(z, u, v);
            S.ray[0][tid] = o.x; S.ray[1][tid] = o.y; S.ray[2][tid] = o.z;
            S.ray[3][tid] = d.x; S.ray[4][tid] = d.y; S.ray[5][tid] = d.z;
        }
        bounds(0, active);
#pragma unroll
        for (int off = 16; off; off >>= 1) z = fminf(z, __shfl_xor_sync(0xffffffffu, z, off));
        if (lane == 0) S.z_min[warp] = z;
    }
    int n_active = __syncthreads_count(active);
    float inv_z = 0.f;
    if (!own_warp) {
        float z = S.z_min[0];
#pragma unroll
        for (int w = 1; w < Sh::kOwnWarps; ++w) z = fminf(z, S.z_min[w]);
        inv_z = bundle_inv_z(cam, z);
    }
    if (!own_warp && n_active > 0)
        stage_pair_batch<PX, NT, B>(S, 0, 0, 0, 1, rg.x, rg.y, ids, recs, cam, inv_z, lq, warp - Sh::kOwnWarps, lane);
    int shape_of = -1;  // the active count that slots and rays are laid out for
    int cur = 0, blk = 0;
    __syncthreads();
    while (n_active > 0 && blk * RB < rg.y - rg.x) {
        const int m = S.n_blk[cur], n = S.start[cur][m];
        if (n_active != shape_of) {  // some pixel ended: close the gaps it left
            float ray[6];
            if (active) {
                for (int w = 0; w < warp; ++w) rank += S.warp_base[w];
#pragma unroll
                for (int k = 0; k < 6; ++k) ray[k] = S.ray[k][slot];
            }
            __syncthreads();
            if (active) {
#pragma unroll
                for (int k = 0; k < 6; ++k) S.ray[k][rank] = ray[k];
                slot = rank;
            }
            shape_of = n_active;
            __syncthreads();
        }
        if (n > 0) {
            // Evaluate.  With more than 32 active slots the warps form two
            // teams, one per half of the slots, sized by the work; a team with
            // few slots splits its warps into groups of `span` lanes (a power
            // of two, at least 4), each group taking its own entry.
            int first = 0, cnt = n_active, team = Sh::kWarps, member = warp;
            if (PX > 32 && n_active > 32) {
                const int rest = n_active - 32;
                const int w1 = rest > 16 ? Sh::kWarps / 2 : rest > 8 ? Sh::kWarps * 3 / 8 : rest > 4 ? Sh::kWarps / 4
                                                                                                    : Sh::kWarps / 8;
                cnt = 32;
                team = Sh::kWarps - w1;
                if (warp >= team) {
                    member = warp - team;
                    first = 32;
                    cnt = rest;
                    team = w1;
                }
            }
            const int span = cnt <= 4 ? 4 : cnt <= 8 ? 8 : cnt <= 16 ? 16 : 32;
            const int groups = 32 / span;
            const int sl = first + (lane & (span - 1));
            if ((lane & (span - 1)) < cnt) {
                const f3 o = {S.ray[0][sl], S.ray[1][sl], S.ray[2][sl]};
                const f3 d = {S.ray[3][sl], S.ray[4][sl], S.ray[5][sl]};
                for (int j = member * groups + lane / span; j < n; j += team * groups)
                    store_result<LOGT>(S, j, sl, eval_entry<LOGT>(S.srec[j], o, d));
            }
            __syncthreads();
        }
        if (!own_warp) {
            const int next = blk + m;
            // blocks to look at: as many as the last batch's yield would need to fill B records
            const int tries = min(Sh::kStageWarps, max(1, B * m / max(n, 1)));
            if (next * RB < rg.y - rg.x)
                stage_pair_batch<PX, NT, B>(S, cur ^ 1, cur, next, tries, rg.x, rg.y, ids, recs, cam, inv_z, lq,
                                            warp - Sh::kOwnWarps, lane);
        } else {
            const bool was = active;
            for (int w = 0; w < m; ++w) {
                const int j1 = S.start[cur][w + 1];
                uint32_t hb = 0;  // bit k: entry k of the block was a hit for this owner's pixel
                if (kMasks && active) write_checkpoint<LOGT>(hm, st, rg.x, rg.x + (blk + w) * RB, sub, subs, p);
                for (int j = S.start[cur][w]; LOGT && j < j1 && active; ++j) {
                    const float a = S.res[0][j][slot];
                    st.logT = st.logT - a;
                    const int at = S.pos[cur][j];
                    hb |= a > 0.f ? 1u << at : 0u;
                    if (st.logT < kTermLogT) {
                        active = false;
                        nc = (blk + w) * RB + at + 1;
                    }
                }
                for (int j = S.start[cur][w]; !LOGT && j < j1 && active; j += 4) {
                    // four entries' results read ahead, whatever they are (rows past
                    // the block's last are there to read and not used)
                    float r[6][4], dens[4];
                    uint32_t bit[4];
                    float logT = st.logT;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int jk = min(j + k, B - 1);
#pragma unroll
                        for (int c = 0; c < 6; ++c) r[c][k] = S.res[c][jk][slot];
                        dens[k] = S.dens[cur][jk];
                        bit[k] = 1u << S.pos[cur][jk];
                        if (j + k >= j1) r[0][k] = r[1][k] = r[2][k] = r[3][k] = r[4][k] = r[5][k] = 0.f;
                        logT = logT - r[0][k];
                    }
                    if (!(logT < kTermLogT)) {  // log T never rises: none of the four ends the walk
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const bool hit = r[0][k] > 0.f;
                            hb |= hit ? bit[k] : 0u;
                            fold_any<kMasks>(st, r[0][k], hit ? dens[k] : 0.f, r[1][k], r[2][k], r[3][k], r[4][k], r[5][k]);
                        }
                    } else {
                        for (int k = 0; k < 4 && j + k < j1; ++k) {
                            const float ak = S.res[0][j + k][slot];
                            if (!(ak > 0.f)) continue;
                            const int at = S.pos[cur][j + k];
                            hb |= 1u << at;
                            fold_any<kMasks>(st, ak, S.dens[cur][j + k], S.res[1][j + k][slot], S.res[2][j + k][slot],
                                     S.res[3][j + k][slot], S.res[4][j + k][slot], S.res[5][j + k][slot]);
                            if (st.logT < kTermLogT) {
                                active = false;
                                nc = (blk + w) * RB + at + 1;
                                break;
                            }
                        }
                    }
                }
                if (kMasks && owner && hm.words) {
                    const int64_t i = mask_word(gtile, rg.x, (blk + w) * RB >> 5, sub, subs, p);
                    if (i < hm.cap) {
                        if (RB == 32) __stcg(hm.words + i, hb);
                        else __stcg((unsigned short*)(hm.words + i) + ((blk + w) & 1), (unsigned short)hb);
                    }
                }
            }
            if (__any_sync(0xffffffffu, was != active))
                bounds(cur ^ 1, active);
            else if (lane < 4)
                S.bnd[cur ^ 1][warp][lane] = S.bnd[cur][warp][lane];
            rank = rank_active();
        }
        blk += m;
        cur ^= 1;
        n_active = __syncthreads_count(active);
    }
    if (inside) {
        out_nc[pix] = nc;
        if (LOGT) return;
        if (kMasks) finish_checkpoints(hm, st, rg.x, nc, sub, subs, p);
        out_img[pix] = make_float4(st.c[0], st.c[1], st.c[2], st.logT);
        float* dd = out_dist + 5 * pix;
#pragma unroll
        for (int k = 0; k < 5; ++k) dd[k] = st.D[k];
    }
}

// Warp forward item: half of a 64-pixel strip (8x4 pixels; a whole strip of
// 16), one lane per pixel, the list walked by one warp on its own: each block
// of 32 records is copied to the warp's shared memory (asynchronous 16-byte
// copies, eight lanes to a record's line; one lane per record took six times
// the L1 lookups), each lane looks at one entry, and those that the warp's
// rays can hit (entry_reaches) are walked in order.  No exchange of results
// and no barrier across warps: a third fewer instructions per ray/tet test
// than the pair items, but a list's walk takes as long as one warp needs, so
// only lists that many other warps outlast come here (order_kernel).
//
// AHEAD: the next block's records are copied while this one is walked, into a
// second buffer.  The batch launches take it, of one view too: 16 views of a
// million tets 33.6 ms (34.8 without), 4 views of 250k 3713 us (3840), one
// served view of 1.6M tets at 1297x840 1336 (1374), at 1920x1080 2174 (2225).
// rm_blend_fwd, whose walks keep what a backward needs, loses more by what the
// second buffers (110 KB an SM) take from the L1: 1297x840 1041 us (1065 with),
// 640x481 738 (752).
template <bool AHEAD>
struct FwdWarpSmem {
    float4 srec[AHEAD ? 2 : 1][32][kRecFloat4 + 1];  // padded: 32 lanes read one record each without conflicts
};

template <int PX, Walk WALK, bool AHEAD>
__device__ __forceinline__ void fwd_warp_item(int tile, int sub, int half, const int32_t* __restrict__ ids,
                                              const int2* __restrict__ ranges, const float4* __restrict__ recs,
                                              const float2* __restrict__ jitter, const rm_camera& cam,
                                              float4* __restrict__ out_img, float* __restrict__ out_dist,
                                              int32_t* __restrict__ out_nc, FwdWarpSmem<AHEAD>& S, const HitMasks& hm,
                                              int subs, int gtile, const Queue& lq) {
    constexpr bool LOGT = WALK == kLogT, kMasks = PX == 64 && WALK != kImage;
    const int lane = threadIdx.x & 31;
    const int2 rg = __ldg(ranges + tile);
    const int p = half * 32 + lane;
    const int tx = tile % cam.grid_width, ty = tile / cam.grid_width;
    int lx, ly;
    strip_pixel<PX>(cam, sub, p, lx, ly);
    const int px = tx * cam.tile_width + lx, py = ty * cam.tile_height + ly;
    const bool inside = p < PX && px < cam.image_width && py < cam.image_height;
    const int64_t pix = (int64_t)py * cam.image_width + px;
    const float* M = cam.world_view;
    f3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f};
    float u = 0.f, v = 0.f, z = 3e38f;
    if (inside) {
        const float2 j = LOGT ? make_float2(0.5f, 0.5f) : __ldg(jitter + pix);
        make_ray(cam, px, py, j.x, j.y, o, d);
        z = dot3(mk3(M[8], M[9], M[10]), d);
        u = dot3(mk3(M[0], M[1], M[2]), d) / z;
        v = dot3(mk3(M[4], M[5], M[6]), d) / z;
        z = bundle_z(z, u, v);
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) z = fminf(z, __shfl_xor_sync(0xffffffffu, z, off));
    const float inv_z = bundle_inv_z(cam, z);
    Bundle bd;
    auto bounds = [&](bool in) {
        bd = {in ? u : 3e38f, in ? u : -3e38f, in ? v : 3e38f, in ? v : -3e38f};
#pragma unroll
        for (int off = 16; off; off >>= 1)
            bd = {fminf(bd.u0, __shfl_xor_sync(0xffffffffu, bd.u0, off)),
                  fmaxf(bd.u1, __shfl_xor_sync(0xffffffffu, bd.u1, off)),
                  fminf(bd.v0, __shfl_xor_sync(0xffffffffu, bd.v0, off)),
                  fmaxf(bd.v1, __shfl_xor_sync(0xffffffffu, bd.v1, off))};
    };
    PixelState st = {{0.f, 0.f, 0.f}, LOGT ? 1.0f : 0.f, {0.f, 0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f, 0.f}};
    int32_t nc = rg.y - rg.x;  // entries walked: all of them unless log T runs out
    bool active = inside && nc > 0;
    bounds(active);
    // This lane's entry of a block, and the copies of a block's records.
    auto entry = [&](int base) { return base + lane < rg.y ? list_id(ids, base + lane, lq) : -1; };
    auto fetch = [&](int b, int32_t g) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int k = 4 * i + (lane >> 3);
            const int32_t gk = __shfl_sync(0xffffffffu, g, k);
            if (gk >= 0) async_copy16(&S.srec[b][k][lane & 7], recs + (int64_t)kRecFloat4 * gk + (lane & 7));
        }
        async_commit();
    };
    int32_t g = entry(rg.x), g_ahead = AHEAD ? entry(rg.x + 32) : -1;
    if (AHEAD && __any_sync(0xffffffffu, active)) fetch(0, g);
    int buf = 0;
    for (int base = rg.x; base < rg.y && __any_sync(0xffffffffu, active); base += 32) {
        if (kMasks && active) write_checkpoint<LOGT>(hm, st, rg.x, base, sub, subs, p);
        const bool valid = g >= 0;
        if (AHEAD) {
            g = g_ahead;
            fetch(buf ^ 1, g);
            g_ahead = entry(base + 64);
            async_wait_but_last();
        } else {
            fetch(0, g);
            g = entry(base + 32);
            async_wait();
        }
        __syncwarp();
        const float4(*rec)[kRecFloat4 + 1] = S.srec[buf];
        const bool keep = valid && rec[lane][0].w > 0.f &&  // a density of zero hits nothing
                          (!(inv_z > 0.f) || entry_reaches(rec[lane], cam, bd, inv_z));
        const uint32_t bal = __ballot_sync(0xffffffffu, keep);
        uint32_t hb = 0;  // bit k: entry k of the block was a hit for this lane's pixel
        bool ended = false;
        if (active) {
            for (uint32_t left = bal; left; left &= left - 1u) {
                const int j = __ffs(left) - 1;
                const EntryResult e = eval_entry<LOGT>(rec[j], o, d);
                if (e.a > 0.f) {
                    hb |= 1u << j;
                    if (LOGT) st.logT = st.logT - e.a;
                    else fold_hit<kMasks>(st, e.a, rec[j][0].w, e.m1, e.d4, e.rgb);
                    if (st.logT < kTermLogT) {
                        nc = base - rg.x + j + 1;
                        ended = true;
                        break;
                    }
                }
            }
        }
        if (kMasks && hm.words) {
            const int64_t i = mask_word(gtile, rg.x, (base - rg.x) >> 5, sub, subs, p);
            if (i < hm.cap) __stcg(hm.words + i, hb);
        }
        if (__any_sync(0xffffffffu, ended)) {
            active = active && !ended;
            bounds(active);
        }
        __syncwarp();  // the walk's reads of the records are done
        if (AHEAD) buf ^= 1;
    }
    if (AHEAD) {  // the copies ahead, before the next item's
        async_wait();
        __syncwarp();
    }
    if (inside) {
        out_nc[pix] = nc;
        if (LOGT) return;
        if (kMasks) finish_checkpoints(hm, st, rg.x, nc, sub, subs, p);
        out_img[pix] = make_float4(st.c[0], st.c[1], st.c[2], st.logT);
        float* dd = out_dist + 5 * pix;
#pragma unroll
        for (int k = 0; k < 5; ++k) dd[k] = st.D[k];
    }
}

// 768 threads per SM (80 registers): at 1024 (64 registers) the spills cost
// more than the warps gain, with the little L1 that the shared memory leaves
// (1.3M tets, 1297x840: 1357 us at 1024, 1024 at 768; a batch of four served
// views 4187 and 3500).
template <int PX, int NT, int B, class V, Walk WALK>
__global__ void __launch_bounds__(NT, 768 / NT) blend_fwd_kernel(
    const int32_t* __restrict__ ids, const int2* __restrict__ ranges, const float4* __restrict__ recs,
    const float2* __restrict__ jitter, const __grid_constant__ V views, float4* __restrict__ out_img,
    float* __restrict__ out_dist, int32_t* __restrict__ out_nc, const Queue q) {
    extern __shared__ __align__(16) unsigned char fwd_smem_raw[];
    FwdPairSmem<PX, B>& S = *reinterpret_cast<FwdPairSmem<PX, B>*>(fwd_smem_raw);
    __shared__ int s_item;
    __shared__ HitMasks hm;  // read once per batch: kept out of the registers
    // first the pair items (the heavy tiles), then each warp on its own
    // the first info[1] tiles of the order go by quarters of their strips
    const int nq = PX == 64 ? __ldg(q.info + 1) : 0;
    const int q_items = nq * q.subs * 4;
    const int n_items = q_items + (__ldg(q.info) - nq) * q.subs;
    if (threadIdx.x == 0)
        hm = live_masks(q.hm, q.subs, WALK == kLogT ? kMaskStats : kMaskValid);  // seen after next_item's barriers
    for (;;) {
        int item = next_item(q, &s_item);
        if (item >= n_items) break;
        int quarter = -1, at = 0;
        if (item < q_items) {
            quarter = item & 3;
            item >>= 2;
        } else {
            item -= q_items;
            at = nq;
        }
        const int t = __ldg(q.order + at + item / q.subs), v = views.find(t);
        const int tb = views.tile_base(v);
        const int64_t pb = views.pixel_base(v);
        fwd_pair_item<PX, NT, B, WALK>(t - tb, item % q.subs, quarter, ids, ranges + tb, recs, jitter + pb, views.camera(v),
                                 out_img + pb, out_dist + 5 * pb, out_nc + pb, S, hm, q.subs, t, q);
    }
    constexpr int kParts = PX / 32 > 0 ? PX / 32 : 1;
    constexpr bool kAhead = V::kViews > 1;
    FwdWarpSmem<kAhead>& W = reinterpret_cast<FwdWarpSmem<kAhead>*>(fwd_smem_raw)[threadIdx.x >> 5];
    const int heavy = __ldg(q.info);
    const int w_items = (q.G - heavy) * q.subs * kParts;
    for (;;) {
        int item = 0;
        if ((threadIdx.x & 31) == 0) item = (int)atomicAdd(q.ticket + 1, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= w_items) return;
        const int part = item % kParts, strip = item / kParts;
        const int t = __ldg(q.order + heavy + strip / q.subs), v = views.find(t);
        const int tb = views.tile_base(v);
        const int64_t pb = views.pixel_base(v);
        fwd_warp_item<PX, WALK, kAhead>(t - tb, strip % q.subs, part, ids, ranges + tb, recs, jitter + pb, views.camera(v),
                          out_img + pb, out_dist + 5 * pb, out_nc + pb, W, hm, q.subs, t, q);
    }
}

// Orders the tiles heaviest first by floor(log2(list length)) (the order
// inside a bucket does not matter), marks as heavy the tiles whose bucket is
// at least heavy_shift above that of the mean non-empty list length and at
// least 2^10 entries (info[0] = their count), and resets the queue tickets.
// One cluster: each CTA counts and places the tiles of its own chunks, and the
// bucket counts are exchanged through distributed shared memory.  What bounds
// it is the chain of matches and shared atomics of a CTA (one CTA of the same
// size took 17.8 us for 17k tiles and 173 for 131k; this 8.8 and 43).
constexpr int kOrderCtas = 8;
__global__ void __cluster_dims__(kOrderCtas, 1, 1) __launch_bounds__(1024)
    order_kernel(const int2* __restrict__ ranges, int G, int32_t* __restrict__ order, int32_t* info, uint32_t* tickets,
                 int heavy_shift, uint32_t* mask_header, const MaskRoom room, const uint32_t* seg_header,
                 int fwd_slots) {
    // Warp-aggregated counting: lanes that share a bucket elect one leader
    // (match_any) for the shared atomic, and the list-length sum and the
    // non-empty count are reduced per warp before one shared update each.
    __shared__ uint32_t cnt[33], all[33], base[33], cur[33];
    __shared__ unsigned long long wtotal[32], total_s;
    __shared__ uint32_t wnonempty[32], nonempty_s;
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 33) cnt[threadIdx.x] = 0, cur[threadIdx.x] = 0;
    __syncthreads();
    unsigned long long total = 0ull;
    uint32_t nonempty = 0u;
    const int G_pad = (G + 31) & ~31;  // whole warps iterate together
    const int t_first = rank * (int)blockDim.x + (int)threadIdx.x, t_step = kOrderCtas * (int)blockDim.x;
    for (int t = t_first; t < G_pad; t += t_step) {
        uint32_t len = 0u;
        if (t < G) {
            const int2 r = __ldg(ranges + t);
            len = (uint32_t)max(r.y - r.x, 0);
        }
        total += len;
        nonempty += __popc(__ballot_sync(0xffffffffu, len != 0u));
        const int b = t < G ? 32 - __clz(len) : 33;
        const unsigned peers = __match_any_sync(0xffffffffu, b);
        if (b < 33 && lane == __ffs(peers) - 1) atomicAdd(&cnt[b], (uint32_t)__popc(peers));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane == 0) wtotal[warp] = total, wnonempty[warp] = nonempty;
    __syncthreads();
    if (warp == 0) {  // one lane a warp of the CTA
        unsigned long long x = wtotal[lane];
#pragma unroll
        for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        const uint32_t y = __reduce_add_sync(0xffffffffu, wnonempty[lane]);
        if (lane == 0) total_s = x, nonempty_s = y;
    }
    cluster.sync();
    if (threadIdx.x < 33) {
        uint32_t sum = 0u, before = 0u;  // of the bucket: all tiles, those of the CTAs before
        for (int k = 0; k < kOrderCtas; ++k) {
            if (k == rank) before = sum;
            sum += cluster.map_shared_rank(cnt, k)[threadIdx.x];
        }
        all[threadIdx.x] = sum;
        base[threadIdx.x] = before;
    }
    unsigned long long sum = 0ull;
    uint32_t ne = 0u;
    if (threadIdx.x == 0)
        for (int k = 0; k < kOrderCtas; ++k)
            sum += *cluster.map_shared_rank(&total_s, k), ne += *cluster.map_shared_rank(&nonempty_s, k);
    cluster.sync();  // the other CTAs' counts are read
    if (warp == 0) {  // heaviest bucket first (32 is empty: lengths are below 2^31)
        const uint32_t x = all[31 - lane];
        uint32_t inc = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        base[31 - lane] += inc - x;
    }
    if (threadIdx.x == 0 && rank == 0) {
        // segments per bucket of the masks' segment length (segment_item)
        int shift = kNoSegments;
        if (seg_header && __ldcg(seg_header) == kMaskValid) shift = (int)__ldcg(seg_header + 1);
        if (mask_header) {
            MaskPlan plan = {kNoSegments, 0, 0};
            if (room.state != 0u) plan = mask_plan(room.words, G, room.subs, (int64_t)sum);
            shift = plan.shift;
            mask_header[0] = room.state;
            mask_header[1] = (uint32_t)shift;
            mask_header[2] = (uint32_t)plan.ck_cap;
            *(int64_t*)(mask_header + 4) = plan.ck_off;
        }
        if (shift >= kMinSegShift && shift <= kNoSegments) {
            uint32_t at = 0;
            for (int b = 32; b > shift; --b) {
                info[kSegInfoOff + 32 - b] = (int32_t)at;
                at += all[b] << (b - shift);
            }
            info[kSegInfoOff + 32 - shift] = (int32_t)at;
        }
        const uint32_t mean = ne ? (uint32_t)(sum / ne) : 0u;
        // heavy_shift 1 sends every tile to the pair kernel, 0 none
        int b_thr = heavy_shift == 1 ? 0 : heavy_shift == 0 ? 33 : max(11, 32 - __clz(mean) + heavy_shift);
        if (heavy_shift == 0 && fwd_slots > 0) {
            // forward, by itself: a strip is walked by two of the 8 warps of a
            // resident CTA unless its list is longer than a warp's share of
            // all entries
            const unsigned long long share = sum / (8ull * fwd_slots);
            while (b_thr > 1 && (1ull << (b_thr - 2)) >= share) --b_thr;
        }
        int heavy = 0;
        for (int b = 32; b >= b_thr; --b) heavy += (int)all[b];
        info[0] = heavy;
        // Tiles whose list is longer than a fourth of one resident CTA's share
        // of all entries go by quarters: walked by one CTA each, they would
        // outlast the launch.  With few strips to a CTA there is little else to
        // fill the launch with and a quarter's overhead counts: a whole share.
        // (1.3M tets, 39 strips to a CTA: 1048 us at a fourth, 1268 at a whole;
        // 27k tets at 256x256, 2.3 strips: 165 and 140.)
        int quarters = 0;
        if (fwd_slots > 0) {
            const unsigned long long share = sum / ((ne >= 8u * fwd_slots ? 4ull : 1ull) * fwd_slots);
            for (int b = 32; b > 0 && (1ull << (b - 1)) >= share; --b) quarters += (int)all[b];
        }
        info[1] = min(quarters, heavy);
        for (int k = 0; k < 4; ++k) tickets[k] = 0u;
    }
    __syncthreads();
    const unsigned lt = (1u << lane) - 1u;
    for (int t = t_first; t < G_pad; t += t_step) {
        int b = 33;
        if (t < G) {
            const int2 r = __ldg(ranges + t);
            b = 32 - __clz((uint32_t)max(r.y - r.x, 0));
        }
        const unsigned peers = __match_any_sync(0xffffffffu, b);
        const int leader = __ffs(peers) - 1;
        uint32_t at = 0u;
        if (b < 33 && lane == leader) at = atomicAdd(&cur[b], (uint32_t)__popc(peers));
        at = __shfl_sync(0xffffffffu, at, leader);
        if (b < 33) order[base[b] + at + __popc(peers & lt)] = t;
    }
}

// --------------------------------------------------------------- backward --
// Warp reduce-scatter by recursive halving over lane offsets OFF, OFF/2, ..., 1:
// after run(), lane l holds in v[0..R) the warp sums of the original value
// indices [slot, slot + R) (indices >= M are padding).
template <int M, int OFF>
struct ReduceScatter {
    static constexpr int H = (M + 1) / 2;
    static constexpr int R = ReduceScatter<H, OFF / 2>::R;
    template <unsigned MASK>
    static __device__ __forceinline__ void run(float* v, int lane, int& slot) {
        const bool up = (lane & OFF) != 0;
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const float lo = v[i];
            const float hi = (H + i < M) ? v[H + i] : 0.f;
            const float send = up ? lo : hi;
            const float keep = up ? hi : lo;
            v[i] = keep + __shfl_xor_sync(MASK, send, OFF);
        }
        if (up) slot += H;
        ReduceScatter<H, OFF / 2>::template run<MASK>(v, lane, slot);
    }
};
template <int M>
struct ReduceScatter<M, 0> {
    static constexpr int R = M;
    template <unsigned MASK>
    static __device__ __forceinline__ void run(float*, int, int&) {}
};

// Warp sum of the 25 per-lane partials of one entry, through shared memory,
// added to the entry's accumulator acc[0..25).  Each lane stores its row as
// seven float4 (row stride 28 floats: the eight lanes of each store phase
// hit distinct banks); then lane k < 25 adds column k over the 32 rows
// (consecutive lanes read consecutive words).  Fewer instructions than the
// 27-shuffle reduce-scatter for full warps.  red: 32 * kRedStride floats,
// 16-byte aligned, private to the warp.
constexpr int kRedStride = 28;

__device__ __forceinline__ void warp_sum_columns(const float* red, int lane, float* __restrict__ acc) {
    __syncwarp();
    if (lane < kNGrad) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
        for (int r = 0; r < 32; r += 4) {
            s0 += red[(r + 0) * kRedStride + lane];
            s1 += red[(r + 1) * kRedStride + lane];
            s2 += red[(r + 2) * kRedStride + lane];
            s3 += red[(r + 3) * kRedStride + lane];
        }
        const float sum = (s0 + s1) + (s2 + s3);
        if (sum != 0.f) atomicAdd(acc + lane, sum);
    }
    __syncwarp();
}

// As warp_sum_columns, from hit_grads_planes' output: gl[12..25) and the two
// planes' normal gradients, stored at the planes' columns (ie, ix: -1 for none
// or a lane without a hit, whose gl[12..25) are zero).
__device__ __forceinline__ void warp_sum_rows_planes(float* __restrict__ red, const float* gl, f3 dne, f3 dnx,
                                                     int ie, int ix, int lane, float* __restrict__ acc) {
    float* rowf = red + lane * kRedStride;
    float4* row = reinterpret_cast<float4*>(rowf);
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    row[0] = z;
    row[1] = z;
    row[2] = z;
#pragma unroll
    for (int c = 3; c < 6; ++c) row[c] = make_float4(gl[4 * c], gl[4 * c + 1], gl[4 * c + 2], gl[4 * c + 3]);
    row[6] = make_float4(gl[24], 0.f, 0.f, 0.f);
    if (ie >= 0) {
        rowf[3 * ie] = dne.x;
        rowf[3 * ie + 1] = dne.y;
        rowf[3 * ie + 2] = dne.z;
    }
    if (ix >= 0) {
        rowf[3 * ix] = dnx.x;
        rowf[3 * ix + 1] = dnx.y;
        rowf[3 * ix + 2] = dnx.z;
    }
    warp_sum_columns(red, lane, acc);
}

// Adjoint of one hit (the Slang autodiff of update_alpha_out,
// evaluate_tetra_interp and load_tet_alphablend_interp, written out by hand).
// Inputs: the entry's intersection and segment, T = exp(log T) and D2, D3 of
// the state before the hit, and dL/d(state after the hit) (dS_c, dS_logT,
// dS_D).  Outputs the 25 per-entry partials gl[] (face normals 0..11, direct
// v0 12..14, v1 15..17, density 18, rgb 19..21, grd 22..24) and returns
// dL/d(log T before the hit); nD2 / nD3 receive dL/d(D2, D3 before the hit).
// a0, a1: v0 - o and v1 - o (the reference vertices of the planes).
//
// hit_grads_planes leaves gl[0..12) alone and returns the gradients of the
// entering and exiting planes' normals (planes is.ie, is.ix) in dne, dnx
// (both zero for a plane index of -1); hit_grads_a scatters them into
// gl[0..12).
__device__ __forceinline__ float hit_grads_planes(const float4* __restrict__ q, f3 a0, f3 a1, f3 d,
                                                  const Isect& is, const Segment& s, float T, float D2_old,
                                                  float D3_old, const float* dS_c, float dS_logT, const float* dS_D,
                                                  float* gl, f3& dne, f3& dnx, float& nD2, float& nD3) {
    const float density = q[0].w;
    const float enter = is.enter, exit = is.exit;
    const float m1 = density * (exit + enter) / 2.0f;
    // update_distortion_state
    const float dm1 = dS_D[0] * 2.0f * D2_old + dS_D[3];
    const float dm0 = dS_D[1] * 2.0f * D3_old + dS_D[2];
    nD2 = dS_D[2] + dS_D[0] * 2.0f * m1;
    nD3 = dS_D[3] + dS_D[1] * 2.0f * density;
    float d_dens = dm0 + dm1 * (exit + enter) * 0.5f;
    float d_enter = dm1 * density * 0.5f;
    float d_exit = d_enter;
    float d_dt = dS_D[4] * density * density * (1.0f / 3.0f);
    d_dens += dS_D[4] * 2.0f * density * s.dt * (1.0f / 3.0f);
    // update_pixel_state
    float d_rgb[3], dT = 0.f, sum_drgb = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        d_rgb[k] = dS_c[k] * T;
        dT = fmaf(dS_c[k], s.rgb[k], dT);
        sum_drgb += d_rgb[k];
    }
    const float d_a = -dS_logT;
    // compute_integral / integrate_tetra_segment
    const float base[3] = {q[1].w, q[2].w, q[3].w};
    float d_w0 = 0.f, d_w1 = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        d_w0 = fmaf(d_rgb[k], s.cx + base[k], d_w0);
        d_w1 = fmaf(d_rgb[k], s.ce + base[k], d_w1);
        gl[19 + k] = d_rgb[k] * (s.w.w0 + s.w.w1);
    }
    const float d_sx = sum_drgb * s.w.w0, d_se = sum_drgb * s.w.w1;
    const float d_x = (d_w0 - d_w1) * dphi_f(s.x, s.w) + d_w0 * s.w.alpha;
    d_dt += (d_x + d_a) * density;
    d_dens += (d_x + d_a) * s.dt;
    const f3 grd = {q[4].w, q[5].w, q[6].w};
    gl[22] = d_se * s.ve.x + d_sx * s.vx.x;
    gl[23] = d_se * s.ve.y + d_sx * s.vx.y;
    gl[24] = d_se * s.ve.z + d_sx * s.vx.z;
    const float d_sum = d_se + d_sx;
    const float gd = dot3(grd, d);
    d_enter += d_se * gd;
    d_exit += d_sx * gd;
    gl[12] = -grd.x * d_sum;
    gl[13] = -grd.y * d_sum;
    gl[14] = -grd.z * d_sum;
    gl[15] = gl[16] = gl[17] = 0.f;
    if (exit - enter > 0.f) {
        d_exit += d_dt;
        d_enter -= d_dt;
    }
    gl[18] = density > 0.f ? d_dens : 0.f;
    float d_tx = 0.f;
    if (is.tx > enter) d_tx = d_exit; else d_enter += d_exit;
    const float d_te = is.te > 0.f ? d_enter : 0.f;
    // plane intersections t = dot(n, vref - o) / dot(n, d)
    // gradient factors only (the hit and its t values are exact above): the
    // approximate quotient (2 ulp) is far inside the gradients' tolerance
    const float ge = __fdividef(d_te, is.dene), gx = __fdividef(d_tx, is.denx);
    // a plane index of -1 (no entering / exiting plane) contributes nothing
    const float gek = is.ie >= 0 ? ge : 0.f, gxk = is.ix >= 0 ? gx : 0.f;
    const f3 ae = is.ie == 3 ? a1 : a0, ax = is.ix == 3 ? a1 : a0;
    dne = {gek * (ae.x - is.te * d.x), gek * (ae.y - is.te * d.y), gek * (ae.z - is.te * d.z)};
    dnx = {gxk * (ax.x - is.tx * d.x), gxk * (ax.y - is.tx * d.y), gxk * (ax.z - is.tx * d.z)};
    // the planes' reference vertices (v1 for plane 3, v0 for the others):
    // gradient +n * g; the normals are read from the staged record by index
    const f3 ne = xyz(q[is.ie < 0 ? 0 : is.ie]), nx = xyz(q[is.ix < 0 ? 0 : is.ix]);
    const float ge0 = is.ie == 3 ? 0.f : gek, ge1 = is.ie == 3 ? gek : 0.f;
    const float gx0 = is.ix == 3 ? 0.f : gxk, gx1 = is.ix == 3 ? gxk : 0.f;
    gl[12] += ne.x * ge0 + nx.x * gx0;
    gl[13] += ne.y * ge0 + nx.y * gx0;
    gl[14] += ne.z * ge0 + nx.z * gx0;
    gl[15] += ne.x * ge1 + nx.x * gx1;
    gl[16] += ne.y * ge1 + nx.y * gx1;
    gl[17] += ne.z * ge1 + nx.z * gx1;
    // safe_exp's clip at log(1e20) never binds: log T <= 0
    return dS_logT + dT * T;
}

__device__ __forceinline__ float hit_grads_a(const float4* __restrict__ q, f3 a0, f3 a1, f3 d, const Isect& is,
                                             const Segment& s, float T, float D2_old, float D3_old,
                                             const float* dS_c, float dS_logT, const float* dS_D, float* gl,
                                             float& nD2, float& nD3) {
    f3 dne, dnx;
    const float r = hit_grads_planes(q, a0, a1, d, is, s, T, D2_old, D3_old, dS_c, dS_logT, dS_D, gl, dne, dnx,
                                     nD2, nD3);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        gl[3 * p + 0] = (is.ie == p ? dne.x : 0.f) + (is.ix == p ? dnx.x : 0.f);
        gl[3 * p + 1] = (is.ie == p ? dne.y : 0.f) + (is.ix == p ? dnx.y : 0.f);
        gl[3 * p + 2] = (is.ie == p ? dne.z : 0.f) + (is.ix == p ? dnx.z : 0.f);
    }
    return r;
}

__device__ __forceinline__ float hit_grads(const float4* __restrict__ q, f3 o, f3 d, const Isect& is,
                                           const Segment& s, float T, float D2_old, float D3_old,
                                           const float* dS_c, float dS_logT, const float* dS_D, float* gl,
                                           float& nD2, float& nD3) {
    return hit_grads_a(q, xyz(q[4]) - o, xyz(q[5]) - o, d, is, s, T, D2_old, D3_old, dS_c, dS_logT, dS_D, gl, nD2,
                       nD3);
}

// Converts the per-entry sums of the 25 partials into vertex and cell-value
// gradients and adds them to global memory (one thread per entry).
template <int NT, int B>
__device__ __forceinline__ void flush_entries(int n, const float4 (*srec)[kRecFloat4], const int32_t* sid,
                                              const float (*sacc)[kNGrad], const int4* __restrict__ indices,
                                              float* __restrict__ gverts, float* __restrict__ gcv) {
    for (int jj = threadIdx.x; jj < n; jj += NT) {
        float v[kNGrad];
        bool any = false;
#pragma unroll
        for (int k = 0; k < kNGrad; ++k) {
            v[k] = sacc[jj][k];
            any |= v[k] != 0.f;
        }
        const int g = sid[jj];
        if (!any || g < 0) continue;
        const float4* q = srec[jj];
        const f3 P[4] = {xyz(q[4]), xyz(q[5]), xyz(q[6]), xyz(q[7])};
        const uint32_t flips = __float_as_uint(q[7].w);
        f3 gv[4] = {{v[12], v[13], v[14]}, {v[15], v[16], v[17]}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
        const int pp[4] = {1, 1, 2, 2}, pq[4] = {0, 0, 0, 1}, pr[4] = {2, 3, 3, 3};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            f3 gc = {v[3 * p], v[3 * p + 1], v[3 * p + 2]};
            if (flips & (1u << p)) gc = neg3(gc);
            const f3 ea = P[pp[p]] - P[pq[p]], eb = P[pr[p]] - P[pq[p]];
            const f3 ga = cross3(eb, gc), gb = cross3(gc, ea);
            gv[pp[p]] = gv[pp[p]] + ga;
            gv[pr[p]] = gv[pr[p]] + gb;
            gv[pq[p]] = gv[pq[p]] - (ga + gb);
        }
        const int4 id = __ldg(indices + g);
        const int vid[4] = {id.x, id.y, id.z, id.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float* dst = gverts + 3 * (int64_t)vid[i];
            if (gv[i].x != 0.f) atomicAdd(dst, gv[i].x);
            if (gv[i].y != 0.f) atomicAdd(dst + 1, gv[i].y);
            if (gv[i].z != 0.f) atomicAdd(dst + 2, gv[i].z);
        }
        float* dc = gcv + 7 * (int64_t)g;
#pragma unroll
        for (int k = 0; k < 7; ++k)
            if (v[18 + k] != 0.f) atomicAdd(dc + k, v[18 + k]);
    }
}

// The state of the reverse walk at the checkpoint at list offset s1, which the
// pixel passed alive: log T, D2, D3 as stored, and the adjoint state after the
// entries from s1 on.  Each of those hits adds T * dot(dL/dc, rgb) to
// dL/dlogT, 2 m1 dL/dD0 to dL/dD2 and 2 m0 dL/dD1 to dL/dD3; the checkpoint
// holds the sums of T * rgb, m0 and m1 over them.
__device__ __forceinline__ void seed_segment(const HitMasks& hm, int x, int s1, int sub, int subs, int p,
                                             float& logT, float& D2, float& D3, const float* dS_c, float& dS_logT,
                                             float* dS_D) {
    const float* c = ck_at(hm, ck_id(x, s1 >> hm.seg_shift, hm.seg_shift), sub, subs, p);
    logT = __ldcg(c);
    D2 = __ldcg(c + 64);
    D3 = __ldcg(c + 2 * 64);
#pragma unroll
    for (int i = 0; i < 3; ++i) dS_logT = fmaf(dS_c[i], __ldcg(c + (3 + i) * 64), dS_logT);
    dS_D[3] = fmaf(2.0f * dS_D[1], __ldcg(c + 6 * 64), dS_D[3]);
    dS_D[2] = fmaf(2.0f * dS_D[0], __ldcg(c + 7 * 64), dS_D[2]);
}

// The lowest n bits of w (none for n <= 0).
__device__ __forceinline__ uint32_t bits_below(uint32_t w, int n) {
    return n <= 0 ? 0u : n >= 32 ? w : w & ((1u << n) - 1u);
}

// Backward item: a 64-pixel strip (16 for 16-pixel strips) over one stretch of
// a tile's list, walked back to front by one warp per 32 pixels (8x4), one
// pixel per lane.  Per block of 32 entries (one mask word per pixel) the
// records of the entries some pixel hit are copied to shared memory; each warp
// walks those that its pixels hit, meets each once, and so has its sums over
// the lanes final when formed (no accumulators to clear, no atomics in shared
// memory).  One of the two warps, in turn, then adds up both warps' sums and
// turns them into vertex and cell-value gradients, one entry per lane.  (Each
// warp adding its own half to global memory saves the barriers, but doubles
// the float additions into the tets and vertices that fill much of the image,
// and with them the rounding of those sums: 1.46e-6 against 0.67e-6 relative
// to 64 bits for the cell values of a 1.3M-tet frame.)
//
// Per hit the lane forms 23 partials: for each face p the sums G_p of
// dL/dt / dot(n_p, d) over the hits that enter or leave through it and H_p of
// the same times the hit point relative to v0, density, rgb and the colour
// gradient.  The gradient of the face normals, of v0 and v1 follow from them
// once per entry (flush_sums): with t_p = dot(n_p, v_ref - o) / dot(n_p, d),
// dt/dn = -(hit point - v_ref) / dot(n, d) and dt/dv_ref = n / dot(n, d).
//
// Bound: instruction issue, about 440 instructions for an entry and up to 32
// pixels, and the shared-memory traffic of the row sums.
template <int NW>
struct BwdSmem {
    float4 srec[32][kRecFloat4 + 1];
    float4 red[NW][32 * kRedStride / 4];  // one row of partials per lane
    float4 sums[NW][32][6];  // per entry: (G, H) of the four faces, density rgb, grd 0
    uint32_t any[2][NW];     // entries that the warp's pixels hit, of this block and the next
    int4 item;
};

// a += v by two packed additions.
__device__ __forceinline__ void add4(float4& a, float4 v) {
    unsigned long long* p = reinterpret_cast<unsigned long long*>(&a);
    const unsigned long long* q = reinterpret_cast<const unsigned long long*>(&v);
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(p[0]) : "l"(q[0]));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(p[1]) : "l"(q[1]));
}
__device__ __forceinline__ float4 shfl_xor4(float4 a, int off) {
    return make_float4(__shfl_xor_sync(0xffffffffu, a.x, off), __shfl_xor_sync(0xffffffffu, a.y, off),
                       __shfl_xor_sync(0xffffffffu, a.z, off), __shfl_xor_sync(0xffffffffu, a.w, off));
}

// Adds up the 24 columns of the lanes' rows: the lane's group (lane / 8) takes
// eight rows, its place in it (< 6) four columns; the groups meet by shuffles.
// Rows of the lanes in bal_a go to a, the others to b (SPLIT) or to a too.
template <bool SPLIT>
__device__ __forceinline__ void warp_sum_rows(const float4* __restrict__ red, int lane, uint32_t bal_a, float4& a,
                                              float4& b) {
    const int quad = lane & 7, row0 = lane & 24;
    a = make_float4(0.f, 0.f, 0.f, 0.f);
    b = a;
    __syncwarp();
    if (quad < 6) {
        const uint32_t in = bal_a >> row0;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float4 v = red[(row0 + r) * (kRedStride / 4) + quad];
            if (!SPLIT || ((in >> r) & 1u)) add4(a, v);
            else add4(b, v);
        }
    }
    __syncwarp();
#pragma unroll
    for (int off = 8; off <= 16; off <<= 1) {
        add4(a, shfl_xor4(a, off));
        if (SPLIT) add4(b, shfl_xor4(b, off));
    }
}

// One entry's sums -> gradients of its four vertices and seven cell values,
// added to global memory by one thread.
__device__ __forceinline__ void flush_sums(const float4* __restrict__ q, const float4* s, int32_t g,
                                           const int4* __restrict__ indices, float* __restrict__ gverts,
                                           float* __restrict__ gcv) {
    const f3 P[4] = {xyz(q[4]), xyz(q[5]), xyz(q[6]), xyz(q[7])};
    const uint32_t flips = __float_as_uint(q[7].w);
    const float4 c = s[4];  // density, r, g, b
    const float4 k = s[5];  // grd
    const float dsum = -(c.y + c.z + c.w);
    f3 gv[4] = {{q[4].w * dsum, q[5].w * dsum, q[6].w * dsum}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    const int pp[4] = {1, 1, 2, 2}, pq[4] = {0, 0, 0, 1}, pr[4] = {2, 3, 3, 3};
    bool any = c.x != 0.f || c.y != 0.f || c.z != 0.f || c.w != 0.f || k.x != 0.f || k.y != 0.f || k.z != 0.f;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const float4 h = s[p];  // (G, H)
        any |= h.x != 0.f || h.y != 0.f || h.z != 0.f || h.w != 0.f;
        const f3 n = xyz(q[p]);
        f3& ref = gv[pq[p]];
        ref = {fmaf(n.x, h.x, ref.x), fmaf(n.y, h.x, ref.y), fmaf(n.z, h.x, ref.z)};
        f3 gc = {-h.y, -h.z, -h.w};  // gradient of the normal
        if (p == 3) {
            const f3 e = P[1] - P[0];
            gc = {fmaf(e.x, h.x, gc.x), fmaf(e.y, h.x, gc.y), fmaf(e.z, h.x, gc.z)};
        }
        if (flips & (1u << p)) gc = neg3(gc);
        const f3 ea = P[pp[p]] - P[pq[p]], eb = P[pr[p]] - P[pq[p]];
        const f3 ga = cross3(eb, gc), gb = cross3(gc, ea);
        gv[pp[p]] = gv[pp[p]] + ga;
        gv[pr[p]] = gv[pr[p]] + gb;
        ref = ref - (ga + gb);
    }
    if (!any) return;
    const int4 id = __ldg(indices + g);
    const int vid[4] = {id.x, id.y, id.z, id.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float* dst = gverts + 3 * (int64_t)vid[i];
        if (gv[i].x != 0.f) atomicAdd(dst, gv[i].x);
        if (gv[i].y != 0.f) atomicAdd(dst + 1, gv[i].y);
        if (gv[i].z != 0.f) atomicAdd(dst + 2, gv[i].z);
    }
    const float out[7] = {c.x, c.y, c.z, c.w, k.x, k.y, k.z};
    float* dc = gcv + 7 * (int64_t)g;
#pragma unroll
    for (int i = 0; i < 7; ++i)
        if (out[i] != 0.f) atomicAdd(dc + i, out[i]);
}

template <int PX>
__device__ __forceinline__ void bwd_item(
    int tile, int sub, int seg, const int32_t* __restrict__ ids, const int2* __restrict__ ranges,
    const float4* __restrict__ recs, const int4* __restrict__ indices, const float2* __restrict__ jitter,
    const rm_camera& cam, const float4* __restrict__ img, const float* __restrict__ dist,
    const int32_t* __restrict__ ncs, const float4* __restrict__ gimg, const float* __restrict__ gdist,
    float* __restrict__ gverts, float* __restrict__ gcv, BwdSmem<PX / 32 + (PX < 32)>& S, const HitMasks& hm, int subs,
    int gtile, const Queue& lq) {
    constexpr int kWarps = PX / 32 + (PX < 32);
    constexpr unsigned kAll = 0xffffffffu;
    const int2 rg = __ldg(ranges + tile);
    const int len = rg.y - rg.x;
    // this item's stretch [s0, s1) of the list, as offsets from its start
    int s0 = 0, s1 = len;
    if (hm.ck && len > (1 << hm.seg_shift)) {
        const int shift = hm.seg_shift;
        if (ck_id(rg.x, (len - 1) >> shift, shift) < hm.ck_cap) {
            s0 = seg << shift;
            s1 = min(len, s0 + (1 << shift));
        } else if (seg) {
            return;  // no room for its checkpoints: item 0 walks the whole list
        }
    } else if (seg) {
        return;
    }
    if (s0 >= s1) return;
    const int p = threadIdx.x, lane = p & 31, warp = p >> 5;
    const int tx = tile % cam.grid_width, ty = tile / cam.grid_width;
    int lx, ly;
    strip_pixel<PX>(cam, sub, p, lx, ly);
    const int px = tx * cam.tile_width + lx, py = ty * cam.tile_height + ly;
    const bool inside = p < PX && px < cam.image_width && py < cam.image_height;
    const int64_t pix = (int64_t)py * cam.image_width + px;
    int32_t nc = inside ? __ldg(ncs + pix) : 0;
    if (nc <= s0) nc = 0;
    // the last block that some pixel's walk reaches (none: they all end before
    // this stretch)
    int last = min((int)__reduce_max_sync(kAll, (unsigned)nc), s1);
    if (kWarps > 1) {
        if (lane == 0) S.any[0][warp] = (uint32_t)last;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kWarps; ++i) last = max(last, (int)S.any[0][i]);
        __syncthreads();
    }
    if (last == 0) return;
    f3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f};
    float logT = 0.f, D2 = 0.f, D3 = 0.f;  // state along the reverse walk
    float dS_c[3] = {0.f, 0.f, 0.f}, dS_logT = 0.f, dS_D[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    if (nc > 0) {
        const float2 j = __ldg(jitter + pix);
        make_ray(cam, px, py, j.x, j.y, o, d);
        const float4 c = __ldg(img + pix);
        logT = c.w;
        D2 = __ldg(dist + 5 * pix + 2);
        D3 = __ldg(dist + 5 * pix + 3);
        const float4 g = __ldg(gimg + pix);
        dS_c[0] = g.x; dS_c[1] = g.y; dS_c[2] = g.z; dS_logT = g.w;
#pragma unroll
        for (int k = 0; k < 5; ++k) dS_D[k] = gdist ? __ldg(gdist + 5 * pix + k) : 0.f;
        if (PX == 64 && nc > s1) {
            seed_segment(hm, rg.x, s1, sub, subs, p, logT, D2, D3, dS_c, dS_logT, dS_D);
            nc = s1;
        }
    }
    // constants of the walk
    const float dS0 = 2.0f * dS_D[0], dS1 = 2.0f * dS_D[1], dS4 = dS_D[4] * (1.0f / 3.0f);
    const float dS_sum = dS_c[0] + dS_c[1] + dS_c[2];
    float dS2 = dS_D[2], dS3 = dS_D[3];
    float4* const row4 = S.red[warp] + lane * (kRedStride / 4);

    // A pixel's hit bits of block k: the forward's word, all entries without
    // one; none at or past n_contributors.
    auto hit_word = [&](int k) {
        uint32_t w = 0xffffffffu;
        if (PX == 64 && hm.words) {
            const int64_t i = mask_word(gtile, rg.x, k, sub, subs, p);
            if (i < hm.cap) w = __ldcg(hm.words + i);
        }
        return bits_below(w, nc - 32 * k);
    };
    int k = (last - 1) >> 5;
    uint32_t w = hit_word(k), mine = __reduce_or_sync(kAll, w);
    if (lane == 0) S.any[k & 1][warp] = mine;
    __syncthreads();
    for (; k >= s0 >> 5; --k) {
        const uint32_t cur = w, own = mine;
        uint32_t any = 0u;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) any |= S.any[k & 1][i];
        const uint32_t any_other = S.any[k & 1][kWarps - 1 - warp];  // the other warp's (its own for one)
        if (k > s0 >> 5) {  // the next block's, ahead of its use
            w = hit_word(k - 1);
            mine = __reduce_or_sync(kAll, w);
            if (lane == 0) S.any[(k - 1) & 1][warp] = mine;
        }
        if (!any) {
            __syncthreads();  // S.any of the next block
            continue;
        }
        int32_t g = -1;
        if ((any >> lane) & 1u) g = list_id(ids, rg.x + 32 * k + lane, lq);
#pragma unroll
        for (int i = 0; i < 8 / kWarps; ++i) {
            const int e = 4 * (warp + kWarps * i) + (lane >> 3);
            const int32_t ge = __shfl_sync(kAll, g, e);
            if (ge >= 0)
                async_copy16(&S.srec[e][lane & 7], recs + (int64_t)kRecFloat4 * ge + (lane & 7));
            else if ((any >> e) & 1u)
                S.srec[e][lane & 7] = make_float4(0.f, 0.f, 0.f, 0.f);  // names no tet: nothing hits it
        }
        async_wait();
        __syncthreads();
        uint32_t left = own;  // entries to walk
        while (left) {
            const int ja = 31 - __clz(left);
            left &= ~(1u << ja);
            bool act = (cur >> ja) & 1u;
            uint32_t bal_a = kAll;
            // When no pixel of the warp hits both this entry and the next one,
            // the warp takes both at once: each lane walks the one it hits
            // (its own order is unchanged), and the rows go to the two
            // entries' sums by lane.
            int je = ja, jb = -1;
            if (left) {
                jb = 31 - __clz(left);
                const uint32_t both = (1u << ja) | (1u << jb);
                if (__any_sync(kAll, (cur & both) == both)) {
                    jb = -1;
                } else {
                    left &= ~(1u << jb);
                    bal_a = __ballot_sync(kAll, act);
                    const bool act_b = (cur >> jb) & 1u;
                    je = act_b ? jb : ja;
                    act |= act_b;
                }
            }
            const float4* q = S.srec[je];
            const Isect is = intersect<true>(q, o, d);
            const float density = q[0].w;
            const float dt = fmaxf(is.exit - is.enter, 0.f);
            const float a = density * dt;
            const bool hit = act && is.geo && a > 0.f;
            const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int c = 0; c < 4; ++c) row4[c] = z4;
            float4 g_val = z4, g_grd = z4;
            if (hit) {
                // the segment (integrate_tetra_segment), the colour linear along the ray
                const f3 a0 = xyz(q[4]) - o;
                const f3 ve = {fmaf(is.enter, d.x, -a0.x), fmaf(is.enter, d.y, -a0.y), fmaf(is.enter, d.z, -a0.z)};
                const f3 vx = {fmaf(is.exit, d.x, -a0.x), fmaf(is.exit, d.y, -a0.y), fmaf(is.exit, d.z, -a0.z)};
                const f3 grd = {q[4].w, q[5].w, q[6].w};
                const f3 base = {q[1].w, q[2].w, q[3].w};
                const float gd = dot3(grd, d);
                const float ce = dot3(grd, ve), cx = dot3(grd, vx);
                const Weights wt = seg_weights<true>(a);
                const float wsum = wt.w0 + wt.w1;
                const float lin = fmaf(wt.w0, cx, wt.w1 * ce);
                // undo_alpha_out (alphablend_shader_interp.slang:128-192): only
                // log T, D2 and D3 of the earlier state enter the adjoint
                const float sum_t = is.exit + is.enter;
                const float m1 = density * sum_t / 2.0f;
                logT = logT + a;
                const float T = exp_approx(logT);
                D2 = D2 - density;
                D3 = D3 - m1;
                // update_distortion_state
                const float dm1 = fmaf(dS0, D2, dS3), dm0 = fmaf(dS1, D3, dS2);
                dS2 = fmaf(dS0, m1, dS2);
                dS3 = fmaf(dS1, density, dS3);
                float d_dens = fmaf(dm1, 0.5f * sum_t, dm0);
                const float half_m = 0.5f * dm1 * density;
                const float d4 = dS4 * density;
                float d_dt = d4 * density;
                d_dens = fmaf(2.0f * d4, dt, d_dens);
                // update_pixel_state, compute_integral
                const f3 d_rgb = {dS_c[0] * T, dS_c[1] * T, dS_c[2] * T};
                const float sum_d = dS_sum * T;
                const float d_base = dot3(d_rgb, base);
                const float dT = fmaf(wsum, d_base, lin * sum_d);  // T times dot(dL/dc, rgb)
                const float d_w0 = fmaf(sum_d, cx, d_base);
                const float d_sx = sum_d * wt.w0, d_se = sum_d * wt.w1;
                const float d_x = fmaf(sum_d * (cx - ce), dphi_f(a, wt), d_w0 * wt.alpha) - dS_logT;
                dS_logT = dS_logT + dT;
                d_dt = fmaf(d_x, density, d_dt);
                d_dens = fmaf(d_x, dt, d_dens);
                // a hit has exit = tx > enter, so both ends move the segment
                const float d_tx = fmaf(d_sx, gd, half_m) + d_dt;
                const float d_te = is.te > 0.f ? fmaf(d_se, gd, half_m) - d_dt : 0.f;
                // gradient factors only (the hit and its t values are exact
                // above): the approximate quotient (2 ulp) is far inside the
                // gradients' tolerance
                const float ge = d_te * rcp_approx(is.dene), gx = d_tx * rcp_approx(is.denx);
                if (is.ie >= 0) row4[is.ie] = make_float4(ge, ge * ve.x, ge * ve.y, ge * ve.z);
                if (is.ix >= 0) row4[is.ix] = make_float4(gx, gx * vx.x, gx * vx.y, gx * vx.z);
                g_val = make_float4(d_dens, d_rgb.x * wsum, d_rgb.y * wsum, d_rgb.z * wsum);
                g_grd = make_float4(fmaf(d_se, ve.x, d_sx * vx.x), fmaf(d_se, ve.y, d_sx * vx.y),
                                    fmaf(d_se, ve.z, d_sx * vx.z), 0.f);
            }
            row4[4] = g_val;
            row4[5] = g_grd;
            float4 sa, sb;
            if (jb < 0) {
                warp_sum_rows<false>(S.red[warp], lane, bal_a, sa, sb);
            } else {
                warp_sum_rows<true>(S.red[warp], lane, bal_a, sa, sb);
                if (lane < 6) S.sums[warp][jb][lane] = sb;
            }
            if (lane < 6) S.sums[warp][ja][lane] = sa;
        }
        __syncthreads();
        if (warp == k % kWarps && g >= 0) {
            float4 sum[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) sum[c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kWarps; ++i) {
                const uint32_t had = i == warp ? own : any_other;
                if ((had >> lane) & 1u) {
#pragma unroll
                    for (int c = 0; c < 6; ++c) add4(sum[c], S.sums[i][lane][c]);
                }
            }
            flush_sums(S.srec[lane], sum, g, indices, gverts, gcv);
        }
        __syncthreads();  // the next block overwrites the records and the sums
    }
}

// Dense backward with the records staged by bulk copies (RM_BLEND_STAGE_TMA;
// 64-pixel items): one thread per pixel, whole lists, sums over the CTA by
// shared-memory atomics (flush_entries).  Each batch is planned one batch ahead: its hit
// masks are OR-ed over the item, the entries some pixel hit are listed, their
// tet ids loaded, and warp 0 starts one 128-byte cp.async.bulk per entry
// (global -> this CTA's shared memory, completing on the buffer's mbarrier).
// Two record buffers alternate, so batch k+1's copies are in flight while
// batch k is walked and flushed; each copy lands in the issuing CTA only.
template <int B>
struct BwdTmaSmem {
    float4 srec[2][B][kRecFloat4];
    float4 red[2][32 * kRedStride / 4];  // warp_sum_rows_planes rows, per warp
    float sacc[B][kNGrad];
    int32_t sid[2][B];
    uint8_t cidx[2][B];
    int32_t n_keep[2];
    uint32_t sor[2][2];  // per warp: OR of its pixels' hit bits (two 32-entry blocks)
    int32_t smax[2];
    uint64_t bar[2];
};

// Pipeline position carried across work items: the buffer the next plan
// fills and the parity of each buffer's next completion.
struct TmaPipe {
    uint32_t buf;
    uint32_t parity;  // bit b: parity to wait for on buffer b
};

template <int B>
__device__ __forceinline__ void bwd_tma_plan(BwdTmaSmem<B>& S, int b, int lo, int top, int rgx,
                                             const int32_t* __restrict__ ids, const float4* __restrict__ recs,
                                             const HitMasks& hm, int gtile, int sub, int subs, uint32_t& hw0,
                                             uint32_t& hw1, const Queue& lq) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = top - lo;
    const int kb0 = (lo - rgx) >> 5, kb1 = (top - 1 - rgx) >> 5;
    hw0 = 0xffffffffu;
    hw1 = 0xffffffffu;
    if (hm.words) {
        const int64_t i0 = mask_word(gtile, rgx, kb0, sub, subs, (int)threadIdx.x);
        const int64_t i1 = mask_word(gtile, rgx, kb1, sub, subs, (int)threadIdx.x);
        if (i0 < hm.cap) hw0 = __ldcg(hm.words + i0);
        if (i1 < hm.cap) hw1 = __ldcg(hm.words + i1);
    }
    uint32_t o0 = hw0, o1 = hw1;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        o0 |= __shfl_xor_sync(0xffffffffu, o0, off);
        o1 |= __shfl_xor_sync(0xffffffffu, o1, off);
    }
    if (lane == 0) {
        S.sor[warp][0] = o0;
        S.sor[warp][1] = o1;
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t c0 = S.sor[0][0] | S.sor[1][0], c1 = S.sor[0][1] | S.sor[1][1];
        int base_c = 0;
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + lane;
            bool keep = false;
            if (k < n) {
                const int off = lo + k - rgx;
                keep = ((((off >> 5) == kb0 ? c0 : c1) >> (off & 31)) & 1u) != 0u;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, keep);
            if (keep) S.cidx[b][base_c + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)k;
            base_c += __popc(bal);
        }
        if (lane == 0) S.n_keep[b] = base_c;
    }
    __syncthreads();
    const int nk = S.n_keep[b];
    for (int k = threadIdx.x; k < nk; k += 64) S.sid[b][k] = list_id(ids, lo + S.cidx[b][k], lq);
    __syncthreads();
    if (warp == 0) {
        // every read of this buffer (the batch two back) is behind the barriers above
        int nv = 0;  // entries with a record to copy (the others are zero-filled)
        for (int k0 = 0; k0 < nk; k0 += 32)
            nv += __popc(__ballot_sync(0xffffffffu, k0 + lane < nk && S.sid[b][k0 + lane] >= 0));
        fence_proxy_async_smem();
        if (lane == 0) mbar_arrive_expect_tx(&S.bar[b], (uint32_t)nv * (uint32_t)(kRecFloat4 * sizeof(float4)));
        __syncwarp();
        for (int k = lane; k < nk; k += 32) {
            const int32_t g = S.sid[b][k];
            if (g >= 0)
                bulk_copy_g2s(&S.srec[b][k][0], recs + (int64_t)kRecFloat4 * g,
                              (uint32_t)(kRecFloat4 * sizeof(float4)), &S.bar[b]);
            else
                for (int c = 0; c < kRecFloat4; ++c) S.srec[b][k][c] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

template <int B>
__device__ __forceinline__ void bwd_dense_item_tma(
    int tile, int sub, const int32_t* __restrict__ ids, const int2* __restrict__ ranges,
    const float4* __restrict__ recs, const int4* __restrict__ indices, const float2* __restrict__ jitter,
    const rm_camera& cam, const float4* __restrict__ img, const float* __restrict__ dist,
    const int32_t* __restrict__ ncs, const float4* __restrict__ gimg, const float* __restrict__ gdist,
    float* __restrict__ gverts, float* __restrict__ gcv, BwdTmaSmem<B>& S, const HitMasks& hm, int subs, int gtile,
    TmaPipe& pipe, const Queue& q) {
    constexpr int NT = 64;
    const int tx = tile % cam.grid_width, ty = tile / cam.grid_width;
    int lx, ly;
    strip_pixel<NT>(cam, sub, (int)threadIdx.x, lx, ly);
    const int px = tx * cam.tile_width + lx, py = ty * cam.tile_height + ly;
    const bool inside = px < cam.image_width && py < cam.image_height;
    const int64_t pix = (int64_t)py * cam.image_width + px;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    f3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f};
    float logT = 0.f, D2 = 0.f, D3 = 0.f;
    float dS_c[3] = {0.f, 0.f, 0.f}, dS_logT = 0.f, dS_D[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    int32_t nc = 0;
    if (inside) {
        const float2 j = __ldg(jitter + pix);
        make_ray(cam, px, py, j.x, j.y, o, d);
        logT = __ldg(img + pix).w;
        D2 = __ldg(dist + 5 * pix + 2);
        D3 = __ldg(dist + 5 * pix + 3);
        const float4 g = __ldg(gimg + pix);
        dS_c[0] = g.x; dS_c[1] = g.y; dS_c[2] = g.z; dS_logT = g.w;
#pragma unroll
        for (int k = 0; k < 5; ++k) dS_D[k] = gdist ? __ldg(gdist + 5 * pix + k) : 0.f;
        nc = __ldg(ncs + pix);
    }
    int32_t m = nc;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
    if (lane == 0) S.smax[warp] = m;
    __syncthreads();
    const int32_t tile_max = max(S.smax[0], S.smax[1]);
    const int2 rg = __ldg(ranges + tile);
    const int end = min(rg.y, rg.x + tile_max);
    if (end <= rg.x) return;  // uniform over the CTA
    // batches aligned to multiples of B from the list start (at most two mask blocks each)
    int ctop = end, clo = rg.x + ((end - 1 - rg.x) / B) * B;
    uint32_t cw0, cw1;
    int cb = (int)pipe.buf;
    bwd_tma_plan<B>(S, cb, clo, ctop, rg.x, ids, recs, hm, gtile, sub, subs, cw0, cw1, q);
    pipe.buf ^= 1u;
    for (;;) {
        const int ntop = clo;
        const bool has_next = ntop > rg.x;
        int nlo = 0, nb = 0;
        uint32_t nw0 = 0u, nw1 = 0u;
        if (has_next) {  // the next batch's copies run while this one is walked
            nlo = rg.x + ((ntop - 1 - rg.x) / B) * B;
            nb = (int)pipe.buf;
            bwd_tma_plan<B>(S, nb, nlo, ntop, rg.x, ids, recs, hm, gtile, sub, subs, nw0, nw1, q);
            pipe.buf ^= 1u;
        }
        const int nk = S.n_keep[cb];
        for (int k = threadIdx.x; k < nk * kNGrad; k += NT) (&S.sacc[0][0])[k] = 0.f;
        if (!mbar_wait(&S.bar[cb], (pipe.parity >> cb) & 1u, q.spin_limit)) {
            if (threadIdx.x == 0 && q.status) atomicOr(q.status, RM_STATUS_QUEUE_TIMEOUT);
            mbar_wait(&S.bar[cb], (pipe.parity >> cb) & 1u, q.spin_limit);  // let the copies land before reuse
        }
        pipe.parity ^= 1u << cb;
        __syncthreads();
        const int kb0 = (clo - rg.x) >> 5;
        for (int jj = nk - 1; jj >= 0; --jj) {
            const int off = clo + S.cidx[cb][jj] - rg.x;
            // with the forward's masks, only its hits are revisited
            const uint32_t hw = (off >> 5) == kb0 ? cw0 : cw1;
            const bool act = inside && off < nc && ((hw >> (off & 31)) & 1u);
            if (!__any_sync(0xffffffffu, act)) continue;
            const float4* qr = S.srec[cb][jj];
            float gl[kNGrad];
#pragma unroll
            for (int k = 0; k < kNGrad; ++k) gl[k] = 0.f;
            const Isect is = intersect<true>(qr, o, d);
            const float density = qr[0].w;
            Segment sg;
            sg.dt = fmaxf(is.exit - is.enter, 0.f);
            sg.a = density * sg.dt;
            const bool hit = act && is.geo && sg.a > 0.f;
            f3 dne = {0.f, 0.f, 0.f}, dnx = {0.f, 0.f, 0.f};
            if (hit) {
                integrate(qr, o, d, is.enter, is.exit, sg);
                const float m1 = density * (is.exit + is.enter) / 2.0f;
                const float logT_old = logT + sg.a;
                const float T = __expf(logT_old);
                D2 = D2 - density;
                D3 = D3 - m1;
                logT = logT_old;
                float nD2, nD3;
                dS_logT = hit_grads_planes(qr, xyz(qr[4]) - o, xyz(qr[5]) - o, d, is, sg, T, D2, D3, dS_c, dS_logT,
                                           dS_D, gl, dne, dnx, nD2, nD3);
                dS_D[2] = nD2;
                dS_D[3] = nD3;
            }
            if (__any_sync(0xffffffffu, hit))
                warp_sum_rows_planes(reinterpret_cast<float*>(S.red[warp]), gl, dne, dnx, hit ? is.ie : -1,
                                     hit ? is.ix : -1, lane, S.sacc[jj]);
        }
        __syncthreads();
        flush_entries<NT, B>(nk, S.srec[cb], S.sid[cb], S.sacc, indices, gverts, gcv);
        __syncthreads();
        if (!has_next) break;
        cb = nb;
        clo = nlo;
        ctop = ntop;
        cw0 = nw0;
        cw1 = nw1;
    }
}

// Pair backward item: the same strip / thread split as the forward.  Per
// batch of B entries (walked back to front) the pixels that still have list
// offsets below their n_contributors are compacted into slots and
//   A. all warps test the (entry, slot) pairs: a (0: no hit), m1 and
//      dot(dL/dcolour, rgb);
//   B. each owner walks its pixel's entries back to front and records, per
//      hit, T and D2, D3 of the state before the hit and dL/d(log T, D2, D3)
//      after it (the only state the adjoint reads; colour and D0, D1, D4 need
//      no undo);
//   C. all warps compute the 25 per-entry partials of every hit pair (warp =
//      entry, lanes = slots), sum them over the warp with a reduce-scatter and
//      add them to the entry's shared accumulator.
template <int PX, int B>
struct BwdPairSmem {
    float4 srec[B][kRecFloat4];
    int32_t sid[B];
    float sacc[B][kNGrad];
    float ray[6][PX];
    float dc[6][PX];      // dL/dcolour (3), dL/dD0, dL/dD1, dL/dD4: constant along the walk
    int32_t nc[PX];
    float resA[3][B][PX];  // a (0: no hit), m1, dot(dL/dcolour, rgb)
    float resB[6][B][PX];  // T, D2, D3 before the hit; dL/d(log T, D2, D3) after it
    uint8_t hit_entry[PX][B];  // per slot: the batch entries it hits
    int32_t hit_pre[PX + 1];   // exclusive prefix of the per-slot hit counts
    int32_t warp_base[(PX + 31) / 32];
    int32_t smax[(PX + 31) / 32];
};

template <int PX, int NT, int B>
__device__ __forceinline__ void bwd_pair_item(
    int tile, int sub, const int32_t* __restrict__ ids, const int2* __restrict__ ranges,
    const float4* __restrict__ recs, const int4* __restrict__ indices, const float2* __restrict__ jitter,
    const rm_camera& cam, const float4* __restrict__ img, const float* __restrict__ dist,
    const int32_t* __restrict__ ncs, const float4* __restrict__ gimg, const float* __restrict__ gdist,
    float* __restrict__ gverts, float* __restrict__ gcv, BwdPairSmem<PX, B>& S, const Queue& lq) {
    constexpr unsigned kOwnMask = WarpShape<PX>::kMask;
    constexpr int kWarps = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool owner = tid < PX;
    const int tx = tile % cam.grid_width, ty = tile / cam.grid_width;
    int lx, ly;
    strip_pixel<PX>(cam, sub, tid, lx, ly);
    const int px = tx * cam.tile_width + lx, py = ty * cam.tile_height + ly;
    const bool inside = owner && px < cam.image_width && py < cam.image_height;
    const int64_t pix = (int64_t)py * cam.image_width + px;
    f3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f};
    float logT = 0.f, D2 = 0.f, D3 = 0.f;  // state along the reverse walk
    float dS_c[3] = {0.f, 0.f, 0.f}, dS_logT = 0.f, dS_D[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    int32_t nc = 0;
    if (inside) {
        const float2 j = __ldg(jitter + pix);
        make_ray(cam, px, py, j.x, j.y, o, d);
        logT = __ldg(img + pix).w;
        D2 = __ldg(dist + 5 * pix + 2);
        D3 = __ldg(dist + 5 * pix + 3);
        const float4 g = __ldg(gimg + pix);
        dS_c[0] = g.x; dS_c[1] = g.y; dS_c[2] = g.z; dS_logT = g.w;
#pragma unroll
        for (int k = 0; k < 5; ++k) dS_D[k] = gdist ? __ldg(gdist + 5 * pix + k) : 0.f;
        nc = __ldg(ncs + pix);
    }
    if (owner) {
        int32_t m = nc;
#pragma unroll
        for (int off = WarpShape<PX>::kTopOffset; off > 0; off >>= 1) m = max(m, __shfl_xor_sync(kOwnMask, m, off));
        if (lane == 0) S.smax[warp] = m;
    }
    __syncthreads();
    int32_t tile_max = 0;
#pragma unroll
    for (int w = 0; w < (PX + 31) / 32; ++w) tile_max = max(tile_max, S.smax[w]);
    const int2 rg = __ldg(ranges + tile);
    const int end = min(rg.y, rg.x + tile_max);
    for (int top = end; top > rg.x; top -= B) {
        const int lo = max(rg.x, top - B);
        const int n = top - lo;
        // pixels with list offsets below n_contributors in this batch
        const bool walking = inside && (lo - rg.x) < nc;
        __syncthreads();  // the previous batch's flush has read sid / srec / sacc
        for (int k = tid; k < n; k += NT) S.sid[k] = list_id(ids, lo + k, lq);
        for (int k = tid; k < n * kNGrad; k += NT) (&S.sacc[0][0])[k] = 0.f;
        int slot = 0;
        if (owner) {
            const unsigned bal = __ballot_sync(kOwnMask, walking);
            if (lane == 0) S.warp_base[warp] = __popc(bal);
            slot = __popc(bal & ((1u << lane) - 1u));
        }
        __syncthreads();
        for (int k = tid; k < n * kRecFloat4; k += NT) {
            const int j = k >> 3, c = k & 7;
            S.srec[j][c] = record_part(recs, S.sid[j], c);
        }
        int k_act = 0;
#pragma unroll
        for (int w = 0; w < (PX + 31) / 32; ++w) k_act += S.warp_base[w];
        if (walking) {
            for (int w = 0; w < warp; ++w) slot += S.warp_base[w];
            S.ray[0][slot] = o.x; S.ray[1][slot] = o.y; S.ray[2][slot] = o.z;
            S.ray[3][slot] = d.x; S.ray[4][slot] = d.y; S.ray[5][slot] = d.z;
            S.dc[0][slot] = dS_c[0]; S.dc[1][slot] = dS_c[1]; S.dc[2][slot] = dS_c[2];
            S.dc[3][slot] = dS_D[0]; S.dc[4][slot] = dS_D[1]; S.dc[5][slot] = dS_D[4];
            S.nc[slot] = nc;
        }
        __syncthreads();
        // A: hit test of every (entry, slot) pair
        for (int j = warp; j < n; j += kWarps) {
            const float4* q = S.srec[j];
            const float density = q[0].w;
            for (int sl = lane; sl < k_act; sl += 32) {
                float ra = 0.f, rm1 = 0.f, rdt = 0.f;
                if (lo + j - rg.x < S.nc[sl]) {
                    const f3 ro = {S.ray[0][sl], S.ray[1][sl], S.ray[2][sl]};
                    const f3 rd = {S.ray[3][sl], S.ray[4][sl], S.ray[5][sl]};
                    const Isect is = intersect<false>(q, ro, rd);
                    Segment s;
                    s.dt = fmaxf(is.exit - is.enter, 0.f);
                    s.a = density * s.dt;
                    if (is.geo && s.a > 0.f) {
                        integrate(q, ro, rd, is.enter, is.exit, s);
                        ra = s.a;
                        rm1 = density * (is.exit + is.enter) / 2.0f;
                        rdt = fmaf(S.dc[2][sl], s.rgb[2], fmaf(S.dc[1][sl], s.rgb[1], S.dc[0][sl] * s.rgb[0]));
                    }
                }
                S.resA[0][j][sl] = ra;
                S.resA[1][j][sl] = rm1;
                S.resA[2][j][sl] = rdt;
            }
        }
        __syncthreads();
        // B: each owner walks its chains back to front and lists its hits
        if (walking) {
            int cnt = 0;
            for (int j = n - 1; j >= 0; --j) {
                const float a = S.resA[0][j][slot];
                if (!(a > 0.f)) continue;
                S.hit_entry[slot][cnt++] = (uint8_t)j;
                const float density = S.srec[j][0].w;
                const float m1 = S.resA[1][j][slot];
                const float logT_old = logT + a;
                const float T = __expf(logT_old);
                D2 = D2 - density;
                D3 = D3 - m1;
                logT = logT_old;
                S.resB[0][j][slot] = T;
                S.resB[1][j][slot] = D2;
                S.resB[2][j][slot] = D3;
                S.resB[3][j][slot] = dS_logT;
                S.resB[4][j][slot] = dS_D[2];
                S.resB[5][j][slot] = dS_D[3];
                dS_logT = dS_logT + S.resA[2][j][slot] * T;
                dS_D[2] = dS_D[2] + dS_D[0] * 2.0f * m1;
                dS_D[3] = dS_D[3] + dS_D[1] * 2.0f * density;
            }
            S.hit_pre[slot + 1] = cnt;
        }
        __syncthreads();
        // exclusive prefix of the hit counts over the k_act slots
        if (warp == 0) {
            int carry = 0;
            for (int s0 = 0; s0 < k_act; s0 += 32) {
                const int v = (s0 + lane < k_act) ? S.hit_pre[s0 + lane + 1] : 0;
                int inc = v;
#pragma unroll
                for (int o2 = 1; o2 < 32; o2 <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, inc, o2);
                    if (lane >= o2) inc += y;
                }
                if (s0 + lane < k_act) S.hit_pre[s0 + lane + 1] = carry + inc;
                carry += __shfl_sync(0xffffffffu, inc, 31);
            }
            if (lane == 0) S.hit_pre[0] = 0;
        }
        __syncthreads();
        // C: adjoint of every hit, one hit per thread (the hits are packed, so
        // all lanes do useful work); consecutive hits belong to one slot and
        // hit different entries, so the per-entry shared accumulators see no
        // address conflicts inside a warp
        const int n_hits = S.hit_pre[k_act];
        for (int h = tid; h < n_hits; h += NT) {
            int lo_s = 0, hi_s = k_act - 1;
            while (lo_s < hi_s) {  // last slot with hit_pre[slot] <= h
                const int mid = (lo_s + hi_s + 1) >> 1;
                if (S.hit_pre[mid] <= h) lo_s = mid; else hi_s = mid - 1;
            }
            const int sl = lo_s;
            const int j = S.hit_entry[sl][h - S.hit_pre[sl]];
            const float4* q = S.srec[j];
            const f3 ro = {S.ray[0][sl], S.ray[1][sl], S.ray[2][sl]};
            const f3 rd = {S.ray[3][sl], S.ray[4][sl], S.ray[5][sl]};
            const Isect is = intersect<true>(q, ro, rd);
            Segment sg;
            sg.dt = fmaxf(is.exit - is.enter, 0.f);
            sg.a = q[0].w * sg.dt;
            integrate(q, ro, rd, is.enter, is.exit, sg);
            const float dsc[3] = {S.dc[0][sl], S.dc[1][sl], S.dc[2][sl]};
            const float dsd[5] = {S.dc[3][sl], S.dc[4][sl], S.resB[4][j][sl], S.resB[5][j][sl], S.dc[5][sl]};
            float gl[kNGrad];
            float nD2, nD3;
            hit_grads(q, ro, rd, is, sg, S.resB[0][j][sl], S.resB[1][j][sl], S.resB[2][j][sl], dsc, S.resB[3][j][sl],
                      dsd, gl, nD2, nD3);
#pragma unroll
            for (int k = 0; k < kNGrad; ++k)
                if (gl[k] != 0.f) atomicAdd(&S.sacc[j][k], gl[k]);
        }
        __syncthreads();
        flush_entries<NT, B>(n, S.srec, S.sid, S.sacc, indices, gverts, gcv);
    }
}

// Resident warps per SM of the backward.
constexpr int kBwdWarpsPerSm = 20;

template <int PX, class V>
__global__ void __launch_bounds__(PX < 32 ? 32 : PX, PX < 32 ? kBwdWarpsPerSm : kBwdWarpsPerSm * 32 / PX)
    blend_bwd_kernel(
    const int32_t* __restrict__ ids, const int2* __restrict__ ranges, const float4* __restrict__ recs,
    const int4* __restrict__ indices, const float2* __restrict__ jitter, const __grid_constant__ V views,
    const float4* __restrict__ img, const float* __restrict__ dist, const int32_t* __restrict__ ncs,
    const float4* __restrict__ gimg, const float* __restrict__ gdist, float* __restrict__ gverts,
    float* __restrict__ gcv, const Queue q) {
    __shared__ BwdSmem<PX / 32 + (PX < 32)> S;
    __shared__ HitMasks hm;  // read once per block: kept out of the registers
    if (threadIdx.x == 0) {
        hm = live_masks(q.hm, q.subs);
        if (__ldg(q.info) != 0) hm.ck = nullptr;  // tiles split off to the pair kernel: the others whole
    }
    __syncthreads();
    // every tile by its segments when the forward left checkpoints, else the
    // queue's tiles whole
    const bool segs = hm.ck != nullptr;
    const int64_t n_items = segs ? segment_items(q.info, q.G, hm.seg_shift) * q.subs : (int64_t)queue_items(q);
    for (;;) {
        if (threadIdx.x == 0) {
            const int item = (int)atomicAdd(q.ticket, 1u);
            SegItem it = {-1, 0, 0};
            if (item < n_items) {
                if (segs) it = segment_item(q, item, hm.seg_shift);
                else it = {queue_tile(q, item), 0, item % q.subs};
            }
            S.item = make_int4(it.tile, it.seg, it.sub, 0);
        }
        __syncthreads();
        const int4 it = S.item;
        __syncthreads();
        if (it.x < 0) return;
        const int v = views.find(it.x);
        const int tb = views.tile_base(v);
        const int64_t pb = views.pixel_base(v);
        bwd_item<PX>(it.x - tb, it.z, it.y, ids, ranges + tb, recs, indices, jitter + pb, views.camera(v), img + pb,
                     dist + 5 * pb, ncs + pb, gimg + pb, gdist ? gdist + 5 * pb : nullptr, gverts, gcv, S, hm, q.subs,
                     it.x, q);
    }
}

template <int B, class V>
__global__ void __launch_bounds__(64, 8) blend_bwd_dense_tma_kernel(
    const int32_t* __restrict__ ids, const int2* __restrict__ ranges, const float4* __restrict__ recs,
    const int4* __restrict__ indices, const float2* __restrict__ jitter, const __grid_constant__ V views,
    const float4* __restrict__ img, const float* __restrict__ dist, const int32_t* __restrict__ ncs,
    const float4* __restrict__ gimg, const float* __restrict__ gdist, float* __restrict__ gverts,
    float* __restrict__ gcv, const Queue q) {
    __shared__ BwdTmaSmem<B> S;
    __shared__ int s_item;
    if (threadIdx.x == 0) {
        mbar_init(&S.bar[0], 1);
        mbar_init(&S.bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    const int n_items = queue_items(q);
    const HitMasks hm = live_masks(q.hm, q.subs);
    TmaPipe pipe = {0u, 0u};
    for (;;) {
        const int item = next_item(q, &s_item);
        if (item >= n_items) return;
        const int t = queue_tile(q, item), v = views.find(t);
        const int tb = views.tile_base(v);
        const int64_t pb = views.pixel_base(v);
        bwd_dense_item_tma<B>(t - tb, item % q.subs, ids, ranges + tb, recs, indices, jitter + pb,
                              views.camera(v), img + pb, dist + 5 * pb, ncs + pb, gimg + pb,
                              gdist ? gdist + 5 * pb : nullptr, gverts, gcv, S, hm, q.subs, t, pipe, q);
    }
}

template <int PX, int NT, int B, class V>
__global__ void __launch_bounds__(NT, 512 / NT) blend_bwd_pair_kernel(
    const int32_t* __restrict__ ids, const int2* __restrict__ ranges, const float4* __restrict__ recs,
    const int4* __restrict__ indices, const float2* __restrict__ jitter, const __grid_constant__ V views,
    const float4* __restrict__ img, const float* __restrict__ dist, const int32_t* __restrict__ ncs,
    const float4* __restrict__ gimg, const float* __restrict__ gdist, float* __restrict__ gverts,
    float* __restrict__ gcv, const Queue q) {
    extern __shared__ __align__(16) unsigned char bwd_smem_raw[];
    BwdPairSmem<PX, B>& S = *reinterpret_cast<BwdPairSmem<PX, B>*>(bwd_smem_raw);
    __shared__ int s_item;
    const int n_items = queue_items(q);
    for (;;) {
        const int item = next_item(q, &s_item);
        if (item >= n_items) return;
        const int t = queue_tile(q, item), v = views.find(t);
        const int tb = views.tile_base(v);
        const int64_t pb = views.pixel_base(v);
        bwd_pair_item<PX, NT, B>(t - tb, item % q.subs, ids, ranges + tb, recs, indices, jitter + pb,
                                 views.camera(v), img + pb, dist + 5 * pb, ncs + pb, gimg + pb,
                                 gdist ? gdist + 5 * pb : nullptr, gverts, gcv, S, q);
    }
}

// ------------------------------------------------------ per-tet statistics --
// calc_tet_err / kern_calc_tet_err (alphablend_shader_interp.slang:433-599):
// the forward walk from each pixel centre, accumulating per hit into
// tet_err[g, c] (float) the weight T = exp(log T) * a and its products with
// the pixel's error, squared error and SSIM error, the entry / exit points
// and the midpoint of the segment, and into tet_count[g] the hit count and
// the maximum of int(65535 * T).  As in the reference the walk starts from
// log T = 1 (its kern_calc_tet_err initialises the state alpha with 1) and
// stops once log T < -5.5.  Sums are formed per list entry across a work
// item (warp reduce-scatter, shared atomics) before one global atomic per
// (item, entry, column), instead of 16 atomics per (pixel, hit).
constexpr int kErrVals = 14;
__constant__ int kErrCol[kErrVals] = {0, 1, 2, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15};

template <int B>
struct ErrSmem {
    float4 srec[B][kRecFloat4];
    int32_t sid[B];
    float sacc[B][kErrVals];
    int32_t scount[B];
    int32_t smax[B];
};

template <int NT, int B>
__device__ __forceinline__ void err_item(int tile, int sub, const int32_t* __restrict__ ids,
                                         const int2* __restrict__ ranges, const float4* __restrict__ recs,
                                         const rm_camera& cam, const float* __restrict__ pixel_err,
                                         const float* __restrict__ ssim_err, float* __restrict__ tet_err,
                                         int32_t* __restrict__ tet_count, ErrSmem<B>& S, const Queue& lq) {
    constexpr unsigned kMask = WarpShape<NT>::kMask;
    const int tx = tile % cam.grid_width, ty = tile / cam.grid_width;
    int lx, ly;
    strip_pixel<NT>(cam, sub, (int)threadIdx.x, lx, ly);
    const int px = tx * cam.tile_width + lx, py = ty * cam.tile_height + ly;
    const bool inside = px < cam.image_width && py < cam.image_height;
    const int64_t pix = (int64_t)py * cam.image_width + px;
    const int lane = threadIdx.x & 31;
    f3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f};
    float err = 0.f, serr = 0.f;
    if (inside) {
        make_ray(cam, px, py, 0.5f, 0.5f, o, d);  // pixel centre
        err = __ldg(pixel_err + pix);
        serr = __ldg(ssim_err + pix);
    }
    float logT = 1.0f;
    bool active = inside;
    const int2 rg = __ldg(ranges + tile);
    for (int base = rg.x; base < rg.y && __syncthreads_or(active); base += B) {
        const int n = min(B, rg.y - base);
        for (int k = threadIdx.x; k < n; k += NT) {
            S.sid[k] = list_id(ids, base + k, lq);
            S.scount[k] = 0;
            S.smax[k] = 0;
        }
        for (int k = threadIdx.x; k < n * kErrVals; k += NT) (&S.sacc[0][0])[k] = 0.f;
        __syncthreads();
        for (int k = threadIdx.x; k < n * kRecFloat4; k += NT) {
            const int j = k >> 3, c = k & 7;
            S.srec[j][c] = record_part(recs, S.sid[j], c);
        }
        __syncthreads();
        for (int j = 0; j < n; ++j) {
            if (!__any_sync(kMask, active)) break;
            const float4* q = S.srec[j];
            const Isect is = intersect<false>(q, o, d);
            const float dt = fmaxf(is.exit - is.enter, 0.f);
            const float a = q[0].w * dt;
            const bool hit = active && is.geo && a > 0.f;
            float v[kErrVals];
#pragma unroll
            for (int k = 0; k < kErrVals; ++k) v[k] = 0.f;
            int tint = 0;
            if (hit) {
                const float T = expf(logT) * a;
                const float mid = 0.5f * (is.enter + is.exit);
                v[0] = T;
                v[1] = T * err;
                v[2] = T * err * err;
                v[3] = T * serr;
                v[4] = T * fmaf(is.enter, d.x, o.x);
                v[5] = T * fmaf(is.enter, d.y, o.y);
                v[6] = T * fmaf(is.enter, d.z, o.z);
                v[7] = T * fmaf(is.exit, d.x, o.x);
                v[8] = T * fmaf(is.exit, d.y, o.y);
                v[9] = T * fmaf(is.exit, d.z, o.z);
                v[10] = T;
                v[11] = T * fmaf(mid, d.x, o.x);
                v[12] = T * fmaf(mid, d.y, o.y);
                v[13] = T * fmaf(mid, d.z, o.z);
                tint = __float2int_rz(65535.0f * T);
                logT = logT - a;
                if (logT < kTermLogT) active = false;
            }
            if (__any_sync(kMask, hit)) {
                using RS = ReduceScatter<kErrVals, WarpShape<NT>::kTopOffset>;
                int slot = 0;
                RS::template run<kMask>(v, lane, slot);
#pragma unroll
                for (int r = 0; r < RS::R; ++r)
                    if (slot + r < kErrVals && v[r] != 0.f) atomicAdd(&S.sacc[j][slot + r], v[r]);
                const unsigned bal = __ballot_sync(kMask, hit);
#pragma unroll
                for (int off = WarpShape<NT>::kTopOffset; off > 0; off >>= 1)
                    tint = max(tint, __shfl_xor_sync(kMask, tint, off));
                if (lane == 0) {
                    atomicAdd(&S.scount[j], __popc(bal));
                    atomicMax(&S.smax[j], tint);
                }
            }
        }
        __syncthreads();
        for (int jj = threadIdx.x; jj < n; jj += NT) {
            const int cnt = S.scount[jj];
            const int64_t g = S.sid[jj];
            if (cnt == 0 || g < 0) continue;
            float* te = tet_err + 16 * g;
#pragma unroll
            for (int k = 0; k < kErrVals; ++k)
                if (S.sacc[jj][k] != 0.f) atomicAdd(te + kErrCol[k], S.sacc[jj][k]);
            atomicAdd(tet_count + 2 * g, cnt);
            atomicMax(tet_count + 2 * g + 1, S.smax[jj]);
        }
    }
}

template <int NT, int B>
__global__ void __launch_bounds__(NT, (NT >= 64 ? 1024 / NT : 32)) err_kernel(
    const int32_t* __restrict__ ids, const int2* __restrict__ ranges, const float4* __restrict__ recs,
    const rm_camera cam, const float* __restrict__ pixel_err, const float* __restrict__ ssim_err,
    float* __restrict__ tet_err, int32_t* __restrict__ tet_count, const Queue q) {
    __shared__ ErrSmem<B> S;
    __shared__ int s_item;
    const int n_items = queue_items(q);
    for (;;) {
        const int item = next_item(q, &s_item);
        if (item >= n_items) return;
        err_item<NT, B>(queue_tile(q, item), item % q.subs, ids, ranges, recs, cam, pixel_err, ssim_err, tet_err,
                        tet_count, S, q);
    }
}

// The statistics from a forward walk's leavings.  The walk itself (which
// pixel hits which entry, until its log T runs out) is the forward kernel with
// log T started at 1 and nothing but a formed (LOGT); it leaves the hit masks,
// n_contributors and log T at every checkpoint.  Each stretch of a list is
// then an item of its own, as in the backward: one warp per 32 pixels goes
// through the entries that its pixels hit, front to back, and the sums of both
// warps of a strip are added to global memory once per entry.  (One kernel
// walking whole lists, as err_kernel does, is bound by its longest list: 4.3
// ms for 653k tets at 1297x840, now 1.66 ms in both kernels.)
constexpr int kErrStride = 20;  // floats per row of 13 values: conflict-free 16-byte stores

struct ErrSegSmem {
    float4 srec[32][kRecFloat4 + 1];
    float4 red[2][32 * kErrStride / 4];
    float4 sums[2][32][4];
    int32_t most[2][32];
    uint8_t count[2][32];
    uint32_t any[2][2];
    int4 item;
};

__device__ __forceinline__ void err_seg_item(int tile, int sub, int seg, const int32_t* __restrict__ ids,
                                             const int2* __restrict__ ranges, const float4* __restrict__ recs,
                                             const rm_camera& cam, const int32_t* __restrict__ ncs,
                                             const float* __restrict__ pixel_err, const float* __restrict__ ssim_err,
                                             float* __restrict__ tet_err, int32_t* __restrict__ tet_count,
                                             ErrSegSmem& S, const HitMasks& hm, int subs, const Queue& lq) {
    constexpr unsigned kAll = 0xffffffffu;
    const int2 rg = __ldg(ranges + tile);
    const int len = rg.y - rg.x;
    int s0 = 0, s1 = len;
    if (hm.ck && len > (1 << hm.seg_shift)) {
        const int shift = hm.seg_shift;
        if (ck_id(rg.x, (len - 1) >> shift, shift) < hm.ck_cap) {
            s0 = seg << shift;
            s1 = min(len, s0 + (1 << shift));
        } else if (seg) {
            return;
        }
    } else if (seg) {
        return;
    }
    if (s0 >= s1) return;
    const int p = threadIdx.x, lane = p & 31, warp = p >> 5;
    const int tx = tile % cam.grid_width, ty = tile / cam.grid_width;
    int lx, ly;
    strip_pixel<64>(cam, sub, p, lx, ly);
    const int px = tx * cam.tile_width + lx, py = ty * cam.tile_height + ly;
    const bool inside = px < cam.image_width && py < cam.image_height;
    const int64_t pix = (int64_t)py * cam.image_width + px;
    int32_t nc = inside ? min(__ldcg(ncs + pix), s1) : 0;
    if (nc <= s0) nc = 0;
    const int mine_last = (int)__reduce_max_sync(kAll, (unsigned)nc);
    if (lane == 0) S.any[0][warp] = (uint32_t)mine_last;
    __syncthreads();
    const int last = max((int)S.any[0][0], (int)S.any[0][1]);
    __syncthreads();
    if (last == 0) return;
    f3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 1.f};
    float err = 0.f, serr = 0.f, logT = 1.0f;
    if (nc > 0) {
        make_ray(cam, px, py, 0.5f, 0.5f, o, d);  // pixel centre
        err = __ldg(pixel_err + pix);
        serr = __ldg(ssim_err + pix);
        if (s0 > 0) logT = __ldcg(ck_at(hm, ck_id(rg.x, seg, hm.seg_shift), sub, subs, p));
    }
    float4* const row4 = S.red[warp] + lane * (kErrStride / 4);
    auto hit_word = [&](int k) {
        const int64_t i = mask_word(tile, rg.x, k, sub, subs, p);
        return bits_below(i < hm.cap ? __ldcg(hm.words + i) : 0xffffffffu, nc - 32 * k);
    };
    int k = s0 >> 5;
    uint32_t w = hit_word(k), mine = __reduce_or_sync(kAll, w);
    if (lane == 0) S.any[k & 1][warp] = mine;
    __syncthreads();
    for (; 32 * k < last; ++k) {
        const uint32_t cur = w, own = mine;
        const uint32_t other = S.any[k & 1][1 - warp], any = own | other;
        w = 32 * (k + 1) < last ? hit_word(k + 1) : 0u;
        mine = __reduce_or_sync(kAll, w);
        if (lane == 0) S.any[(k + 1) & 1][warp] = mine;
        if (!any) {
            __syncthreads();  // S.any of the next block
            continue;
        }
        int32_t g = -1;
        if ((any >> lane) & 1u) g = list_id(ids, rg.x + 32 * k + lane, lq);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = 4 * (warp + 2 * i) + (lane >> 3);
            const int32_t ge = __shfl_sync(kAll, g, e);
            if (ge >= 0)
                async_copy16(&S.srec[e][lane & 7], recs + (int64_t)kRecFloat4 * ge + (lane & 7));
            else if ((any >> e) & 1u)
                S.srec[e][lane & 7] = make_float4(0.f, 0.f, 0.f, 0.f);  // names no tet: nothing hits it
        }
        async_wait();
        __syncthreads();
        for (uint32_t left = own; left; left &= left - 1u) {
            const int j = __ffs(left) - 1;
            const float4* q = S.srec[j];
            const Isect is = intersect<false>(q, o, d);
            const float a = q[0].w * fmaxf(is.exit - is.enter, 0.f);
            const bool hit = ((cur >> j) & 1u) && is.geo && a > 0.f;
            const float T = hit ? expf(logT) * a : 0.f;
            logT = hit ? logT - a : logT;
            // a lane without a hit adds zeros (its distances may be infinite)
            const float enter = hit ? is.enter : 0.f, exit = hit ? is.exit : 0.f, mid = 0.5f * (enter + exit);
            const float Te = T * err;
            row4[0] = make_float4(T, Te, Te * err, T * serr);
            row4[1] = make_float4(T * fmaf(enter, d.x, o.x), T * fmaf(enter, d.y, o.y), T * fmaf(enter, d.z, o.z),
                                  T * fmaf(exit, d.x, o.x));
            row4[2] = make_float4(T * fmaf(exit, d.y, o.y), T * fmaf(exit, d.z, o.z), T * fmaf(mid, d.x, o.x),
                                  T * fmaf(mid, d.y, o.y));
            row4[3] = make_float4(T * fmaf(mid, d.z, o.z), 0.f, 0.f, 0.f);
            const unsigned bal = __ballot_sync(kAll, hit);
            const int most = __reduce_max_sync(kAll, __float2int_rz(65535.0f * T));
            __syncwarp();
            // four columns of four rows per lane, then over the eight groups
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            const int quad = lane & 3, row0 = lane & 28;
#pragma unroll
            for (int r = 0; r < 4; ++r) add4(s, S.red[warp][(row0 + r) * (kErrStride / 4) + quad]);
            __syncwarp();
#pragma unroll
            for (int off = 4; off <= 16; off <<= 1) add4(s, shfl_xor4(s, off));
            if (lane < 4) S.sums[warp][j][lane] = s;
            if (lane == 0) {
                S.most[warp][j] = most;
                S.count[warp][j] = (uint8_t)__popc(bal);
            }
        }
        __syncthreads();
        if (warp == (k & 1) && g >= 0) {
            float v[16];
            float4* v4 = reinterpret_cast<float4*>(v);
            int count = 0, most = 0;
#pragma unroll
            for (int c = 0; c < 4; ++c) v4[c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (((i == warp ? own : other) >> lane) & 1u) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) add4(v4[c], S.sums[i][lane][c]);
                    count += S.count[i][lane];
                    most = max(most, S.most[i][lane]);
                }
            }
            if (count > 0) {
                float* te = tet_err + 16 * (int64_t)g;
                const int col[13] = {0, 1, 2, 5, 6, 7, 8, 9, 10, 11, 13, 14, 15};
#pragma unroll
                for (int c = 0; c < 13; ++c)
                    if (v[c] != 0.f) atomicAdd(te + col[c], v[c]);
                if (v[0] != 0.f) atomicAdd(te + 12, v[0]);
                atomicAdd(tet_count + 2 * (int64_t)g, count);
                atomicMax(tet_count + 2 * (int64_t)g + 1, most);
            }
        }
        __syncthreads();  // the next block overwrites the records and the sums
    }
}

__global__ void __launch_bounds__(64, 12) err_seg_kernel(const int32_t* __restrict__ ids,
                                                         const int2* __restrict__ ranges,
                                                         const float4* __restrict__ recs, const rm_camera cam,
                                                         const int32_t* __restrict__ ncs,
                                                         const float* __restrict__ pixel_err,
                                                         const float* __restrict__ ssim_err,
                                                         float* __restrict__ tet_err, int32_t* __restrict__ tet_count,
                                                         const Queue q) {
    __shared__ ErrSegSmem S;
    __shared__ HitMasks hm;
    if (threadIdx.x == 0) hm = live_masks(q.hm, q.subs, kMaskStats);
    __syncthreads();
    const int64_t n_items = segment_items(q.info, q.G, hm.seg_shift) * q.subs;
    for (;;) {
        if (threadIdx.x == 0) {
            const int item = (int)atomicAdd(q.ticket, 1u);
            SegItem it = {-1, 0, 0};
            if (item < n_items) it = segment_item(q, item, hm.seg_shift);
            S.item = make_int4(it.tile, it.seg, it.sub, 0);
        }
        __syncthreads();
        const int4 it = S.item;
        __syncthreads();
        if (it.x < 0) return;
        err_seg_item(it.x, it.z, it.y, ids, ranges, recs, cam, ncs, pixel_err, ssim_err, tet_err, tet_count, S, hm,
                     q.subs, q);
    }
}

struct BlendWs {
    float4* recs;
    int32_t* order;
    int32_t* info;
    uint32_t* tickets;
    uint32_t* status;       // the pass's status word when the caller passes none

    uint32_t* mask_header;  // nullptr: the workspace has no room for hit masks
    uint32_t* mask_words;
    int64_t mask_cap;       // words for the masks and, after them, the checkpoints
};

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// Byte offset of the status word inside the 256-byte header that follows the
// records and the tile order (info at 0, queue tickets at 64).
constexpr size_t kBlendStatusOff = 128;

size_t blend_ws_bytes(int64_t n_tets, int64_t n_tiles) {
    const size_t rec = align256((size_t)(n_tets > 0 ? n_tets : 1) * kRecFloat4 * sizeof(float4));
    const size_t ord = align256((size_t)(n_tiles > 0 ? n_tiles : 1) * sizeof(int32_t));
    return rec + ord + 256;
}

// Hit masks, when the caller's workspace is larger than blend_ws_bytes: a
// 256-byte header, the mask words (mask_word), the checkpoints (ck_at).
BlendWs blend_ws(void* base, int64_t n_tets, int64_t n_tiles, size_t workspace_bytes) {
    char* p = (char*)base;
    const size_t rec = align256((size_t)(n_tets > 0 ? n_tets : 1) * kRecFloat4 * sizeof(float4));
    const size_t ord = align256((size_t)(n_tiles > 0 ? n_tiles : 1) * sizeof(int32_t));
    BlendWs w = {(float4*)p, (int32_t*)(p + rec), (int32_t*)(p + rec + ord), (uint32_t*)(p + rec + ord + 64),
                 (uint32_t*)(p + rec + ord + kBlendStatusOff), nullptr, nullptr, 0};
    const size_t end = rec + ord + 256;
    if (workspace_bytes >= end + 256 + 64 * sizeof(uint32_t)) {
        w.mask_header = (uint32_t*)(p + end);
        w.mask_words = (uint32_t*)(p + end + 256);
        w.mask_cap = (int64_t)((workspace_bytes - end - 256) / sizeof(uint32_t));
    }
    return w;
}

// Persistent grid: as many CTAs as fit on the device at once (cached per
// kernel instantiation and device).
// Resident CTAs of a persistent kernel on the current device (SMs x CTAs per
// SM), cached per (kernel, device, block shape): kernels of one signature
// differ in their resource use, so the kernel's address is part of the key.
struct GridKey {
    const void* kernel;
    int dev, threads, smem, blocks;
};
std::mutex g_grid_mu;
GridKey g_grid_cache[64];
int g_grid_used = 0;

template <typename K>
int persistent_grid(K kernel, int threads, int smem, int n_items) {
    int dev = 0;
    cudaGetDevice(&dev);
    const void* kp = (const void*)kernel;
    int blocks = -1;
    {
        std::lock_guard<std::mutex> lock(g_grid_mu);
        for (int i = 0; i < g_grid_used; ++i) {
            const GridKey& k = g_grid_cache[i];
            if (k.kernel == kp && k.dev == dev && k.threads == threads && k.smem == smem) blocks = k.blocks;
        }
    }
    if (blocks < 0) {
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
        blocks = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
        std::lock_guard<std::mutex> lock(g_grid_mu);
        if (g_grid_used < 64) g_grid_cache[g_grid_used++] = {kp, dev, threads, smem, blocks};
    }
    return n_items < blocks ? n_items : blocks;
}

int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

// When a pass splits its tiles between the two kernels, the pair kernel runs
// on a side stream forked from and joined back into the caller's stream with
// events (capturable in a CUDA graph).  Each (device, caller stream) gets its
// own side stream, so callers on different streams stay independent.
struct SideStream {
    int dev = -1;
    cudaStream_t caller = nullptr;
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
constexpr int kSideStreams = 64;
std::mutex g_side_mu;
SideStream g_side[kSideStreams];

// Caller holds g_side_mu.
int side_stream(cudaStream_t caller, SideStream** out) {
    int dev = 0;
    cudaGetDevice(&dev);
    SideStream* free_slot = nullptr;
    for (SideStream& e : g_side) {
        if (e.stream && e.dev == dev && e.caller == caller) {
            *out = &e;
            return RM_OK;
        }
        if (!e.stream && !free_slot) free_slot = &e;
    }
    if (!free_slot) {  // table full: share the first side stream of this device
        for (SideStream& e : g_side)
            if (e.dev == dev) {
                *out = &e;
                return RM_OK;
            }
        return rm_host::fail(RM_ECUDA, "rm_blend: no side stream slot left");
    }
    SideStream& e = *free_slot;
    if (cudaStreamCreateWithFlags(&e.stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&e.fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&e.join, cudaEventDisableTiming) != cudaSuccess)
        return rm_host::fail(RM_ECUDA, "rm_blend: side stream: %s", cudaGetErrorString(cudaGetLastError()));
    e.dev = dev;
    e.caller = caller;
    *out = &e;
    return RM_OK;
}

int launch_order(const int32_t* ranges, int G, const BlendWs& w, int heavy_shift, cudaStream_t s,
                 uint32_t* mask_header = nullptr, MaskRoom room = MaskRoom{}, const uint32_t* seg_header = nullptr,
                 int fwd_slots = 0) {
    order_kernel<<<kOrderCtas, 1024, 0, s>>>((const int2*)ranges, G, w.order, w.info, w.tickets, heavy_shift, mask_header, room,
                                    seg_header, fwd_slots);
    return rm_host::check_launch("rm_blend order");
}

int fork_side(cudaStream_t s, SideStream* side) {
    if (cudaEventRecord(side->fork, s) != cudaSuccess || cudaStreamWaitEvent(side->stream, side->fork, 0) != cudaSuccess)
        return rm_host::fail(RM_ECUDA, "rm_blend: fork: %s", cudaGetErrorString(cudaGetLastError()));
    return RM_OK;
}

int join_side(cudaStream_t s, SideStream* side) {
    if (cudaEventRecord(side->join, side->stream) != cudaSuccess || cudaStreamWaitEvent(s, side->join, 0) != cudaSuccess)
        return rm_host::fail(RM_ECUDA, "rm_blend: join: %s", cudaGetErrorString(cudaGetLastError()));
    return RM_OK;
}

// Launch tunables carried in the flags word (include/rm_capi.h).
struct Tuning {
    int heavy_shift;       // heavy tiles: list-length bucket >= bucket(mean) + heavy_shift; 1: all tiles, 0: none
    int pair_ctas_per_sm;  // resident CTAs of the pair kernel per SM
    bool hit_masks;        // RM_BLEND_HIT_MASKS
    bool tma;              // RM_BLEND_STAGE_TMA
    uint32_t* status;      // where a staging wait that gives up is reported
    int64_t n_recs;        // records the list ids may name
};

Tuning tuning_from_flags(int flags, int def_shift, int def_ctas) {
    Tuning t;
    t.tma = (flags & RM_BLEND_STAGE_TMA) != 0;
    t.status = nullptr;
    t.n_recs = 0;
    const int hs = (flags >> RM_BLEND_HEAVY_SHIFT) & 0xf;
    const int pc = (flags >> RM_BLEND_PAIR_CTAS_SHIFT) & 0xf;
    t.heavy_shift = hs ? hs : def_shift;
    t.pair_ctas_per_sm = pc ? pc : def_ctas;
    t.hit_masks = (flags & RM_BLEND_HIT_MASKS) != 0;
    return t;
}

// Shape of one blend launch: G global tiles of tile_px pixels each.
struct Shape {
    int G;
    int tile_px;
};

// Forward pass: order kernel, then one persistent kernel for the heavy tiles
// (pair items) and the others (warp items).
template <int PX, int NT, int B, Walk WALK, class V>
int launch_fwd(const int32_t* ids, const int32_t* ranges, const BlendWs& w, const float* jitter, const V& views,
               const Shape& sh, float* img, float* dist, int32_t* nc, const Tuning& tn, cudaStream_t s) {
    const int G = sh.G;
    // hit masks need 64-pixel items; the header records whether this forward
    // wrote them, so a backward never reads stale masks
    const bool masks = WALK != kImage && w.mask_header;
    const int subs = sh.tile_px / PX;
    const int cap = tn.pair_ctas_per_sm * sm_count();
    const MaskRoom room = {!masks ? 0u : WALK == kLogT ? kMaskStats : kMaskValid, subs, w.mask_cap};
    int rc = launch_order(ranges, G, w, PX == 64 ? tn.heavy_shift : tn.heavy_shift == 0 ? 1 : tn.heavy_shift, s,
                          w.mask_header, room, nullptr, PX == 64 ? (cap > subs ? cap / subs : 1) : 0);
    if (rc) return rc;
    const HitMasks hm = {masks ? w.mask_words : nullptr, w.mask_cap, w.mask_header, nullptr, 0, kNoSegments};
    const Queue q = {w.order, w.info, w.tickets + 0, G, subs, true, hm, tn.status, rm_host::wait_limit(), tn.n_recs};
    auto kernel = blend_fwd_kernel<PX, NT, B, V, WALK>;
    constexpr int kPairSmem = (int)sizeof(FwdPairSmem<PX, B>),
                  kWarpSmem = NT / 32 * (int)sizeof(FwdWarpSmem<(V::kViews > 1)>);
    constexpr int smem = kPairSmem > kWarpSmem ? kPairSmem : kWarpSmem;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const int64_t items = (int64_t)G * subs * (PX == 64 ? 4 : 1);
    const int grid = items < cap ? (int)items : cap;
    kernel<<<grid, NT, smem, s>>>(ids, (const int2*)ranges, w.recs, (const float2*)jitter, views, (float4*)img, dist,
                                  nc, q);
    return rm_host::check_launch("rm_blend_fwd");
}

template <int PX, int B_DENSE, int PX_PAIR, int NT_PAIR, int B_PAIR, class V>
int launch_bwd(const int32_t* ids, const int32_t* ranges, const BlendWs& w, const int32_t* indices,
               const float* jitter, const V& views, const Shape& sh, const float* img, const float* dist,
               const int32_t* nc, const float* gimg, const float* gdist, float* gverts, float* gcv,
               const Tuning& tn, cudaStream_t s) {
    const int G = sh.G;
    const int subs = sh.tile_px / PX;
    const int subs_pair = sh.tile_px / PX_PAIR;
    const bool masks = tn.hit_masks && PX == 64 && w.mask_header;
    int rc = launch_order(ranges, G, w, tn.heavy_shift, s, nullptr, MaskRoom{}, masks ? w.mask_header : nullptr);
    if (rc) return rc;
    const HitMasks hm = {masks ? w.mask_words : nullptr, w.mask_cap, w.mask_header, nullptr, 0, kNoSegments};
    const Queue qd = {w.order, w.info, w.tickets + 2, G, subs, false, hm, tn.status, rm_host::wait_limit(),
                      tn.n_recs};
    const Queue qp = {w.order, w.info, w.tickets + 3, G, subs_pair, true, HitMasks{},
                      tn.status, rm_host::wait_limit(), tn.n_recs};
    auto pair_kernel = blend_bwd_pair_kernel<PX_PAIR, NT_PAIR, B_PAIR, V>;
    const int smem = (int)sizeof(BwdPairSmem<PX_PAIR, B_PAIR>);
    cudaFuncSetAttribute(pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const int pair_cap = tn.pair_ctas_per_sm * sm_count();
    const int pair_grid = G * subs_pair < pair_cap ? G * subs_pair : pair_cap;
    const bool tma = PX == 64 && tn.tma;  // records staged by bulk copies, two batches in flight
    auto launch_dense = [&]() {
        if (tma) {
            auto tma_kernel = blend_bwd_dense_tma_kernel<B_DENSE, V>;
            const int grid = persistent_grid(tma_kernel, 64, 0, G * subs);
            tma_kernel<<<grid, 64, 0, s>>>(ids, (const int2*)ranges, w.recs, (const int4*)indices,
                                           (const float2*)jitter, views, (const float4*)img, dist, nc,
                                           (const float4*)gimg, gdist, gverts, gcv, qd);
            return rm_host::check_launch("rm_blend_bwd (dense, bulk-copy staging)");
        }
        auto kernel = blend_bwd_kernel<PX, V>;
        constexpr int threads = PX < 32 ? 32 : PX;
        // segments make more items than tiles: always the resident grid
        const int grid = persistent_grid(kernel, threads, 0, masks ? 1 << 30 : G * subs);
        kernel<<<grid, threads, 0, s>>>(ids, (const int2*)ranges, w.recs, (const int4*)indices, (const float2*)jitter,
                                        views, (const float4*)img, dist, nc, (const float4*)gimg, gdist, gverts, gcv,
                                        qd);
        return rm_host::check_launch("rm_blend_bwd");
    };
    if (tn.heavy_shift == 0) return launch_dense();
    if (tn.heavy_shift == 1) {
        pair_kernel<<<pair_grid, NT_PAIR, smem, s>>>(ids, (const int2*)ranges, w.recs, (const int4*)indices,
                                                     (const float2*)jitter, views, (const float4*)img, dist, nc,
                                                     (const float4*)gimg, gdist, gverts, gcv, qp);
        return rm_host::check_launch("rm_blend_bwd (pair)");
    }
    std::lock_guard<std::mutex> lock(g_side_mu);
    SideStream* side = nullptr;
    if ((rc = side_stream(s, &side)) || (rc = fork_side(s, side))) return rc;
    pair_kernel<<<pair_grid, NT_PAIR, smem, side->stream>>>(ids, (const int2*)ranges, w.recs, (const int4*)indices,
                                                            (const float2*)jitter, views, (const float4*)img, dist,
                                                            nc, (const float4*)gimg, gdist, gverts, gcv, qp);
    if ((rc = rm_host::check_launch("rm_blend_bwd (pair)"))) return rc;
    if ((rc = launch_dense())) return rc;
    return join_side(s, side);
}

// Strip of pixels handled by one CTA: flags may request 2^k pixels
// (RM_BLEND_STRIP_SHIFT); default 64.  Must divide the tile and be a multiple
// of the tile width.
int strip_pixels(const rm_camera* cam, int flags) {
    const int tile_px = cam->tile_width * cam->tile_height;
    const int req = (flags >> RM_BLEND_STRIP_SHIFT) & 0xff;
    int strip = req ? (1 << req) : 64;
    if (tile_px < strip) strip = tile_px;
    return strip;
}

// Tets per shared-memory batch: flags may request 2^k (RM_BLEND_BATCH_SHIFT).
int batch_size(int flags, int def) {
    const int req = (flags >> RM_BLEND_BATCH_SHIFT) & 0xf;
    return req ? (1 << req) : def;
}

int pack(const int32_t* indices, const float* vertices, int64_t n_verts, const float* cv, int64_t n_tets,
         const int32_t* tiles, float4* recs, cudaStream_t s) {
    const int threads = 256;
    const int64_t blocks = (n_tets + threads - 1) / threads;
    pack_kernel<<<(unsigned)blocks, threads, 0, s>>>((const int4*)indices, vertices, n_verts, cv, n_tets, tiles, recs);
    return rm_host::check_launch("rm_blend pack");
}

// Checks shared by all blend entry points; cam0 is the (first) camera, G the
// total tile count of the launch.
int check_blend_args(const char* who, const int32_t* indices, const float* vertices, const float* cv, int64_t n_tets,
                     const float* jitter, const rm_camera* cam0, int64_t G, void* workspace, size_t workspace_bytes,
                     int flags) {
    int rc = rm_host::check_cam(cam0);
    if (rc) return rc;
    if (n_tets < 0) return rm_host::fail(RM_EINVAL, "%s: negative size", who);
    if (!indices || !vertices || !cv || !jitter || !workspace)
        return rm_host::fail(RM_EINVAL, "%s: NULL pointer", who);
    if ((uintptr_t)indices & 15) return rm_host::fail(RM_EINVAL, "%s: indices must be 16-byte aligned", who);
    if ((uintptr_t)workspace & 15) return rm_host::fail(RM_EINVAL, "%s: workspace must be 16-byte aligned", who);
    if (workspace_bytes < blend_ws_bytes(n_tets, G))
        return rm_host::fail(RM_EINVAL, "%s: workspace %zu < %zu bytes", who, workspace_bytes,
                             blend_ws_bytes(n_tets, G));
    const int nt = cam0->tile_width * cam0->tile_height;
    if (nt != 16 && nt != 64 && nt != 256 && nt != 1024)
        return rm_host::fail(RM_EINVAL, "%s: tile of %d pixels unsupported (16, 64, 256 or 1024)", who, nt);
    const int strip = strip_pixels(cam0, flags);
    if ((strip != 16 && strip != 64) || nt % strip)
        return rm_host::fail(RM_EINVAL, "%s: strip of %d pixels does not fit a %dx%d tile", who, strip,
                             cam0->tile_width, cam0->tile_height);
    return RM_OK;
}

// The pass's status word: the caller's, else the workspace's own (cleared here).
int pass_status(const char* who, BlendWs& w, uint32_t* status_dev, cudaStream_t s, uint32_t** out) {
    if (status_dev) {
        *out = status_dev;
        return RM_OK;
    }
    cudaError_t e = cudaMemsetAsync(w.status, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return rm_host::fail(RM_ECUDA, "%s: %s", who, cudaGetErrorString(e));
    *out = w.status;
    return RM_OK;
}

template <class V>
int blend_fwd_any(const char* who, const int32_t* sorted_ids, const int32_t* ranges, const int32_t* indices,
                  const float* vertices, const float* cell_values, int64_t n_tets, int64_t n_verts,
                  const int32_t* tiles_touched,
                  const float* ray_jitter, const rm_camera* cam0, const V& views, const Shape& sh, float* out_img,
                  float* out_distortion, int32_t* n_contrib, const void* records, void* workspace,
                  size_t workspace_bytes, int flags, uint32_t* status_dev, void* stream) {
    int rc = check_blend_args(who, indices, vertices, cell_values, records ? 0 : n_tets, ray_jitter, cam0, sh.G,
                              workspace, workspace_bytes, flags);
    if (rc) return rc;
    if (!ranges || !out_img || !out_distortion || !n_contrib) return rm_host::fail(RM_EINVAL, "%s: NULL pointer", who);
    if (((uintptr_t)out_img & 15) || ((uintptr_t)ranges & 7) || ((uintptr_t)ray_jitter & 7))
        return rm_host::fail(RM_EINVAL, "%s: misaligned image / ranges / jitter", who);
    cudaStream_t s = (cudaStream_t)stream;
    BlendWs w = blend_ws(workspace, records ? 0 : n_tets, sh.G, workspace_bytes);
    if (records) {
        if ((uintptr_t)records & 15) return rm_host::fail(RM_EINVAL, "%s: records must be 16-byte aligned", who);
        w.recs = (float4*)records;  // packed by rm_blend_pack_records
    } else if (!(flags & RM_BLEND_REUSE_RECORDS) && n_tets > 0) {
        rc = pack(indices, vertices, n_verts, cell_values, n_tets, tiles_touched, w.recs, s);
        if (rc) return rc;
    }
    Tuning tn = tuning_from_flags(flags, 0, 3);
    tn.n_recs = n_tets;
    if ((rc = pass_status(who, w, status_dev, s, &tn.status))) return rc;
    // tets per shared-memory batch of the pair items: 16, 32 (default) or 64
    const int key = strip_pixels(cam0, flags) * 1000 + batch_size(flags, 32);
    const bool masks = tn.hit_masks && w.mask_header;
#define RM_FWD_CALL(PX, NT, BP, WALK)                                                                             \
    launch_fwd<PX, NT, BP, WALK>(sorted_ids, ranges, w, ray_jitter, views, sh, out_img, out_distortion, n_contrib, \
                                 tn, s)
#define RM_FWD_STRIP(BP)              \
    case 16 * 1000 + BP:              \
        return RM_FWD_CALL(16, 64, BP, kImage); \
    case 64 * 1000 + BP:              \
        return masks ? RM_FWD_CALL(64, 256, BP, kImageAndMasks) : RM_FWD_CALL(64, 256, BP, kImage);
    switch (key) {
        RM_FWD_STRIP(16)
        RM_FWD_STRIP(32)
        RM_FWD_STRIP(64)
        default:
            return rm_host::fail(RM_EINVAL, "%s: tets per batch %d unsupported (16, 32 or 64)", who, key % 1000);
    }
#undef RM_FWD_STRIP
#undef RM_FWD_CALL
}

template <class V>
int blend_bwd_any(const char* who, const int32_t* sorted_ids, const int32_t* ranges, const int32_t* indices,
                  const float* vertices, const float* cell_values, int64_t n_tets, int64_t n_verts,
                  const int32_t* tiles_touched,
                  const float* ray_jitter, const rm_camera* cam0, const V& views, const Shape& sh,
                  const float* out_img, const float* out_distortion, const int32_t* n_contrib, const float* grad_img,
                  const float* grad_distortion, float* grad_vertices, float* grad_cell_values, const void* records,
                  void* workspace, size_t workspace_bytes, int flags, uint32_t* status_dev, void* stream) {
    int rc = check_blend_args(who, indices, vertices, cell_values, records ? 0 : n_tets, ray_jitter, cam0, sh.G,
                              workspace, workspace_bytes, flags);
    if (rc) return rc;
    if (!ranges || !out_img || !out_distortion || !n_contrib || !grad_img || !grad_vertices || !grad_cell_values)
        return rm_host::fail(RM_EINVAL, "%s: NULL pointer", who);
    if (((uintptr_t)out_img & 15) || ((uintptr_t)grad_img & 15) || ((uintptr_t)ranges & 7) ||
        ((uintptr_t)ray_jitter & 7))
        return rm_host::fail(RM_EINVAL, "%s: misaligned image / grad / ranges / jitter", who);
    cudaStream_t s = (cudaStream_t)stream;
    BlendWs w = blend_ws(workspace, records ? 0 : n_tets, sh.G, workspace_bytes);
    if (records) {
        if ((uintptr_t)records & 15) return rm_host::fail(RM_EINVAL, "%s: records must be 16-byte aligned", who);
        w.recs = (float4*)records;  // packed by rm_blend_pack_records
    } else if (!(flags & RM_BLEND_REUSE_RECORDS) && n_tets > 0) {
        rc = pack(indices, vertices, n_verts, cell_values, n_tets, tiles_touched, w.recs, s);
        if (rc) return rc;
    }
    // no tile is heavy unless asked for: long lists are cut at the checkpoints
    // (the pair kernel, for all tiles or the longest ones, measured slower)
    Tuning tn = tuning_from_flags(flags, 0, 1);
    tn.n_recs = n_tets;
    if ((rc = pass_status(who, w, status_dev, s, &tn.status))) return rc;
    // tets per shared-memory batch of the bulk-copy staging: 16, 32 or 64 (default)
    const int key = strip_pixels(cam0, flags) * 1000 + batch_size(flags, 64);
#define RM_BWD_CASE(PX, NT, BD)                                                                                  \
    case PX * 1000 + BD:                                                                                         \
        return launch_bwd<PX, BD, PX, NT, 16>(sorted_ids, ranges, w, indices, ray_jitter, views, sh, out_img,       \
                                              out_distortion, n_contrib, grad_img, grad_distortion, grad_vertices,  \
                                              grad_cell_values, tn, s);
    switch (key) {
        RM_BWD_CASE(16, 64, 16)
        RM_BWD_CASE(16, 64, 32)
        RM_BWD_CASE(16, 64, 64)
        RM_BWD_CASE(64, 256, 16)
        RM_BWD_CASE(64, 256, 32)
        RM_BWD_CASE(64, 256, 64)
        default:
            return rm_host::fail(RM_EINVAL, "%s: tets per batch %d unsupported (16, 32 or 64)", who, key % 1000);
    }
#undef RM_BWD_CASE
}

}  // namespace
}  // namespace rm

extern "C" {

size_t rm_blend_workspace_size(int64_t n_tets, int64_t n_tiles) { return rm::blend_ws_bytes(n_tets, n_tiles); }

size_t rm_blend_status_offset(int64_t n_tets, int64_t n_tiles) {
    return rm::blend_ws_bytes(n_tets, n_tiles) - 256 + rm::kBlendStatusOff;
}

size_t rm_blend_hit_mask_bytes(int64_t n_pairs, int64_t n_tiles, int tile_pixels) {
    const int64_t subs = tile_pixels > 64 ? tile_pixels / 64 : 1;
    const int64_t P = n_pairs > 0 ? n_pairs : 0, G = n_tiles > 0 ? n_tiles : 0;
    // no less than any shorter lists need
    int64_t words = 0;
    for (int64_t n : {P < rm::kShortLists ? P : rm::kShortLists, P < rm::kLongLists ? P : rm::kLongLists, P}) {
        const int64_t w = rm::mask_word_count(n, G, subs) + rm::ck_words(n, subs, rm::seg_shift_for(n));
        words = w > words ? w : words;
    }
    return 256 + (size_t)words * sizeof(uint32_t);
}

int rm_calc_tet_err(const int32_t* sorted_ids, const int32_t* ranges, const int32_t* indices, const float* vertices,
                    const float* cell_values, int64_t n_tets, int64_t n_verts, const int32_t* tiles_touched,
                    const rm_camera* cam, const float* pixel_err, const float* ssim_err, float* tet_err,
                    int32_t* tet_count, void* workspace, size_t workspace_bytes, int flags, void* stream) {
    using namespace rm;
    int rc = rm_host::check_cam(cam);
    if (rc) return rc;
    const int64_t G = (int64_t)cam->grid_width * cam->grid_height;
    // the camera check of the blend calls; jitter is unused (pixel centres)
    rc = check_blend_args("rm_calc_tet_err", indices, vertices, cell_values, n_tets, pixel_err, cam, G, workspace,
                          workspace_bytes, flags);
    if (rc) return rc;
    if (!ranges || !ssim_err || !tet_err || !tet_count) return rm_host::fail(RM_EINVAL, "rm_calc_tet_err: NULL pointer");
    cudaStream_t s = (cudaStream_t)stream;
    const BlendWs w = blend_ws(workspace, n_tets, G, workspace_bytes);
    if (!(flags & RM_BLEND_REUSE_RECORDS) && n_tets > 0) {
        rc = pack(indices, vertices, n_verts, cell_values, n_tets, tiles_touched, w.recs, s);
        if (rc) return rc;
    }
    const int strip = strip_pixels(cam, flags);
    const int subs = cam->tile_width * cam->tile_height / strip;
    // with room for hit masks and n_contributors that is the call's own: the
    // forward's walk, then the statistics by stretches.  Otherwise that part of
    // the workspace is left as it is: a backward may still need its masks.
    const size_t nc_bytes = (size_t)cam->image_height * cam->image_width * sizeof(int32_t);
    if ((flags & RM_BLEND_OWN_SCRATCH) && strip == 64 && workspace_bytes > blend_ws_bytes(n_tets, G) + nc_bytes + 512) {
        const size_t nc_off = (workspace_bytes - nc_bytes) / 256 * 256;
        const BlendWs wm = blend_ws(workspace, n_tets, G, nc_off);
        if (wm.mask_header) {
            int32_t* nc = (int32_t*)((char*)workspace + nc_off);
            const OneView one = {*cam};
            const Shape sh = {(int)G, cam->tile_width * cam->tile_height};
            Tuning tn = tuning_from_flags(flags, 0, 3);
            tn.hit_masks = true;
            tn.n_recs = n_tets;
            rc = launch_fwd<64, 256, 32, kLogT>(sorted_ids, ranges, wm, nullptr, one, sh, nullptr, nullptr, nc,
                                                        tn, s);
            if (rc) return rc;
            const HitMasks hm = {wm.mask_words, wm.mask_cap, wm.mask_header, nullptr, 0, kNoSegments};
            const Queue q = {wm.order, wm.info, wm.tickets + 2, (int)G, subs, true, hm, nullptr,
                             rm_host::wait_limit(), n_tets};
            const int grid = persistent_grid(err_seg_kernel, 64, 0, 1 << 30);
            err_seg_kernel<<<grid, 64, 0, s>>>(sorted_ids, (const int2*)ranges, wm.recs, *cam, nc, pixel_err, ssim_err,
                                               tet_err, tet_count, q);
            return rm_host::check_launch("rm_calc_tet_err");
        }
    }
    // every tile in one heavy-first queue (heavy_shift 1 marks all tiles heavy)
    if ((rc = launch_order(ranges, (int)G, w, 1, s))) return rc;
    const Queue qd = {w.order, w.info, w.tickets + 0, (int)G, subs, true, HitMasks{}, nullptr,
                      rm_host::wait_limit(), n_tets};
    if (strip == 16) {
        const int grid = persistent_grid(err_kernel<16, 32>, 16, 0, (int)G * subs);
        err_kernel<16, 32><<<grid, 16, 0, s>>>(sorted_ids, (const int2*)ranges, w.recs, *cam, pixel_err, ssim_err,
                                                tet_err, tet_count, qd);
    } else {
        const int grid = persistent_grid(err_kernel<64, 32>, 64, 0, (int)G * subs);
        err_kernel<64, 32><<<grid, 64, 0, s>>>(sorted_ids, (const int2*)ranges, w.recs, *cam, pixel_err, ssim_err,
                                                tet_err, tet_count, qd);
    }
    return rm_host::check_launch("rm_calc_tet_err");
}

size_t rm_blend_records_size(int64_t n_tets) {
    return (size_t)(n_tets > 0 ? n_tets : 0) * rm::kRecFloat4 * sizeof(float4);
}

int rm_blend_pack_records(const int32_t* indices, const float* vertices, const float* cell_values, int64_t n_tets,
                          int64_t n_verts, const int32_t* tiles_touched, void* records, void* stream) {
    if (n_tets < 0 || n_verts < 0) return rm_host::fail(RM_EINVAL, "rm_blend_pack_records: negative size");
    if (n_tets == 0) return RM_OK;
    if (!indices || !vertices || !cell_values || !records)
        return rm_host::fail(RM_EINVAL, "rm_blend_pack_records: NULL pointer");
    if (((uintptr_t)indices & 15) || ((uintptr_t)records & 15))
        return rm_host::fail(RM_EINVAL, "rm_blend_pack_records: indices and records must be 16-byte aligned");
    return rm::pack(indices, vertices, n_verts, cell_values, n_tets, tiles_touched, (float4*)records,
                    (cudaStream_t)stream);
}

int rm_blend_fwd(const int32_t* sorted_ids, const int32_t* ranges, const int32_t* indices, const float* vertices,
                 const float* cell_values, int64_t n_tets, int64_t n_verts, const int32_t* tiles_touched,
                 const float* ray_jitter, const rm_camera* cam, float* out_img, float* out_distortion,
                 int32_t* n_contrib, void* workspace, size_t workspace_bytes, int flags, uint32_t* status_dev,
                 void* stream) {
    int rc = rm_host::check_cam(cam);
    if (rc) return rc;
    const rm::OneView one = {*cam};
    const rm::Shape sh = {cam->grid_width * cam->grid_height, cam->tile_width * cam->tile_height};
    return rm::blend_fwd_any("rm_blend_fwd", sorted_ids, ranges, indices, vertices, cell_values, n_tets, n_verts,
                             tiles_touched, ray_jitter, cam, one, sh, out_img, out_distortion, n_contrib, nullptr,
                             workspace, workspace_bytes, flags, status_dev, stream);
}

int rm_blend_bwd(const int32_t* sorted_ids, const int32_t* ranges, const int32_t* indices, const float* vertices,
                 const float* cell_values, int64_t n_tets, int64_t n_verts, const int32_t* tiles_touched,
                 const float* ray_jitter, const rm_camera* cam, const float* out_img, const float* out_distortion,
                 const int32_t* n_contrib, const float* grad_img, const float* grad_distortion, float* grad_vertices,
                 float* grad_cell_values, void* workspace, size_t workspace_bytes, int flags, uint32_t* status_dev,
                 void* stream) {
    int rc = rm_host::check_cam(cam);
    if (rc) return rc;
    const rm::OneView one = {*cam};
    const rm::Shape sh = {cam->grid_width * cam->grid_height, cam->tile_width * cam->tile_height};
    return rm::blend_bwd_any("rm_blend_bwd", sorted_ids, ranges, indices, vertices, cell_values, n_tets, n_verts,
                             tiles_touched, ray_jitter, cam, one, sh, out_img, out_distortion, n_contrib, grad_img,
                             grad_distortion, grad_vertices, grad_cell_values, nullptr, workspace, workspace_bytes,
                             flags, status_dev, stream);
}

int rm_blend_fwd_multi(const int32_t* sorted_ids, const int32_t* ranges, const int32_t* indices,
                       const float* vertices, const float* cell_values, int64_t n_tets, int64_t n_verts,
                       const int32_t* tiles_touched, const float* ray_jitter, const rm_camera* cams, int n_views,
                       float* out_img, float* out_distortion, int32_t* n_contrib, const void* records,
                       void* workspace, size_t workspace_bytes, int flags, uint32_t* status_dev, void* stream) {
    rm::ViewSet views;
    int rc = rm_host::make_views("rm_blend_fwd_multi", cams, n_views, &views);
    if (rc) return rc;
    const rm::Shape sh = {views.tiles[n_views], cams[0].tile_width * cams[0].tile_height};
    return rm::blend_fwd_any("rm_blend_fwd_multi", sorted_ids, ranges, indices, vertices, cell_values, n_tets, n_verts,
                             tiles_touched, ray_jitter, cams, views, sh, out_img, out_distortion, n_contrib,
                             records, workspace, workspace_bytes, flags, status_dev, stream);
}

int rm_blend_bwd_multi(const int32_t* sorted_ids, const int32_t* ranges, const int32_t* indices,
                       const float* vertices, const float* cell_values, int64_t n_tets, int64_t n_verts,
                       const int32_t* tiles_touched, const float* ray_jitter, const rm_camera* cams, int n_views,
                       const float* out_img, const float* out_distortion, const int32_t* n_contrib,
                       const float* grad_img, const float* grad_distortion, float* grad_vertices,
                       float* grad_cell_values, const void* records, void* workspace, size_t workspace_bytes,
                       int flags, uint32_t* status_dev, void* stream) {
    rm::ViewSet views;
    int rc = rm_host::make_views("rm_blend_bwd_multi", cams, n_views, &views);
    if (rc) return rc;
    const rm::Shape sh = {views.tiles[n_views], cams[0].tile_width * cams[0].tile_height};
    return rm::blend_bwd_any("rm_blend_bwd_multi", sorted_ids, ranges, indices, vertices, cell_values, n_tets, n_verts,
                             tiles_touched, ray_jitter, cams, views, sh, out_img, out_distortion, n_contrib,
                             grad_img, grad_distortion, grad_vertices, grad_cell_values, records, workspace,
                             workspace_bytes, flags, status_dev, stream);
}

}  // extern "C"
