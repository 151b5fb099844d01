// Per-tile alpha compositing, forward and backward (instruction-issue bound).
//
// One CTA (256 threads, one pixel each) per 16x16 tile, like the reference, but:
//  * the five per-Gaussian inputs are first packed into one 64-byte record per Gaussian
//    [x y, cull extents | a b c opacity | r g b m0 | m1..m4];
//  * the CTA culls 512 entries of the tile's list at a time against the tile's eight 8x4 pixel blocks, one warp each,
//    with exact-safe bounds (a Gaussian or a pixel is dropped only if alpha < 1/255 is guaranteed there); after that one
//    barrier the warps are on their own;
//  * each warp collects the Gaussians that may reach its block ("visits") with the mask of the pixels they may reach in
//    a queue of 32 that spans the culled stretches; only those fetch their colours and plane maps;
//  * a full queue is walked by pixel: every lane takes only its OWN visits, in list order, so the expensive part is
//    executed as often as the busiest pixel of the block contributes, not once per visit: on aerial scenes a visit has
//    1-5 contributing pixels out of 32;
//  * the backward then walks the queue once more by visit: a lane sums the 16 gradient terms of its Gaussian over the
//    pixels in registers and issues ONE atomic per term per Gaussian per warp straight into the caller's tensors;
//  * the per-tile statistics (sum of per-pixel counters) are reduced in the forward's epilogue.
#include "cgx_common.cuh"

namespace cgx {

struct __align__(16) Record {
    float4 q0;  // x, y, cull half-extent x, y (see cull_extent)
    float4 q1;  // conic a, b, c, opacity
    float4 q2;  // r, g, b, m0
    float4 q3;  // m1, m2, m3, m4
};

// A record in a warp's queue: 80-byte pitch.  In the walks every lane reads the record of a DIFFERENT Gaussian; at
// the natural 64-byte pitch eight lanes of a quarter-warp would hit the same two groups of four banks, at 80 bytes
// consecutive records fall into all eight groups.
struct __align__(16) RecSlot : Record {
    float4 pad;
};

// 16-byte asynchronous global -> shared copy, and the wait for all of this thread's copies.
__device__ __forceinline__ void copy_async_16(void* dst_smem, const void* src_gmem)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)),
                 "l"(src_gmem)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Half extents of the axis-aligned box outside of which opacity * exp(power) < 1/255 for certain.
// power = -0.5 (a dx^2 + c dy^2) - b dx dy >= -tau bounds |dx| <= sqrt(2 tau c / (ac - b^2)), same for dy with a.
// The box is inflated (1 % + 0.01 px) so float rounding in the per-pixel test can never keep a pixel the box drops.
__device__ __forceinline__ float2 cull_extent(float a, float b, float c, float o)
{
    const float inf = __int_as_float(0x7f800000);
    if (!(o >= 1.0f / 255.0f)) return {-1.f, -1.f};  // alpha <= o < 1/255 everywhere (NaN opacity: never kept either)
    const float det = a * c - b * b;
    if (!(det > 0.f) || !(a > 0.f) || !(c > 0.f)) return {inf, inf};
    const float tau = __logf(255.0f * o) * 1.01f + 0.01f;
    const float ex = sqrtf(2.f * tau * c / det) * 1.01f + 0.01f;
    const float ey = sqrtf(2.f * tau * a / det) * 1.01f + 0.01f;
    if (!(ex == ex) || !(ey == ey)) return {inf, inf};
    return {ex, ey};
}

// alpha of one Gaussian at one pixel, in the reference's operation order (cuda_rasterizer/forward.cu:376-389), with
// the contractions written out so that the compiler cannot choose others from one use to the next.
// Returns false when the pixel is skipped (power > 0 or alpha < 1/255).
// `rows_first`: the product that is fused into the sum a dx^2 + c dy^2 is the second instead of the first.  Never in
// the forward; in the backward on scenes of small splats (see scene_is_dense), where its kernel has always rounded that way: a contribution whose alpha lies
// within an ulp of 1/255 is kept or dropped as it was, and a kept or dropped one shifts the transmittance of
// everything in front of it by 0.4 %.
__device__ __forceinline__ bool eval_alpha(const float2 xy, const float4 con_o, const float2 pixf, float2& d, float& G,
                                           float& alpha, const bool rows_first = false)
{
    d = {xy.x - pixf.x, xy.y - pixf.y};
    const float ax = __fmul_rn(con_o.x, d.x), cy = __fmul_rn(con_o.z, d.y);
    const float q = rows_first ? __fmaf_rn(cy, d.y, __fmul_rn(ax, d.x)) : __fmaf_rn(ax, d.x, __fmul_rn(cy, d.y));
    const float power = __fmaf_rn(-0.5f, q, -__fmul_rn(__fmul_rn(con_o.y, d.x), d.y));
    if (power > 0.0f) return false;
    G = exp(power);
    alpha = min(0.99f, con_o.w * G);
    return !(alpha < 1.0f / 255.0f);
}

// How densely the scene's splats cover the 8x4 pixel blocks they meet, measured by the forward pass behind its P
// records: pairs (pixels reached, Gaussians that meet a block), spread over slots so that there is no hot address.
constexpr int DENSITY_SLOTS = 32;
constexpr size_t DENSITY_BYTES = DENSITY_SLOTS * 2 * sizeof(unsigned long long);
constexpr int DENSE_PIXELS_PER_VISIT = 6;
__device__ __forceinline__ bool scene_is_dense(const Record* records, int P, int lane)
{
    const ulonglong2 slot = reinterpret_cast<const ulonglong2*>(records + P)[lane];
    float excess = (float)slot.x - (float)DENSE_PIXELS_PER_VISIT * (float)slot.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) excess += __shfl_xor_sync(0xffffffffu, excess, o);
    return excess > 0.f;
}

// Pixels of a warp's 8x4 block (bit y * 8 + x = lane of that pixel) that a Gaussian may reach: per pixel row, the
// interval of the ellipse "alpha = 1/255" inflated like its bounding box (ex, ey).  A superset of the pixels that pass
// eval_alpha: the walks test each of them.  Lane = Gaussian, so 32 are bounded at once for about 90 instructions;
// evaluating alpha at the pixels of the box instead cost 25 instructions per pixel of the widest of the 32 boxes
// (40 % of the forward kernel's instructions on a scene of 2-pixel splats).
// Where the conic is close to singular (a thin splat, slanted) the interval would be lost to rounding: whole box.
__device__ __forceinline__ uint32_t block_mask(const float4 q0, const float4 q1, const float sx0, const float sy0)
{
    const float ex = q0.z, ey = q0.w, a = q1.x, b = q1.y, c = q1.z;
    const float rel_det = 1.f - __fdividef(b * b, a * c);
    // on the row at offset dy the pixels within hx * sqrt(1 - (dy / ey)^2) of x + slope * dy
    const bool slanted = rel_det > 1e-3f && ex < 1e6f;
    const float hx = slanted ? ex * sqrtf(rel_det) : ex;
    const float slope = slanted ? __fdividef(b, a) : 0.f;
    const float inv_ey2 = slanted ? __fdividef(1.f, ey * ey) : 0.f;
    const float x = q0.x - sx0, y = q0.y - sy0;
    uint32_t pm = 0;
#pragma unroll
    for (int row = 0; row < 4; row++) {
        const float dy = y - (float)row;
        const float t = 1.f - dy * dy * inv_ey2;
        const float half = hx * sqrtf(fmaxf(t, 0.f)) + 0.01f;
        const float mid = x + slope * dy;
        const int x0 = min(8, max(0, __float2int_ru(mid - half)));
        const int x1 = max(-1, min(7, __float2int_rd(mid + half)));
        const uint32_t bits = (0xFFu << x0) & (0xFFu >> (7 - x1)) & 0xFFu;
        pm |= (fabsf(dy) <= ey ? bits : 0u) << (8 * row);
    }
    return pm;
}

// 32 x 32 bit matrix held one row per lane -> one column per lane (five exchanges of off-diagonal blocks).  Turns
// "lane v holds the pixel mask of visit v" into "lane p holds the visit mask of pixel p" and back.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t a, const int lane)
{
#pragma unroll
    for (int s = 0; s < 5; s++) {
        const int j = 16 >> s;
        const uint32_t m0 = s == 0 ? 0x0000FFFFu : s == 1 ? 0x00FF00FFu : s == 2 ? 0x0F0F0F0Fu
                          : s == 3 ? 0x33333333u : 0x55555555u;
        const uint32_t other = __shfl_xor_sync(0xffffffffu, a, j);
        a = (lane & j) ? ((a & ~m0) | ((other >> j) & m0)) : ((a & m0) | ((other & m0) << j));
    }
    return a;
}

// ------------------------------------------------------------------------------------------------ pack
__global__ void __launch_bounds__(256)
pack_records_kernel(int P, const int* __restrict__ radii, const float2* __restrict__ means2D,
                    const float4* __restrict__ conic_opacity, const float* __restrict__ rgb,
                    const float* __restrict__ all_map, int render_geo, Record* __restrict__ records,
                    int* __restrict__ out_observe)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 2 * DENSITY_SLOTS) reinterpret_cast<unsigned long long*>(records + P)[i] = 0ull;
    if (i >= P) return;
    if (out_observe) out_observe[i] = 0;
    // Gaussians without a radius never enter a tile list: their record is never read, so it is not written
    if (radii && radii[i] <= 0) return;
    const float2 xy = means2D[i];
    const float4 co = conic_opacity[i];
    const float r = rgb[3 * i], g = rgb[3 * i + 1], b = rgb[3 * i + 2];
    float m[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    if (render_geo) {
#pragma unroll
        for (int k = 0; k < 5; k++) m[k] = all_map[5 * i + k];
    }
    Record rec;
    const float2 ext = cull_extent(co.x, co.y, co.z, co.w);
    rec.q0 = {xy.x, xy.y, ext.x, ext.y};
    rec.q1 = co;
    rec.q2 = {r, g, b, m[0]};
    rec.q3 = {m[1], m[2], m[3], m[4]};
    records[i] = rec;
}

constexpr int RENDER_THREADS = CGX_BLOCK_SIZE;
constexpr int RENDER_WARPS = RENDER_THREADS / 32;

#ifndef CGX_SCAN_SLOTS
#define CGX_SCAN_SLOTS 256
#endif
constexpr int SCAN_SLOTS = CGX_SCAN_SLOTS;          // list entries a CTA culls at a time (512: 2-4 % slower, by its memory)
static_assert(SCAN_SLOTS % 32 == 0 && SCAN_SLOTS <= 256, "slots are kept as bytes");

// What the warps of a CTA share about the entries of the tile's list that were culled together.
template <int WARPS>
struct ScanSmem {
    float4 q0[SCAN_SLOTS], q1[SCAN_SLOTS];
    int id[SCAN_SLOTS];
    uint32_t bits[WARPS][SCAN_SLOTS / 32];      // entry meets the 8x4 block of warp w
    uint8_t hits[WARPS][SCAN_SLOTS];
};

// The Gaussians that a warp has collected for its 8x4 block.
struct QueueSmem {
    RecSlot rec[32];
    uint32_t mask[32];         // pixels it may reach
    int id[32];
    int idx[32];               // its position in the tile's list
};

// Culls entries first, first + step, ... (n of them, n <= SCAN_SLOTS) of a tile's list against the tile's eight
// blocks: a thread tests one entry against all eight (every warp for itself would read each entry eight times from
// shared memory), ballots turn the answers into one bit list per warp.  Callers put a barrier before and after.
template <int WARPS>
__device__ __forceinline__ void scan_entries(ScanSmem<WARPS>& sm, const uint32_t* __restrict__ list, int step, int n,
                                             const Record* __restrict__ records, float x0, float y0)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 2
    for (int slot = threadIdx.x; slot < ((n + 31) & ~31); slot += 32 * WARPS) {
        uint32_t meets = 0;
        if (slot < n) {
            const int id = list[(ptrdiff_t)slot * step];
            const float4 q0 = records[id].q0;
            sm.q0[slot] = q0;
            sm.q1[slot] = records[id].q1;
            sm.id[slot] = id;
            const float l = q0.x - q0.z - x0, r = q0.x + q0.z - x0, t = q0.y - q0.w - y0, b = q0.y + q0.w - y0;
            const uint32_t cols = (r >= 0.f && l <= 7.f ? 0x55u : 0u) | (r >= 8.f && l <= 15.f ? 0xAAu : 0u);
            uint32_t rows = 0;
#pragma unroll
            for (int k = 0; k < WARPS / 2; k++)
                if (b >= 4.f * k && t <= 4.f * k + 3.f) rows |= 3u << (2 * k);
            meets = cols & rows;
        }
        uint32_t word = 0;
#pragma unroll
        for (int w = 0; w < WARPS; w++) {
            const uint32_t m = __ballot_sync(0xffffffffu, (meets >> w) & 1u);
            if (lane == w) word = m;
        }
        if (lane < WARPS) sm.bits[lane][slot >> 5] = word;
    }
}

// Slots >= first of the scanned entries that meet this warp's block, in order; returns their number.
template <int WARPS>
__device__ __forceinline__ int collect_hits(ScanSmem<WARPS>& sm, int warp, int lane, int first, int n)
{
    int n_hits = 0;
    for (int w = first >> 5; w < (n + 31) >> 5; w++) {
        uint32_t m = sm.bits[warp][w];
        if (w == first >> 5) m &= 0xffffffffu << (first & 31);
        if ((m >> lane) & 1u) sm.hits[warp][n_hits + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(w * 32 + lane);
        n_hits += __popc(m);
    }
    __syncwarp();
    return n_hits;
}

// Appends up to 32 hits, one per lane, to the queue.  `fresh`: lanes whose hit still waits (the lowest go first, order
// is kept); returns those that found no place.  The second half of a record is fetched asynchronously.
__device__ __forceinline__ uint32_t queue_push(QueueSmem& q, int& nq, uint32_t fresh, int lane, uint32_t mask,
                                               const float4 q0, const float4 q1, int id, int idx,
                                               const Record* __restrict__ records)
{
    const int rank = __popc(fresh & ((1u << lane) - 1u));
    const int take = min(32 - nq, __popc(fresh));
    const bool mine = (fresh >> lane) & 1u;
    if (mine && rank < take) {
        const int k = nq + rank;
        copy_async_16(&q.rec[k].q2, &records[id].q2);
        copy_async_16(&q.rec[k].q3, &records[id].q3);
        q.rec[k].q0 = q0;
        q.rec[k].q1 = q1;
        q.mask[k] = mask;
        q.id[k] = id;
        q.idx[k] = idx;
    }
    nq += take;
    return __ballot_sync(0xffffffffu, mine && rank >= take);
}

#ifndef CGX_FWD_MIN_CTAS
#define CGX_FWD_MIN_CTAS 4
#endif

struct FwdSmem {
    ScanSmem<RENDER_WARPS> scan;
    QueueSmem queue[RENDER_WARPS];
    int red[4][RENDER_WARPS];
};

// One CTA per 16x16 tile.  CULL = false: every pixel looks at every Gaussian of the batch (the reference's loop; the
// yardstick of the tests).  CULL = true: every warp collects the Gaussians that may reach its 8x4 pixel block in a
// queue of 32 (across the staged batches) and every pixel then walks its own bits of the queue's masks, in list
// order: the blending is run as often as the busiest pixel of the block has contributors, not once per Gaussian.
// Both take every decision on the same bits (eval_alpha) and blend in the same order: identical outputs.
// Bound by instruction issue (64 %) and shared-memory wavefronts (51 %).  Per camera of 6 M Gaussians at 1600x1200:
// 0.53 -> 0.38 ms; 4 M at 3840x2160: 0.77 -> 0.50 ms; 150 k large splats at 1280x720: 0.21 -> 0.12 ms.
template <bool CULL>
__global__ void __launch_bounds__(RENDER_THREADS, CGX_FWD_MIN_CTAS)
render_fwd_kernel(const uint2* __restrict__ ranges, const uint32_t* __restrict__ point_list, int W, int H,
                  const float focal_x, const float focal_y, const float cx, const float cy,
                  const Record* __restrict__ records, float* __restrict__ final_T, uint32_t* __restrict__ n_contrib,
                  uint32_t* __restrict__ n_contrib2loss, const uint8_t* __restrict__ compute_locally,
                  const float* __restrict__ bg_color, float* __restrict__ out_color, int* __restrict__ out_observe,
                  float* __restrict__ out_all_map, float* __restrict__ out_plane_depth, const bool render_geo,
                  int* __restrict__ n_render_t, int* __restrict__ n_consider_t, int* __restrict__ n_contrib_t,
                  unsigned long long* __restrict__ density)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    FwdSmem& sm = *reinterpret_cast<FwdSmem*>(smem_raw);

    const uint32_t block_id = blockIdx.y * gridDim.x + blockIdx.x;
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    // warp w owns the 8x4 pixel block (w & 1, w >> 1) of the tile: compact footprints keep a small splat
    // inside few warps, which is what the per-warp culling (and the backward's per-warp sums) pays for
    const uint32_t lx = (warp & 1) * 8 + (lane & 7), ly = (warp >> 1) * 4 + (lane >> 3);

    const uint2 pix_min = {blockIdx.x * CGX_BLOCK_X, blockIdx.y * CGX_BLOCK_Y};
    const uint2 pix = {pix_min.x + lx, pix_min.y + ly};
    const uint32_t pix_id = W * pix.y + pix.x;
    const float2 pixf = {(float)pix.x, (float)pix.y};
    const bool inside = pix.x < W && pix.y < H;
    const size_t HW = (size_t)H * W;

    if (!compute_locally[block_id]) {
        // tiles owned by another rank: defined zeros in every image output
        if (inside) {
            final_T[pix_id] = 0.f;
            n_contrib[pix_id] = 0;
            n_contrib2loss[pix_id] = 0;
            for (int ch = 0; ch < CGX_NCH; ch++) out_color[ch * HW + pix_id] = 0.f;
            for (int ch = 0; ch < CGX_NMAP; ch++) out_all_map[ch * HW + pix_id] = 0.f;
            out_plane_depth[pix_id] = 0.f;
        }
        if (tid == 0) {
            const uint2 rg = ranges[block_id];
            n_render_t[block_id] = rg.y - rg.x;
            n_consider_t[block_id] = 0;
            n_contrib_t[block_id] = 0;
        }
        return;
    }

    bool done = !inside;
    const uint2 range = ranges[block_id];
    const int total = range.y - range.x;
    // first pixel of this warp's block
    const float sx0 = (float)(pix_min.x + (warp & 1) * 8), sy0 = (float)(pix_min.y + (warp >> 1) * 4);

    float T = 1.0f;
    uint32_t last_contributor = 0;
    uint32_t thread_n_contrib2loss = 0;
    float C[CGX_NCH] = {0};
    float All_map[CGX_NMAP] = {0};
    int reached = 0, visits = 0;       // pixels that this lane's Gaussians may reach; Gaussians that meet the block

    // Blends one Gaussian into this pixel unless its alpha is below the threshold there (cuda_rasterizer/
    // forward.cu:376-416).  Returns whether it was blended while the transmittance was above one half.
    auto blend = [&](const Record& r, const int idx) -> bool {
        float2 d;
        float G, alpha;
        if (!eval_alpha(*reinterpret_cast<const float2*>(&r.q0), r.q1, pixf, d, G, alpha)) return false;
        const float test_T = T * (1 - alpha);
        if (test_T < 0.0001f) {
            done = true;
            return false;
        }
        thread_n_contrib2loss++;
        const float4 q2 = r.q2;
        const float feat[CGX_NCH] = {q2.x, q2.y, q2.z};
#pragma unroll
        for (int ch = 0; ch < CGX_NCH; ch++) C[ch] += feat[ch] * alpha * T;
        if (render_geo) {
            const float4 q3 = r.q3;
            const float am[CGX_NMAP] = {q2.w, q3.x, q3.y, q3.z, q3.w};
#pragma unroll
            for (int ch = 0; ch < CGX_NMAP; ch++) All_map[ch] += am[ch] * alpha * T;
        }
        const bool clear = T > 0.5;
        T = test_T;
        last_contributor = idx + 1;
        return clear;
    };

    if (!CULL) {
        for (int k = 0; !done && k < total; k++) {
            const int id = point_list[range.x + k];
            if (blend(records[id], k)) atomicAdd(&out_observe[id], 1);
        }
    } else {
        QueueSmem& queue = sm.queue[warp];
        int nq = 0;                        // visits in the queue (warp-uniform)
        for (int start = 0; start < total; start += SCAN_SLOTS) {
            // ends when every pixel of the tile is done (and orders the reuse of the scan's memory)
            if (__syncthreads_count(done) == RENDER_THREADS) break;
            const int n = min(SCAN_SLOTS, total - start);
            scan_entries(sm.scan, point_list + range.x + start, 1, n, records, (float)pix_min.x, (float)pix_min.y);
            __syncthreads();
            if (__all_sync(0xffffffffu, done)) continue;
            const bool last = start + SCAN_SLOTS >= total;
            const int n_hits = collect_hits(sm.scan, warp, lane, 0, n);
            visits += n_hits;
            for (int base = 0; base < n_hits || (last && nq > 0); base += 32) {
                uint32_t pm = 0;
                int slot = 0;
                float4 q0, q1;
                if (base + lane < n_hits) {
                    slot = sm.scan.hits[warp][base + lane];
                    q0 = sm.scan.q0[slot];
                    q1 = sm.scan.q1[slot];
                    pm = block_mask(q0, q1, sx0, sy0);
                    reached += __popc(pm);
                }
                uint32_t fresh = __ballot_sync(0xffffffffu, pm != 0);
                do {
                    fresh = queue_push(queue, nq, fresh, lane, pm, q0, q1, sm.scan.id[slot], start + slot, records);
                    // on with the next hits until the queue is full or the list has ended
                    if (nq < 32 && !(last && base + 32 >= n_hits)) break;
                    copy_async_wait();
                    __syncwarp();
                    // lane = pixel, front to back
                    uint32_t mine = warp_transpose32(lane < nq ? queue.mask[lane] : 0u, lane);
                    uint32_t seen_clear = 0;      // visits this pixel blended while its transmittance was above 0.5
                    for (; mine && !done; mine &= mine - 1) {
                        const int v = __ffs(mine) - 1;
                        if (blend(queue.rec[v], queue.idx[v])) seen_clear |= 1u << v;
                    }
                    // out_observe: one atomic per Gaussian with the number of such pixels
                    if (__any_sync(0xffffffffu, seen_clear != 0)) {
                        const int cnt = __popc(warp_transpose32(seen_clear, lane));   // lane = visit: its pixels
                        if (cnt) atomicAdd(&out_observe[queue.id[lane]], cnt);
                    }
                    __syncwarp();
                    nq = 0;
                } while (fresh);
            }
        }
        copy_async_wait();     // what a saturated block had in its queue
    }

    if (inside) {
        final_T[pix_id] = T;
        n_contrib[pix_id] = last_contributor;
        n_contrib2loss[pix_id] = thread_n_contrib2loss;
        for (int ch = 0; ch < CGX_NCH; ch++) out_color[ch * HW + pix_id] = C[ch] + T * bg_color[ch];
        if (render_geo) {
            const float2 ray = {(pixf.x - cx) / focal_x, (pixf.y - cy) / focal_y};
            for (int ch = 0; ch < CGX_NMAP; ch++) out_all_map[ch * HW + pix_id] = All_map[ch];
            out_plane_depth[pix_id] = All_map[4] / -(All_map[0] * ray.x + All_map[1] * ray.y + All_map[2] + 1.0e-8);
        } else {
            for (int ch = 0; ch < CGX_NMAP; ch++) out_all_map[ch * HW + pix_id] = 0.f;
            out_plane_depth[pix_id] = 0.f;
        }
    }

    // per-tile sums of the two per-pixel counters (pixels outside the image count as 0)
    const int a = __reduce_add_sync(0xffffffffu, inside ? (int)last_contributor : 0);
    const int b = __reduce_add_sync(0xffffffffu, inside ? (int)thread_n_contrib2loss : 0);
    reached = __reduce_add_sync(0xffffffffu, reached);
    if (lane == 0) {
        sm.red[0][warp] = a;
        sm.red[1][warp] = b;
        sm.red[2][warp] = reached;
        sm.red[3][warp] = visits;
    }
    __syncthreads();
    if (tid == 0) {
        int sa = 0, sb = 0;
        unsigned long long sr = 0, sv = 0;
        for (int w = 0; w < RENDER_WARPS; w++) {
            sa += sm.red[0][w];
            sb += sm.red[1][w];
            sr += (unsigned)sm.red[2][w];
            sv += (unsigned)sm.red[3][w];
        }
        if (density && sv) {
            atomicAdd(density + 2 * (block_id % DENSITY_SLOTS), sr);
            atomicAdd(density + 2 * (block_id % DENSITY_SLOTS) + 1, sv);
        }
        n_render_t[block_id] = total;
        n_consider_t[block_id] = sa;
        n_contrib_t[block_id] = sb;
    }
}

__global__ void __launch_bounds__(RENDER_THREADS)
tile_stats_kernel(int W, int H, const uint2* __restrict__ ranges, const uint32_t* __restrict__ n_contrib_px,
                  const uint32_t* __restrict__ n_c2l_px, const uint8_t* __restrict__ compute_locally,
                  int* __restrict__ n_render, int* __restrict__ n_consider, int* __restrict__ n_contrib)
{
    __shared__ int red[2][RENDER_WARPS];
    const uint32_t block_id = blockIdx.y * gridDim.x + blockIdx.x;
    const int tid = threadIdx.y * CGX_BLOCK_X + threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const bool local = compute_locally[block_id];
    const uint32_t px = blockIdx.x * CGX_BLOCK_X + threadIdx.x, py = blockIdx.y * CGX_BLOCK_Y + threadIdx.y;
    const bool inside = px < (uint32_t)W && py < (uint32_t)H;
    int a = (local && inside) ? (int)n_contrib_px[(size_t)W * py + px] : 0;
    int b = (local && inside) ? (int)n_c2l_px[(size_t)W * py + px] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
        red[0][warp] = a;
        red[1][warp] = b;
    }
    __syncthreads();
    if (tid == 0) {
        int sa = 0, sb = 0;
        for (int w = 0; w < RENDER_WARPS; w++) {
            sa += red[0][w];
            sb += red[1][w];
        }
        const uint2 rg = ranges[block_id];
        n_render[block_id] = rg.y - rg.x;
        n_consider[block_id] = sa;
        n_contrib[block_id] = sb;
    }
}

// ------------------------------------------------------------------------------------------------ backward
#ifndef CGX_BWD_CAP
#define CGX_BWD_CAP 288
#endif
#ifndef CGX_BWD_MIN_CTAS
#define CGX_BWD_MIN_CTAS 6
#endif
// (pixel, Gaussian) contributions a warp keeps between its two steps.  Small splats fill 150 of them per queue, splats
// that fill the block a thousand; what is left beside six CTAs per SM.
constexpr int BWD_CAP = CGX_BWD_CAP;
static_assert(BWD_CAP >= 32, "a group must hold at least one full visit");

struct BwdOut {
    float *means2D, *abs2D, *conic, *rgb, *all_map;   // (P,2) (P,3) (P,4) (P,3) (P,5)
    bool vec;                                         // means2D 8-byte and conic 16-byte aligned: vector atomics
    float4* table;                                    // P rows of 16 floats, or null: see bwd_add
};

// What one pixel carries from one contributor to the next, back to front (cuda_rasterizer/backward.cu:408-443).
// The reference keeps the blended colour / plane map behind the pixel per channel and multiplies each difference by
// its cotangent; only the sum over the channels is ever used, and the blend is linear, so this walk keeps the blend
// of the dot products <features, cotangents>: one recurrence instead of eight.
struct BwdPixel {
    float T, T_final_bg;                 // transmittance in front of the next contributor; T_final * <bg, dL/dC>
    Pair behind[4];                      // the features blended behind the next contributor: r g | b m0 | m1 m2 | m3 m4
    float d[CGX_NCH + CGX_NMAP];         // cotangents: colour, plane map (with the plane depth's folded in)
};

// Loads the pixel's cotangents and folds the plane-depth cotangent into the plane-map channels
// (cuda_rasterizer/backward.cu:379-443).
__device__ __forceinline__ void bwd_pixel_init(BwdPixel& px, bool inside, uint32_t pix_id, size_t HW, float2 ray,
                                               const float* __restrict__ bg_color, const float* __restrict__ final_Ts,
                                               const float* __restrict__ all_map_pixels,
                                               const float* __restrict__ dL_dpixels,
                                               const float* __restrict__ dL_dout_all_maps,
                                               const float* __restrict__ dL_dout_plane_depths, bool render_geo)
{
    px.T = inside ? final_Ts[pix_id] : 0;
#pragma unroll
    for (int k = 0; k < 4; k++) px.behind[k] = pack(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < CGX_NCH + CGX_NMAP; i++) px.d[i] = 0.f;
    float bg_dot = 0.f;
    if (inside) {
#pragma unroll
        for (int i = 0; i < CGX_NCH; i++) {
            px.d[i] = dL_dpixels[i * HW + pix_id];
            bg_dot += bg_color[i] * px.d[i];
        }
        if (render_geo) {
            float* m = px.d + CGX_NCH;
#pragma unroll
            for (int i = 0; i < CGX_NMAP; i++) m[i] = dL_dout_all_maps[i * HW + pix_id];
            const float3 normal = {all_map_pixels[pix_id], all_map_pixels[HW + pix_id], all_map_pixels[2 * HW + pix_id]};
            const float distance = all_map_pixels[4 * HW + pix_id];
            const float tmp = (normal.x * ray.x + normal.y * ray.y + normal.z + 1.0e-8);
            const float dd = dL_dout_plane_depths[pix_id];
            m[CGX_NMAP - 1] += (-dd / tmp);
            m[0] += dd * (distance / (tmp * tmp) * ray.x);
            m[1] += dd * (distance / (tmp * tmp) * ray.y);
            m[2] += dd * (distance / (tmp * tmp));
        }
    }
    px.T_final_bg = px.T * bg_dot;
}

// One contribution (cuda_rasterizer/backward.cu:476-563): advances the pixel and returns
//   x = alpha * T              (dL/drgb, dL/dall_map are this times the pixel's cotangents)
//   y = opacity * G * dL/dalpha (every geometric term is this times a polynomial of the offset d)
__device__ __forceinline__ float2 bwd_contribution(BwdPixel& px, const Record& r, const float opacity, const float G,
                                                   const float alpha)
{
    // one reciprocal serves both quotients: the hardware's approximation and a Newton step (within 0.51 ulp for these
    // arguments, 0.01 to 1, without the special cases that a general correctly rounded reciprocal carries along)
    const float one_ma = 1.f - alpha;
    float inv_1ma;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv_1ma) : "f"(one_ma));
    inv_1ma = fmaf(inv_1ma, fmaf(-one_ma, inv_1ma, 1.f), inv_1ma);
    px.T = px.T * inv_1ma;
    // Channel by channel and in this order: behind the blended normal's projection on the ray the eight products cancel
    // to four digits in places, and any other order of the same sum has other digits left there.
    const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(&r.q2), q3 = *reinterpret_cast<const ulonglong2*>(&r.q3);
    const Pair feature[4] = {Pair{q2.x}, Pair{q2.y}, Pair{q3.x}, Pair{q3.y}};
    const Pair minus_one = pack(-1.f, -1.f), alpha2 = pack(alpha, alpha), one_ma2 = pack(one_ma, one_ma);
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 ahead = unpack(fma2(px.behind[k], minus_one, feature[k]));
        sum = fmaf(ahead.x, px.d[2 * k], sum);
        sum = fmaf(ahead.y, px.d[2 * k + 1], sum);
        px.behind[k] = fma2(alpha2, feature[k], mul2(one_ma2, px.behind[k]));
    }
    const float dL_dalpha = sum * px.T - px.T_final_bg * inv_1ma;
    return make_float2(alpha * px.T, opacity * G * dL_dalpha);
}

// The 16 gradient terms of one Gaussian, summed over pixels.
struct BwdSums {
    float x, y, ax, ay;          // h (a dx + b dy), h (c dy + b dx) and their absolute values
    float xx, xy, yy, o;         // h dx dx, h dx dy, h dy dy, h
    float f[CGX_NCH + CGX_NMAP];
};

__device__ __forceinline__ void bwd_accumulate(BwdSums& s, const float2 wh, const float dx, const float dy,
                                               const float ca, const float cb, const float cc, const float4 d0,
                                               const float4 d1)
{
    const float hx = wh.y * dx, hy = wh.y * dy;
    const float tx = hx * ca + hy * cb, ty = hy * cc + hx * cb;
    s.x += tx;
    s.y += ty;
    s.ax += fabsf(tx);
    s.ay += fabsf(ty);
    s.xx += hx * dx;
    s.xy += hx * dy;
    s.yy += hy * dy;
    s.o += wh.y;
    s.f[0] += wh.x * d0.x;
    s.f[1] += wh.x * d0.y;
    s.f[2] += wh.x * d0.z;
    s.f[3] += wh.x * d0.w;
    s.f[4] += wh.x * d1.x;
    s.f[5] += wh.x * d1.y;
    s.f[6] += wh.x * d1.z;
    s.f[7] += wh.x * d1.w;
}

// Adds the sums of the lane `o` away.
__device__ __forceinline__ void bwd_combine(BwdSums& s, int o)
{
    float* p = &s.x;
    static_assert(sizeof(BwdSums) == 16 * sizeof(float), "sixteen terms");
#pragma unroll
    for (int k = 0; k < 16; k++) p[k] += __shfl_xor_sync(0xffffffffu, p[k], o);
}

// Adds the sums of one Gaussian, either straight to the caller's tensors (12 atomics to 5-7 sectors of memory) or to
// its row of a table (4 atomics of 16 bytes to 2 sectors) that bwd_unpack_kernel spreads over the tensors afterwards.
template <bool TABLE>
__device__ __forceinline__ void bwd_add(const BwdOut& out, const BwdSums& s, const size_t id, const float opacity,
                                        const float ddelx_dx, const float ddely_dy, const bool render_geo)
{
    const float gx = -ddelx_dx * s.x, gy = -ddely_dy * s.y, ax = ddelx_dx * s.ax, ay = ddely_dy * s.ay;
    const float4 con = make_float4(-0.5f * s.xx, -0.5f * s.xy, -0.5f * s.yy, s.o / opacity);
    if (TABLE) {
        float4* row = out.table + 4 * id;
        atomicAdd(row, make_float4(gx, gy, ax, ay));
        atomicAdd(row + 1, con);
        atomicAdd(row + 2, make_float4(s.f[0], s.f[1], s.f[2], s.f[3]));
        if (render_geo) atomicAdd(row + 3, make_float4(s.f[4], s.f[5], s.f[6], s.f[7]));
        return;
    }
    if (out.vec) {
        atomicAdd(reinterpret_cast<float2*>(out.means2D) + id, make_float2(gx, gy));
        atomicAdd(reinterpret_cast<float4*>(out.conic) + id, con);
    } else {
        atomicAdd(out.means2D + 2 * id, gx);
        atomicAdd(out.means2D + 2 * id + 1, gy);
        atomicAdd(out.conic + 4 * id, con.x);
        atomicAdd(out.conic + 4 * id + 1, con.y);
        atomicAdd(out.conic + 4 * id + 2, con.z);
        atomicAdd(out.conic + 4 * id + 3, con.w);
    }
    atomicAdd(out.abs2D + 3 * id, ax);
    atomicAdd(out.abs2D + 3 * id + 1, ay);
#pragma unroll
    for (int k = 0; k < CGX_NCH; k++) atomicAdd(out.rgb + 3 * id + k, s.f[k]);
    if (render_geo) {
#pragma unroll
        for (int k = 0; k < CGX_NMAP; k++) atomicAdd(out.all_map + 5 * id + k, s.f[CGX_NCH + k]);
    }
}

// Clears the table rows of the Gaussians that are in some tile's list (the others are neither added to nor read).
// A warp looks at 128 flags at a time and then clears the rows among them eight at a time, four lanes each.
__global__ void __launch_bounds__(256)
bwd_clear_kernel(int P, const uint32_t* __restrict__ tiles_touched, float4* __restrict__ table, const int vec_ok)
{
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * 8;
    for (int base = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 128; base < P; base += warps * 128) {
        uint32_t f[4];
        const int i = base + 4 * lane;
        if (vec_ok && i + 4 <= P) {
            const uint4 v = *reinterpret_cast<const uint4*>(tiles_touched + i);
            f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) f[k] = i + k < P ? tiles_touched[i + k] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t m = __ballot_sync(0xffffffffu, f[k] != 0);      // lanes whose k-th Gaussian has tiles
            while (m) {
                uint32_t t = m;
#pragma unroll
                for (int q = 0; q < 7; q++)
                    if (q < (lane >> 2)) t &= t - 1;
                if (t) table[4 * (size_t)(base + 4 * (__ffs(t) - 1) + k) + (lane & 3)] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int q = 0; q < 8; q++) m &= m - 1;
            }
        }
    }
}

// One CTA's slice of the five tensors, as it lies in memory.
constexpr int UNPACK_ROWS = 256;
struct __align__(16) UnpackSlice {
    float xy[2 * UNPACK_ROWS], abs2D[3 * UNPACK_ROWS], con[4 * UNPACK_ROWS], rgb[3 * UNPACK_ROWS], map[5 * UNPACK_ROWS];
};

__device__ __forceinline__ void bulk_store(void* dst_gmem, const void* src_smem, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst_gmem),
                 "r"((uint32_t)__cvta_generic_to_shared(src_smem)), "r"(bytes)
                 : "memory");
}

// Table -> the caller's tensors, every element written (zeros for Gaussians without tiles): HBM-bound, 68 B per
// Gaussian out, 4 in, 64 more where it has tiles.  Persistent CTAs rearrange 256 rows at a time in shared memory and
// send each tensor's slice off as one bulk copy, which runs beside the next 256 rows' loads (two buffers).
__global__ void __launch_bounds__(UNPACK_ROWS)
bwd_unpack_kernel(int P, const uint32_t* __restrict__ tiles_touched, const BwdOut out, const bool render_geo,
                  const int vec_ok)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    UnpackSlice* buf = reinterpret_cast<UnpackSlice*>(smem_raw);
    const int t = threadIdx.x;
    int which = 0;
    for (int base = blockIdx.x * UNPACK_ROWS; base < P; base += gridDim.x * UNPACK_ROWS, which ^= 1) {
        UnpackSlice& s = buf[which];
        const int n = min(UNPACK_ROWS, P - base);
        float4 r[4] = {};
        if (t < n && tiles_touched[base + t]) {
            const float4* row = out.table + 4 * (size_t)(base + t);
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < 3 || render_geo) r[k] = __ldcs(row + k);
            if (!render_geo) r[2].w = 0.f;
        }
        // the copies that still read this buffer were queued two rounds ago
        if (t == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        __syncthreads();
        *reinterpret_cast<float2*>(s.xy + 2 * t) = make_float2(r[0].x, r[0].y);
        s.abs2D[3 * t] = r[0].z, s.abs2D[3 * t + 1] = r[0].w, s.abs2D[3 * t + 2] = 0.f;
        *reinterpret_cast<float4*>(s.con + 4 * t) = r[1];
        s.rgb[3 * t] = r[2].x, s.rgb[3 * t + 1] = r[2].y, s.rgb[3 * t + 2] = r[2].z;
        const float m[5] = {r[2].w, r[3].x, r[3].y, r[3].z, r[3].w};
#pragma unroll
        for (int k = 0; k < 5; k++) s.map[5 * t + k] = m[k];
        if (n == UNPACK_ROWS && vec_ok) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
            if (t == 0) {
                bulk_store(out.means2D + (size_t)base * 2, s.xy, sizeof(s.xy));
                bulk_store(out.abs2D + (size_t)base * 3, s.abs2D, sizeof(s.abs2D));
                bulk_store(out.conic + (size_t)base * 4, s.con, sizeof(s.con));
                bulk_store(out.rgb + (size_t)base * 3, s.rgb, sizeof(s.rgb));
                bulk_store(out.all_map + (size_t)base * 5, s.map, sizeof(s.map));
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        } else {
            __syncthreads();
            block_store_rows<2>(out.means2D + (size_t)base * 2, s.xy, n, vec_ok);
            block_store_rows<3>(out.abs2D + (size_t)base * 3, s.abs2D, n, vec_ok);
            block_store_rows<4>(out.conic + (size_t)base * 4, s.con, n, vec_ok);
            block_store_rows<3>(out.rgb + (size_t)base * 3, s.rgb, n, vec_ok);
            block_store_rows<5>(out.all_map + (size_t)base * 5, s.map, n, vec_ok);
            if (t == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");    // an empty group: keeps the count
        }
    }
    if (t == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Plain walk, one tile per CTA: every pixel looks at every Gaussian of its list, every contribution is added with
// its own atomics.  Slow; the yardstick of the tests (cgx_set_render_variant(0)).
__global__ void __launch_bounds__(RENDER_THREADS)
render_bwd_plain_kernel(const uint2* __restrict__ ranges, const uint32_t* __restrict__ point_list, int W, int H,
                        float fx, float fy, const float* __restrict__ bg_color, const Record* __restrict__ records,
                        const float* __restrict__ all_map_pixels, const float* __restrict__ final_Ts,
                        const uint32_t* __restrict__ n_contrib, const uint8_t* __restrict__ compute_locally,
                        const float* __restrict__ dL_dpixels, const float* __restrict__ dL_dout_all_maps,
                        const float* __restrict__ dL_dout_plane_depths, const bool render_geo, BwdOut out, int P,
                        int walk)
{
    const uint32_t block_id = blockIdx.y * gridDim.x + blockIdx.x;
    const uint32_t x = blockIdx.x * CGX_BLOCK_X + threadIdx.x % CGX_BLOCK_X;
    const uint32_t y = blockIdx.y * CGX_BLOCK_Y + threadIdx.x / CGX_BLOCK_X;
    const bool rows_first = walk ? walk == 1 : !scene_is_dense(records, P, threadIdx.x & 31);
    if (!compute_locally[block_id] || x >= W || y >= H) return;
    const uint32_t pix_id = W * y + x;
    const float2 pixf = {(float)x, (float)y};
    const float2 ray = {(float)((pixf.x - W * 0.5) / fx), (float)((pixf.y - H * 0.5) / fy)};
    BwdPixel px;
    bwd_pixel_init(px, true, pix_id, (size_t)H * W, ray, bg_color, final_Ts, all_map_pixels, dL_dpixels,
                   dL_dout_all_maps, dL_dout_plane_depths, render_geo);
    const uint32_t start = ranges[block_id].x;
    for (int k = (int)n_contrib[pix_id] - 1; k >= 0; k--) {
        const uint32_t id = point_list[start + k];
        const Record r = records[id];
        float2 d;
        float G, alpha;
        if (!eval_alpha(make_float2(r.q0.x, r.q0.y), r.q1, pixf, d, G, alpha, rows_first)) continue;
        const float2 wh = bwd_contribution(px, r, r.q1.w, G, alpha);
        BwdSums s = {};
        bwd_accumulate(s, wh, d.x, d.y, r.q1.x, r.q1.y, r.q1.z, make_float4(px.d[0], px.d[1], px.d[2], px.d[3]),
                       make_float4(px.d[4], px.d[5], px.d[6], px.d[7]));
        bwd_add<false>(out, s, id, r.q1.w, 0.5f * W, 0.5f * H, render_geo);
    }
}

#ifndef CGX_BWD_WARPS
#define CGX_BWD_WARPS 4
#endif
constexpr int BWD_WARPS = CGX_BWD_WARPS;
constexpr int BWD_SPLIT = RENDER_WARPS / BWD_WARPS;      // CTAs per tile

struct BwdSmem {
    ScanSmem<BWD_WARPS> scan;
    QueueSmem queue[BWD_WARPS];
    float4 pix[BWD_WARPS][2][32];           // cotangents of the warp's pixels: first and second four
    float2 wh[BWD_WARPS][BWD_CAP];
    uint2 visit[BWD_WARPS][32];             // pixels of a visit that contribute, its first entry in wh
    int last;                                  // the tile's last contributor
};

// Half a 16x16 tile per CTA, back to front over the tile's list.  Every warp owns an 8x4 pixel block and collects the
// Gaussians that may reach it ("visits") in a queue of 32, across the culled stretches of the list, so that the two
// steps below run on full queues:
//   step A, lane = pixel:  walks its own contributors, keeps (alpha T, opacity G dL/dalpha) of each in shared memory;
//   step B, lane = visit:  sums the 16 gradient terms of its Gaussian over the visit's pixels in registers, then adds
//                          them with one atomic per term (or per four).
// Bound by instruction issue and by shared-memory bandwidth (every lane reads another record or pixel): step A is run
// as often as the busiest of 32 pixels contributes (8.6 times per queue on the 6 M-Gaussian ring views, 4.8 being the
// average), step B as often as the widest of 32 visits has pixels (13.8 against 5.5).  Keeping two numbers per
// contribution and summing by visit replaced staging all sixteen terms per contribution and summing them by rows.
// Four warps per CTA: with eight a fifth of the time went into waiting for the slowest at the barriers.  Per camera of
// 6 M Gaussians at 1600x1200: 1.21 -> 0.70 ms; one 1920x1080 view of 1 M: 0.35 -> 0.26; two 3840x2160 views of a
// 20 M-Gaussian city: 2.34 -> 1.70 (of that 0.62 against 0.44 by the table's clearing and unpacking).
template <bool TABLE>
__global__ void __launch_bounds__(32 * BWD_WARPS, CGX_BWD_MIN_CTAS)
render_bwd_kernel(const uint2* __restrict__ ranges, const uint32_t* __restrict__ point_list, int W, int H, float fx,
                  float fy, const float* __restrict__ bg_color, const Record* __restrict__ records,
                  const float* __restrict__ all_map_pixels, const float* __restrict__ final_Ts,
                  const uint32_t* __restrict__ n_contrib, const uint8_t* __restrict__ compute_locally,
                  const float* __restrict__ dL_dpixels, const float* __restrict__ dL_dout_all_maps,
                  const float* __restrict__ dL_dout_plane_depths, const bool render_geo, BwdOut out, int P,
                  int walk)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    BwdSmem& sm = *reinterpret_cast<BwdSmem*>(smem_raw);
    const uint32_t tile_y = blockIdx.y / BWD_SPLIT;
    const uint32_t block_id = tile_y * gridDim.x + blockIdx.x;
    if (!compute_locally[block_id]) return;
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const uint32_t lx = (warp & 1) * 8 + (lane & 7), ly = (warp >> 1) * 4 + (lane >> 3);   // 8x4 block per warp
    const uint2 pix_min = {blockIdx.x * CGX_BLOCK_X, blockIdx.y * (CGX_BLOCK_Y / BWD_SPLIT)};
    const uint2 pix = {pix_min.x + lx, pix_min.y + ly};
    const uint32_t pix_id = W * pix.y + pix.x;
    const float2 pixf = {(float)pix.x, (float)pix.y};
    const bool inside = pix.x < W && pix.y < H;
    const uint2 range = ranges[block_id];
    if (range.x >= range.y) return;
    // pixels outside the image take part in the votes only: nothing is ever "before their last contributor"
    const int last_contributor = inside ? n_contrib[pix_id] : 0;
    const int warp_last = __reduce_max_sync(0xffffffffu, last_contributor);
    const bool rows_first = walk ? walk == 1 : !scene_is_dense(records, P, lane);      // see eval_alpha
    if (tid == 0) sm.last = 0;
    __syncthreads();
    if (lane == 0) atomicMax(&sm.last, warp_last);
    __syncthreads();
    // what lies behind the tile's last contributor is never looked at: the walk starts there
    const int total = sm.last;
    // first pixel of this warp's block
    const float sx0 = (float)(pix_min.x + (warp & 1) * 8), sy0 = (float)(pix_min.y + (warp >> 1) * 4);

    BwdPixel px;
    {
        // double arithmetic (W * 0.5 is a double expression), narrowed to float afterwards
        const float2 ray = {(float)((pixf.x - W * 0.5) / fx), (float)((pixf.y - H * 0.5) / fy)};
        bwd_pixel_init(px, inside, pix_id, (size_t)H * W, ray, bg_color, final_Ts, all_map_pixels, dL_dpixels,
                       dL_dout_all_maps, dL_dout_plane_depths, render_geo);
    }
    sm.pix[warp][0][lane] = make_float4(px.d[0], px.d[1], px.d[2], px.d[3]);
    sm.pix[warp][1][lane] = make_float4(px.d[4], px.d[5], px.d[6], px.d[7]);
    const uint32_t lanes_below = (1u << lane) - 1u;
    QueueSmem& queue = sm.queue[warp];
    float2* wh_rows = sm.wh[warp];
    int nq = 0;                        // visits in the queue (warp-uniform)

    for (int start = 0; start < total; start += SCAN_SLOTS) {
        const int n = min(SCAN_SLOTS, total - start);
        const int base_idx = total - 1 - start;              // slot s is entry base_idx - s of the tile's list
        if (start) __syncthreads();
        scan_entries(sm.scan, point_list + range.x + base_idx, -1, n, records, (float)pix_min.x, (float)pix_min.y);
        __syncthreads();
        // nearer to the back than the warp's last contributor: none of its pixels sees it
        const int first = max(0, base_idx - warp_last + 1);
        const bool last = start + SCAN_SLOTS >= total;
        const int n_hits = first < n ? collect_hits(sm.scan, warp, lane, first, n) : 0;
        for (int base = 0; base < n_hits || (last && nq > 0); base += 32) {
            uint32_t pm = 0;
            int slot = 0;
            float4 q0, q1;
            if (base + lane < n_hits) {
                slot = sm.scan.hits[warp][base + lane];
                q0 = sm.scan.q0[slot];
                q1 = sm.scan.q1[slot];
                pm = block_mask(q0, q1, sx0, sy0);
            }
            uint32_t fresh = __ballot_sync(0xffffffffu, pm != 0);
            do {
                fresh = queue_push(queue, nq, fresh, lane, pm, q0, q1, sm.scan.id[slot], base_idx - slot, records);
                // on with the next hits until the queue is full or the list has ended
                if (nq < 32 && !(last && base + 32 >= n_hits)) break;
                copy_async_wait();
                __syncwarp();

                uint32_t vmask = lane < nq ? queue.mask[lane] : 0u;          // lane = visit: its pixels
                uint32_t mine_all = warp_transpose32(vmask, lane);           // lane = pixel: its visits
                // a pixel that saturated stops before the end of the list: drop the visits behind its last contributor
                if (__any_sync(0xffffffffu, mine_all != 0 && queue.idx[0] >= last_contributor)) {
                    int lo = 0, hi = nq;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (queue.idx[mid] >= last_contributor) lo = mid + 1;
                        else hi = mid;
                    }
                    mine_all = lo >= 32 ? 0u : (mine_all & (0xffffffffu << lo));
                    vmask = warp_transpose32(mine_all, lane);
                }
                const int cnt = __popc(vmask);
                int cum = cnt;
#pragma unroll
                for (int dd = 1; dd < 32; dd <<= 1) {
                    const int up = __shfl_up_sync(0xffffffffu, cum, dd);
                    if (lane >= dd) cum += up;
                }
                int v0 = 0;            // visits [v0, v0 + g): as many as the table holds
                while (v0 < nq) {
                    const int before = v0 ? __shfl_sync(0xffffffffu, cum, v0 - 1) : 0;
                    const uint32_t group = __ballot_sync(0xffffffffu, lane >= v0 && lane < nq && cum - before <= BWD_CAP);
                    const int g = __popc(group);
                    sm.visit[warp][lane] = make_uint2(vmask, (uint32_t)(cum - cnt - before));
                    __syncwarp();
                    // ---- step A (the cotangents come from shared memory: no registers for them in step B)
                    const float4 d0 = sm.pix[warp][0][lane], d1 = sm.pix[warp][1][lane];
                    const float dd[CGX_NCH + CGX_NMAP] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
                    for (int k = 0; k < CGX_NCH + CGX_NMAP; k++) px.d[k] = dd[k];
                    for (uint32_t mine = mine_all & group; mine; mine &= mine - 1) {
                        const int v = __ffs(mine) - 1;
                        const Record& r = queue.rec[v];
                        const uint2 vs = sm.visit[warp][v];
                        const float4 con_o = r.q1;
                        float2 d, wh = make_float2(0.f, 0.f);
                        float G, alpha;
                        if (eval_alpha(*reinterpret_cast<const float2*>(&r.q0), con_o, pixf, d, G, alpha, rows_first))
                            wh = bwd_contribution(px, r, con_o.w, G, alpha);
                        wh_rows[vs.y + __popc(vs.x & lanes_below)] = wh;
                    }
                    __syncwarp();
                    // ---- step B: few visits (large splats, whose pixels fill the table, or the end of a list) are
                    // summed by two or four lanes each, every one half or a quarter of the block's rows
                    const int split = g <= 8 ? 4 : g <= 16 ? 2 : 1;
                    const int v = v0 + (split == 4 ? lane >> 2 : split == 2 ? lane >> 1 : lane);
                    const int part = lane & (split - 1);
                    uint32_t bits = 0;
                    BwdSums s = {};
                    float opacity = 1.f;
                    if (v < v0 + g) {
                        const uint2 vs = sm.visit[warp][v];
                        const uint32_t part_mask = split == 4 ? 0xFFu << (8 * part) : split == 2 ? 0xFFFFu << (16 * part)
                                                                                              : 0xffffffffu;
                        bits = vs.x & part_mask;
                        const float2 xy = *reinterpret_cast<const float2*>(&queue.rec[v].q0);
                        const float4 con = queue.rec[v].q1;
                        opacity = con.w;
                        const float2* row = wh_rows + vs.y + __popc(vs.x & ((part_mask & (0u - part_mask)) - 1u));
                        for (uint32_t left = bits; left; left &= left - 1) {
                            const int p = __ffs(left) - 1;
                            // the pixel's coordinates, exactly: 2^23 + (p & 7) by its bits, minus 2^23
                            const float dx = xy.x - (__uint_as_float(0x4B000000u | (p & 7)) + (sx0 - 8388608.f));
                            const float dy = xy.y - (__uint_as_float(0x4B000000u | (p >> 3)) + (sy0 - 8388608.f));
                            bwd_accumulate(s, *row++, dx, dy, con.x, con.y, con.z, sm.pix[warp][0][p],
                                           sm.pix[warp][1][p]);
                        }
                        bits = part ? 0u : vs.x;
                    }
                    if (split >= 2) bwd_combine(s, 1);
                    if (split == 4) bwd_combine(s, 2);
                    if (bits) bwd_add<TABLE>(out, s, (size_t)queue.id[v], opacity, 0.5f * W, 0.5f * H, render_geo);
                    __syncwarp();
                    v0 += g;
                }
                nq = 0;
            } while (fresh);
        }
    }
}

// Clears up to five float arrays in one launch (grid-stride over the concatenated index space).
struct ZeroJobs {
    float* ptr[5];
    long long n[5];
};
__global__ void __launch_bounds__(256) zero_arrays_kernel(ZeroJobs z)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        float* p = z.ptr[k];
        const long long n = z.n[k];
        if (!p) continue;
        if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
            float4* p4 = reinterpret_cast<float4*>(p);
            const long long n4 = n >> 2;
            for (long long i = t0; i < n4; i += stride) p4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (long long i = (n4 << 2) + t0; i < n; i += stride) p[i] = 0.f;
        } else {
            for (long long i = t0; i < n; i += stride) p[i] = 0.f;
        }
    }
}

}  // namespace cgx

using namespace cgx;

// P records, then the density counters the forward pass leaves for the backward pass
extern "C" int cgx_render_density_words(void) { return 2 * DENSITY_SLOTS; }
extern "C" int cgx_render_dense_threshold(void) { return DENSE_PIXELS_PER_VISIT; }

extern "C" size_t cgx_render_records_bytes(int P) { return (size_t)(P > 0 ? P : 0) * sizeof(Record) + DENSITY_BYTES; }

// Test-only switch (cgx_raster_testing.h): bit 0 clear = the plain walks (every pixel looks at every Gaussian).
static int g_render_variant = 1;

extern "C" int cgx_set_render_variant(int variant)
{
    g_render_variant = variant;
    return CGX_OK;
}

static int render_fwd(bool pack_first, int P, int W, int H, float tanfovx, float tanfovy, const uint32_t* ranges,
                              const uint32_t* point_list, const int32_t* radii, const float* means2D, const float* rgb, const float* all_map,
                              const float* conic_opacity, const uint8_t* compute_locally, const float* bg,
                              int render_geo, void* records, float* final_T, uint32_t* n_contrib,
                              uint32_t* n_contrib2loss, float* out_color, int32_t* out_observe, float* out_all_map,
                              float* out_plane_depth, int32_t* n_render_t, int32_t* n_consider_t, int32_t* n_contrib_t,
                              void* stream)
{
    if (P < 0 || W <= 0 || H <= 0) return CGX_EINVAL;
    if (!ranges || !compute_locally || !bg || !final_T || !n_contrib || !n_contrib2loss || !out_color ||
        !out_all_map || !out_plane_depth || !n_render_t || !n_consider_t || !n_contrib_t)
        return CGX_EINVAL;
    if (P > 0 && (!means2D || !rgb || !conic_opacity || !records || !out_observe || (render_geo && !all_map)))
        return CGX_EINVAL;
    if (P > 0 && (((uintptr_t)means2D & 7) || !aligned16(conic_opacity) || !aligned16(records))) return CGX_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    if (P > 0 && pack_first)
        pack_records_kernel<<<(P + 255) / 256, 256, 0, st>>>(P, radii, (const float2*)means2D,
                                                             (const float4*)conic_opacity, rgb, all_map, render_geo,
                                                             (Record*)records, out_observe);
    const float focal_y = H / (2.0f * tanfovy);
    const float focal_x = W / (2.0f * tanfovx);
    const dim3 grid((W + CGX_BLOCK_X - 1) / CGX_BLOCK_X, (H + CGX_BLOCK_Y - 1) / CGX_BLOCK_Y, 1);
    const dim3 block(RENDER_THREADS, 1, 1);
    const bool cull = g_render_variant & 1;
    auto kernel = cull ? render_fwd_kernel<true> : render_fwd_kernel<false>;
    if (!(cull ? allow_shared<render_fwd_kernel<true>>((int)sizeof(FwdSmem))
               : allow_shared<render_fwd_kernel<false>>((int)sizeof(FwdSmem))))
        return CGX_ECUDA;
    kernel<<<grid, block, sizeof(FwdSmem), st>>>(
        (const uint2*)ranges, point_list, W, H, focal_x, focal_y, float(W * 0.5f), float(H * 0.5f),
        (const Record*)records, final_T, n_contrib, n_contrib2loss, compute_locally, bg, out_color, out_observe,
        out_all_map, out_plane_depth, render_geo != 0, n_render_t, n_consider_t, n_contrib_t,
        P > 0 ? reinterpret_cast<unsigned long long*>((Record*)records + P) : nullptr);
    return check_launch(P > 0 && pack_first ? 2 : 1);
}

extern "C" int cgx_render_fwd(int P, int W, int H, float tanfovx, float tanfovy, const uint32_t* ranges,
                              const uint32_t* point_list, const int32_t* radii, const float* means2D,
                              const float* rgb, const float* all_map, const float* conic_opacity,
                              const uint8_t* compute_locally, const float* bg, int render_geo, void* records,
                              float* final_T, uint32_t* n_contrib, uint32_t* n_contrib2loss, float* out_color,
                              int32_t* out_observe, float* out_all_map, float* out_plane_depth, int32_t* n_render_t,
                              int32_t* n_consider_t, int32_t* n_contrib_t, void* stream)
{
    return render_fwd(true, P, W, H, tanfovx, tanfovy, ranges, point_list, radii, means2D, rgb, all_map, conic_opacity, compute_locally,
                      bg, render_geo, records, final_T, n_contrib, n_contrib2loss, out_color, out_observe, out_all_map,
                      out_plane_depth, n_render_t, n_consider_t, n_contrib_t, stream);
}

extern "C" int cgx_render_fwd_packed(int P, int W, int H, float tanfovx, float tanfovy, const uint32_t* ranges,
                                     const uint32_t* point_list, const int32_t* radii, const float* means2D,
                                     const float* rgb, const float* all_map, const float* conic_opacity,
                                     const uint8_t* compute_locally, const float* bg, int render_geo, void* records,
                                     float* final_T, uint32_t* n_contrib, uint32_t* n_contrib2loss, float* out_color,
                                     int32_t* out_observe, float* out_all_map, float* out_plane_depth,
                                     int32_t* n_render_t, int32_t* n_consider_t, int32_t* n_contrib_t, void* stream)
{
    return render_fwd(false, P, W, H, tanfovx, tanfovy, ranges, point_list, radii, means2D, rgb, all_map, conic_opacity, compute_locally,
                      bg, render_geo, records, final_T, n_contrib, n_contrib2loss, out_color, out_observe, out_all_map,
                      out_plane_depth, n_render_t, n_consider_t, n_contrib_t, stream);
}

extern "C" int cgx_render_pack(int P, const int32_t* radii, const float* means2D, const float* rgb, const float* all_map,
                               const float* conic_opacity, int render_geo, void* records, int32_t* out_observe,
                               void* stream)
{
    if (P < 0) return CGX_EINVAL;
    if (P == 0) return CGX_OK;
    if (!means2D || !rgb || !conic_opacity || !records || !out_observe || (render_geo && !all_map)) return CGX_EINVAL;
    if (((uintptr_t)means2D & 7) || !aligned16(conic_opacity) || !aligned16(records)) return CGX_EINVAL;
    pack_records_kernel<<<(P + 255) / 256, 256, 0, (cudaStream_t)stream>>>(P, radii, (const float2*)means2D,
                                                                           (const float4*)conic_opacity, rgb, all_map,
                                                                           render_geo, (Record*)records, out_observe);
    return check_launch();
}

extern "C" int cgx_tile_stats(int W, int H, const uint32_t* ranges, const uint32_t* n_contrib_px,
                              const uint32_t* n_contrib2loss_px, const uint8_t* compute_locally, int32_t* n_render,
                              int32_t* n_consider, int32_t* n_contrib, void* stream)
{
    if (W <= 0 || H <= 0 || !ranges || !n_contrib_px || !n_contrib2loss_px || !compute_locally || !n_render ||
        !n_consider || !n_contrib)
        return CGX_EINVAL;
    const dim3 grid((W + CGX_BLOCK_X - 1) / CGX_BLOCK_X, (H + CGX_BLOCK_Y - 1) / CGX_BLOCK_Y, 1);
    const dim3 block(CGX_BLOCK_X, CGX_BLOCK_Y, 1);
    tile_stats_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(W, H, (const uint2*)ranges, n_contrib_px,
                                                               n_contrib2loss_px, compute_locally, n_render,
                                                               n_consider, n_contrib);
    return check_launch();
}

extern "C" size_t cgx_render_bwd_workspace_bytes(int P) { return (size_t)(P > 0 ? P : 0) * 16 * sizeof(float); }

extern "C" int cgx_render_bwd_table(int P, int W, int H, float tanfovx, float tanfovy, const uint32_t* ranges,
                              const uint32_t* point_list, const float* bg, const void* records,
                              const float* all_map_pixels, const float* final_T, const uint32_t* n_contrib,
                              const uint8_t* compute_locally, const float* dL_dcolor, const float* dL_dout_all_map,
                              const float* dL_dout_plane_depth, int render_geo, float* dL_dmeans2D,
                              float* dL_dmeans2D_abs, float* dL_dconic_opacity, float* dL_drgb, float* dL_dall_map,
                              int walk, const uint32_t* tiles_touched, void* workspace, size_t workspace_bytes, void* stream)
{
    if (P < 0 || W <= 0 || H <= 0 ) return CGX_EINVAL;
    if (P == 0) return CGX_OK;
    if (!ranges) return CGX_EINVAL;
    if (!bg || !records || !final_T || !n_contrib || !compute_locally || !dL_dcolor || !dL_dmeans2D ||
        !dL_dmeans2D_abs || !dL_dconic_opacity || !dL_drgb || !dL_dall_map)
        return CGX_EINVAL;
    if (render_geo && (!all_map_pixels || !dL_dout_all_map || !dL_dout_plane_depth)) return CGX_EINVAL;
    if (!aligned16(records)) return CGX_EINVAL;
    if (workspace && (!tiles_touched || !aligned16(workspace))) return CGX_EINVAL;
    if (workspace && workspace_bytes < cgx_render_bwd_workspace_bytes(P)) return CGX_ENOMEM;
    cudaStream_t st = (cudaStream_t)stream;
    const bool plain = !(g_render_variant & 1);
    const bool table = workspace && !plain;
    if (table) {
        bwd_clear_kernel<<<min((P + 1023) / 1024, 148 * 8), 256, 0, st>>>(P, tiles_touched, (float4*)workspace,
                                                                          aligned16(tiles_touched));
    } else {
        // the five gradient arrays start at zero: one launch clears all of them
        ZeroJobs z;
        float* arrs[5] = {dL_dmeans2D, dL_dmeans2D_abs, dL_dconic_opacity, dL_drgb, dL_dall_map};
        const int widths[5] = {2, 3, 4, 3, 5};
        for (int k = 0; k < 5; k++) {
            z.ptr[k] = arrs[k];
            z.n[k] = (long long)P * widths[k];
        }
        zero_arrays_kernel<<<148 * 8, 256, 0, st>>>(z);
    }

    BwdOut out = {dL_dmeans2D, dL_dmeans2D_abs, dL_dconic_opacity, dL_drgb, dL_dall_map,
                  ((uintptr_t)dL_dmeans2D & 7) == 0 && aligned16(dL_dconic_opacity), (float4*)workspace};
    const float focal_y = H / (2.0f * tanfovy);
    const float focal_x = W / (2.0f * tanfovx);
    const dim3 grid((W + CGX_BLOCK_X - 1) / CGX_BLOCK_X, (H + CGX_BLOCK_Y - 1) / CGX_BLOCK_Y, 1);
    const dim3 block(RENDER_THREADS, 1, 1);
    if (plain) {
        render_bwd_plain_kernel<<<grid, block, 0, st>>>(
            (const uint2*)ranges, point_list, W, H, focal_x, focal_y, bg, (const Record*)records, all_map_pixels,
            final_T, n_contrib, compute_locally, dL_dcolor, dL_dout_all_map, dL_dout_plane_depth, render_geo != 0, out, P,
        walk);
        return check_launch(2);
    }
    auto kernel = table ? render_bwd_kernel<true> : render_bwd_kernel<false>;
    if (!(table ? allow_shared<render_bwd_kernel<true>>((int)sizeof(BwdSmem))
                : allow_shared<render_bwd_kernel<false>>((int)sizeof(BwdSmem))))
        return CGX_ECUDA;
    kernel<<<dim3(grid.x, grid.y * BWD_SPLIT), 32 * BWD_WARPS, sizeof(BwdSmem), st>>>(
        (const uint2*)ranges, point_list, W, H, focal_x, focal_y, bg, (const Record*)records, all_map_pixels, final_T,
        n_contrib, compute_locally, dL_dcolor, dL_dout_all_map, dL_dout_plane_depth, render_geo != 0, out, P,
        walk);
    if (table) {
        const int vec_ok = aligned16(dL_dmeans2D) && aligned16(dL_dmeans2D_abs) && aligned16(dL_dconic_opacity) &&
                           aligned16(dL_drgb) && aligned16(dL_dall_map);
        const int smem = 2 * sizeof(UnpackSlice);        // six CTAs per SM
        if (!allow_shared<bwd_unpack_kernel>(smem)) return CGX_ECUDA;
        bwd_unpack_kernel<<<min((P + UNPACK_ROWS - 1) / UNPACK_ROWS, 148 * 6), UNPACK_ROWS, smem, st>>>(
            P, tiles_touched, out, render_geo != 0, vec_ok);
    }
    return check_launch(table ? 3 : 2);
}

extern "C" int cgx_render_bwd(int P, int W, int H, float tanfovx, float tanfovy, const uint32_t* ranges,
                              const uint32_t* point_list, const float* bg, const void* records,
                              const float* all_map_pixels, const float* final_T, const uint32_t* n_contrib,
                              const uint8_t* compute_locally, const float* dL_dcolor, const float* dL_dout_all_map,
                              const float* dL_dout_plane_depth, int render_geo, float* dL_dmeans2D,
                              float* dL_dmeans2D_abs, float* dL_dconic_opacity, float* dL_drgb, float* dL_dall_map,
                              int walk, void* stream)
{
    return cgx_render_bwd_table(P, W, H, tanfovx, tanfovy, ranges, point_list, bg, records, all_map_pixels, final_T,
                                n_contrib, compute_locally, dL_dcolor, dL_dout_all_map, dL_dout_plane_depth, render_geo,
                                dL_dmeans2D, dL_dmeans2D_abs, dL_dconic_opacity, dL_drgb, dL_dall_map, walk, nullptr,
                                nullptr, 0, stream);
}
