// Statistics that the densifier reads (the consumer side of the rasterizer's contract): per Gaussian the screen-space
// gradient norms and visits over a batch's cameras, and per anchor / per slot the sums of the anchor model.
// HBM-bound; what they replaced was a dozen tensor operations per camera, and four masked scatters (each a device-wide
// scan of its mask) per iteration.
#include "cgx_common.cuh"

namespace cgx {

constexpr int STAT_CAMS = 16;
struct DensifyBatch {
    int B;
    const int* radii[STAT_CAMS];
    const float2* grad[STAT_CAMS];
};

// 400 k Gaussians, four cameras: one launch of 11 us instead of 24 of 95 us together.
__global__ void __launch_bounds__(256)
densify_kernel(int P, const __grid_constant__ DensifyBatch d, float* __restrict__ grad_accum, float* __restrict__ denom,
               int* __restrict__ max_radii)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= P) return;
    float sum = grad_accum[i], visits = denom[i];
    int largest = max_radii ? max_radii[i] : 0;
    for (int b = 0; b < d.B; b++) {
        const int r = __ldg(d.radii[b] + i);
        if (r > 0) {
            const float2 g = __ldg(d.grad[b] + i);
            sum += sqrtf(g.x * g.x + g.y * g.y);
            visits += 1.f;
        }
        largest = max(largest, r);
    }
    grad_accum[i] = sum;
    denom[i] = visits;
    if (max_radii) max_radii[i] = largest;
}

constexpr int ANCHORS = 256;         // anchors per CTA, and per warp that counts
constexpr int SLOT_CHUNK = 4096;     // slots per partial count

// Sum of n <= 4096 bytes that are 0 or 1, over the CTA's 256 threads.
__device__ __forceinline__ int count_bytes(const uint8_t* __restrict__ p, int n, int* s_red)
{
    int c = 0;
    if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
        for (int i = threadIdx.x; i < n >> 4; i += 256) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p) + i);
            c += __popc(v.x & 0x01010101u) + __popc(v.y & 0x01010101u) + __popc(v.z & 0x01010101u) +
                 __popc(v.w & 0x01010101u);
        }
        for (int i = (n & ~15) + threadIdx.x; i < n; i += 256) c += p[i] != 0;
    } else {
        for (int i = threadIdx.x; i < n; i += 256) c += p[i] != 0;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = c;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) total += s_red[w];
    return total;
}
__device__ __forceinline__ long long sum_counts(const int* __restrict__ counts, int n, long long* s_red)
{
    long long c = 0;
    for (int i = threadIdx.x; i < n; i += 256) c += counts[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = c;
    __syncthreads();
    long long total = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) total += s_red[w];
    return total;
}

// Partial counts: visible anchors per ANCHORS of the first mask, selected slots per SLOT_CHUNK of the second.
__global__ void __launch_bounds__(256)
anchor_count_kernel(int n_anchors, long long n_slots, int anchor_blocks, const uint8_t* __restrict__ seen,
                    const uint8_t* __restrict__ selected, int* __restrict__ counts)
{
    __shared__ int s_red[8];
    const int count_blocks = (anchor_blocks + 7) / 8;
    if ((int)blockIdx.x < count_blocks) {
        const int b = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
        const int64_t first = (int64_t)b * ANCHORS;
        int c = 0;
        if (first + ANCHORS <= n_anchors && (reinterpret_cast<uintptr_t>(seen) & 7u) == 0) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(seen + first) + lane);
            c = __popc(v.x & 0x01010101u) + __popc(v.y & 0x01010101u);
        } else {
            for (int64_t i = first + lane; i < min(first + ANCHORS, (int64_t)n_anchors); i += 32) c += seen[i] != 0;
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0 && b < anchor_blocks) counts[b] = c;
        return;
    }
    const int b = blockIdx.x - count_blocks;
    const long long start = (long long)b * SLOT_CHUNK;
    const int c = count_bytes(selected + start, (int)min((long long)SLOT_CHUNK, n_slots - start), s_red);
    if (threadIdx.x == 0) counts[anchor_blocks + b] = c;
}

// Per CTA of ANCHORS anchors: its visible ones (in order) own consecutive slots, the selected among those consecutive
// Gaussians; where both begin follows from the partial counts.  Bound by the latency of its chains of dependent loads
// (mask, rank, Gaussian, sum): few anchors per CTA, and a warp has 128 slots in flight.  500 k anchors of ten slots, with
// the counting launch: 270 us (34 launches, four device-wide scans) -> 46 with 1024 anchors and 32 slots -> 34.
__global__ void __launch_bounds__(256, 5)
anchor_stats_kernel(int n_anchors, int n_off, long long n_slots, long long n_gaussians, int anchor_blocks,
                    const int* __restrict__ counts, const uint8_t* __restrict__ seen,
                    const uint8_t* __restrict__ selected, const uint8_t* __restrict__ on_screen,
                    const float* __restrict__ opacity, const float* __restrict__ grad, int grad_stride,
                    float* __restrict__ opacity_accum, float* __restrict__ anchor_demon,
                    float* __restrict__ gradient_accum, float* __restrict__ denom)
{
    __shared__ uint16_t s_anchor[ANCHORS];         // visible anchors of the CTA
    __shared__ int s_red[8];
    __shared__ long long s_red64[8];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int a0 = blockIdx.x * ANCHORS;
    if (counts[blockIdx.x] == 0) return;
    const long long v0 = sum_counts(counts, blockIdx.x, s_red64);          // visible anchors before this CTA's
    const long long slot0 = v0 * n_off;
    const int chunk = (int)(slot0 / SLOT_CHUNK);
    long long g0 = sum_counts(counts + anchor_blocks, chunk, s_red64);     // selected slots before this CTA's
    g0 += count_bytes(selected + (long long)chunk * SLOT_CHUNK, (int)(slot0 - (long long)chunk * SLOT_CHUNK), s_red);

    // list the visible anchors: a warp takes 128 consecutive ones
    int mine = 0;
    uint32_t m[ANCHORS / 256];
#pragma unroll
    for (int k = 0; k < ANCHORS / 256; k++) {
        const int a = a0 + warp * (ANCHORS / 8) + 32 * k + lane;
        m[k] = __ballot_sync(0xffffffffu, a < n_anchors && seen[a]);
        mine += __popc(m[k]);
    }
    __syncthreads();
    if (lane == 0) s_red[warp] = mine;
    __syncthreads();
    int at = 0, n_seen = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
        if (w < warp) at += s_red[w];
        n_seen += s_red[w];
    }
#pragma unroll
    for (int k = 0; k < ANCHORS / 256; k++) {
        if ((m[k] >> lane) & 1u)
            s_anchor[at + __popc(m[k] & ((1u << lane) - 1u))] = (uint16_t)(warp * (ANCHORS / 8) + 32 * k + lane);
        at += __popc(m[k]);
    }
    __syncthreads();

    for (int j = t; j < n_seen; j += 256) {
        const float* o = opacity + slot0 + (long long)j * n_off;
        float sum = 0.f;
#pragma unroll 5
        for (int k = 0; k < n_off; k++) sum += fmaxf(o[k], 0.f);
        const int a = a0 + s_anchor[j];
        opacity_accum[a] += sum;
        anchor_demon[a] += 1.f;
    }

    // slots: a warp takes a contiguous share, counts its selected ones, then visits them with their ranks known
    const int slots = (int)min((long long)n_seen * n_off, n_slots - slot0);
    const int share = (slots + 255) / 256 * 32, s_begin = min(slots, warp * share), s_end = min(slots, s_begin + share);
    int chosen = 0;
    for (int s = s_begin + lane; s < s_end; s += 32) chosen += selected[slot0 + s] != 0;
    chosen = __reduce_add_sync(0xffffffffu, chosen);
    __syncthreads();
    if (lane == 0) s_red[warp] = chosen;
    __syncthreads();
    int rank = 0;                                  // from the CTA's first Gaussian
#pragma unroll
    for (int w = 0; w < 8; w++)
        if (w < warp) rank += s_red[w];
    constexpr int FLIGHT = 4;
    on_screen += g0;
    grad += g0 * grad_stride;
    gradient_accum += (long long)a0 * n_off;
    denom += (long long)a0 * n_off;
    const int here = (int)max(0ll, min(n_gaussians - g0, (long long)slots));
    for (int s0 = s_begin; s0 < s_end; s0 += 32 * FLIGHT) {
        bool sel[FLIGHT], seen_g[FLIGHT];
        int to[FLIGHT];
        float x[FLIGHT], y[FLIGHT], sum[FLIGHT], visits[FLIGHT];
#pragma unroll
        for (int f = 0; f < FLIGHT; f++) {
            const int s = s0 + 32 * f + lane;
            sel[f] = s < s_end && selected[slot0 + s];
        }
#pragma unroll
        for (int f = 0; f < FLIGHT; f++) {
            const uint32_t sm = __ballot_sync(0xffffffffu, sel[f]);
            const int g = rank + __popc(sm & ((1u << lane) - 1u));
            rank += __popc(sm);
            sel[f] = sel[f] && g < here;
            if (!sel[f]) continue;
            const int s = s0 + 32 * f + lane, j = s / n_off;
            to[f] = s_anchor[j] * n_off + (s - j * n_off);
            seen_g[f] = on_screen[g];
            x[f] = grad[(long long)g * grad_stride], y[f] = grad[(long long)g * grad_stride + 1];
            sum[f] = gradient_accum[to[f]], visits[f] = denom[to[f]];
        }
#pragma unroll
        for (int f = 0; f < FLIGHT; f++)
            if (sel[f] && seen_g[f]) {
                gradient_accum[to[f]] = sum[f] + sqrtf(x[f] * x[f] + y[f] * y[f]);
                denom[to[f]] = visits[f] + 1.f;
            }
    }
}

}  // namespace cgx

using namespace cgx;

extern "C" int cgx_densify_update(int P, int B, const int32_t* const* radii, const float* const* dL_dmeans2D,
                                  float* grad_accum, float* denom, int32_t* max_radii, void* stream)
{
    if (P < 0 || B < 0 || B > STAT_CAMS) return CGX_EINVAL;
    if (P == 0 || B == 0) return CGX_OK;
    if (!radii || !dL_dmeans2D || !grad_accum || !denom) return CGX_EINVAL;
    DensifyBatch d;
    d.B = B;
    for (int b = 0; b < B; b++) {
        if (!radii[b] || !dL_dmeans2D[b] || ((uintptr_t)dL_dmeans2D[b] & 7)) return CGX_EINVAL;
        d.radii[b] = radii[b];
        d.grad[b] = (const float2*)dL_dmeans2D[b];
    }
    densify_kernel<<<(P + 255) / 256, 256, 0, (cudaStream_t)stream>>>(P, d, grad_accum, denom, max_radii);
    return check_launch();
}

extern "C" size_t cgx_anchor_stats_workspace_bytes(int n_anchors, int64_t n_slots)
{
    if (n_anchors <= 0 || n_slots < 0) return 0;
    return (size_t)((n_anchors + ANCHORS - 1) / ANCHORS + (n_slots + SLOT_CHUNK - 1) / SLOT_CHUNK) * sizeof(int);
}

extern "C" int cgx_anchor_stats(int n_anchors, int n_offsets, int64_t n_slots, int64_t n_gaussians, const float* grad,
                                int grad_stride, const float* opacity, const uint8_t* on_screen, const uint8_t* selected,
                                const uint8_t* seen, float* opacity_accum, float* anchor_demon, float* gradient_accum,
                                float* denom, void* workspace, size_t workspace_bytes, void* stream)
{
    if (n_anchors < 0 || n_offsets <= 0 || n_slots < 0 || n_gaussians < 0 || grad_stride < 2) return CGX_EINVAL;
    if (n_anchors == 0) return CGX_OK;
    if (!seen || !opacity_accum || !anchor_demon || !gradient_accum || !denom || !workspace) return CGX_EINVAL;
    if (n_slots && (!opacity || !selected)) return CGX_EINVAL;
    if (n_gaussians && (!grad || !on_screen)) return CGX_EINVAL;
    if (workspace_bytes < cgx_anchor_stats_workspace_bytes(n_anchors, n_slots)) return CGX_ENOMEM;
    const int anchor_blocks = (n_anchors + ANCHORS - 1) / ANCHORS;
    const int slot_blocks = (int)((n_slots + SLOT_CHUNK - 1) / SLOT_CHUNK);
    cudaStream_t st = (cudaStream_t)stream;
    anchor_count_kernel<<<(anchor_blocks + 7) / 8 + slot_blocks, 256, 0, st>>>(n_anchors, n_slots, anchor_blocks, seen, selected,
                                                                     (int*)workspace);
    anchor_stats_kernel<<<anchor_blocks, 256, 0, st>>>(n_anchors, n_offsets, n_slots, n_gaussians, anchor_blocks,
                                                       (const int*)workspace, seen, selected, on_screen, opacity, grad,
                                                       grad_stride, opacity_accum, anchor_demon, gradient_accum, denom);
    return check_launch(2);
}
