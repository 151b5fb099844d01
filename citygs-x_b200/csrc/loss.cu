// Strip loss: masked L1 and masked 11x11 Gaussian-window SSIM of a rendered strip against its ground truth, with the
// gradient towards the rendered strip.  Restates, as two fused kernels, what the reference computes with five grouped
// convolutions and a dozen element-wise tensor ops per strip per step (utils/loss_utils.py:88-132
// pixelwise_l1_with_mask / pixelwise_ssim_with_mask, driven by gaussian_renderer/loss_distribution.py:2835-2885); the
// time of this stage also feeds the tile-row balancer (workload_division.py, `forward_loss_time`).
//
// Both directions run the separable 11-tap window as a stream: a warp owns 32 columns of a channel and walks down a
// segment of rows.  Per row it convolves horizontally out of a row buffer in shared memory and adds the result to the
// eleven output rows it belongs to, which sit in registers (eleven accumulators per map, the roles rotating by
// unrolling); an output row is complete when its eleventh row has been added.  No barrier, no intermediate image, rows
// read once (plus ten at a segment's head).  Zero padding outside the strip, like conv2d(padding=5); the order of every
// sum is that of the plain double loop.
// Forward: forms the SSIM value, accumulates the two masked sums, and stores the three partial derivatives of the SSIM
// value with respect to the window moments E[x], E[x^2], E[xy] (already masked) for the backward.
// Backward: dL/dx(q) = w_l1 * mask(q) * sign(x(q) - y(q))
//                     + w_ssim * sum_p win(p - q) * [D_mu(p) + 2 x(q) D_xx(p) + y(q) D_xy(p)],
// i.e. the same separable window over the three stored maps.
#include <algorithm>
#include <cmath>

#include "cgx_common.cuh"

namespace cgx {

constexpr int LR = 5;                  // window radius
constexpr int TAPS = 2 * LR + 1;
constexpr int LOSS_WARPS = 4;          // warps per CTA, each on its own
constexpr int ROW = 32 + 2 * LR;       // columns a warp reads for its 32

// gauss(11, sigma 1.5) normalised, in float as the reference builds it (utils/loss_utils.py:27-35)
__constant__ float c_win[11];
static float h_win[11];
static bool h_win_ready[64] = {false};

// The warp's piece of the image: channel, first column, rows [row0, row1) of output.  False when there is none.
struct Strip {
    int c, x0, row0, row1;
};
__device__ __forceinline__ bool my_strip(Strip& st, int C, int H, int W, int seg_rows)
{
    const int cols = (W + 31) / 32, segs = (H + seg_rows - 1) / seg_rows;
    const int w = blockIdx.x * LOSS_WARPS + (threadIdx.x >> 5);
    if (w >= cols * segs * C) return false;
    const int s = w / cols;                        // neighbouring warps: neighbouring columns of the same rows
    st.x0 = (w - s * cols) * 32;
    st.c = s / segs;
    st.row0 = (s - st.c * segs) * seg_rows;
    st.row1 = min(H, st.row0 + seg_rows);
    return true;
}

// Reads row y of N images into registers: columns x0 - 5 + lane, and for ten lanes x0 + 27 + lane; zero outside.
template <int N>
__device__ __forceinline__ void fetch_row(float (&v)[N][2], const float* const (&src)[N], int y, int x0, int H, int W,
                                          int lane)
{
    const int xa = x0 - LR + lane, xb = xa + 32;
    const bool in = y >= 0 && y < H, a = in && xa >= 0 && xa < W, b = in && lane < 2 * LR && xb < W;
#pragma unroll
    for (int n = 0; n < N; n++) {
        v[n][0] = a ? src[n][(size_t)y * W + xa] : 0.f;
        v[n][1] = b ? src[n][(size_t)y * W + xb] : 0.f;
    }
}
// The mask byte at the warp's pixel of output row y; 1 without a mask, 0 where there is no pixel.  The byte itself: it
// is fetched a row ahead, and whatever is computed from it at once would wait for it at once.
__device__ __forceinline__ uint32_t fetch_mask(const uint8_t* __restrict__ mask, int y, int x, int W, const Strip& st)
{
    if (y < st.row0 || x >= W) return 0u;
    return mask ? mask[(size_t)y * W + x] : 1u;
}

// Bound by instruction issue: 77 horizontal and 55 vertical multiply-adds a pixel, in 77 instructions.  3x1200x1600: 170 -> 78 us.
__global__ void __launch_bounds__(32 * LOSS_WARPS, 4)
strip_loss_fwd_kernel(int C, int H, int W, int seg_rows, const float* __restrict__ img, const float* __restrict__ gt,
                      const uint8_t* __restrict__ mask, double* __restrict__ sums, float* __restrict__ d_mu,
                      float* __restrict__ d_xx, float* __restrict__ d_xy)
{
    __shared__ Pair s_rows[LOSS_WARPS][TAPS][ROW];      // (rendered, ground truth) of the last eleven rows
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Strip st;
    if (!my_strip(st, C, H, W, seg_rows)) return;
    const size_t plane = (size_t)st.c * H * W;
    const float* const src[2] = {img + plane, gt + plane};
    const int x = st.x0 + lane;
    Pair half[LR + 1];                                  // the window is symmetric, to the bit
#pragma unroll
    for (int k = 0; k <= LR; k++) half[k] = pack(c_win[k], c_win[k]);
    auto w = [&](int k) { return half[k <= LR ? k : 2 * LR - k]; };
    Pair acc[TAPS][2];                                  // slot of output row r: (r - row0) mod 11; (x, y), (xx, yy)
    float acc_xy[TAPS];
#pragma unroll
    for (int j = 0; j < TAPS; j++) acc[j][0] = acc[j][1] = pack(0.f, 0.f), acc_xy[j] = 0.f;
    float l1 = 0.f, ss = 0.f;

    float next[2][2];
    uint32_t next_m = 0;
    fetch_row<2>(next, src, st.row0 - LR, st.x0, H, W, lane);
    const int n_in = st.row1 - st.row0 + 2 * LR;        // input row i is image row row0 - 5 + i
    for (int base = 0; base < n_in; base += TAPS) {
#pragma unroll
        for (int u = 0; u < TAPS; u++) {
            const int i = base + u;
            if (i < n_in) {
                Pair* row = s_rows[warp][u];
                row[lane] = pack(next[0][0], next[1][0]);
                if (lane < 2 * LR) row[32 + lane] = pack(next[0][1], next[1][1]);
                const float m = next_m ? 1.f : 0.f;
                __syncwarp();
                if (i + 1 < n_in) next_m = fetch_mask(mask, st.row0 + i + 1 - 2 * LR, x, W, st);
                if (i + 1 < n_in) fetch_row<2>(next, src, st.row0 - LR + i + 1, st.x0, H, W, lane);
                Pair h0 = pack(0.f, 0.f), h1 = h0;
                float h_xy = 0.f;
#pragma unroll
                for (int k = 0; k < TAPS; k++) {
                    const Pair v = row[lane + k], wv = mul2(w(k), v);
                    h0 = fma2(w(k), v, h0);
                    h1 = fma2(wv, v, h1);
                    h_xy = fmaf(unpack(wv).x, unpack(v).y, h_xy);
                }
                // tap k of output i - k; slots of outputs not begun yet (negative) hold nothing that is used
#pragma unroll
                for (int k = 0; k < TAPS; k++) {
                    const int j = (u - k + TAPS) % TAPS;
                    acc[j][0] = k == 0 ? mul2(w(0), h0) : fma2(w(k), h0, acc[j][0]);
                    acc[j][1] = k == 0 ? mul2(w(0), h1) : fma2(w(k), h1, acc[j][1]);
                    acc_xy[j] = k == 0 ? unpack(w(0)).x * h_xy : fmaf(unpack(w(k)).x, h_xy, acc_xy[j]);
                }
                const int y = st.row0 + i - 2 * LR;     // the output row that this input row completes
                if (i >= 2 * LR && x < W) {
                    const float2 mu = unpack(acc[(u + 1) % TAPS][0]), e2 = unpack(acc[(u + 1) % TAPS][1]);
                    const float mu1 = mu.x, mu2 = mu.y, exx = e2.x, eyy = e2.y, exy = acc_xy[(u + 1) % TAPS];
                    const float C1 = 0.01f * 0.01f, C2 = 0.03f * 0.03f;
                    const float s1 = exx - mu1 * mu1, s2 = eyy - mu2 * mu2, s12 = exy - mu1 * mu2;
                    const float A1 = 2.f * mu1 * mu2 + C1, A2 = 2.f * s12 + C2;
                    const float B1 = mu1 * mu1 + mu2 * mu2 + C1, B2 = s1 + s2 + C2;
                    const float inv = 1.f / (B1 * B2);
                    const float val = A1 * A2 * inv;
                    const size_t o = (size_t)y * W + x;
                    if (d_mu) {
                        // derivatives with respect to the window moments, E[x^2] and E[xy] held fixed for the first one
                        const float dnum = 2.f * mu2 * A2 - 2.f * mu2 * A1;              // d(A1 A2)/d mu1
                        const float dden = 2.f * mu1 * B2 - 2.f * mu1 * B1;              // d(B1 B2)/d mu1
                        d_mu[plane + o] = m * (dnum - val * dden) * inv;
                        d_xx[plane + o] = m * (-val / B2);
                        d_xy[plane + o] = m * (2.f * A1 * inv);
                    }
                    const float2 centre = unpack(s_rows[warp][(u + TAPS - LR) % TAPS][lane + LR]);
                    l1 += m * fabsf(centre.x - centre.y);
                    ss += m * val;
                }
            }
        }
    }
    // thousands of partial sums: accumulated in double so that their order does not matter
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        l1 += __shfl_xor_sync(0xffffffffu, l1, o);
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
    }
    if (lane == 0) {
        atomicAdd(sums, (double)l1);
        atomicAdd(sums + 1, (double)ss);
    }
}

// Bound by instruction issue and by waiting for rows with 16 to 20 warps per SM (60 % issued).  3x1200x1600: 152 -> 77 us.
__global__ void __launch_bounds__(32 * LOSS_WARPS)
strip_loss_bwd_kernel(int C, int H, int W, int seg_rows, const float* __restrict__ img, const float* __restrict__ gt,
                      const uint8_t* __restrict__ mask, const float* __restrict__ weights,
                      const float* __restrict__ d_mu, const float* __restrict__ d_xx, const float* __restrict__ d_xy,
                      float* __restrict__ dL_dimg)
{
    __shared__ Pair s_rows[LOSS_WARPS][2][ROW];         // (d_mu, d_xx)
    __shared__ float s_xy[LOSS_WARPS][2][ROW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Strip st;
    if (!my_strip(st, C, H, W, seg_rows)) return;
    const size_t plane = (size_t)st.c * H * W;
    const float* const src[3] = {d_mu + plane, d_xx + plane, d_xy + plane};
    const int x = st.x0 + lane;
    const float w_l1 = weights[0], w_ssim = weights[1];
    Pair half[LR + 1];                                  // the window is symmetric, to the bit
#pragma unroll
    for (int k = 0; k <= LR; k++) half[k] = pack(c_win[k], c_win[k]);
    auto w = [&](int k) { return half[k <= LR ? k : 2 * LR - k]; };
    Pair acc[TAPS];
    float acc_xy[TAPS];
#pragma unroll
    for (int j = 0; j < TAPS; j++) acc[j] = pack(0.f, 0.f), acc_xy[j] = 0.f;

    uint32_t next_m = 0;
    float next[3][2], next_v = 0.f, next_y = 0.f;
    fetch_row<3>(next, src, st.row0 - LR, st.x0, H, W, lane);
    const int n_in = st.row1 - st.row0 + 2 * LR;
    for (int base = 0; base < n_in; base += TAPS) {
#pragma unroll
        for (int u = 0; u < TAPS; u++) {
            const int i = base + u;
            if (i < n_in) {
                Pair* row = s_rows[warp][i & 1];
                float* row_xy = s_xy[warp][i & 1];
                row[lane] = pack(next[0][0], next[1][0]);
                row_xy[lane] = next[2][0];
                if (lane < 2 * LR) {
                    row[32 + lane] = pack(next[0][1], next[1][1]);
                    row_xy[32 + lane] = next[2][1];
                }
                __syncwarp();
                const float m = next_m ? 1.f : 0.f, v = next_v, y = next_y;
                if (i + 1 < n_in) {
                    const int out = st.row0 + i + 1 - 2 * LR;
                    next_m = fetch_mask(mask, out, x, W, st);
                    if (out >= st.row0 && x < W) {
                        next_v = img[plane + (size_t)out * W + x];
                        next_y = gt[plane + (size_t)out * W + x];
                    }
                    fetch_row<3>(next, src, st.row0 - LR + i + 1, st.x0, H, W, lane);
                }
                Pair h = pack(0.f, 0.f);
                float h_xy = 0.f;
#pragma unroll
                for (int k = 0; k < TAPS; k++) {
                    h = fma2(w(k), row[lane + k], h);
                    h_xy = fmaf(unpack(w(k)).x, row_xy[lane + k], h_xy);
                }
#pragma unroll
                for (int k = 0; k < TAPS; k++) {
                    const int j = (u - k + TAPS) % TAPS;
                    acc[j] = k == 0 ? mul2(w(0), h) : fma2(w(k), h, acc[j]);
                    acc_xy[j] = k == 0 ? unpack(w(0)).x * h_xy : fmaf(unpack(w(k)).x, h_xy, acc_xy[j]);
                }
                if (i >= 2 * LR && x < W) {
                    const float2 e = unpack(acc[(u + 1) % TAPS]);
                    const float e_xy = acc_xy[(u + 1) % TAPS];
                    const size_t o = (size_t)(st.row0 + i - 2 * LR) * W + x;
                    const float diff = v - y;
                    const float sgn = diff > 0.f ? 1.f : (diff < 0.f ? -1.f : 0.f);
                    dL_dimg[plane + o] = w_l1 * m * sgn + w_ssim * (e.x + 2.f * v * e.y + y * e_xy);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Normal image from a depth image (render_normal, gaussian_renderer/__init__.py:1311-1323 with scale = 1 and no
// offsets -> normal_from_depth_image / depth_pcd2normal, utils/graphics_utils.py:87-152): camera-space points
// p(x,y) = z * ((x - cx)/fx, (y - cy)/fy, 1), normal = normalize((p_right - p_left) x (p_top - p_bottom)) with
// bottom = row + 1, top = row - 1, zero on the one-pixel border.
struct Pinhole {
    float fx, fy, cx, cy;
};

__device__ __forceinline__ float3 cross3(const float3 a, const float3 b)
{
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

constexpr int NT_ROWS = 32;       // a CTA of 256 threads takes 32 x 32 pixels: four rows per thread keep loads in flight

// A pixel block with a margin of M pixels: depths and the ray coordinates of its columns and rows, each fetched or
// divided once.
template <int M>
struct DepthTile {
    float z[NT_ROWS + 2 * M][32 + 2 * M], rx[32 + 2 * M], ry[NT_ROWS + 2 * M];

    __device__ __forceinline__ void load(const float* __restrict__ depth, int H, int W, int x0, int y0, const Pinhole k)
    {
        constexpr int TW = 32 + 2 * M, TH = NT_ROWS + 2 * M;
#pragma unroll
        for (int e = threadIdx.x; e < TW * TH; e += 256) {
            const int r = e / TW, q = e - r * TW, y = y0 - M + r, x = x0 - M + q;
            z[r][q] = (y >= 0 && y < H && x >= 0 && x < W) ? depth[(size_t)y * W + x] : 0.f;
        }
        if (threadIdx.x < TW) rx[threadIdx.x] = ((float)(x0 - M + (int)threadIdx.x) - k.cx) / k.fx;
        else if (threadIdx.x >= 64 && threadIdx.x < 64 + TH)
            ry[threadIdx.x - 64] = ((float)(y0 - M + (int)threadIdx.x - 64) - k.cy) / k.fy;
    }
    // a = right - left, b = top - bottom, c = a x b of the tile's pixel (r, q).  Differences of neighbouring points lose
    // most of their digits, so the roundings are written out: they are those of the point-wise form.
    __device__ __forceinline__ void frame(int r, int q, float3& a, float3& b, float3& c) const
    {
        const float zr = z[r][q + 1], zl = z[r][q - 1], zt = z[r - 1][q], zb = z[r + 1][q];
        a = make_float3(__fsub_rn(__fmul_rn(zr, rx[q + 1]), __fmul_rn(zl, rx[q - 1])),
                        __fsub_rn(__fmul_rn(zr, ry[r]), __fmul_rn(zl, ry[r])), zr - zl);
        b = make_float3(__fsub_rn(__fmul_rn(zt, rx[q]), __fmul_rn(zb, rx[q])),
                        __fmaf_rn(-zb, ry[r + 1], __fmul_rn(zt, ry[r - 1])), zt - zb);
        c = make_float3(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
                        __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
    }
    static __device__ __forceinline__ float length(const float3 c)
    {
        return sqrtf(__fmaf_rn(c.z, c.z, __fmaf_rn(c.x, c.x, __fmul_rn(c.y, c.y))));
    }
};

// HBM-bound.  1200x1600: 18 -> 14 us.
__global__ void __launch_bounds__(256)
depth_normal_fwd_kernel(int H, int W, Pinhole k, const float* __restrict__ depth, float* __restrict__ normal)
{
    __shared__ DepthTile<1> t;
    t.load(depth, H, W, blockIdx.x * 32, blockIdx.y * NT_ROWS, k);
    __syncthreads();
    const int q = threadIdx.x & 31, x = blockIdx.x * 32 + q;
    const size_t HW = (size_t)H * W;
#pragma unroll
    for (int r = threadIdx.x >> 5; r < NT_ROWS; r += 8) {
        const int y = blockIdx.y * NT_ROWS + r;
        if (x >= W || y >= H) continue;
        float3 n = make_float3(0.f, 0.f, 0.f);
        if (x > 0 && x < W - 1 && y > 0 && y < H - 1) {
            float3 a, b, c;
            t.frame(r + 1, q + 1, a, b, c);
            const float len = fmaxf(t.length(c), 1e-12f);
            n = make_float3(c.x / len, c.y / len, c.z / len);
        }
        const size_t o = (size_t)y * W + x;
        normal[o] = n.x;
        normal[HW + o] = n.y;
        normal[2 * HW + o] = n.z;
    }
}

// Gather form: a depth pixel is the right / left / top / bottom point of four neighbouring normals.  Each normal's
// frame and cotangent are worked out once per block (1.13 times per pixel with the margin) and left in shared memory;
// every pixel doing so for its four neighbours took four times the square roots and quotients.
// 1200x1600: 72 -> 31 us.
struct NormalGradSmem {
    DepthTile<2> t;
    float a[3][NT_ROWS + 2][34], b[3][NT_ROWS + 2][34], gc[3][NT_ROWS + 2][34];
};
__global__ void __launch_bounds__(256)
depth_normal_bwd_kernel(int H, int W, Pinhole k, const float* __restrict__ depth, const float* __restrict__ g,
                        float* __restrict__ dL_ddepth)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    NormalGradSmem& sm = *reinterpret_cast<NormalGradSmem*>(smem_raw);
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * NT_ROWS;
    const size_t HW = (size_t)H * W;
    sm.t.load(depth, H, W, x0, y0, k);
    __syncthreads();
    for (int e = threadIdx.x; e < 34 * (NT_ROWS + 2); e += 256) {
        const int r = e / 34, q = e - r * 34, x = x0 - 1 + q, y = y0 - 1 + r;
        float3 a = make_float3(0.f, 0.f, 0.f), b = a, gc = a;
        if (x > 0 && x < W - 1 && y > 0 && y < H - 1) {
            float3 c;
            sm.t.frame(r + 1, q + 1, a, b, c);
            const float len = sm.t.length(c);
            if (len > 1e-12f) {                   // else a clamped norm: the direction carries no gradient
                const size_t o = (size_t)y * W + x;
                const float3 gn = make_float3(g[o], g[HW + o], g[2 * HW + o]);
                const float3 n = make_float3(c.x / len, c.y / len, c.z / len);
                const float d = n.x * gn.x + n.y * gn.y + n.z * gn.z;
                gc = make_float3((gn.x - n.x * d) / len, (gn.y - n.y * d) / len, (gn.z - n.z * d) / len);
            }
        }
        sm.a[0][r][q] = a.x, sm.a[1][r][q] = a.y, sm.a[2][r][q] = a.z;
        sm.b[0][r][q] = b.x, sm.b[1][r][q] = b.y, sm.b[2][r][q] = b.z;
        sm.gc[0][r][q] = gc.x, sm.gc[1][r][q] = gc.y, sm.gc[2][r][q] = gc.z;
    }
    __syncthreads();
    const int q = threadIdx.x & 31, x = x0 + q;
    auto get = [](const float (&m)[3][NT_ROWS + 2][34], int r, int c) {
        return make_float3(m[0][r][c], m[1][r][c], m[2][r][c]);
    };
#pragma unroll
    for (int r = threadIdx.x >> 5; r < NT_ROWS; r += 8) {
        const int y = y0 + r;
        if (x >= W || y >= H) continue;
        // c = a x b:  dL/da = b x gc,  dL/db = gc x a
        float3 gp = cross3(get(sm.b, r + 1, q), get(sm.gc, r + 1, q));             // right point of (x-1, y): +dL/da
        float3 t = cross3(get(sm.b, r + 1, q + 2), get(sm.gc, r + 1, q + 2));      // left point of (x+1, y): -dL/da
        gp.x -= t.x; gp.y -= t.y; gp.z -= t.z;
        t = cross3(get(sm.gc, r + 2, q + 1), get(sm.a, r + 2, q + 1));             // top point of (x, y+1): +dL/db
        gp.x += t.x; gp.y += t.y; gp.z += t.z;
        t = cross3(get(sm.gc, r, q + 1), get(sm.a, r, q + 1));                     // bottom point of (x, y-1): -dL/db
        gp.x -= t.x; gp.y -= t.y; gp.z -= t.z;
        dL_ddepth[(size_t)y * W + x] = gp.x * sm.t.rx[q + 2] + gp.y * sm.t.ry[r + 2] + gp.z;
    }
}

// Rows per warp: ten more are read than written, so long segments waste least; what counts is rows read times the
// rounds in which the chip takes the warps (16 per SM).
static int loss_segment(int C, int H, int W)
{
    const long long cols = (long long)((W + 31) / 32) * C, room = 148 * 16;
    long long best = -1;
    int best_rows = 0;
    for (int rows = 128; rows >= 8; rows -= 2) {
        const long long rounds = (cols * ((H + rows - 1) / rows) + room - 1) / room;
        const long long cost = rounds * (std::min(rows, H) + 2 * LR);
        if (best < 0 || cost < best) best = cost, best_rows = rows;
    }
    return best_rows;
}
static int loss_blocks(int C, int H, int W, int rows)
{
    const long long warps = (long long)((W + 31) / 32) * C * ((H + rows - 1) / rows);
    return (int)((warps + LOSS_WARPS - 1) / LOSS_WARPS);
}

static int upload_window()
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return CGX_ECUDA;
    }
    if (dev < 0 || dev >= 64) return CGX_EINVAL;
    if (h_win_ready[dev]) return CGX_OK;
    float g[11], sum = 0.f;
    for (int x = 0; x < 11; x++) {
        g[x] = (float)exp(-(double)((x - 5) * (x - 5)) / (2.0 * 1.5 * 1.5));   // stored to float first, as torch.Tensor does
        sum += g[x];                                                          // float sum, ascending
    }
    for (int x = 0; x < 11; x++) h_win[x] = g[x] / sum;
    e = cudaMemcpyToSymbol(c_win, h_win, sizeof(h_win));
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return CGX_ECUDA;
    }
    h_win_ready[dev] = true;
    return CGX_OK;
}

}  // namespace cgx

using namespace cgx;

extern "C" int cgx_strip_loss_fwd(int C, int H, int W, const float* img, const float* gt, const uint8_t* mask,
                                  double* sums, float* d_mu, float* d_xx, float* d_xy, void* stream)
{
    if (C <= 0 || H <= 0 || W <= 0 || !img || !gt || !sums) return CGX_EINVAL;
    if ((d_mu != nullptr) != (d_xx != nullptr) || (d_mu != nullptr) != (d_xy != nullptr)) return CGX_EINVAL;
    int st = upload_window();
    if (st != CGX_OK) return st;
    cudaError_t e = cudaMemsetAsync(sums, 0, 2 * sizeof(double), (cudaStream_t)stream);
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return CGX_ECUDA;
    }
    const int rows = loss_segment(C, H, W);
    strip_loss_fwd_kernel<<<loss_blocks(C, H, W, rows), 32 * LOSS_WARPS, 0, (cudaStream_t)stream>>>(
        C, H, W, rows, img, gt, mask, sums, d_mu, d_xx, d_xy);
    return check_launch();
}

extern "C" int cgx_strip_loss_bwd(int C, int H, int W, const float* img, const float* gt, const uint8_t* mask,
                                  const float* weights, const float* d_mu, const float* d_xx, const float* d_xy,
                                  float* dL_dimg, void* stream)
{
    if (C <= 0 || H <= 0 || W <= 0 || !img || !gt || !weights || !d_mu || !d_xx || !d_xy || !dL_dimg)
        return CGX_EINVAL;
    int st = upload_window();
    if (st != CGX_OK) return st;
    const int rows = loss_segment(C, H, W);
    strip_loss_bwd_kernel<<<loss_blocks(C, H, W, rows), 32 * LOSS_WARPS, 0, (cudaStream_t)stream>>>(
        C, H, W, rows, img, gt, mask, weights, d_mu, d_xx, d_xy, dL_dimg);
    return check_launch();
}

extern "C" int cgx_depth_normal_fwd(int H, int W, float fx, float fy, float cx, float cy, const float* depth,
                                    float* normal, void* stream)
{
    if (H <= 0 || W <= 0 || !depth || !normal || fx == 0.f || fy == 0.f) return CGX_EINVAL;
    dim3 grid((W + 31) / 32, (H + NT_ROWS - 1) / NT_ROWS);
    depth_normal_fwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(H, W, Pinhole{fx, fy, cx, cy}, depth, normal);
    return check_launch();
}

extern "C" int cgx_depth_normal_bwd(int H, int W, float fx, float fy, float cx, float cy, const float* depth,
                                    const float* dL_dnormal, float* dL_ddepth, void* stream)
{
    if (H <= 0 || W <= 0 || !depth || !dL_dnormal || !dL_ddepth || fx == 0.f || fy == 0.f) return CGX_EINVAL;
    dim3 grid((W + 31) / 32, (H + NT_ROWS - 1) / NT_ROWS);
    static_assert(sizeof(NormalGradSmem) <= 48 * 1024, "fits without an opt-in");
    depth_normal_bwd_kernel<<<grid, 256, sizeof(NormalGradSmem), (cudaStream_t)stream>>>(H, W, Pinhole{fx, fy, cx, cy}, depth, dL_dnormal,
                                                                    dL_ddepth);
    return check_launch();
}
