// sift.cu — SIFT feature extraction on sm_100a.
//
// Restates sfm-lite/src/sift.rs (extract_sift, :435-555) for one image:
//
//   resize      load-time resize to max_dim (resize.cu; `.max(1)` sides)
//   pyramid     the reference's per-octave levels (sift.rs:51-134) have sigma
//               1.6 (1 << int(l / 3)): levels 1, 2 repeat level 0's and 4, 5
//               level 3's, and the blur between equal sigmas (0.01) has the taps
//               0, 1, 0 exactly, so those levels equal the one before bit for
//               bit, every DoG but number 2 is zero, and no extremum can lie in
//               a zero DoG.  Level 0 (blurred once, from the grey image), level
//               3 and DoG 2 are all that is made (identity_taps checks it)
//   octave      one kernel per octave: level 3 (separable f32 blur with
//               clamped edges, f64 kernel weights cast to f32, taps summed in
//               order) and DoG 2 of a tile in shared memory, the 2x2 box
//               downsample that is the next octave's level 0, and per pixel
//               the 24-neighbour test, the quadratic fit (nalgebra's cofactor
//               3x3 inverse, f64), the contrast and curvature tests
//               (sift.rs:176-262); keypoints are appended with their place in
//               the reference's (octave, level, y, x) order
//   selection   the reference sorts its descriptors by response (stable) and
//               keeps the first max_features (sift.rs:543-544).  A descriptor's
//               response is its keypoint's, so that order is the keypoints of
//               all octaves by (response descending, place) with each
//               keypoint's peaks in turn.  A histogram of the responses picks a
//               threshold for the first max_features and some, and those are
//               ranked by counting
//   orientation one block per keypoint in that order: its threads evaluate the
//               window's samples (atan2, exp in f64), thread b adds bin b's in
//               window order, so every bin is the reference's sequential f64 sum;
//               a warp smooths and picks up to four peaks (sift.rs:274-334)
//   descriptor  one block per (keypoint, peak): the threads evaluate the
//               window's samples (bilinear gradients, rotation, trilinear
//               parameters) into shared memory; then thread t owns bin t and
//               walks the list of its cell's samples, in window order; L2 -> clip 0.2 -> L2 in f32 with the
//               reference's serial sums (sift.rs:340-431)
//
// All of it is queued without waiting: the counts stay on the device until
// one read at the end.  Where that read shows that the first keypoints did not
// fill max_features (or max_features is past QUICK_CAP), the general path
// continues: all keypoints sorted by CUB, orientations and descriptors in
// chunks until max_features valid ones exist.
//
// The library builds with --fmad=false: every f32/f64 product and sum rounds
// as written, so the pyramid, the DoGs and the extrema with their fitted
// positions and responses are those of the CPU restatement bit for bit.  Orientation and
// descriptor use the device's f64 exp / atan2 / sin / cos, which may differ
// from the host libm in the last bit; their results agree with the CPU
// restatement to a tolerance, and a histogram bin or peak decision at an exact boundary can
// differ.
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <cub/cub.cuh>
#include <string>
#include <vector>

#include "ctx_internal.cuh"

namespace rcmvs {

namespace {

constexpr int NSPO = 3;
constexpr int NLEV = NSPO + 3;  // blurred levels per octave
constexpr int DESC_LEN = 128;
constexpr int MAX_TAPS = 32;
constexpr double SIGMA0 = 1.6;
constexpr double ASSUMED_BLUR = 0.5;
constexpr double EDGE_THR = 10.0;
constexpr double PI = 3.14159265358979323846;
constexpr int WARPS = 4;  // warps per block in the keypoint kernels

struct BlurTaps {
    int radius;
    float k[MAX_TAPS];
};

struct KpArrays {  // raw keypoints, in no order
    double* x;       // octave coordinates
    double* y;
    double* resp;
    uint32_t* place; // in the reference's (octave, level, y, x) order
    int32_t* oct;
};

constexpr int KP_LEVEL = 2;  // the DoG level every keypoint lies in
constexpr int MAX_OCT = 8;
struct OctTable {  // per octave: level 0 (= levels 1 and 2, whose gradients the keypoints use), size, scale
    const float* img[MAX_OCT];
    int w[MAX_OCT], h[MAX_OCT];
    double scale[MAX_OCT];
};

struct Counts {  // on the device
    uint32_t kp;     // raw keypoints
    uint32_t kept;   // of them past the selection's threshold
    uint32_t pairs;  // (keypoint, peak) pairs of the first keypoints
    uint32_t valid;  // valid descriptors among the first max_features pairs
};

__device__ __host__ __forceinline__ double level_sigma(int l) {
    return SIGMA0 * (double)(1 << (int)((double)l / (double)NSPO));
}

// ---- separable blur of one tile (sift.rs:65-90): BX x BY outputs whose
// first is at (x0, y0), the source clamped at the image's edges.  Each thread
// makes eight neighbouring sums from one run of loads.  in: [BY + 2R][BX + 2R]
// (pitch IN_P), mid: [BY + 2R][BX] (pitch MID_P).
constexpr int BX = 64, BY = 32, BLUR_THREADS = 256;
template <int R>
struct BlurSmem {
    static constexpr int IN_W = BX + 2 * R, IN_H = BY + 2 * R, IN_P = IN_W | 1, MID_P = BX + 1;
    float in[IN_H * IN_P];
    float mid[IN_H * MID_P];
};

template <int R, class Load, class Store>
__device__ __forceinline__ void blur_tile(BlurSmem<R>& sm, int x0, int y0, int w, int h, const BlurTaps& taps, Load load,
                                          Store store) {
    using S = BlurSmem<R>;
    const int tid = threadIdx.x;
    // a warp per row; all of a thread's loads are in flight together
    {
        constexpr int ROWS = (S::IN_H + BLUR_THREADS / 32 - 1) / (BLUR_THREADS / 32), COLS = (S::IN_W + 31) / 32;
        const int lane = tid & 31;
        int gx[COLS];
#pragma unroll
        for (int c = 0; c < COLS; ++c) gx[c] = min(max(x0 - R + lane + 32 * c, 0), w - 1);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int iy = (tid >> 5) + r * (BLUR_THREADS / 32);
            const int64_t row = (int64_t)min(max(y0 - R + iy, 0), h - 1) * w;
#pragma unroll
            for (int c = 0; c < COLS; ++c)
                if (iy < S::IN_H && lane + 32 * c < S::IN_W) sm.in[iy * S::IN_P + lane + 32 * c] = load(row + gx[c]);
        }
    }
    __syncthreads();
    // horizontal: lanes on different rows (odd pitches: no bank conflicts)
    for (int i = tid; i < 64 * (BX / 8); i += BLUR_THREADS) {
        const int row = i & 63, g = i >> 6;
        if (row >= S::IN_H) continue;
        const float* src = sm.in + row * S::IN_P + 8 * g;
        float v[8 + 2 * R];
#pragma unroll
        for (int k = 0; k < 8 + 2 * R; ++k) v[k] = src[k];
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k <= 2 * R; ++k) acc = acc + taps.k[k] * v[o + k];
            sm.mid[row * S::MID_P + 8 * g + o] = acc;
        }
    }
    __syncthreads();
    // vertical
    {
        const int col = tid & (BX - 1), g = tid / BX;
        float v[8 + 2 * R];
#pragma unroll
        for (int k = 0; k < 8 + 2 * R; ++k) v[k] = sm.mid[(8 * g + k) * S::MID_P + col];
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k <= 2 * R; ++k) acc = acc + taps.k[k] * v[o + k];
            store(col, 8 * g + o, acc);
        }
    }
}
static_assert(BLUR_THREADS == BX * BY / 8 && BY + 2 * 9 <= 64, "blur tile");

constexpr int R_BASE = 5, R_LEVEL = 9;  // radii of the base blur and of level 3's

// Level 0 of the first octave from the grey image (sift.rs:446-457).
__global__ void __launch_bounds__(BLUR_THREADS) base_kernel(const uint8_t* __restrict__ gray, int w, int h,
                                                            const __grid_constant__ BlurTaps taps,
                                                            float* __restrict__ out) {
    __shared__ BlurSmem<R_BASE> sm;
    const int tiles_x = (w + BX - 1) / BX;
    const int x0 = (int)(blockIdx.x % tiles_x) * BX, y0 = (int)(blockIdx.x / tiles_x) * BY;
    blur_tile<R_BASE>(
        sm, x0, y0, w, h, taps, [&](int64_t i) { return (float)gray[i] / 255.0f; },
        [&](int x, int y, float v) {
            if (x0 + x < w && y0 + y < h) out[(int64_t)(y0 + y) * w + x0 + x] = v;
        });
}

// nalgebra 0.32 Matrix3::try_inverse: cofactors over the determinant
__device__ __forceinline__ bool inverse3(const double m[9], double o[9]) {
    const double m11 = m[0], m12 = m[1], m13 = m[2], m21 = m[3], m22 = m[4], m23 = m[5], m31 = m[6], m32 = m[7],
                 m33 = m[8];
    const double a = m22 * m33 - m32 * m23;
    const double b = m21 * m33 - m31 * m23;
    const double c = m21 * m32 - m31 * m22;
    const double det = m11 * a - m12 * b + m13 * c;
    if (det == 0.0) return false;
    o[0] = a / det;
    o[1] = (m13 * m32 - m33 * m12) / det;
    o[2] = (m12 * m23 - m22 * m13) / det;
    o[3] = -b / det;
    o[4] = (m11 * m33 - m31 * m13) / det;
    o[5] = (m13 * m21 - m23 * m11) / det;
    o[6] = c / det;
    o[7] = (m12 * m31 - m32 * m11) / det;
    o[8] = (m11 * m22 - m21 * m12) / det;
    return true;
}

// One octave (see the file's head).  A block makes the DoG of BX x BY pixels
// and answers for the inner (BX - 2) x (BY - 2): their extrema (sift.rs:176-262,
// the DoGs above and below being zero) and their part of the next octave's
// level 0 (sift.rs:95-110; next may be null).  1600x1200, six octaves: five blurs
// each, DoGs, extrema over three levels, gradients and their selections took
// 124 launches and 590 us; 78 us here with the base (the fits in a second
// pass over the tile's candidates; 150 us with them in the first).
__global__ void __launch_bounds__(BLUR_THREADS) octave_kernel(const float* __restrict__ lev0, int w, int h,
                                                              const __grid_constant__ BlurTaps taps, double thr,
                                                              float* __restrict__ next, int nw, int nh, int octave,
                                                              uint32_t place0, KpArrays kp, Counts* __restrict__ counts) {
    __shared__ BlurSmem<R_LEVEL> sm;
    __shared__ float lev3[BY][BX];
    __shared__ float dog[BY][BX + 1];
    // strict extrema: at most one maximum and one minimum in any 2 x 2 pixels
    __shared__ uint16_t cand[2 * (BX / 2 - 1) * (BY / 2 - 1)];
    __shared__ int n_cand;
    if (threadIdx.x == 0) n_cand = 0;
    const int tiles_x = (w + BX - 3) / (BX - 2);
    const int x0 = (int)(blockIdx.x % tiles_x) * (BX - 2);  // the first inner pixel
    const int y0 = (int)(blockIdx.x / tiles_x) * (BY - 2);
    blur_tile<R_LEVEL>(
        sm, x0 - 1, y0 - 1, w, h, taps, [&](int64_t i) { return __ldg(lev0 + i); },
        [&](int x, int y, float v) {
            lev3[y][x] = v;
            dog[y][x] = v - sm.in[(y + R_LEVEL) * BlurSmem<R_LEVEL>::IN_P + x + R_LEVEL];
        });
    __syncthreads();
    const double edge_lim = (EDGE_THR + 1.0) * (EDGE_THR + 1.0) / EDGE_THR;
    for (int i = threadIdx.x; i < (BX - 2) * (BY - 2); i += BLUR_THREADS) {
        const int cx = 1 + i % (BX - 2), cy = 1 + i / (BX - 2);
        const int x = x0 + cx - 1, y = y0 + cy - 1;
        if (x < 1 || y < 1 || x + 1 >= w || y + 1 >= h) continue;
        const float v = dog[cy][cx];
        if ((double)fabsf(v) < thr) continue;
        // a neighbour of the zero DoGs is 0
        bool is_max = !(0.0f >= v), is_min = !(0.0f <= v);
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                if (dy == 0 && dx == 0) continue;
                const float n = dog[cy + dy][cx + dx];
                if (n >= v) is_max = false;
                if (n <= v) is_min = false;
            }
        if (is_max || is_min) cand[atomicAdd(&n_cand, 1)] = (uint16_t)(cy * BX + cx);
    }
    __syncthreads();
    // the fits, of all candidates at once: one f64 chain per block, not per warp
    for (int i = threadIdx.x; i < n_cand; i += BLUR_THREADS) {
        const int cx = cand[i] % BX, cy = cand[i] / BX;
        const int x = x0 + cx - 1, y = y0 + cy - 1;
        const float v = dog[cy][cx];
        auto d = [&](int dx, int dy) { return dog[cy + dy][cx + dx]; };
        const float zero = 0.0f;
        const float fdx = 0.5f * (d(1, 0) - d(-1, 0));
        const float fdy = 0.5f * (d(0, 1) - d(0, -1));
        const float fds = 0.5f * (zero - zero);
        const float dxx = d(1, 0) + d(-1, 0) - 2.0f * v;
        const float dyy = d(0, 1) + d(0, -1) - 2.0f * v;
        const float dss = zero + zero - 2.0f * v;
        const float dxy = 0.25f * (d(1, 1) + d(-1, -1) - d(-1, 1) - d(1, -1));
        const float dxs = 0.25f * (zero + zero - zero - zero);
        const float dys = 0.25f * (zero + zero - zero - zero);
        const double hm[9] = {dxx, dxy, dxs, dxy, dyy, dys, dxs, dys, dss};
        double hi[9];
        if (!inverse3(hm, hi)) continue;
        const double g0 = -(double)fdx, g1 = -(double)fdy, g2 = -(double)fds;
        const double ox = hi[0] * g0 + hi[1] * g1 + hi[2] * g2;
        const double oy = hi[3] * g0 + hi[4] * g1 + hi[5] * g2;
        const double os = hi[6] * g0 + hi[7] * g1 + hi[8] * g2;
        if (fabs(ox) > 1.0 || fabs(oy) > 1.0 || fabs(os) > 1.0) continue;
        const double contrast = (double)v + 0.5 * ((double)fdx * ox + (double)fdy * oy + (double)fds * os);
        const double tr = (double)(dxx + dyy);
        const double det = (double)(dxx * dyy - dxy * dxy);
        if (fabs(contrast) < thr || det <= 0.0 || tr * tr / det > edge_lim) continue;
        const uint32_t k = atomicAdd(&counts->kp, 1u);
        kp.x[k] = (double)x + ox;
        kp.y[k] = (double)y + oy;
        kp.resp[k] = fabs(contrast);
        kp.place[k] = place0 + (uint32_t)y * (uint32_t)w + (uint32_t)x;
        kp.oct[k] = octave;
    }
    if (next) {
        for (int i = threadIdx.x; i < (BX / 2 - 1) * (BY / 2 - 1); i += BLUR_THREADS) {
            const int tx = i % (BX / 2 - 1), ty = i / (BX / 2 - 1);
            const int x = x0 / 2 + tx, y = y0 / 2 + ty;
            if (x >= nw || y >= nh) continue;
            const int ax = 1 + 2 * tx, ay = 1 + 2 * ty;
            const int bx = min(2 * x + 1, w - 1) - x0 + 1, by = min(2 * y + 1, h - 1) - y0 + 1;
            const float sum = lev3[ay][ax] + lev3[ay][bx] + lev3[by][ax] + lev3[by][bx];
            next[(int64_t)y * nw + x] = 0.25f * sum;
        }
    }
}

// ---- selection of the first `want` keypoints by (response descending, place)
constexpr int SEL_BINS = 2048, SEL_CAP = 16384;
struct Kept {  // SEL_CAP entries each
    long long* key;
    uint32_t* place;
    uint32_t* kp;
};

// A response's order: it is never negative, so its bits are ordered as it is.
__device__ __forceinline__ long long resp_key(double r) { return __double_as_longlong(r); }

// Monotone in the key: 256 bins per octave from 2^-9, clamped.
__device__ __forceinline__ int resp_bin(double r) {
    const int b = (__float_as_int((float)r) - 0x3B000000) >> 15;
    return min(max(b, 0), SEL_BINS - 1);
}

__global__ void __launch_bounds__(256) hist_kernel(const double* __restrict__ resp, const Counts* __restrict__ counts,
                                                   uint32_t* __restrict__ hist) {
    __shared__ uint32_t s_hist[SEL_BINS];
    for (int i = threadIdx.x; i < SEL_BINS; i += 256) s_hist[i] = 0;
    __syncthreads();
    const uint32_t n = counts->kp;
    for (uint32_t k = blockIdx.x * 256 + threadIdx.x; k < n; k += gridDim.x * 256) atomicAdd(&s_hist[resp_bin(resp[k])], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < SEL_BINS; i += 256)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// The keypoints whose bin is at least the highest one with `want` keypoints
// at or above it.
__global__ void __launch_bounds__(256) keep_kernel(const double* __restrict__ resp, const uint32_t* __restrict__ hist,
                                                   const uint32_t* __restrict__ place, uint32_t want,
                                                   Counts* __restrict__ counts, Kept kept) {
    __shared__ uint32_t s_sum[256];
    __shared__ int s_bin;
    constexpr int PER = SEL_BINS / 256;
    // thread t: bins from the top, [t * PER, (t + 1) * PER)
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        c[i] = hist[SEL_BINS - 1 - (threadIdx.x * PER + i)];
        sum += c[i];
    }
    s_sum[threadIdx.x] = sum;
    if (threadIdx.x == 0) s_bin = 0;
    __syncthreads();
    for (int o = 1; o < 256; o <<= 1) {
        const uint32_t v = (int)threadIdx.x >= o ? s_sum[threadIdx.x - o] : 0;
        __syncthreads();
        s_sum[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t above = s_sum[threadIdx.x] - sum;
    if (above < want && s_sum[threadIdx.x] >= want) {
        int bin = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (above < want) {
                above += c[i];
                bin = SEL_BINS - 1 - (threadIdx.x * PER + i);
            }
        s_bin = bin;
    }
    __syncthreads();
    const int bin = s_bin;  // 0 with fewer than `want`
    const uint32_t n = counts->kp;
    for (uint32_t k = blockIdx.x * 256 + threadIdx.x; k < n; k += gridDim.x * 256)
        if (resp_bin(resp[k]) >= bin) {
            const uint32_t at = atomicAdd(&counts->kept, 1u);
            if (at < SEL_CAP) {
                kept.key[at] = resp_key(resp[k]);
                kept.place[at] = place[k];
                kept.kp[at] = k;
            }
        }
}

// Rank of each kept keypoint by counting; skp[rank] = keypoint.  One warp each.
__global__ void __launch_bounds__(256) rank_kernel(const Kept kept, const Counts* __restrict__ counts,
                                                   uint32_t* __restrict__ skp) {
    const uint32_t n = counts->kept;
    if (n > SEL_CAP) return;
    const int lane = threadIdx.x & 31;
    for (uint32_t i = (blockIdx.x * 256 + threadIdx.x) >> 5; i < n; i += gridDim.x * 8) {
        const uint32_t place = kept.place[i];
        const long long key = kept.key[i];
        uint32_t before = 0;
#pragma unroll 8
        for (uint32_t j = lane; j < n; j += 32) {
            const long long q = __ldg(kept.key + j);
            const uint32_t qp = __ldg(kept.place + j);
            before += q > key || (q == key && qp < place);
        }
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        if (lane == 0) skp[before] = kept.kp[i];
    }
}

__device__ __forceinline__ double rem_euclid(double a, double b) {
    // fmod(a, b), b > 0: below 2 b in magnitude the subtraction is exact
    const double m = fabs(a);
    const double r = m < b ? a : m < 2.0 * b ? copysign(m - b, a) : fmod(a, b);
    return r < 0.0 ? r + fabs(b) : r;
}

// sift.rs:274-334.  One block per keypoint, for the keypoints at sorted
// positions base .. base + gridDim.x - 1 (skp[pos] = keypoint), or with `counts`
// as many of them as were kept; theta[4 pos ..] and cnt[pos] (0 when the keypoint
// is outside the 8-pixel margin of the image, sift.rs:519-521, or there is none).
// Bound by the latency of a sample's f64 chain (atan2, exp): five warps take
// the window in two rounds where one warp took ten.  2432 keypoints: 37 -> 29 us.
constexpr int ORI_BINS = 36, ORI_RADIUS = 8, ORI_SIDE = 2 * ORI_RADIUS + 1, ORI_SAMPLES = ORI_SIDE * ORI_SIDE;
constexpr int ORI_THREADS = 160;
__global__ void __launch_bounds__(ORI_THREADS) orient_kernel(KpArrays kp, const uint32_t* __restrict__ skp, int64_t base,
                                                             const Counts* __restrict__ counts,
                                                             const __grid_constant__ OctTable oct, int img_w, int img_h,
                                                             double* __restrict__ theta, int32_t* __restrict__ cnt) {
    __shared__ int sbin[ORI_SAMPLES];
    __shared__ double sval[ORI_SAMPLES];
    __shared__ double shist[2][ORI_BINS];
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t k = base + blockIdx.x;  // output position
    if (counts && (counts->kept > SEL_CAP || blockIdx.x >= counts->kept)) {
        if (tid == 0) cnt[k] = 0;
        return;
    }
    const uint32_t kk = skp[k];
    const double kx = kp.x[kk], ky = kp.y[kk];
    const int o = kp.oct[kk];
    const double scale = oct.scale[o];
    const double x0 = kx * scale, y0 = ky * scale;
    if (x0 < 8.0 || y0 < 8.0 || x0 >= (double)img_w - 8.0 || y0 >= (double)img_h - 8.0) {
        if (tid == 0) cnt[k] = 0;
        return;
    }
    const int w = oct.w[o], h = oct.h[o];
    const float* img = oct.img[o];
    const double sigma = 1.5 * level_sigma(KP_LEVEL);  // 2.4: a radius of ceil(3 sigma) = ORI_RADIUS
    const double s2 = 2.0 * sigma * sigma;
    const long long xr = (long long)round(kx), yr = (long long)round(ky);
    for (int s = tid; s < ORI_SAMPLES; s += ORI_THREADS) {
        int bin = -1;
        double val = 0.0;
        const int dy = s / ORI_SIDE - ORI_RADIUS, dx = s % ORI_SIDE - ORI_RADIUS;
        const long long sx = xr + dx, sy = yr + dy;
        if (!(sx < 1 || sy < 1 || sx >= w - 1 || sy >= h - 1)) {
            const int64_t i = sy * w + sx;
            const float a = img[i + 1] - img[i - 1], b = img[i + w] - img[i - w];  // sift.rs:137-149
            const double mag = sqrt((double)(a * a + b * b));
            const double ang = atan2((double)b, (double)a);
            const double wgt = exp((-((double)dx * (double)dx) - (double)dy * (double)dy) / s2);
            const double fb = floor((ang + PI) / (2.0 * PI) * 36.0);
            bin = !(fb > 0.0) ? 0 : (int)((long long)fb % 36);
            val = wgt * mag;
        }
        sbin[s] = bin;
        sval[s] = val;
    }
    __syncthreads();
    // thread b's bin: its samples in window order
    if (tid < ORI_BINS) {
        double acc = 0.0;
#pragma unroll 17
        for (int t = 0; t < ORI_SAMPLES; ++t) {
            const double v = sval[t];
            if (sbin[t] == tid) acc += v;
        }
        shist[0][tid] = acc;
    }
    __syncthreads();
    for (int it = 0; it < 2; ++it) {
        const double* from = shist[it];
        if (tid < ORI_BINS)
            shist[it ^ 1][tid] = (from[(tid + 35) % 36] + 2.0 * from[tid] + from[(tid + 1) % 36]) / 4.0;
        __syncthreads();
    }
    if (tid >= 32) return;
    // the peaks, in bin order
    const int b0 = lane, b1 = lane + 32;
    const double* hist = shist[0];
    double maxv = fmax(hist[b0], b1 < 36 ? hist[b1] : 0.0);
    for (int o = 16; o > 0; o >>= 1) maxv = fmax(maxv, __shfl_xor_sync(0xffffffffu, maxv, o));
    maxv = fmax(0.0, maxv);
    if (maxv < 1e-12) {
        if (lane == 0) {
            theta[4 * k] = 0.0;
            cnt[k] = 1;
        }
        return;
    }
    const double thresh = 0.8 * maxv;
    auto peak = [&](int b, double& th) -> bool {
        if (b >= 36) return false;
        const double prev = hist[(b + 35) % 36], next = hist[(b + 1) % 36];
        if (!(hist[b] > prev && hist[b] > next && hist[b] >= thresh)) return false;
        const double denom = hist[b] * 2.0 - prev - next;
        const double d = fabs(denom) > 1e-12 ? 0.5 * (prev - next) / denom : 0.0;
        th = rem_euclid(((double)b + d) / 36.0 * 2.0 * PI - PI, 2.0 * PI);
        return true;
    };
    double t0 = 0.0, t1 = 0.0;
    const unsigned m0 = __ballot_sync(0xffffffffu, peak(b0, t0)), m1 = __ballot_sync(0xffffffffu, peak(b1, t1));
    const int at0 = __popc(m0 & ((1u << lane) - 1u)), at1 = __popc(m0) + __popc(m1 & ((1u << lane) - 1u));
    if (((m0 >> lane) & 1u) && at0 < 4) theta[4 * k + at0] = t0;
    if (((m1 >> lane) & 1u) && at1 < 4) theta[4 * k + at1] = t1;
    if (lane == 0) {
        const int np = min(__popc(m0) + __popc(m1), 4);
        if (np == 0) theta[4 * k] = 0.0;
        cnt[k] = max(np, 1);
    }
}

// The pairs of the first n positions in one block: offsets by a scan of cnt,
// then pairs_kernel's entries; counts->pairs.
__global__ void __launch_bounds__(1024) first_pairs_kernel(const uint32_t* __restrict__ skp, int n,
                                                           const int32_t* __restrict__ cnt,
                                                           const double* __restrict__ theta,
                                                           int32_t* __restrict__ pair_kp,
                                                           double* __restrict__ pair_theta, Counts* __restrict__ counts) {
    __shared__ int warp_sum[32];
    __shared__ int s_base;
    if (threadIdx.x == 0) s_base = 0;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int b = 0; b < n; b += 1024) {
        const int pos = b + threadIdx.x;
        const int c = pos < n ? cnt[pos] : 0;
        int x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int v = warp_sum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += y;
            }
            warp_sum[lane] = v;
        }
        __syncthreads();
        const int at = s_base + (wid ? warp_sum[wid - 1] : 0) + x - c;
        for (int p = 0; p < c; ++p) {
            pair_kp[at + p] = (int32_t)skp[pos];
            pair_theta[at + p] = theta[4 * (int64_t)pos + p];
        }
        __syncthreads();
        if (threadIdx.x == 0) s_base += warp_sum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) counts->pairs = (uint32_t)s_base;
}

// (keypoint, peak) pairs of the keypoints at sorted positions base ..
// base + n - 1, peaks in order, appended at pair index at + off[i] + p.
__global__ void pairs_kernel(const uint32_t* __restrict__ skp, int64_t base, int n, const int32_t* __restrict__ cnt,
                             const int32_t* __restrict__ off, const double* __restrict__ theta, int64_t at,
                             int32_t* __restrict__ pair_kp, double* __restrict__ pair_theta) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int64_t pos = base + i;
        for (int p = 0; p < cnt[pos]; ++p) {
            pair_kp[at + off[i] + p] = (int32_t)skp[pos];
            pair_theta[at + off[i] + p] = theta[4 * pos + p];
        }
    }
}

__global__ void gather_resp_kernel(const double* __restrict__ resp, const uint32_t* __restrict__ idx, int64_t n,
                                   double* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = resp[idx[i]];
}

__global__ void iota_kernel(uint32_t* __restrict__ out, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (uint32_t)i;
}

// sift.rs:340-431.  One block per (keypoint, peak) pair, for the pairs
// base .. base + gridDim.x - 1 (in output order), or with `counts` those of
// them that exist; descriptor and validity stored at the pair's index.  Bound
// by the samples' f64 functions, so the samples of the rotated window (three
// fifths of the square) are first packed, by an approximate test with a margin,
// and each cell walks a list of its own samples (about 90).  2048 descriptors:
// 187 us without the two, 73 us.
//
// Lattice points in a square of side s number at most (s + sqrt 2)^2 (their
// unit squares are disjoint and lie within sqrt(1/2) of it): 645 in the window,
// of 5 cells' side, and 121 that touch one cell, in 2 cells' side.
constexpr int DESC_RADIUS = 15, DESC_SIDE = 2 * DESC_RADIUS + 1, DESC_SAMPLES = DESC_SIDE * DESC_SIDE;
constexpr int DESC_HITS = 648, CELL_HITS = 124;
struct DescSmem {
    double w[DESC_HITS], fx[DESC_HITS], fy[DESC_HITS], fo[DESC_HITS];
    uint16_t hdr[DESC_HITS + 32];  // (by0 + 2, bx0 + 2, ob0 mod 8) of 4 bits each, or 0xFFFF
    union {
        uint16_t cand[DESC_HITS];         // the samples of the window, in order
        uint16_t cell[16][CELL_HITS];     // a cell's: index, ob0 << 10, upper column << 13, upper row << 14
    };
    float sq[DESC_LEN];
    double cos_t, sin_t;
    float norm;
    int count[4];
};
__global__ void __launch_bounds__(DESC_LEN, 8) desc_kernel(KpArrays kp, int64_t base, const int32_t* __restrict__ pair_kp,
                                                          const double* __restrict__ pair_theta,
                                                          const Counts* __restrict__ counts,
                                                          const __grid_constant__ OctTable oct, float* __restrict__ desc,
                                                          uint8_t* __restrict__ valid) {
    constexpr int D = 4, N = 8, ROUNDS = (DESC_SAMPLES + DESC_LEN - 1) / DESC_LEN;
    __shared__ DescSmem sm;
    const int64_t pos = base + blockIdx.x;
    if (counts && pos >= (int64_t)counts->pairs) return;
    const int k = pair_kp[pos];
    const double x = kp.x[k], y = kp.y[k], th = pair_theta[pos];
    const int o = kp.oct[k];
    const int w = oct.w[o], h = oct.h[o];
    const float* img = oct.img[o];
    // 4.8: a radius of ceil(sqrt(1.5) cell (D + 1) / 2) = DESC_RADIUS
    const double cell = 3.0 * level_sigma(KP_LEVEL);
    const double half = (double)D * 0.5;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (wid == 0) sm.cos_t = cos(th);
    if (wid == 1) sm.sin_t = sin(th);
    __syncthreads();
    const double cos_t = sm.cos_t, sin_t = sm.sin_t;
    {
        // warp w: samples [32 ROUNDS w, 32 ROUNDS (w + 1))
        const double inv = 1.0 / cell, lo = -1.0 - 1e-6, hi = (double)D + 1e-6;
        unsigned m[ROUNDS];
        int n = 0;
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            const int s = (wid * ROUNDS + r) * 32 + lane;
            const int dy = s / DESC_SIDE - DESC_RADIUS, dx = s % DESC_SIDE - DESC_RADIUS;
            const double sx = x + (double)dx, sy = y + (double)dy;
            const double bx = (cos_t * (double)dx + sin_t * (double)dy) * inv + half - 0.5;
            const double by = (-sin_t * (double)dx + cos_t * (double)dy) * inv + half - 0.5;
            m[r] = __ballot_sync(0xffffffffu, s < DESC_SAMPLES && !(sx < 1.0 || sy < 1.0 || sx >= (double)w - 2.0 ||
                                                                   sy >= (double)h - 2.0) &&
                                                  bx >= lo && by >= lo && bx <= hi && by <= hi);
            n += __popc(m[r]);
        }
        if (lane == 0) sm.count[wid] = n;
        __syncthreads();
        int at = 0;
        for (int i = 0; i < wid; ++i) at += sm.count[i];
#pragma unroll
        for (int r = 0; r < ROUNDS; ++r) {
            if ((m[r] >> lane) & 1u) sm.cand[at + __popc(m[r] & ((1u << lane) - 1u))] = (uint16_t)((wid * ROUNDS + r) * 32 + lane);
            at += __popc(m[r]);
        }
    }
    const int n = sm.count[0] + sm.count[1] + sm.count[2] + sm.count[3];
    __syncthreads();
    const double exp_scale = -1.0 / ((double)(D * D) * 0.5);
    for (int i = tid; i < n + 32; i += DESC_LEN) {
        int hd = 0xFFFF;
        const int s = i < n ? sm.cand[i] : 0;
        const int dy = s / DESC_SIDE - DESC_RADIUS, dx = s % DESC_SIDE - DESC_RADIUS;
        const double rx = cos_t * (double)dx + sin_t * (double)dy;
        const double ry = -sin_t * (double)dx + cos_t * (double)dy;
        const double bx = rx / cell + half - 0.5;
        const double by = ry / cell + half - 0.5;
        if (i < n && !(bx < -1.0 || by < -1.0 || bx > (double)D || by > (double)D)) {
            // sift.rs:137-166: bilinear gradients; 1 <= x0, x0 + 1 <= w - 2, so no
            // clamp applies and every gradient is a central difference
            const double sx = x + (double)dx, sy = y + (double)dy;
            const int x0 = (int)floor(sx), y0 = (int)floor(sy);
            const float fx = (float)(sx - (double)x0), fy = (float)(sy - (double)y0);
            const float* p = img + (int64_t)y0 * w + x0;
            const float a0 = p[-1], a1 = p[0], a2 = p[1], a3 = p[2];
            const float b0 = p[w - 1], b1 = p[w], b2 = p[w + 1], b3 = p[w + 2];
            const float u1 = p[-w], u2 = p[-w + 1], d1 = p[2 * w], d2 = p[2 * w + 1];
            const float gxa = (a2 - a0) * (1.0f - fx) + (a3 - a1) * fx, gxb = (b2 - b0) * (1.0f - fx) + (b3 - b1) * fx;
            const float gya = (b1 - u1) * (1.0f - fx) + (b2 - u2) * fx, gyb = (d1 - a1) * (1.0f - fx) + (d2 - a2) * fx;
            const double gx = (double)(gxa * (1.0f - fy) + gxb * fy);
            const double gy = (double)(gya * (1.0f - fy) + gyb * fy);
            const double mag = sqrt(gx * gx + gy * gy);
            if (!(mag < 1e-12)) {
                const double ang = atan2(gy, gx) - th;
                const double ob = rem_euclid(ang, 2.0 * PI) / (2.0 * PI) * (double)N;
                double wgt = ((bx - half + 0.5) * (bx - half + 0.5) + (by - half + 0.5) * (by - half + 0.5)) * exp_scale;
                wgt = exp(wgt) * mag;
                // bx, by in [-1, 4], ob in [0, 8]
                const int bx0 = (int)floor(bx), by0 = (int)floor(by), ob0 = (int)floor(ob);
                sm.w[i] = wgt;
                sm.fx[i] = bx - (double)bx0;
                sm.fy[i] = by - (double)by0;
                sm.fo[i] = ob - (double)ob0;
                hd = ((by0 + 2) << 8) | ((bx0 + 2) << 4) | (ob0 & 7);
            }
        }
        sm.hdr[i] = (uint16_t)hd;
    }
    __syncthreads();
    // Warp q makes the lists of cell row q.
    const int cx = lane >> 3, co = lane & 7, q = wid;
    int hits = 0;  // of this lane's cell
    {
        int at[4] = {0, 0, 0, 0};
        for (int b = 0; b < n; b += 32) {
            const int hv = sm.hdr[b + lane];
            const int row = q + 2 - (hv >> 8), col = ((hv >> 4) & 15) - 2;  // row 0xFFFF: negative
            const int e = (b + lane) | (hv & 7) << 10 | row << 14;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const bool mine = (unsigned)row <= 1u && (unsigned)(c - col) <= 1u;
                const unsigned m = __ballot_sync(0xffffffffu, mine);
                if (mine) sm.cell[4 * q + c][at[c] + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(e | (c - col) << 13);
                at[c] += __popc(m);
            }
        }
        hits = cx == 0 ? at[0] : cx == 1 ? at[1] : cx == 2 ? at[2] : at[3];
    }
    __syncwarp();
    // Thread t owns bin t: cell row q, cell column lane / 8, orientation lane % 8.
    // A sample adds to a bin at most once, in window order.
    double acc = 0.0;
    const uint16_t* list = sm.cell[4 * q + cx];
#pragma unroll 4
    for (int j = 0; j < hits; ++j) {
        const int e = list[j];
        const int s = e & 1023, io = (co - (e >> 10)) & 7;
        const double wgt = sm.w[s], fx = sm.fx[s], fy = sm.fy[s], fo = sm.fo[s];
        if (io <= 1) {
            const double wy = e & (1 << 14) ? fy : 1.0 - fy;
            const double wx = e & (1 << 13) ? fx : 1.0 - fx;
            const double wo = io ? fo : 1.0 - fo;
            acc += wgt * wx * wy * wo;
        }
    }
    // the serial f32 sums of the reference; the elementwise steps by all
    float d = (float)acc;
    auto norm = [&]() -> float {
        sm.sq[tid] = d * d;
        __syncthreads();
        if (tid == 0) {
            float ss = 0.0f;
#pragma unroll 16
            for (int i = 0; i < DESC_LEN; ++i) ss = ss + sm.sq[i];
            sm.norm = sqrtf(ss);
        }
        __syncthreads();
        return sm.norm;
    };
    float nm = norm();
    bool ok = !(nm < 1e-6f);
    if (ok) {
        d = d / nm;
        if (d > 0.2f) d = 0.2f;
        nm = norm();  // sm.norm and sm.sq are read before the next writes: both sides synchronise
        ok = !(nm < 1e-6f);
        if (ok) d = d / nm;
    }
    desc[pos * DESC_LEN + tid] = d;
    if (tid == 0) valid[pos] = ok ? 1 : 0;
}

// The valid ones among the first min(counts->pairs, cap) pairs, in order, in
// one block; counts->valid.
__global__ void __launch_bounds__(1024) first_valid_kernel(const uint8_t* __restrict__ valid, int cap,
                                                           uint32_t* __restrict__ sel, Counts* __restrict__ counts) {
    __shared__ int warp_sum[32];
    __shared__ int s_base;
    if (threadIdx.x == 0) s_base = 0;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n = (int)min(counts->pairs, (uint32_t)cap);
    __syncthreads();
    for (int b = 0; b < n; b += 1024) {
        const int i = b + threadIdx.x;
        const bool v = i < n && valid[i];
        const unsigned m = __ballot_sync(0xffffffffu, v);
        if (lane == 0) warp_sum[wid] = __popc(m);
        __syncthreads();
        int before = s_base;
        for (int k = 0; k < wid; ++k) before += warp_sum[k];
        if (v) sel[before + __popc(m & ((1u << lane) - 1u))] = (uint32_t)i;
        __syncthreads();
        if (threadIdx.x == 1023) s_base = before + __popc(m);
        __syncthreads();
    }
    if (threadIdx.x == 0) counts->valid = (uint32_t)s_base;
}

// sift.rs:543-554: output i is the pair sel[i] (the i-th valid descriptor in
// response order), of n or with `counts` of the valid ones; clamped position,
// descriptor, colour.
__global__ void final_kernel(const uint32_t* __restrict__ sel, int n, const Counts* __restrict__ counts,
                             const int32_t* __restrict__ pair_kp, KpArrays kp, const __grid_constant__ OctTable oct,
                             const float* __restrict__ desc, const uint8_t* __restrict__ rgb, int w, int h,
                             double* __restrict__ pts, float* __restrict__ odesc, uint8_t* __restrict__ col) {
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (wid >= n || (counts && (uint32_t)wid >= counts->valid)) return;
    const uint32_t pos = sel[wid];
    if (lane == 0) {
        const int k = pair_kp[pos];
        const double scale = oct.scale[kp.oct[k]];
        const double x = fmin(fmax(kp.x[k] * scale, 0.0), (double)(w - 1));
        const double y = fmin(fmax(kp.y[k] * scale, 0.0), (double)(h - 1));
        const long long px = min((long long)round(x), (long long)(w - 1));
        const long long py = min((long long)round(y), (long long)(h - 1));
        pts[2 * wid] = x;
        pts[2 * wid + 1] = y;
        for (int c = 0; c < 3; ++c) col[3 * wid + c] = rgb[3 * (py * w + px) + c];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
        odesc[(int64_t)wid * DESC_LEN + lane + 32 * q] = desc[(int64_t)pos * DESC_LEN + lane + 32 * q];
}

unsigned grid_of(int64_t n, int threads = 256) {
    const int64_t b = (n + threads - 1) / threads;
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 16));
}

// sift.rs:51-63: f64 kernel weights, normalised, cast to f32 per tap
bool blur_taps(double sigma, BlurTaps& t) {
    const int radius = (int)std::max(std::ceil(sigma * 3.0), 1.0);
    if (2 * radius + 1 > MAX_TAPS) return false;
    std::vector<double> k(2 * radius + 1);
    const double s2 = 2.0 * sigma * sigma;
    double sum = 0.0;
    for (int i = 0; i < 2 * radius + 1; ++i) {
        const double x = (double)i - (double)radius;
        k[i] = std::exp(-x * x / s2);
        sum += k[i];
    }
    t.radius = radius;
    for (int i = 0; i < 2 * radius + 1; ++i) t.k[i] = (float)(k[i] / sum);
    return true;
}

// Taps that return their input: exactly 0 but for a 1 in the middle (0 x + a
// and 1 x are exact for finite x).
bool identity_taps(const BlurTaps& t) {
    for (int i = 0; i <= 2 * t.radius; ++i)
        if (t.k[i] != (i == t.radius ? 1.0f : 0.0f)) return false;
    return true;
}

int sfail(rcmvs_ctx* ctx, int code, const std::string& msg) {
    if (ctx) ctx->err = msg;
    return code;
}

#define SCK(x)                                                                                 \
    do {                                                                                       \
        cudaError_t e_ = (x);                                                                  \
        if (e_ != cudaSuccess)                                                                 \
            return sfail(ctx, e_ == cudaErrorMemoryAllocation ? RCMVS_E_NOMEM : RCMVS_E_CUDA,    \
                         std::string(#x) + ": " + cudaGetErrorString(e_));                     \
    } while (0)

// max_features up to which the first keypoints are selected, oriented and
// described without waiting for their counts, and how many keypoints that
// takes beyond max_features (margins drop some, extra peaks add some).
constexpr int64_t QUICK_CAP = 8192;
int64_t quick_keypoints(int64_t cap) { return cap + cap / 8 + 64; }

// Context arena slots 80-159.
enum {
    F_IN = 80, F_GRAY, F_RGB, F_KPX, F_KPY, F_KPRESP, F_KPPLACE, F_KPOCT, F_TEMP, F_THETA, F_CNT, F_OFF, F_PKP, F_PTH,
    F_PIDX, F_PLACE2, F_PIDX2, F_SRESP, F_SRESP2, F_SIDX, F_DESC, F_VALID, F_OSEL, F_PTS, F_FDESC, F_COL, F_COUNTS,
    F_HIST, F_KEPT, F_NSEL,
    F_LEV = 130  // + octave: its level 0 (octaves 0..7)
};

// Grows an arena slot to `need` bytes keeping its first `keep` bytes: a
// device-to-device copy into a buffer of twice the need when the slot is too
// small, else the slot as it is.
int grow_copy(rcmvs_ctx* ctx, int slot, size_t need, size_t keep, void** p) {
    DeviceArena& A = ctx->arena;
    if ((int)A.slots.size() <= slot) A.slots.resize(slot + 1);
    DeviceArena::Slot& s = A.slots[slot];
    if (s.p && s.bytes >= need) {
        *p = s.p;
        return RCMVS_OK;
    }
    void* np_ = nullptr;
    const size_t cap = std::max<size_t>(2 * need, 1 << 20);
    SCK(cudaMalloc(&np_, cap));
    if (keep && s.p) SCK(cudaMemcpyAsync(np_, s.p, keep, cudaMemcpyDeviceToDevice, ctx->stream));
    SCK(cudaStreamSynchronize(ctx->stream));
    if (s.p) SCK(cudaFree(s.p));
    s.p = np_;
    s.bytes = cap;
    *p = np_;
    return RCMVS_OK;
}

}  // namespace
}  // namespace rcmvs

using namespace rcmvs;

extern "C" {

void rcmvs_sift_options_default(rcmvs_sift_options* o) {
    if (!o) return;
    o->max_dim = 1600;  // sift.rs:28-31
    o->max_features = 2048;
    o->reserved = 0;
    o->reserved2 = 0;
    o->contrast_thr = 0.0067;
}

void rcmvs_sift_frame_free(rcmvs_sift_frame* f) {
    if (!f) return;
    std::free(f->pts);
    std::free(f->desc);
    std::free(f->colors);
    f->pts = nullptr;
    f->desc = nullptr;
    f->colors = nullptr;
    f->n = 0;
}

int rcmvs_extract_sift(rcmvs_ctx* ctx, const uint8_t* img, int32_t w0, int32_t h0, int32_t channels,
                       const rcmvs_sift_options* opts, rcmvs_sift_frame* out) {
    if (!ctx || !img || !opts || !out) return sfail(ctx, RCMVS_E_ARG, "rcmvs_extract_sift: bad argument");
    std::memset(out, 0, sizeof(*out));
    // sift.rs:436-444: resize so the long side is at most max_dim (sides >= 1)
    int32_t w = w0, h = h0;
    const int32_t m = std::max(w0, h0);
    if (m > 0 && (uint32_t)m > opts->max_dim) {
        const double s = (double)opts->max_dim / (double)m;
        w = (int32_t)std::max(std::round((double)w0 * s), 1.0);
        h = (int32_t)std::max(std::round((double)h0 * s), 1.0);
    }
    int rc = resize_check(ctx, w0, h0, channels, w, h);
    if (rc) return rc;
    SCK(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    DeviceArena& A = ctx->arena;
    const int64_t n_in = (int64_t)w0 * h0, npx0 = (int64_t)w * h;
    if (NSPO * npx0 > (int64_t)UINT32_MAX) return sfail(ctx, RCMVS_E_LIMIT, "sift: octave too large");
    void *p_in, *p_gray, *p_rgb;
    SCK(A.get(F_IN, (size_t)n_in * channels, &p_in));
    SCK(A.get(F_GRAY, (size_t)npx0, &p_gray));
    SCK(A.get(F_RGB, 3 * (size_t)npx0, &p_rgb));
    SCK(host_upload(p_in, img, (size_t)n_in * channels, st));
    const int* d_err = nullptr;
    rc = resize_device(ctx, (const uint8_t*)p_in, w0, h0, channels, w, h, (uint8_t*)p_gray, (uint8_t*)p_rgb, &d_err);
    if (rc) return rc;

    int n_oct = 1;  // sift.rs:458-461
    while ((std::max(w, h) >> n_oct) >= 40 && n_oct < 8) ++n_oct;
    if (n_oct > MAX_OCT) return sfail(ctx, RCMVS_E_LIMIT, "sift: too many octaves");
    BlurTaps first{}, inc[NLEV];
    const double fs = std::sqrt(std::max(SIGMA0 * SIGMA0 - ASSUMED_BLUR * ASSUMED_BLUR, 1e-4));
    if (!blur_taps(fs, first)) return sfail(ctx, RCMVS_E_LIMIT, "sift: blur kernel too wide");
    for (int l = 1; l < NLEV; ++l) {
        const double sp = level_sigma(l - 1), sc = level_sigma(l);
        if (!blur_taps(std::sqrt(std::max(sc * sc - sp * sp, 1e-4)), inc[l]))
            return sfail(ctx, RCMVS_E_LIMIT, "sift: blur kernel too wide");
        if (l != NSPO && !identity_taps(inc[l])) return sfail(ctx, RCMVS_E_STATE, "sift: levels of one sigma differ");
    }
    if (first.radius != R_BASE || inc[NSPO].radius != R_LEVEL) return sfail(ctx, RCMVS_E_STATE, "sift: blur radius");

    const SpanHook& hook = ctx->hook();
    const int64_t cap = (int64_t)opts->max_features;
    // keypoint arrays sized for every pixel of every octave
    OctTable table{};
    int64_t kcap = 0;
    for (int o = 0, tw = w, th = h; o < n_oct; ++o, tw = std::max(tw / 2, 1), th = std::max(th / 2, 1)) {
        void* p;
        SCK(A.get(F_LEV + o, sizeof(float) * (size_t)tw * th, &p));
        table.img[o] = (const float*)p;
        table.w[o] = tw;
        table.h[o] = th;
        table.scale[o] = std::pow(2.0, o);
        kcap += (int64_t)tw * th;
    }
    KpArrays kp{};
    Counts* d_counts;
    uint32_t* d_hist;
    {
        void *p_x, *p_y, *p_r, *p_l, *p_o, *p_c;
        SCK(A.get(F_KPX, 8 * (size_t)kcap, &p_x));
        SCK(A.get(F_KPY, 8 * (size_t)kcap, &p_y));
        SCK(A.get(F_KPRESP, 8 * (size_t)kcap, &p_r));
        SCK(A.get(F_KPPLACE, 4 * (size_t)kcap, &p_l));
        SCK(A.get(F_KPOCT, 4 * (size_t)kcap, &p_o));
        kp = KpArrays{(double*)p_x, (double*)p_y, (double*)p_r, (uint32_t*)p_l, (int32_t*)p_o};
        SCK(A.get(F_COUNTS, sizeof(Counts) + sizeof(uint32_t) * SEL_BINS, &p_c));
        d_counts = (Counts*)p_c;
        d_hist = (uint32_t*)(d_counts + 1);
    }
    SCK(cudaMemsetAsync(d_counts, 0, sizeof(Counts) + sizeof(uint32_t) * SEL_BINS, st));
    hook.begin("sift_pyramid");
    base_kernel<<<((w + BX - 1) / BX) * ((h + BY - 1) / BY), BLUR_THREADS, 0, st>>>((const uint8_t*)p_gray, w, h, first,
                                                                                   const_cast<float*>(table.img[0]));
    SCK(cudaGetLastError());
    hook.end("sift_pyramid");
    hook.begin("sift_extrema");
    int64_t place = 0;
    for (int o = 0; o < n_oct; ++o) {
        const int ow = table.w[o], oh = table.h[o];
        const bool more = o + 1 < n_oct;
        octave_kernel<<<((ow + BX - 3) / (BX - 2)) * ((oh + BY - 3) / (BY - 2)), BLUR_THREADS, 0, st>>>(
            table.img[o], ow, oh, inc[NSPO], opts->contrast_thr, more ? const_cast<float*>(table.img[o + 1]) : nullptr,
            more ? table.w[o + 1] : 0, more ? table.h[o + 1] : 0, o, (uint32_t)place, kp, d_counts);
        SCK(cudaGetLastError());
        place += (int64_t)ow * oh;
    }
    hook.end("sift_extrema");

    int64_t n_valid = 0;
    void *p_skp = nullptr, *p_th = nullptr, *p_cnt = nullptr, *p_pkp = nullptr, *p_pth = nullptr, *p_desc = nullptr,
         *p_valid = nullptr, *p_osel = nullptr, *p_pts = nullptr, *p_fdesc = nullptr, *p_col = nullptr;
    const bool quick = cap > 0 && cap <= QUICK_CAP;
    const int64_t want = quick_keypoints(cap);
    if (quick) {
        void* p_kept;
        SCK(A.get(F_KEPT, 16 * (size_t)SEL_CAP, &p_kept));
        SCK(A.get(F_SIDX, sizeof(uint32_t) * SEL_CAP, &p_skp));
        SCK(A.get(F_THETA, sizeof(double) * 4 * (size_t)want, &p_th));
        SCK(A.get(F_CNT, sizeof(int32_t) * (size_t)want, &p_cnt));
        SCK(A.get(F_PKP, sizeof(int32_t) * 4 * (size_t)want, &p_pkp));
        SCK(A.get(F_PTH, sizeof(double) * 4 * (size_t)want, &p_pth));
        SCK(A.get(F_VALID, (size_t)cap, &p_valid));
        SCK(A.get(F_OSEL, sizeof(uint32_t) * (size_t)cap, &p_osel));
        if ((rc = grow_copy(ctx, F_DESC, sizeof(float) * DESC_LEN * (size_t)cap, 0, &p_desc))) return rc;
        SCK(A.get(F_PTS, sizeof(double) * 2 * cap, &p_pts));
        SCK(A.get(F_FDESC, sizeof(float) * DESC_LEN * cap, &p_fdesc));
        SCK(A.get(F_COL, 3 * (size_t)cap, &p_col));
        hist_kernel<<<64, 256, 0, st>>>(kp.resp, d_counts, d_hist);
        SCK(cudaGetLastError());
        const Kept kept{(long long*)p_kept, (uint32_t*)((long long*)p_kept + SEL_CAP),
                        (uint32_t*)((long long*)p_kept + SEL_CAP) + SEL_CAP};
        keep_kernel<<<64, 256, 0, st>>>(kp.resp, d_hist, kp.place, (uint32_t)want, d_counts, kept);
        SCK(cudaGetLastError());
        rank_kernel<<<148 * 2, 256, 0, st>>>(kept, d_counts, (uint32_t*)p_skp);
        SCK(cudaGetLastError());
        hook.begin("sift_orient");
        orient_kernel<<<(unsigned)want, ORI_THREADS, 0, st>>>(
            kp, (const uint32_t*)p_skp, 0, d_counts, table, w, h, (double*)p_th, (int32_t*)p_cnt);
        SCK(cudaGetLastError());
        hook.end("sift_orient");
        first_pairs_kernel<<<1, 1024, 0, st>>>((const uint32_t*)p_skp, (int)want, (const int32_t*)p_cnt,
                                               (const double*)p_th, (int32_t*)p_pkp, (double*)p_pth, d_counts);
        SCK(cudaGetLastError());
        hook.begin("sift_desc");
        desc_kernel<<<(unsigned)cap, DESC_LEN, 0, st>>>(kp, 0, (const int32_t*)p_pkp, (const double*)p_pth, d_counts,
                                                        table, (float*)p_desc, (uint8_t*)p_valid);
        SCK(cudaGetLastError());
        hook.end("sift_desc");
        first_valid_kernel<<<1, 1024, 0, st>>>((const uint8_t*)p_valid, (int)cap, (uint32_t*)p_osel, d_counts);
        SCK(cudaGetLastError());
        final_kernel<<<(int)((cap + WARPS - 1) / WARPS), 32 * WARPS, 0, st>>>(
            (const uint32_t*)p_osel, (int)cap, d_counts, (const int32_t*)p_pkp, kp, table, (const float*)p_desc,
            (const uint8_t*)p_rgb, w, h, (double*)p_pts, (float*)p_fdesc, (uint8_t*)p_col);
        SCK(cudaGetLastError());
    }
    int bad = 0;
    Counts hc{};
    if (d_err) SCK(cudaMemcpyAsync(&bad, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    SCK(cudaMemcpyAsync(&hc, d_counts, sizeof(Counts), cudaMemcpyDeviceToHost, st));
    SCK(cudaStreamSynchronize(st));
    if (bad) return sfail(ctx, RCMVS_E_CUDA, "sift: resize tap table overflow");
    const int64_t nkp = hc.kp;  // keypoints of all octaves
    const uint64_t n_raw = (uint64_t)nkp;
    if (nkp > INT32_MAX / 4) return sfail(ctx, RCMVS_E_LIMIT, "sift: too many keypoints");
    // the quick path's answer stands when it filled the cap, or when it took
    // every keypoint and described every pair of them
    const bool all_taken = hc.kept == hc.kp && nkp <= want && (int64_t)hc.pairs <= cap;
    const bool done_quick = quick && hc.kept <= (uint32_t)SEL_CAP && ((int64_t)hc.valid == cap || all_taken);
    if (done_quick) {
        n_valid = hc.valid;
    } else if (nkp > 0 && cap > 0) {
        // The general path: all keypoints by (response descending, place), then
        // orientations, pairs and descriptors in that order until max_features
        // valid descriptors exist (a descriptor that normalises to nothing is
        // dropped, as in the reference).
        thrust::counting_iterator<uint32_t> it(0);
        void *p_temp, *p_off, *p_kidx, *p_place2, *p_kidx2, *p_r1, *p_r2, *p_nsel;
        int64_t kdone = 0, np = 0, done = 0;
        SCK(A.get(F_NSEL, sizeof(int) * 4, &p_nsel));
        SCK(A.get(F_PIDX, sizeof(uint32_t) * (size_t)nkp, &p_kidx));
        SCK(A.get(F_PLACE2, sizeof(uint32_t) * (size_t)nkp, &p_place2));
        SCK(A.get(F_PIDX2, sizeof(uint32_t) * (size_t)nkp, &p_kidx2));
        SCK(A.get(F_SRESP, sizeof(double) * (size_t)nkp, &p_r1));
        SCK(A.get(F_SRESP2, sizeof(double) * (size_t)nkp, &p_r2));
        SCK(A.get(F_SIDX, sizeof(uint32_t) * (size_t)std::max<int64_t>(nkp, SEL_CAP), &p_skp));
        SCK(A.get(F_THETA, sizeof(double) * 4 * (size_t)nkp, &p_th));
        SCK(A.get(F_CNT, sizeof(int32_t) * (size_t)nkp, &p_cnt));
        SCK(A.get(F_OFF, sizeof(int32_t) * (size_t)nkp, &p_off));
        SCK(A.get(F_PKP, sizeof(int32_t) * 4 * (size_t)nkp, &p_pkp));
        SCK(A.get(F_PTH, sizeof(double) * 4 * (size_t)nkp, &p_pth));
        SCK(A.get(F_VALID, 4 * (size_t)nkp, &p_valid));
        SCK(A.get(F_OSEL, sizeof(uint32_t) * 4 * (size_t)nkp, &p_osel));
        iota_kernel<<<grid_of(nkp), 256, 0, st>>>((uint32_t*)p_kidx, nkp);
        SCK(cudaGetLastError());
        size_t tb1 = 0, tb2 = 0;
        SCK(cub::DeviceRadixSort::SortPairs(nullptr, tb1, (const uint32_t*)kp.place, (uint32_t*)p_place2,
                                            (const uint32_t*)p_kidx, (uint32_t*)p_kidx2, (int)nkp, 0, 32, st));
        SCK(cub::DeviceRadixSort::SortPairsDescending(nullptr, tb2, (const double*)p_r1, (double*)p_r2,
                                                      (const uint32_t*)p_kidx2, (uint32_t*)p_skp, (int)nkp, 0, 64, st));
        SCK(A.get(F_TEMP, std::max(tb1, tb2), &p_temp));
        SCK(cub::DeviceRadixSort::SortPairs(p_temp, tb1, (const uint32_t*)kp.place, (uint32_t*)p_place2,
                                            (const uint32_t*)p_kidx, (uint32_t*)p_kidx2, (int)nkp, 0, 32, st));
        gather_resp_kernel<<<grid_of(nkp), 256, 0, st>>>(kp.resp, (const uint32_t*)p_kidx2, nkp, (double*)p_r1);
        SCK(cudaGetLastError());
        SCK(cub::DeviceRadixSort::SortPairsDescending(p_temp, tb2, (const double*)p_r1, (double*)p_r2,
                                                      (const uint32_t*)p_kidx2, (uint32_t*)p_skp, (int)nkp, 0, 64, st));
        while (n_valid < cap && (done < np || kdone < nkp)) {
            if (done == np) {
                // orientations of the next keypoints in response order, and their pairs
                const int64_t ck = std::min<int64_t>(nkp - kdone, std::max<int64_t>(cap - n_valid, 64));
                hook.begin("sift_orient");
                orient_kernel<<<(unsigned)ck, ORI_THREADS, 0, st>>>(
                    kp, (const uint32_t*)p_skp, kdone, nullptr, table, w, h, (double*)p_th, (int32_t*)p_cnt);
                SCK(cudaGetLastError());
                hook.end("sift_orient");
                size_t tb = 0;
                SCK(cub::DeviceScan::ExclusiveSum(nullptr, tb, (const int32_t*)p_cnt + kdone, (int32_t*)p_off, (int)ck,
                                                  st));
                SCK(A.get(F_TEMP, tb, &p_temp));
                SCK(cub::DeviceScan::ExclusiveSum(p_temp, tb, (const int32_t*)p_cnt + kdone, (int32_t*)p_off, (int)ck,
                                                  st));
                pairs_kernel<<<grid_of(ck), 256, 0, st>>>((const uint32_t*)p_skp, kdone, (int)ck, (const int32_t*)p_cnt,
                                                          (const int32_t*)p_off, (const double*)p_th, np,
                                                          (int32_t*)p_pkp, (double*)p_pth);
                SCK(cudaGetLastError());
                int last_off = 0, last_cnt = 0;
                SCK(cudaMemcpyAsync(&last_off, (int32_t*)p_off + ck - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
                SCK(cudaMemcpyAsync(&last_cnt, (int32_t*)p_cnt + kdone + ck - 1, sizeof(int), cudaMemcpyDeviceToHost,
                                    st));
                SCK(cudaStreamSynchronize(st));
                kdone += ck;
                np += (int64_t)last_off + last_cnt;
                continue;
            }
            const int64_t chunk = std::min<int64_t>(np - done, std::max<int64_t>(cap - n_valid, 32));
            if ((rc = grow_copy(ctx, F_DESC, sizeof(float) * DESC_LEN * (size_t)(done + chunk),
                                sizeof(float) * DESC_LEN * (size_t)done, &p_desc)))
                return rc;
            hook.begin("sift_desc");
            desc_kernel<<<(unsigned)chunk, DESC_LEN, 0, st>>>(kp, done, (const int32_t*)p_pkp, (const double*)p_pth,
                                                              nullptr, table, (float*)p_desc, (uint8_t*)p_valid);
            SCK(cudaGetLastError());
            hook.end("sift_desc");
            done += chunk;
            size_t tb = 0;
            SCK(cub::DeviceSelect::Flagged(nullptr, tb, it, (const uint8_t*)p_valid, (uint32_t*)p_osel, (int*)p_nsel,
                                           (int)done, st));
            SCK(A.get(F_TEMP, tb, &p_temp));
            SCK(cub::DeviceSelect::Flagged(p_temp, tb, it, (const uint8_t*)p_valid, (uint32_t*)p_osel, (int*)p_nsel,
                                           (int)done, st));
            int nv = 0;
            SCK(cudaMemcpyAsync(&nv, (int*)p_nsel, sizeof(int), cudaMemcpyDeviceToHost, st));
            SCK(cudaStreamSynchronize(st));
            n_valid = nv;
        }
    }

    // sift.rs:543-544: the first max_features
    const int64_t n_out = std::min<int64_t>(n_valid, cap);
    out->width = w;
    out->height = h;
    out->n_raw = n_raw;
    out->n = (uint64_t)n_out;
    out->pts = (double*)ctx->result(RCMVS_RESULT_PTS, n_out, sizeof(double) * 2);
    out->desc = (float*)ctx->result(RCMVS_RESULT_DESC, n_out, sizeof(float) * DESC_LEN);
    out->colors = (uint8_t*)ctx->result(RCMVS_RESULT_COLORS, n_out, 3);
    if (!out->pts || !out->desc || !out->colors) {
        ctx->drop(out);
        return sfail(ctx, RCMVS_E_NOMEM, "sift: host allocation failed");
    }
    if (n_out == 0) return RCMVS_OK;
    if (!done_quick) {
        SCK(A.get(F_PTS, sizeof(double) * 2 * n_out, &p_pts));
        SCK(A.get(F_FDESC, sizeof(float) * DESC_LEN * n_out, &p_fdesc));
        SCK(A.get(F_COL, 3 * (size_t)n_out, &p_col));
        final_kernel<<<(int)((n_out + WARPS - 1) / WARPS), 32 * WARPS, 0, st>>>(
            (const uint32_t*)p_osel, (int)n_out, nullptr, (const int32_t*)p_pkp, kp, table, (const float*)p_desc,
            (const uint8_t*)p_rgb, w, h, (double*)p_pts, (float*)p_fdesc, (uint8_t*)p_col);
        SCK(cudaGetLastError());
    }
    SCK(host_download(out->pts, p_pts, sizeof(double) * 2 * n_out, st));
    SCK(host_download(out->desc, p_fdesc, sizeof(float) * DESC_LEN * n_out, st));
    SCK(host_download(out->colors, p_col, 3 * (size_t)n_out, st));
    SCK(cudaStreamSynchronize(st));
    return RCMVS_OK;
}

}  // extern "C"
