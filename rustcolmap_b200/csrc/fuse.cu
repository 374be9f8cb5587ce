// fuse.cu — geometric-consistency fusion + voxel dedup on sm_100a.
//
// Restates mvs/src/fuse.rs:
//   sample_depth        fuse.rs:32-62    (device function sample_depth)
//   per-pixel check     fuse.rs:96-167   (candidates_kernel, one thread/pixel,
//                                          f64 as the reference)
//   voxel dedup         fuse.rs:176-214  (sort + in-order segmented sums)
//   PLY vertex records  fuse.rs:232-237  (reduce_kernel packs 15-byte records)
//
// The reference accumulates each voxel sequentially in view-then-pixel
// order.  Here candidates keep their global pixel index (views are
// concatenated in order), are compacted stably, keyed by the packed voxel
// index and radix-sorted stably, so each voxel's members stay in that order
// and one lane per coordinate reproduces the reference's f64 sums bit for bit.
// Output order is the sorted key order (the reference's HashMap order is
// unspecified).
#include <thrust/iterator/counting_iterator.h>

#include <climits>
#include <cmath>
#include <limits>
#include <cub/cub.cuh>

#include "hostcopy.cuh"
#include "rcmvs_internal.cuh"

namespace rcmvs {

namespace {

constexpr int FT = 256;  // threads per block for pixel kernels
constexpr int VPX = 4 * FT;  // pixels per block of valid_kernel

__device__ __forceinline__ int find_item(const int32_t* start, int n, int b) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (start[mid] <= b)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// Quotients by one divisor, correctly rounded as a / b is: with y the
// correctly rounded 1 / b and q within one unit in the last place of a / b,
// q + fma(-b, q, a) y rounds to RN(a / b) (P. Markstein, IBM J. Res. Dev. 34,
// 1990, theorem on division).  The first correction brings a y within one
// unit, the second one rounds.  Exponents are kept to where no step can
// overflow or lose bits to the subnormals; zero and what lies outside is
// divided.  Five operations where a division takes about thirty.
struct Recip {
    double b, y;
    bool ok;
};
__device__ __forceinline__ bool exponent_in(double x, int lo, int hi) {
    return (unsigned)(((__double2hiint(x) >> 20) & 0x7FF) - (1023 + lo)) < (unsigned)(hi - lo);
}
__device__ __forceinline__ Recip recip(double b) { return Recip{b, __drcp_rn(b), exponent_in(b, -100, 100)}; }
__device__ __forceinline__ Recip recip(double b, double y) { return Recip{b, y, exponent_in(b, -100, 100)}; }
__device__ __forceinline__ double quot(double a, const Recip& r) {
    if (!(r.ok && exponent_in(a, -900, 900))) return a / r.b;
    double q = a * r.y;
    q = __fma_rn(__fma_rn(-r.b, q, a), r.y, q);
    return __fma_rn(__fma_rn(-r.b, q, a), r.y, q);
}

// sfm-lite/src/geom.rs:28-42
__device__ __forceinline__ void cam_normalize(const FuseView& v, double u, double w, double& xn, double& yn) {
    const Recip f = recip(v.f, v.rf);
    xn = quot(u - v.cx, f);
    yn = quot(w - v.cy, f);
    // with k = 0 and a finite radius, d = 1 + 0 * r2 is exactly 1, f * d = f,
    // and both iterations give back xn, yn: skipped
    if (v.k == 0.0 && isfinite(xn * xn + yn * yn)) return;
    for (int it = 0; it < 2; ++it) {
        double r2 = xn * xn + yn * yn;
        double d = 1.0 + v.k * r2;
        if (fabs(d) < 1e-12) break;
        const Recip fd = recip(v.f * d);
        xn = quot(u - v.cx, fd);
        yn = quot(w - v.cy, fd);
    }
}

struct Pose {
    double m[12];  // R by rows, then t
    __device__ __forceinline__ const double* R() const { return m; }
    __device__ __forceinline__ double t(int i) const { return m[9 + i]; }
};
__device__ __forceinline__ Pose load_pose(const FuseView& v) {
    Pose p;
    const double2* s = reinterpret_cast<const double2*>(v.pose);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double2 q = __ldg(s + i);
        p.m[2 * i] = q.x;
        p.m[2 * i + 1] = q.y;
    }
    return p;
}

// nalgebra 3x3 products, k ascending
__device__ __forceinline__ void mat_vec(const double* m, const double* x, double* o) {
    for (int i = 0; i < 3; ++i) o[i] = m[3 * i] * x[0] + m[3 * i + 1] * x[1] + m[3 * i + 2] * x[2];
}
__device__ __forceinline__ void matt_vec(const double* m, const double* x, double* o) {
    for (int i = 0; i < 3; ++i) o[i] = m[i] * x[0] + m[3 + i] * x[1] + m[6 + i] * x[2];
}

// World -> camera (sfm-lite/src/geom.rs:64-66)
__device__ __forceinline__ void to_cam(const Pose& p, const double* x, double* xc) {
    mat_vec(p.R(), x, xc);
    for (int i = 0; i < 3; ++i) xc[i] = xc[i] + p.t(i);
}

// Camera -> pixel (sfm-lite/src/geom.rs:67-75); z is recip(xc[2])
__device__ __forceinline__ void project(const FuseView& v, const double* xc, const Recip& z, double& u, double& w) {
    const double xn = quot(xc[0], z), yn = quot(xc[1], z);
    const double r2 = xn * xn + yn * yn;
    const double d = 1.0 + v.k * r2;
    u = v.f * xn * d + v.cx;
    w = v.f * yn * d + v.cy;
}

// fuse.rs:32-62.  The reference truncates floor(u) to an i32 and tests
// 0 <= u0, u0 + 1 < w (a NaN counts as 0, and the weights it makes give 0):
// the same tests on u itself need no conversion, and below 2^31 adding 1.5 2^52
// rounded down leaves floor(u) in the low word.
__device__ __forceinline__ double sample_depth(const float* __restrict__ dm, int w, int h, double u, double v) {
    if (!(u >= 0.0 && v >= 0.0 && u < (double)(w - 1) && v < (double)(h - 1))) return 0.0;
    const double big = 6755399441055744.0;
    const double ub = __dadd_rd(u, big), vb = __dadd_rd(v, big);
    const int u0 = __double2loint(ub), v0 = __double2loint(vb);
    const float fx = (float)(u - (ub - big));
    const float fy = (float)(v - (vb - big));
    const float* p = dm + (size_t)v0 * w + u0;
    const float d00 = __ldg(p), d10 = __ldg(p + 1);
    const float d01 = __ldg(p + w), d11 = __ldg(p + w + 1);
    const float ds[4] = {d00, d10, d01, d11};
    const float wt[4] = {(1.0f - fx) * (1.0f - fy), fx * (1.0f - fy), (1.0f - fx) * fy, fx * fy};
    float acc = 0.f, wsum = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (ds[q] > 0.0f) {
            acc += ds[q] * wt[q];
            wsum += wt[q];
        }
    if (wsum > 1e-6f) return (double)(acc / wsum);
    return 0.0;
}

// Marks the pixels with a depth (z > 0) of the views that have a map; the
// consistency kernel then runs on the compacted list of these pixels only.
__global__ void __launch_bounds__(FT) valid_kernel(const FuseView* __restrict__ views,
                                                   const int32_t* __restrict__ blk_start,
                                                   const int32_t* __restrict__ blk_view, int n_items,
                                                   const float* __restrict__ depth, uint8_t* __restrict__ flag) {
    const int item = find_item(blk_start, n_items, blockIdx.x);
    const FuseView& v = views[blk_view[item]];
    const int64_t n = (int64_t)v.w * v.h;
    const int64_t local = (int64_t)(blockIdx.x - blk_start[item]) * VPX + threadIdx.x;
    const size_t gi = (size_t)v.off + (size_t)local;
    float d[VPX / FT];
#pragma unroll
    for (int k = 0; k < VPX / FT; ++k) d[k] = local + k * FT < n ? __ldg(depth + gi + k * FT) : 0.0f;
#pragma unroll
    for (int k = 0; k < VPX / FT; ++k)
        if (local + k * FT < n) flag[gi + k * FT] = d[k] > 0.0f ? 1 : 0;
}

// fuse.rs:96-167 for one pixel with a depth: flag + averaged point.  One
// thread per entry of the list of such pixels (global indices; view k of
// the map-holding views starts at voff[k]).  Bound by issued instructions: the
// f64 divisions of a check (two per projection, the relative difference, two
// per back-projection) share reciprocals (quot), the reprojection distance is
// compared under its square (reproj_sq: the largest double whose root is
// within the limit), and poses are read 16 bytes at a time.  24 views of
// 960 x 720, 8 sources, a third of the pixels with a depth: 1640 -> 1490 us.
__global__ void __launch_bounds__(FT, 4) candidates_kernel(const FuseView* __restrict__ views,
                                                           const int64_t* __restrict__ voff,
                                                           const int32_t* __restrict__ vidx, int n_items,
                                                           const uint32_t* __restrict__ work, uint32_t n_work,
                                                           const int32_t* __restrict__ order,
                                                           const float* __restrict__ depth, uint32_t min_consistent,
                                                           double depth_diff, bool gate, double reproj_sq,
                                                           uint8_t* __restrict__ flag, double* __restrict__ pts) {
    const uint32_t t = blockIdx.x * FT + threadIdx.x;
    if (t >= n_work) return;
    const size_t gi = work[t];
    int lo = 0, hi = n_items - 1;  // the map-holding view that owns gi
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (voff[mid] <= (int64_t)gi)
            lo = mid;
        else
            hi = mid - 1;
    }
    const FuseView& v = views[vidx[lo]];
    const int64_t local = (int64_t)gi - v.off;
    const int px = (int)(local % v.w), py = (int)(local / v.w);
    const double zr = (double)depth[gi];
    uint8_t ok = 0;
    {
        double nx, ny;
        cam_normalize(v, (double)px, (double)py, nx, ny);
        const double xr[3] = {nx * zr, ny * zr, 1.0 * zr};
        const Pose ref = load_pose(v);
        const double dd[3] = {xr[0] - ref.t(0), xr[1] - ref.t(1), xr[2] - ref.t(2)};
        double xw[3];
        matt_vec(ref.R(), dd, xw);
        double acc[3] = {xw[0], xw[1], xw[2]};
        uint32_t n_cons = 0;
        for (int q = v.order_begin; q < v.order_end; ++q) {
            const FuseView& sv = views[order[q]];
            const Pose sp = load_pose(sv);
            double xs[3];
            to_cam(sp, xw, xs);
            if (xs[2] <= 1e-6) continue;
            const Recip z = recip(xs[2]);
            double us, vs;
            project(sv, xs, z, us, vs);
            const double zs = sample_depth(depth + sv.off, sv.w, sv.h, us, vs);
            if (zs <= 0.0) continue;
            const double rel = fabs(quot(xs[2] - zs, z));
            if (rel < depth_diff) {
                double sx, sy;
                cam_normalize(sv, us, vs, sx, sy);
                const double xs2[3] = {sx * zs, sy * zs, 1.0 * zs};
                const double d2[3] = {xs2[0] - sp.t(0), xs2[1] - sp.t(1), xs2[2] - sp.t(2)};
                double xw2[3];
                matt_vec(sp.R(), d2, xw2);
                if (gate) {  // extension: forward-backward reprojection gate
                    double xc[3], ru, rv;
                    to_cam(load_pose(v), xw2, xc);
                    if (xc[2] <= 1e-9) continue;
                    project(v, xc, recip(xc[2]), ru, rv);
                    const double ex = ru - (double)px, ey = rv - (double)py;
                    if (!(ex * ex + ey * ey <= reproj_sq)) continue;
                }
                for (int a = 0; a < 3; ++a) acc[a] += xw2[a];
                ++n_cons;
            }
        }
        if (n_cons >= min_consistent) {
            const Recip m = recip((double)(n_cons + 1));
            pts[3 * gi] = quot(acc[0], m);
            pts[3 * gi + 1] = quot(acc[1], m);
            pts[3 * gi + 2] = quot(acc[2], m);
            ok = 1;
        }
    }
    flag[gi] = ok;
}

// Rust `f64 as i64` (saturating, NaN -> 0): cvt.rzi.s64.f64
__device__ __forceinline__ long long vkey(double p, const Recip& cell) { return __double2ll_rz(floor(quot(p, cell))); }

__global__ void keys_minmax_kernel(const uint32_t* __restrict__ cand, uint32_t n, const double* __restrict__ pts,
                                   double cell, long long* __restrict__ kmin, long long* __restrict__ kmax) {
    __shared__ long long smin[3][FT / 32], smax[3][FT / 32];
    const Recip rc = recip(cell);
    long long lo[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, hi[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
    for (uint32_t c = blockIdx.x * FT + threadIdx.x; c < n; c += gridDim.x * FT) {
        const size_t g = cand[c];
        for (int a = 0; a < 3; ++a) {
            long long k = vkey(pts[3 * g + a], rc);
            lo[a] = min(lo[a], k);
            hi[a] = max(hi[a], k);
        }
    }
    for (int a = 0; a < 3; ++a)
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = min(lo[a], __shfl_down_sync(0xffffffffu, lo[a], o));
            hi[a] = max(hi[a], __shfl_down_sync(0xffffffffu, hi[a], o));
        }
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int a = 0; a < 3; ++a) {
            smin[a][wid] = lo[a];
            smax[a][wid] = hi[a];
        }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int a = threadIdx.x;
        long long l = LLONG_MAX, h = LLONG_MIN;
        for (int q = 0; q < FT / 32; ++q) {
            l = min(l, smin[a][q]);
            h = max(h, smax[a][q]);
        }
        atomicMin(kmin + a, l);
        atomicMax(kmax + a, h);
    }
}

__global__ void pack_keys_kernel(const uint32_t* __restrict__ cand, uint32_t n, const double* __restrict__ pts,
                                 double cell, const long long* __restrict__ kmin, int ybits, int zbits,
                                 uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const uint32_t c = blockIdx.x * FT + threadIdx.x;
    if (c >= n) return;
    const size_t g = cand[c];
    const Recip rc = recip(cell);
    uint64_t key = 0;
    for (int a = 0; a < 3; ++a) {
        const uint64_t k = (uint64_t)(vkey(pts[3 * g + a], rc) - kmin[a]);
        key = (key << (a == 0 ? 0 : a == 1 ? ybits : zbits)) | k;  // x in the high bits: lexicographic (x, y, z)
    }
    keys[c] = key;
    vals[c] = c;
}

// fuse.rs:194-213: in-order sums per voxel (u16 colour sums wrap), means,
// and the 15-byte PLY vertex record of fuse.rs:232-237.  G lanes per voxel
// fetch G members at a time (sorted position -> candidate -> point, the next
// ones before the last are added); lanes 0-2 add one coordinate each in member
// order.  Bound by that chain: with a thread per voxel the voxel of most members
// set the time.  24 views of 960 x 720: 350 us with a thread per voxel, 81 us
// with a warp (G = 32).  G = 8 where the mean is under 8 members: 212 k voxels
// of 3 members 26 us against 75 us.
template <int G>
__global__ void __launch_bounds__(FT) reduce_kernel(const uint32_t* __restrict__ run_off,
                                                    const uint32_t* __restrict__ run_len, uint32_t n_runs,
                                                    const uint32_t* __restrict__ sorted_vals,
                                                    const uint32_t* __restrict__ cand, const double* __restrict__ pts,
                                                    const uint8_t* __restrict__ rgb, double* __restrict__ out_xyz,
                                                    uint8_t* __restrict__ out_rgb, uint8_t* __restrict__ ply) {
    __shared__ double s_pt[FT / G][3][G];
    const uint32_t r = blockIdx.x * (FT / G) + threadIdx.x / G;
    const int lane = threadIdx.x % G;
    const unsigned mask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G);
    if (r >= n_runs) return;
    const uint32_t b = run_off[r], n = run_len[r];
    double(*pt)[G] = s_pt[threadIdx.x / G];
    uint32_t cr = 0, cg = 0, cb = 0;
    double x = 0.0, y = 0.0, z = 0.0, sum = 0.0;
    auto fetch = [&](uint32_t m) {
        if (m >= n) return;
        const size_t g = cand[sorted_vals[b + m]];
        x = pts[3 * g];
        y = pts[3 * g + 1];
        z = pts[3 * g + 2];
        cr += rgb[3 * g];
        cg += rgb[3 * g + 1];
        cb += rgb[3 * g + 2];
    };
    fetch(lane);
    for (uint32_t base = 0; base < n; base += G) {
        pt[0][lane] = x;
        pt[1][lane] = y;
        pt[2][lane] = z;
        __syncwarp(mask);
        fetch(base + G + lane);
        if (lane < 3) {
            const int m = (int)min((uint32_t)G, n - base);
            if (m == G) {
#pragma unroll
                for (int t = 0; t < G; ++t) sum += pt[lane][t];
            } else {
                for (int t = 0; t < m; ++t) sum += pt[lane][t];
            }
        }
        __syncwarp(mask);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        cr += __shfl_xor_sync(mask, cr, o);
        cg += __shfl_xor_sync(mask, cg, o);
        cb += __shfl_xor_sync(mask, cb, o);
    }
    if (lane >= 3) return;
    const double nn = (double)n;
    const double mean = sum / nn;
    out_xyz[3 * (size_t)r + lane] = mean;
    const uint16_t cs = (uint16_t)(lane == 0 ? cr : lane == 1 ? cg : cb);
    const double q = round((double)cs / nn);  // half away from zero, as f64::round
    const uint8_t c = q <= 0.0 ? 0 : (q >= 255.0 ? 255 : (uint8_t)q);
    out_rgb[3 * (size_t)r + lane] = c;
    uint8_t* o = ply + 15 * (size_t)r;
    const uint32_t bits = __float_as_uint((float)mean);
    for (int i = 0; i < 4; ++i) o[4 * lane + i] = (uint8_t)(bits >> (8 * i));
    o[12 + lane] = c;
}

__global__ void init_minmax_kernel(long long* kmin, long long* kmax) {
    if (threadIdx.x < 3) {
        kmin[threadIdx.x] = LLONG_MAX;
        kmax[threadIdx.x] = LLONG_MIN;
    }
}

struct CountingIt {
    using value_type = uint32_t;
};

__global__ void iota_kernel(uint32_t* __restrict__ out, uint32_t n) {
    for (uint32_t i = blockIdx.x * FT + threadIdx.x; i < n; i += gridDim.x * FT) out[i] = i;
}

// Compacts the candidates' points and reference colours in list order.
__global__ void gather_cand_kernel(const uint32_t* __restrict__ cand, uint32_t n, const double* __restrict__ pts,
                                   const uint8_t* __restrict__ rgb, double* __restrict__ out_xyz,
                                   uint8_t* __restrict__ out_rgb) {
    for (uint32_t c = blockIdx.x * FT + threadIdx.x; c < n; c += gridDim.x * FT) {
        const size_t g = cand[c];
        for (int a = 0; a < 3; ++a) {
            out_xyz[3 * (size_t)c + a] = pts[3 * g + a];
            out_rgb[3 * (size_t)c + a] = rgb[3 * g + a];
        }
    }
}

}  // namespace

#define FCK(x)                                                                   \
    do {                                                                         \
        cudaError_t e_ = (x);                                                    \
        if (e_ != cudaSuccess) {                                                 \
            *err = std::string(#x) + ": " + cudaGetErrorString(e_);              \
            return RCMVS_E_CUDA;                                                 \
        }                                                                        \
    } while (0)

// Arena slots used by fusion (the stereo path uses slots below 16): 16-37
// and 70-74.
enum {
    S_FLAG = 16, S_PTS, S_CAND, S_NSEL, S_KMIN, S_KEYS, S_VALS, S_KEYS2, S_VALS2, S_RUNKEY, S_RUNLEN,
    S_RUNOFF, S_NRUNS, S_TEMP, S_OUTXYZ, S_OUTRGB, S_PLY, S_FVIEWS, S_ORDER, S_BLK, S_WORK, S_VOFF
};
enum { S_INXYZ = 70, S_INRGB, S_IOTA, S_GXYZ, S_GRGB };

unsigned fgrid(uint32_t n) { return (unsigned)std::max<uint32_t>(1, std::min<uint32_t>((n + FT - 1) / FT, 148u * 8u)); }

int fuse_candidates_device(DeviceArena& A, const FuseView* h_views, int n_views, const int32_t* h_order,
                           int n_order, const float* depth, uint32_t min_consistent, double depth_diff,
                           double reproj_px, const uint32_t** d_cand, uint32_t* n_cand_out, const double** d_pts,
                           cudaStream_t st, std::string* err, const SpanHook& hook) {
    // pixel-block table over the reference views that have a depth map
    std::vector<int32_t> blk_start, blk_view;
    int64_t total_blocks = 0, total_px = 0;
    for (int v = 0; v < n_views; ++v) {
        total_px = std::max<int64_t>(total_px, h_views[v].off + (int64_t)h_views[v].w * h_views[v].h);
        if (!h_views[v].has_depth || !h_views[v].is_ref) continue;
        blk_start.push_back((int32_t)total_blocks);
        blk_view.push_back(v);
        total_blocks += ((int64_t)h_views[v].w * h_views[v].h + VPX - 1) / VPX;
    }
    *n_cand_out = 0;
    *d_cand = nullptr;
    *d_pts = nullptr;
    if (blk_view.empty() || total_px == 0) return RCMVS_OK;
    if (total_blocks > INT32_MAX || total_px > (int64_t)UINT32_MAX) {
        *err = "fusion: scene too large for 32-bit candidate indices";
        return RCMVS_E_LIMIT;
    }
    const int n_items = (int)blk_view.size();
    blk_start.push_back((int32_t)total_blocks);
    void *p_views, *p_order, *p_blk, *p_flag, *p_pts;
    FCK(A.get(S_FVIEWS, sizeof(FuseView) * n_views, &p_views));
    FCK(A.get(S_ORDER, sizeof(int32_t) * std::max(1, n_order), &p_order));
    FCK(A.get(S_BLK, sizeof(int32_t) * (2 * n_items + 1), &p_blk));
    FCK(A.get(S_FLAG, (size_t)total_px, &p_flag));
    FCK(A.get(S_PTS, sizeof(double) * 3 * (size_t)total_px, &p_pts));
    FCK(cudaMemcpyAsync(p_views, h_views, sizeof(FuseView) * n_views, cudaMemcpyHostToDevice, st));
    if (n_order > 0) FCK(cudaMemcpyAsync(p_order, h_order, sizeof(int32_t) * n_order, cudaMemcpyHostToDevice, st));
    std::vector<int32_t> blk(blk_start);
    blk.insert(blk.end(), blk_view.begin(), blk_view.end());
    FCK(cudaMemcpyAsync(p_blk, blk.data(), sizeof(int32_t) * blk.size(), cudaMemcpyHostToDevice, st));
    uint8_t* flag = (uint8_t*)p_flag;
    double* pts = (double*)p_pts;
    // pixels of views without a depth map are never read: zero all flags
    FCK(cudaMemsetAsync(flag, 0, (size_t)total_px, st));
    const uint32_t npx = (uint32_t)total_px;
    void *p_cand, *p_nsel, *p_temp, *p_work, *p_voff;
    FCK(A.get(S_CAND, sizeof(uint32_t) * npx, &p_cand));
    FCK(A.get(S_WORK, sizeof(uint32_t) * npx, &p_work));
    FCK(A.get(S_NSEL, sizeof(uint32_t) * 4, &p_nsel));
    FCK(A.get(S_VOFF, sizeof(int64_t) * n_items, &p_voff));
    std::vector<int64_t> voff(n_items);
    for (int k = 0; k < n_items; ++k) voff[k] = h_views[blk_view[k]].off;
    FCK(cudaMemcpyAsync(p_voff, voff.data(), sizeof(int64_t) * n_items, cudaMemcpyHostToDevice, st));
    thrust::counting_iterator<uint32_t> it(0);
    size_t tb = 0;
    FCK(cub::DeviceSelect::Flagged(nullptr, tb, it, flag, (uint32_t*)p_cand, (uint32_t*)p_nsel, npx, st));
    FCK(A.get(S_TEMP, tb, &p_temp));
    hook.begin("fuse_candidates");
    // the pixels with a depth, compacted, then one thread each
    valid_kernel<<<(unsigned)total_blocks, FT, 0, st>>>((const FuseView*)p_views, (const int32_t*)p_blk,
                                                       (const int32_t*)p_blk + n_items + 1, n_items, depth, flag);
    FCK(cudaGetLastError());
    FCK(cub::DeviceSelect::Flagged(p_temp, tb, it, flag, (uint32_t*)p_work, (uint32_t*)p_nsel + 1, npx, st));
    uint32_t n_work = 0;
    FCK(cudaMemcpyAsync(&n_work, (uint32_t*)p_nsel + 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    FCK(cudaStreamSynchronize(st));
    // sqrt rounds correctly and grows with its argument: sqrt(s) <= reproj_px
    // exactly where s is at most the largest double with that
    const bool gate = reproj_px > 0.0;
    double reproj_sq = reproj_px * reproj_px;
    if (gate && std::isfinite(reproj_px)) {
        const double inf = std::numeric_limits<double>::infinity();
        while (std::sqrt(reproj_sq) > reproj_px) reproj_sq = std::nextafter(reproj_sq, 0.0);
        while (std::sqrt(std::nextafter(reproj_sq, inf)) <= reproj_px) reproj_sq = std::nextafter(reproj_sq, inf);
    }
    if (n_work > 0)
        candidates_kernel<<<(n_work + FT - 1) / FT, FT, 0, st>>>(
            (const FuseView*)p_views, (const int64_t*)p_voff, (const int32_t*)p_blk + n_items + 1, n_items,
            (const uint32_t*)p_work, n_work, (const int32_t*)p_order, depth, min_consistent, depth_diff, gate,
            reproj_sq, flag, pts);
    FCK(cudaGetLastError());
    hook.end("fuse_candidates");

    // stable compaction of candidate pixel indices (view-then-pixel order)
    FCK(cub::DeviceSelect::Flagged(p_temp, tb, it, flag, (uint32_t*)p_cand, (uint32_t*)p_nsel, npx, st));
    uint32_t n_cand = 0;
    FCK(cudaMemcpyAsync(&n_cand, p_nsel, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    FCK(cudaStreamSynchronize(st));
    *n_cand_out = n_cand;
    *d_cand = (const uint32_t*)p_cand;
    *d_pts = pts;
    return RCMVS_OK;
}

int fuse_reduce_device(DeviceArena& A, const uint32_t* d_cand, uint32_t n_cand, const double* pts,
                       const uint8_t* rgb, double cell, double** d_xyz, uint8_t** d_rgb, uint8_t** d_ply,
                       uint64_t* n_points, cudaStream_t st, std::string* err, const SpanHook& hook) {
    *n_points = 0;
    if (n_cand == 0) return RCMVS_OK;
    const void* p_cand = d_cand;
    void* p_temp;
    size_t tb = 0;
    // voxel keys, packed; at most 21 bits per axis
    void* p_kmin;
    FCK(A.get(S_KMIN, sizeof(long long) * 6, &p_kmin));
    long long* kmin = (long long*)p_kmin;
    long long* kmax = kmin + 3;
    init_minmax_kernel<<<1, 32, 0, st>>>(kmin, kmax);
    const unsigned gb = (unsigned)std::min<uint32_t>((n_cand + FT - 1) / FT, 148u * 8u);
    keys_minmax_kernel<<<gb, FT, 0, st>>>((const uint32_t*)p_cand, n_cand, pts, cell, kmin, kmax);
    FCK(cudaGetLastError());
    int bits[3];
    long long hk[6];
    FCK(cudaMemcpyAsync(hk, kmin, sizeof(hk), cudaMemcpyDeviceToHost, st));
    FCK(cudaStreamSynchronize(st));
    for (int a = 0; a < 3; ++a) {
        unsigned long long span = (unsigned long long)(hk[3 + a] - hk[a]);
        if (hk[3 + a] < hk[a] || span >= (1ull << 21)) {
            *err = "fusion: voxel index range exceeds 2^21 cells per axis (cell too small for the cloud)";
            return RCMVS_E_LIMIT;
        }
        for (bits[a] = 0; (span >> bits[a]) != 0;) ++bits[a];
    }
    // the sort's passes go by the bits that the ranges need
    const int key_bits = std::max(1, bits[0] + bits[1] + bits[2]);
    void *p_keys, *p_vals, *p_keys2, *p_vals2;
    FCK(A.get(S_KEYS, sizeof(uint64_t) * n_cand, &p_keys));
    FCK(A.get(S_VALS, sizeof(uint32_t) * n_cand, &p_vals));
    FCK(A.get(S_KEYS2, sizeof(uint64_t) * n_cand, &p_keys2));
    FCK(A.get(S_VALS2, sizeof(uint32_t) * n_cand, &p_vals2));
    pack_keys_kernel<<<(n_cand + FT - 1) / FT, FT, 0, st>>>((const uint32_t*)p_cand, n_cand, pts, cell, kmin,
                                                            bits[1], bits[2], (uint64_t*)p_keys, (uint32_t*)p_vals);
    FCK(cudaGetLastError());
    // stable LSD radix sort
    tb = 0;
    FCK(cub::DeviceRadixSort::SortPairs(nullptr, tb, (const uint64_t*)p_keys, (uint64_t*)p_keys2,
                                        (const uint32_t*)p_vals, (uint32_t*)p_vals2, n_cand, 0, key_bits, st));
    FCK(A.get(S_TEMP, tb, &p_temp));
    FCK(cub::DeviceRadixSort::SortPairs(p_temp, tb, (const uint64_t*)p_keys, (uint64_t*)p_keys2,
                                        (const uint32_t*)p_vals, (uint32_t*)p_vals2, n_cand, 0, key_bits, st));
    // runs of equal keys = voxels
    void *p_runkey, *p_runlen, *p_runoff, *p_nruns;
    FCK(A.get(S_RUNKEY, sizeof(uint64_t) * n_cand, &p_runkey));
    FCK(A.get(S_RUNLEN, sizeof(uint32_t) * n_cand, &p_runlen));
    FCK(A.get(S_RUNOFF, sizeof(uint32_t) * n_cand, &p_runoff));
    FCK(A.get(S_NRUNS, sizeof(uint32_t) * 4, &p_nruns));
    tb = 0;
    FCK(cub::DeviceRunLengthEncode::Encode(nullptr, tb, (const uint64_t*)p_keys2, (uint64_t*)p_runkey,
                                           (uint32_t*)p_runlen, (uint32_t*)p_nruns, n_cand, st));
    size_t tb2 = 0;
    FCK(cub::DeviceScan::ExclusiveSum(nullptr, tb2, (const uint32_t*)p_runlen, (uint32_t*)p_runoff, n_cand, st));
    FCK(A.get(S_TEMP, std::max(tb, tb2), &p_temp));
    FCK(cub::DeviceRunLengthEncode::Encode(p_temp, tb, (const uint64_t*)p_keys2, (uint64_t*)p_runkey,
                                           (uint32_t*)p_runlen, (uint32_t*)p_nruns, n_cand, st));
    uint32_t n_runs = 0;
    FCK(cudaMemcpyAsync(&n_runs, p_nruns, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    FCK(cudaStreamSynchronize(st));
    FCK(cub::DeviceScan::ExclusiveSum(p_temp, tb2, (const uint32_t*)p_runlen, (uint32_t*)p_runoff, n_runs, st));
    void *p_oxyz, *p_orgb, *p_ply;
    FCK(A.get(S_OUTXYZ, sizeof(double) * 3 * n_runs, &p_oxyz));
    FCK(A.get(S_OUTRGB, 3 * (size_t)n_runs, &p_orgb));
    FCK(A.get(S_PLY, 15 * (size_t)n_runs, &p_ply));
    hook.begin("fuse_reduce");
    auto reduce = [&](auto kernel, uint32_t per_block) {
        kernel<<<(n_runs + per_block - 1) / per_block, FT, 0, st>>>(
            (const uint32_t*)p_runoff, (const uint32_t*)p_runlen, n_runs, (const uint32_t*)p_vals2,
            (const uint32_t*)p_cand, pts, rgb, (double*)p_oxyz, (uint8_t*)p_orgb, (uint8_t*)p_ply);
    };
    if (n_cand / 8 < n_runs)
        reduce(reduce_kernel<8>, FT / 8);
    else
        reduce(reduce_kernel<32>, FT / 32);
    FCK(cudaGetLastError());
    hook.end("fuse_reduce");
    *d_xyz = (double*)p_oxyz;
    *d_rgb = (uint8_t*)p_orgb;
    *d_ply = (uint8_t*)p_ply;
    *n_points = n_runs;
    return RCMVS_OK;
}

int fuse_reduce_host(DeviceArena& A, const double* h_xyz, const uint8_t* h_rgb, uint64_t n, double cell,
                     double** d_xyz, uint8_t** d_rgb, uint8_t** d_ply, uint64_t* n_points, cudaStream_t st,
                     std::string* err, const SpanHook& hook) {
    *n_points = 0;
    if (n == 0) return RCMVS_OK;
    if (n > (uint64_t)UINT32_MAX) {
        *err = "fusion: more than 2^32 candidates";
        return RCMVS_E_LIMIT;
    }
    void *p_xyz, *p_rgb, *p_iota;
    FCK(A.get(S_INXYZ, sizeof(double) * 3 * n, &p_xyz));
    FCK(A.get(S_INRGB, 3 * n, &p_rgb));
    FCK(A.get(S_IOTA, sizeof(uint32_t) * n, &p_iota));
    FCK(host_upload(p_xyz, h_xyz, sizeof(double) * 3 * n, st));
    FCK(host_upload(p_rgb, h_rgb, 3 * n, st));
    iota_kernel<<<fgrid((uint32_t)n), FT, 0, st>>>((uint32_t*)p_iota, (uint32_t)n);
    FCK(cudaGetLastError());
    return fuse_reduce_device(A, (const uint32_t*)p_iota, (uint32_t)n, (const double*)p_xyz, (const uint8_t*)p_rgb,
                              cell, d_xyz, d_rgb, d_ply, n_points, st, err, hook);
}

int fuse_reduce_devptr(DeviceArena& A, const double* d_in_xyz, const uint8_t* d_in_rgb, uint64_t n, double cell,
                       double** d_xyz, uint8_t** d_rgb, uint8_t** d_ply, uint64_t* n_points, cudaStream_t st,
                       std::string* err, const SpanHook& hook) {
    *n_points = 0;
    if (n == 0) return RCMVS_OK;
    if (n > (uint64_t)UINT32_MAX) {
        *err = "fusion: more than 2^32 candidates";
        return RCMVS_E_LIMIT;
    }
    void* p_iota;
    FCK(A.get(S_IOTA, sizeof(uint32_t) * n, &p_iota));
    iota_kernel<<<fgrid((uint32_t)n), FT, 0, st>>>((uint32_t*)p_iota, (uint32_t)n);
    FCK(cudaGetLastError());
    return fuse_reduce_device(A, (const uint32_t*)p_iota, (uint32_t)n, d_in_xyz, d_in_rgb, cell, d_xyz, d_rgb, d_ply,
                              n_points, st, err, hook);
}

int fuse_gather_device(DeviceArena& A, const uint32_t* d_cand, uint32_t n, const double* pts, const uint8_t* rgb,
                       double** d_xyz, uint8_t** d_rgb, cudaStream_t st, std::string* err) {
    void *p_xyz, *p_rgb;
    FCK(A.get(S_GXYZ, sizeof(double) * 3 * std::max<uint32_t>(n, 1), &p_xyz));
    FCK(A.get(S_GRGB, 3 * (size_t)std::max<uint32_t>(n, 1), &p_rgb));
    if (n > 0) {
        gather_cand_kernel<<<fgrid(n), FT, 0, st>>>(d_cand, n, pts, rgb, (double*)p_xyz, (uint8_t*)p_rgb);
        FCK(cudaGetLastError());
    }
    *d_xyz = (double*)p_xyz;
    *d_rgb = (uint8_t*)p_rgb;
    return RCMVS_OK;
}

int fuse_device(DeviceArena& A, const FuseView* h_views, int n_views, const int32_t* h_order, int n_order,
                const float* depth, const uint8_t* rgb, double cell, uint32_t min_consistent, double depth_diff,
                double reproj_px, double** d_xyz, uint8_t** d_rgb, uint8_t** d_ply, FuseResult* res,
                cudaStream_t st, std::string* err, const SpanHook& hook) {
    res->n_candidates = res->n_points = 0;
    const uint32_t* cand = nullptr;
    const double* pts = nullptr;
    uint32_t n_cand = 0;
    int rc = fuse_candidates_device(A, h_views, n_views, h_order, n_order, depth, min_consistent, depth_diff,
                                    reproj_px, &cand, &n_cand, &pts, st, err, hook);
    if (rc) return rc;
    res->n_candidates = n_cand;
    return fuse_reduce_device(A, cand, n_cand, pts, rgb, cell, d_xyz, d_rgb, d_ply, &res->n_points, st, err, hook);
}

}  // namespace rcmvs
