// match.cu — SIFT descriptor matching on sm_100a.
//
// Restates sfm-lite/src/matching.rs:22-95 (match_pair) for a batch of image
// pairs: for every descriptor of A the nearest and second-nearest descriptor
// of B by squared L2 distance, the same from B to A, Lowe's ratio test both
// ways and the mutual-best check.
//
// The reference sums (a_k - b_k)^2 serially over k = 0..127 in f32.  Its
// result is only which descriptors pass the tests on the nearest and
// second-nearest distance, so a tensor-core product with an error bound
// decides every descriptor that is not within the bound of a test's edge,
// and only the rest are summed as written:
//
//   pack_kernel   every frame as FP16 hi + lo (x = 2^-6 (hi + lo) to 2^-22) in
//                 the tensor cores' operand order, blocks of 128 descriptors,
//                 and squared norms
//   nearest_kernel  one CTA per 128 descriptors of one frame (queries) against
//                 all descriptors of the other, both directions of each pair:
//                 |t|^2 - 2 q.t, the products as hi.lo + lo.hi + hi.hi on
//                 tcgen05.mma with FP32 accumulation in tensor memory; one
//                 thread keeps the two smallest of its query and half of the
//                 targets
//   outcome_kernel  per query: certainly refused, certainly accepted (then the
//                 two targets of the smallest's column pair are summed
//                 serially and the nearer is the answer), or listed
//   rescan_kernel the listed queries against all targets, serially summed, and
//                 the reference's tests
//   mutual_kernel the reference's mutual check per row of A
//
// Error bound (u = 2^-24; |q|, |t| norms, S = |q| + max |t|, so |q||t| <= S^2 / 4).
// In the distance, 2 q.t counts twice:
//   operands to 2^-22 relative or 2^-31 absolute per component   4 u S^2 + 2^-26 S
//   lo.lo dropped (2^-22 |q||t|)                                 2 u S^2
//   sums of the products                                        42 u S^2
//   norms (summed in f64), |t|^2 - 2 q.t and + |q|^2 rounded     4 u S^2
// together 52 u S^2 + 2^-26 S; search_bound takes 80 u.  The sums' part rests on
// a measurement, since PTX leaves the rounding of kind::f16 open: an MMA cuts its
// 16 products and the accumulator toward zero to 2^-25 of the largest one's power
// of two, adds them, and cuts the sum toward zero to FP32 (this model gave all of
// 26389 products, magnitudes over 2^-28 .. 1 and both signs, bit for bit).  So an
// MMA loses at most 17 u / 2 + 2 u of the largest term.  The products with a lo are
// summed first, while all terms are below 2^-10 |q||t|; after them come 8 MMAs of
// hi.hi: 84 u |q||t|.  (With hi.lo last there were 16 at full size: 168 u, of
// which up to 95 u were measured.)  The reference's own serial sum is within
// 131 u d < 7.9e-6 d of the exact distance.
//
// Frames with components past 1000 or not finite, and chunks in which many
// queries are listed (repeated descriptors), run on the FP32 pipes instead:
//
//   dist_kernel   64x64 distances per block, 4x4 per thread; 32-wide k chunks
//                 of both tiles staged k-major in shared memory (float4 reads,
//                 conflict-free), each distance accumulated in k order; with
//                 --fmad=false every difference, square and sum rounds as in
//                 the reference.  The distances never leave the block: it
//                 writes, for each of its rows and columns, the (best, index,
//                 second) over the tile, merged through shuffles and shared
//                 memory.  One distance serves both directions: (a - b)^2 and
//                 the reference's backward (a - b)^2 are the same number.
//   rows_kernel   one thread per row: the tiles' partials merged by value
//   cols_kernel   with the lower index winning ties -- the first minimum and
//                 the second smallest value, exactly what the reference's
//                 sequential scan keeps (the merge is associative, so the
//                 order of the tiles does not matter)
//
// Pairs run in chunks whose tile partials (the per-tile best/second entries
// of every row and column, 12 bytes each; no distance matrix is written)
// fit P_BUDGET; results come back as per-pair lists in the reference's order
// (ascending index in A).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_fp16.h>

#include "ctx_internal.cuh"
#include "tc.cuh"

namespace rcmvs {

namespace {

constexpr int DESC_LEN = 128;
constexpr int TILE = 64;
constexpr int KC = 32;
constexpr size_t P_BUDGET = size_t(1) << 28;  // bytes of tile partials per chunk

struct PairJob {
    int64_t a_off, b_off;      // first descriptor of each frame (in descriptors)
    int64_t prow_off, pcol_off;  // tile partials: [column tile][na] rows, [row tile][nb] columns
    int32_t na, nb;
    int32_t row_off, col_off;  // into the chunk's forward / backward results
    int32_t fa, fb;            // frames
    int32_t pair;              // of the chunk
};

struct Nearest {
    uint32_t idx;
    float d1, d2;
};

// Sequential-scan state: the first minimum and the second smallest value.
__device__ __forceinline__ void push(float s, uint32_t j, float& best, uint32_t& bi, float& second) {
    if (s < best) {
        second = best;
        best = s;
        bi = j;
    } else if (s < second) {
        second = s;
    }
}

// The same state of a union of two disjoint parts: the smaller best (the
// lower index among equal values) and the second smallest value of the union.
__device__ __forceinline__ void merge(float& best, uint32_t& bi, float& second, float ob, uint32_t oi, float os) {
    const float nsec = fminf(fmaxf(best, ob), fminf(second, os));
    if (ob < best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
    }
    second = nsec;
}

__global__ void __launch_bounds__(256) dist_kernel(const float* __restrict__ desc, const PairJob* __restrict__ jobs,
                                                   Nearest* __restrict__ rowpart, Nearest* __restrict__ colpart) {
    __shared__ __align__(16) float As[KC][TILE];
    __shared__ __align__(16) float Bs[KC][TILE];
    __shared__ Nearest cpart[8][TILE];
    const PairJob J = jobs[blockIdx.z];
    const int r0 = blockIdx.y * TILE, c0 = blockIdx.x * TILE;
    if (r0 >= J.na || c0 >= J.nb) return;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const float* A = desc + J.a_off * DESC_LEN;
    const float* B = desc + J.b_off * DESC_LEN;
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.0f;
    for (int k0 = 0; k0 < DESC_LEN; k0 += KC) {
        // 64 rows x 8 float4 per tile; a warp covers 32 rows of one float4
        for (int e = threadIdx.x; e < TILE * (KC / 4); e += 256) {
            const int row = e % TILE, q = e / TILE;
            float4 va = make_float4(0.f, 0.f, 0.f, 0.f), vb = va;
            if (r0 + row < J.na) va = *reinterpret_cast<const float4*>(A + (int64_t)(r0 + row) * DESC_LEN + k0 + 4 * q);
            if (c0 + row < J.nb) vb = *reinterpret_cast<const float4*>(B + (int64_t)(c0 + row) * DESC_LEN + k0 + 4 * q);
            As[4 * q][row] = va.x;
            As[4 * q + 1][row] = va.y;
            As[4 * q + 2][row] = va.z;
            As[4 * q + 3][row] = va.w;
            Bs[4 * q][row] = vb.x;
            Bs[4 * q + 1][row] = vb.y;
            Bs[4 * q + 2][row] = vb.z;
            Bs[4 * q + 3][row] = vb.w;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < KC; ++kk) {
            const float4 a4 = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 b4 = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w};
            const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float d = a[r] - b[c];
                    acc[r][c] = acc[r][c] + d * d;
                }
        }
        __syncthreads();
    }
    // Rows: each of this thread's 4 rows over its 4 columns, then over the
    // 16 threads of the row group (lanes 0-15 or 16-31 of the warp).
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int ia = r0 + ty * 4 + r;
        float best = INFINITY, second = INFINITY;
        uint32_t bi = UINT32_MAX;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int ib = c0 + tx * 4 + c;
            if (ia < J.na && ib < J.nb) push(acc[r][c], (uint32_t)ib, best, bi, second);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
            merge(best, bi, second, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o),
                  __shfl_xor_sync(0xffffffffu, second, o));
        if (tx == 0 && ia < J.na) rowpart[J.prow_off + (int64_t)blockIdx.x * J.na + ia] = Nearest{bi, best, second};
    }
    // Columns: each of this thread's 4 columns over its 4 rows, then the two
    // row groups of the warp, then the 8 warps through shared memory.
    const int wid = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int ib = c0 + tx * 4 + c;
        float best = INFINITY, second = INFINITY;
        uint32_t bi = UINT32_MAX;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int ia = r0 + ty * 4 + r;
            if (ia < J.na && ib < J.nb) push(acc[r][c], (uint32_t)ia, best, bi, second);
        }
        merge(best, bi, second, __shfl_xor_sync(0xffffffffu, best, 16), __shfl_xor_sync(0xffffffffu, bi, 16),
              __shfl_xor_sync(0xffffffffu, second, 16));
        if ((threadIdx.x & 16) == 0) cpart[wid][tx * 4 + c] = Nearest{bi, best, second};
    }
    __syncthreads();
    if (threadIdx.x < TILE) {
        const int ib = c0 + threadIdx.x;
        Nearest m = cpart[0][threadIdx.x];
        for (int q = 1; q < 8; ++q) {
            const Nearest o = cpart[q][threadIdx.x];
            merge(m.d1, m.idx, m.d2, o.d1, o.idx, o.d2);
        }
        if (ib < J.nb) colpart[J.pcol_off + (int64_t)blockIdx.y * J.nb + ib] = m;
    }
}

// The tiles' partials of each row (over column tiles) and of each column
// (over row tiles), merged into the nearest and second-nearest of the row or
// column; one thread each.
__global__ void __launch_bounds__(256) rows_kernel(const PairJob* __restrict__ jobs, const Nearest* __restrict__ rowpart,
                                                   Nearest* __restrict__ fwd) {
    const PairJob J = jobs[blockIdx.y];
    const int ia = blockIdx.x * 256 + threadIdx.x;
    if (ia >= J.na) return;
    const int nct = (J.nb + TILE - 1) / TILE;
    Nearest m{UINT32_MAX, INFINITY, INFINITY};
    for (int t = 0; t < nct; ++t) {
        const Nearest o = rowpart[J.prow_off + (int64_t)t * J.na + ia];
        merge(m.d1, m.idx, m.d2, o.d1, o.idx, o.d2);
    }
    fwd[J.row_off + ia] = m;
}

__global__ void __launch_bounds__(256) cols_kernel(const PairJob* __restrict__ jobs, const Nearest* __restrict__ colpart,
                                                   Nearest* __restrict__ bwd) {
    const PairJob J = jobs[blockIdx.y];
    const int ib = blockIdx.x * 256 + threadIdx.x;
    if (ib >= J.nb) return;
    const int nrt = (J.na + TILE - 1) / TILE;
    Nearest m{UINT32_MAX, INFINITY, INFINITY};
    for (int t = 0; t < nrt; ++t) {
        const Nearest o = colpart[J.pcol_off + (int64_t)t * J.nb + ib];
        merge(m.d1, m.idx, m.d2, o.d1, o.idx, o.d2);
    }
    bwd[J.col_off + ib] = m;
}

// ------------------------------------------------------ tensor-core search
constexpr int QB = 128;                      // descriptors per packed block
constexpr int QB_HALF = QB * DESC_LEN * 2;   // bytes of a block's hi (or lo) half
constexpr int QB_BYTES = 2 * QB_HALF;
constexpr float PACK_SCALE = 64.0f;          // keeps lo clear of FP16 subnormals for unit descriptors
constexpr float PACK_LIMIT = 1000.0f;        // larger components overflow FP16 after scaling
constexpr int RESCAN_MAX = 2048;             // listed queries a chunk may have

struct Frame {
    int64_t off;   // first descriptor
    int64_t blk;   // first packed block (and 128 * blk: first norm)
    int32_t n;
};

struct MatchStatus {
    int wild;   // a component past PACK_LIMIT or not finite
    int listed; // queries for rescan_kernel
    int fault;  // the context's fault word was set (outcome_kernel)
};

// Block b of 128 descriptors: half (hi, lo) h, descriptor r, component k at
// h * QB_HALF + (k / 8) * 2048 + r * 16 + (k % 8) * 2: [8-component group]
// [descriptor][8], a canonical K-major operand.  Past the frame's end:
// zeros with an infinite norm.
__global__ void __launch_bounds__(256) pack_kernel(const float* __restrict__ desc, const Frame* __restrict__ frames,
                                                   const int32_t* __restrict__ blk_start, int n_frames, int first,
                                                   unsigned char* __restrict__ packed, float* __restrict__ norms,
                                                   int* __restrict__ max_norm, MatchStatus* __restrict__ st) {
    __shared__ double part[2][QB];
    const int block = first + (int)blockIdx.x;
    int lo = 0, hi = n_frames - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (blk_start[mid] <= block)
            lo = mid;
        else
            hi = mid - 1;
    }
    const Frame F = frames[lo];
    const int r = threadIdx.x & (QB - 1), half = threadIdx.x >> 7;
    const int row = (block - blk_start[lo]) * QB + r;
    const bool in = row < F.n;
    const float* src = desc + (F.off + row) * DESC_LEN;
    unsigned char* out = packed + (size_t)block * QB_BYTES + r * 16;
    double sum = 0.0;
    bool wild = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int g = 2 * i + half;
        float x[8] = {};
        if (in) {
            const float4 a = *reinterpret_cast<const float4*>(src + 8 * g), b = *reinterpret_cast<const float4*>(src + 8 * g + 4);
            x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w, x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
        }
        __half h[8], l[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            wild = wild || !(fabsf(x[c]) <= PACK_LIMIT);
            sum = __fma_rn((double)x[c], (double)x[c], sum);
            const float v = x[c] * PACK_SCALE;
            h[c] = __float2half_rn(v);
            l[c] = __float2half_rn(v - __half2float(h[c]));
        }
        *reinterpret_cast<uint4*>(out + g * (QB * 16)) = *reinterpret_cast<const uint4*>(h);
        *reinterpret_cast<uint4*>(out + QB_HALF + g * (QB * 16)) = *reinterpret_cast<const uint4*>(l);
    }
    part[half][r] = sum;
    if (wild) st->wild = 1;
    __syncthreads();
    if (half == 0) {
        const float n = (float)(part[0][r] + part[1][r]);
        norms[(size_t)block * QB + r] = in ? n : INFINITY;
        float m = in ? n : 0.0f;
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) == 0) atomicMax(&max_norm[lo], __float_as_int(m));  // norms are not negative
    }
}

struct Two {  // the two smallest values and the column pair (target / 2) of the smallest
    float v0, v1;
    int32_t pair;
};

// One direction of a pair: queries q against targets t; entry at `out`.
__device__ __forceinline__ void direction(const PairJob& J, const Frame* frames, int dir, Frame& q, Frame& t, int& out) {
    q = frames[dir ? J.fb : J.fa];
    t = frames[dir ? J.fa : J.fb];
    out = dir ? J.col_off : J.row_off;
}

// One CTA: up to two query blocks (256 queries) against every target block.
// Shared memory holds the query blocks (128 KB) and a ring of three 32 KB
// slots for the halves (hi, lo) of the target blocks; tensor memory two
// accumulators per query block (128 columns each), one multiplying while the
// other is read.  Warp 8's first thread loads and multiplies: step 2c is
// block c's lo (queries hi), step 2c + 1 its hi (queries lo, then hi: the small
// terms first, for the error bound); the load of step s + 2 starts when step
// s - 1's products are done, two steps ahead of its use.  Warps 0-3 scan the
// first query block's values, 4-7 the second's, one thread per query.  Bound by
// the tensor pipe (48 MMAs of 128 x 128 x 16 per target block; 56% active over
// 170 pairs of 2048, 41% with one query block per CTA) and the L2 reads of the
// target blocks.  12 frames of 2048, 66 pairs (both directions): 429 us (FP32
// pipes: 4158); one query block per CTA and 64 KB target blocks in two buffers:
// 547 us (the load of a block had one scan's time to arrive); with the four
// smallest kept in branches: 1040 us.
constexpr int NSLOT = 3;
constexpr int kNearestThreads = 288;
constexpr int kNearestSmem = 2 * QB_BYTES + NSLOT * QB_HALF + 128;

__global__ void __launch_bounds__(kNearestThreads, 1)
    nearest_kernel(const PairJob* __restrict__ jobs, const Frame* __restrict__ frames,
                   const unsigned char* __restrict__ packed, const float* __restrict__ norms, int blocks_per_cta,
                   Two* __restrict__ fwd, Two* __restrict__ bwd, int* fault) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[1 + 2 * NSLOT + 4];  // queries; slot full, slot free; values full, values free
    __shared__ uint32_t s_taddr;
    const int dir = blockIdx.y & 1;
    const PairJob J = jobs[blockIdx.y >> 1];
    Frame q, t;
    int out0;
    direction(J, frames, dir, q, t, out0);
    const int qb0 = blockIdx.x * blocks_per_cta;
    const int nq = min(blocks_per_cta, (q.n + QB - 1) / QB - qb0);
    const int n = (t.n + QB - 1) / QB;
    if (nq <= 0 || n == 0) return;  // without targets the queries' entries are not read
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sq = (smem_u32(smem) + 127u) & ~127u, ring = sq + 2 * QB_BYTES;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int k) { return bar0 + 8u + 8u * k; };
    auto slot_free = [&](int k) { return bar0 + 8u + 8u * (NSLOT + k); };
    auto acc_full = [&](int k) { return bar0 + 8u + 8u * (2 * NSLOT + k); };
    auto acc_free = [&](int k) { return bar0 + 8u + 8u * (2 * NSLOT + 2 + k); };
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_taddr)),
                     "r"(4 * QB));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int k = 0; k < 1 + 2 * NSLOT + 2; ++k) mbar_init(bar0 + 8u * k, 1);
        for (int k = 0; k < 2; ++k) mbar_init(acc_free(k), 4 * nq);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t taddr = s_taddr;
    if (warp == 8) {
        if (lane == 0) {
            const int steps = 2 * n;
            int loaded = 0, landed = 0, issued = 0, freed = 0;  // steps
            auto load = [&](uint32_t dst, const unsigned char* src, uint32_t bytes, uint32_t bar) {
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                             "l"(src), "r"(bytes), "r"(bar)
                             : "memory");
            };
            auto load_step = [&](int s) {
                mbar_expect_tx(full(s % NSLOT), QB_HALF);
                load(ring + (s % NSLOT) * QB_HALF, packed + (t.blk + (s >> 1)) * (int64_t)QB_BYTES + ((s & 1) ^ 1) * QB_HALF,
                     QB_HALF, full(s % NSLOT));
                ++loaded;
            };
            mbar_expect_tx(bar0, nq * QB_BYTES);
            load(sq, packed + (q.blk + qb0) * (int64_t)QB_BYTES, nq * QB_BYTES, bar0);
            load_step(0);
            load_step(1);
            bool ok = mbar_wait(bar0, 0, TC_WAIT_NS);
            const bool q_in = ok;
            for (int s = 0; s < steps && ok; ++s) {
                const int c = s >> 1, slot = s % NSLOT;
                if (!(ok = mbar_wait(full(slot), (s / NSLOT) & 1, TC_WAIT_NS))) break;
                ++landed;
                if ((s & 1) == 0 && c >= 2 && !(ok = mbar_wait(acc_free(c & 1), ((c >> 1) - 1) & 1, TC_WAIT_NS))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                constexpr uint32_t IDESC = (1u << 4) | ((QB >> 3) << 17) | ((QB >> 4) << 24);  // F16 in, F32 out, 128 x 128
                const uint32_t sb = ring + slot * QB_HALF;
                for (int b = 0; b < nq; ++b) {
                    const uint32_t d = taddr + (2 * b + (c & 1)) * QB;
                    for (int term = (s & 1) ? 0 : 1; term < 2; ++term) {  // queries lo, then hi; only hi against lo
                        const uint32_t a0 = sq + b * QB_BYTES + (term == 0 ? QB_HALF : 0);
#pragma unroll
                        for (int kc = 0; kc < DESC_LEN / 16; ++kc)
                            umma_f16(d, umma_desc(a0 + kc * (2 * QB * 16), QB * 16, 128),
                                     umma_desc(sb + kc * (2 * QB * 16), QB * 16, 128), IDESC,
                                     ((s & 1) | kc) != 0 ? 1u : 0u);
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(slot_free(slot))
                             : "memory");
                if (s & 1)
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(acc_full(c & 1))
                                 : "memory");
                ++issued;
                if (s + 2 < steps) {
                    if (s >= 1) {  // step s - 1's products have read the slot
                        if (!(ok = mbar_wait(slot_free((s - 1) % NSLOT), ((s - 1) / NSLOT) & 1, TC_WAIT_NS))) break;
                        freed = s;
                    }
                    load_step(s + 2);
                }
            }
            // everything in flight ends before the memory is released
            if (!ok) atomicExch(fault, 1);
            if (!q_in) mbar_wait(bar0, 0, TC_WAIT_NS);
            for (; landed < loaded; ++landed) mbar_wait(full(landed % NSLOT), (landed / NSLOT) & 1, TC_WAIT_NS);
            for (; freed < issued; ++freed) {
                if (!mbar_wait(slot_free(freed % NSLOT), (freed / NSLOT) & 1, TC_WAIT_NS)) atomicExch(fault, 1);
            }
        }
        __syncwarp();
    } else if ((warp >> 2) < nq) {
        const int b = warp >> 2;
        const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
        const float4* tn = reinterpret_cast<const float4*>(norms + t.blk * QB);
        Two f{INFINITY, INFINITY, -1};
        bool ok = true;
        for (int c = 0; c < n; ++c) {
            if (!(ok = __all_sync(0xffffffffu, mbar_wait(acc_full(c & 1), (c >> 1) & 1, TC_WAIT_NS)))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int part = 0; part < QB / 32; ++part) {
                uint32_t v[32];
                tmem_ld_32x32b<32>(taddr + lanes + (uint32_t)((2 * b + (c & 1)) * QB + 32 * part), v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                constexpr float M2 = -2.0f / (PACK_SCALE * PACK_SCALE);
                const int pair0 = (c * QB + 32 * part) / 2;
#pragma unroll
                for (int k = 0; k < 32; k += 4) {
                    const float4 nb = __ldg(tn + (c * QB + 32 * part + k) / 4);
                    auto scan = [&](float x, float y, int pair) {  // branch-free; column pairs halve the index work
                        const float lo = fminf(x, y);
                        f.v1 = fminf(fminf(f.v1, fmaxf(x, y)), fmaxf(f.v0, lo));
                        f.pair = lo < f.v0 ? pair : f.pair;
                        f.v0 = fminf(f.v0, lo);
                    };
                    scan(__fmaf_rn(M2, __uint_as_float(v[k]), nb.x), __fmaf_rn(M2, __uint_as_float(v[k + 1]), nb.y),
                         pair0 + k / 2);
                    scan(__fmaf_rn(M2, __uint_as_float(v[k + 2]), nb.z), __fmaf_rn(M2, __uint_as_float(v[k + 3]), nb.w),
                         pair0 + k / 2 + 1);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_free(c & 1)) : "memory");
        }
        if (!ok && lane == 0) atomicExch(fault, 1);
        const int row = (qb0 + b) * QB + 32 * (warp & 3) + lane;
        if (ok && row < q.n) (dir ? bwd : fwd)[out0 + row] = f;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(4 * QB));
}

// What an approximate distance may be off (see the file's head), with 2% slack;
// qn, tm: |q|^2 and the largest |t|^2.
__device__ __forceinline__ float search_bound(float qn, float tm) {
    const float s = sqrtf(qn) + sqrtf(tm);
    return 1.02f * ((3.82e-6f + 9.6e-7f) * s * s + 1.5e-8f * s);
}

// The reference's distance (matching.rs:27-33).
__device__ __forceinline__ float serial_dist(const float* __restrict__ a, const float* __restrict__ b) {
    float s = 0.0f;
#pragma unroll 8
    for (int k = 0; k < DESC_LEN / 4; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(a + 4 * k), y = *reinterpret_cast<const float4*>(b + 4 * k);
        const float d0 = x.x - y.x, d1 = x.y - y.y, d2 = x.z - y.z, d3 = x.w - y.w;
        s = s + d0 * d0;
        s = s + d1 * d1;
        s = s + d2 * d2;
        s = s + d3 * d3;
    }
    return s;
}

// matching.rs:74-90 for one query: its answer, or UINT32_MAX.  The 0.9 cap is
// the forward direction's.
__device__ __forceinline__ uint32_t answer(uint32_t idx, float d1, float d2, float ratio, int dir) {
    if (idx == UINT32_MAX || !isfinite(d2)) return UINT32_MAX;
    if (dir == 0 && d1 > 0.9f) return UINT32_MAX;
    return d1 > ratio * d2 ? UINT32_MAX : idx;
}

// With *fault set (a wait of nearest_kernel gave up, so some of its entries were
// not written) this kernel and the two after it read and answer nothing; the
// host then reports the fault.
__global__ void __launch_bounds__(256) outcome_kernel(const PairJob* __restrict__ jobs, const Frame* __restrict__ frames,
                                                      const float* __restrict__ desc, const float* __restrict__ norms,
                                                      const int* __restrict__ max_norm, const Two* __restrict__ fwd2,
                                                      const Two* __restrict__ bwd2, float ratio,
                                                      uint32_t* __restrict__ fwd, uint32_t* __restrict__ bwd,
                                                      int2* __restrict__ list, MatchStatus* __restrict__ st,
                                                      const int* __restrict__ fault) {
    if (*fault) {
        st->fault = 1;  // the host reads one block
        return;
    }
    const int dir = blockIdx.y & 1;
    const PairJob J = jobs[blockIdx.y >> 1];
    Frame q, t;
    int out0;
    direction(J, frames, dir, q, t, out0);
    const int row = blockIdx.x * 256 + threadIdx.x;
    if (row >= q.n) return;
    uint32_t out = UINT32_MAX;
    if (t.n > 1) {  // with fewer targets the second distance is infinite: refused
        const Two f = (dir ? bwd2 : fwd2)[out0 + row];
        const float qn = norms[q.blk * QB + row], tm = __int_as_float(max_norm[dir ? J.fa : J.fb]);
        const float d1 = f.v0 + qn, d2 = f.v1 + qn;
        // the reference's own error at the larger of the two distances
        const float e = search_bound(qn, tm) + 8.16e-6f * fmaxf(d2, 0.0f);
        const float r_lo = ratio * 0.9999995f, r_hi = ratio * 1.0000005f;
        const bool refused = (dir == 0 && d1 - e > 0.9000002f) || d1 - e > r_hi * (d2 + e);
        const bool accepted = (dir != 0 || d1 + e < 0.8999998f) && d1 + e < r_lo * (d2 - e) && d2 - d1 > 2.0f * e;
        if (accepted) {
            const int i = 2 * f.pair;
            const float* a = desc + (q.off + row) * DESC_LEN;
            const float* b = desc + (t.off + i) * DESC_LEN;
            out = (uint32_t)i;
            if (i + 1 < t.n && serial_dist(a, b + DESC_LEN) < serial_dist(a, b)) ++out;
        } else if (!refused) {
            const int at = atomicAdd(&st->listed, 1);
            if (at < RESCAN_MAX) list[at] = make_int2((int)blockIdx.y, row);
        }
    }
    (dir ? bwd : fwd)[out0 + row] = out;
}

// The smaller distance of each query of frame 0 (rcmvs_diag_match_distances) and
// its bound.
__global__ void distances_kernel(const Two* __restrict__ two, const float* __restrict__ norms,
                                 const int* __restrict__ max_norm, int n, float* __restrict__ approx,
                                 float* __restrict__ bound) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    approx[i] = two[i].v0 + norms[i];
    bound[i] = search_bound(norms[i], __int_as_float(max_norm[1]));
}

// Listed queries against all targets; one block each.
__global__ void __launch_bounds__(256) rescan_kernel(const PairJob* __restrict__ jobs, const Frame* __restrict__ frames,
                                                     const float* __restrict__ desc, float ratio,
                                                     uint32_t* __restrict__ fwd, uint32_t* __restrict__ bwd,
                                                     const int2* __restrict__ list, const MatchStatus* __restrict__ st,
                                                     const int* __restrict__ fault) {
    __shared__ Nearest part[8];
    if (*fault) return;
    const int n = st->listed;
    if (n > RESCAN_MAX || st->wild) return;  // the chunk runs again on the FP32 pipes
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const int dir = list[e].x & 1, row = list[e].y;
        Frame q, t;
        int out0;
        direction(jobs[list[e].x >> 1], frames, dir, q, t, out0);
        float best = INFINITY, second = INFINITY;
        uint32_t bi = UINT32_MAX;
        for (int i = threadIdx.x; i < t.n; i += 256)
            push(serial_dist(desc + (q.off + row) * DESC_LEN, desc + (t.off + i) * DESC_LEN), (uint32_t)i, best, bi, second);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            merge(best, bi, second, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o),
                  __shfl_xor_sync(0xffffffffu, second, o));
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = Nearest{bi, best, second};
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < 8; ++k) merge(best, bi, second, part[k].d1, part[k].idx, part[k].d2);
            (dir ? bwd : fwd)[out0 + row] = answer(bi, best, second, ratio, dir);
        }
        __syncthreads();
    }
}

// matching.rs:90-94: mutual answers.
__global__ void mutual_kernel(const PairJob* __restrict__ jobs, const uint32_t* __restrict__ fwd,
                              const uint32_t* __restrict__ bwd, uint32_t* __restrict__ match_b,
                              const int* __restrict__ fault) {
    if (*fault) return;
    const PairJob J = jobs[blockIdx.y];
    const int ia = blockIdx.x * 256 + threadIdx.x;
    if (ia >= J.na) return;
    const uint32_t f = fwd[J.row_off + ia];
    match_b[J.row_off + ia] = f != UINT32_MAX && bwd[J.col_off + f] == (uint32_t)ia ? f : UINT32_MAX;
}

// The matches of a chunk packed in pair order: how many each pair has, where
// they begin, and (second pass) the indices.  From COMPACT_MIN rows on: 135 k
// rows of 66 pairs collected on the host from one entry per row took 400 us of
// 1760.
constexpr int64_t COMPACT_MIN = 16384;
__device__ __forceinline__ int block_matches(const uint32_t* __restrict__ mb, int na, int base, uint32_t& b) {
    const int ia = base + (int)threadIdx.x;
    b = ia < na ? mb[ia] : UINT32_MAX;
    return __syncthreads_count(b != UINT32_MAX);
}
__global__ void __launch_bounds__(256) count_kernel(const PairJob* __restrict__ jobs, const uint32_t* __restrict__ match_b,
                                                    uint32_t* __restrict__ counts) {
    const PairJob J = jobs[blockIdx.x];
    int n = 0;
    uint32_t b;
    for (int base = 0; base < J.na; base += 256) n += block_matches(match_b + J.row_off, J.na, base, b);
    if (threadIdx.x == 0) counts[J.pair] = (uint32_t)n;
}
__global__ void __launch_bounds__(1024) begin_kernel(const uint32_t* __restrict__ counts, int n, uint32_t* __restrict__ begin) {
    __shared__ uint32_t s_sum[1024];
    uint32_t before = 0;
    for (int base = 0; base < n; base += 1024) {
        const int i = base + (int)threadIdx.x;
        const uint32_t c = i < n ? counts[i] : 0;
        s_sum[threadIdx.x] = c;
        __syncthreads();
        for (int o = 1; o < 1024; o <<= 1) {
            const uint32_t v = (int)threadIdx.x >= o ? s_sum[threadIdx.x - o] : 0;
            __syncthreads();
            s_sum[threadIdx.x] += v;
            __syncthreads();
        }
        if (i < n) begin[i] = before + s_sum[threadIdx.x] - c;
        before += s_sum[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0) begin[n] = before;
}
__global__ void __launch_bounds__(256) compact_kernel(const PairJob* __restrict__ jobs,
                                                      const uint32_t* __restrict__ match_b,
                                                      const uint32_t* __restrict__ begin, uint32_t* __restrict__ a,
                                                      uint32_t* __restrict__ b) {
    __shared__ int s_warp[8];
    const PairJob J = jobs[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    size_t at = begin[J.pair];
    for (int base = 0; base < J.na; base += 256) {
        uint32_t v;
        const int n = block_matches(match_b + J.row_off, J.na, base, v);
        const unsigned m = __ballot_sync(0xffffffffu, v != UINT32_MAX);
        if (lane == 0) s_warp[warp] = __popc(m);
        __syncthreads();
        int before = __popc(m & ((1u << lane) - 1u));
        for (int k = 0; k < warp; ++k) before += s_warp[k];
        if (v != UINT32_MAX) {
            a[at + before] = (uint32_t)(base + (int)threadIdx.x);
            b[at + before] = v;
        }
        at += n;
        __syncthreads();
    }
}

// matching.rs:74-94
__global__ void decide_kernel(const PairJob* __restrict__ jobs, const Nearest* __restrict__ fwd,
                              const Nearest* __restrict__ bwd, float ratio, uint32_t* __restrict__ match_b) {
    const PairJob J = jobs[blockIdx.y];
    const int ia = blockIdx.x * 256 + threadIdx.x;
    if (ia >= J.na) return;
    uint32_t out = UINT32_MAX;
    const Nearest f = fwd[J.row_off + ia];
    if (f.idx != UINT32_MAX && isfinite(f.d2) && !(f.d1 > 0.9f || f.d1 > ratio * f.d2)) {
        const Nearest g = bwd[J.col_off + f.idx];
        if (g.idx == (uint32_t)ia && isfinite(g.d2) && !(g.d1 > ratio * g.d2)) out = f.idx;
    }
    match_b[J.row_off + ia] = out;
}

int mfail(rcmvs_ctx* ctx, int code, const std::string& msg) {
    if (ctx) ctx->err = msg;
    return code;
}

#define MCK(x)                                                                                 \
    do {                                                                                       \
        cudaError_t e_ = (x);                                                                  \
        if (e_ != cudaSuccess)                                                                 \
            return mfail(ctx, e_ == cudaErrorMemoryAllocation ? RCMVS_E_NOMEM : RCMVS_E_CUDA,    \
                         std::string(#x) + ": " + cudaGetErrorString(e_));                     \
    } while (0)

// Context arena slots 160-175.
enum { M_DESC = 160, M_JOBS, M_ROWP, M_FWD, M_BWD, M_MB, M_COLP, M_FRAMES, M_PACK, M_NORM, M_MAXN, M_TWO, M_LIST, M_STATUS, M_BEGIN, M_AB };

// Chunks of fewer distances run on the FP32 pipes: there the tensor-core
// search's extra launches cost more than its products save.  Whole calls,
// FP32 / tensor: one pair of 512 122 / 145 us, of 1024 158 / 179, of 2048 290 /
// 275; 10 pairs of up to 1100 385 / 301, 66 pairs of 2048 5350 / 1315.
constexpr int64_t TENSOR_MIN = int64_t(1) << 22;
constexpr int64_t GROUP_BYTES = 1 << 20;  // descriptors uploaded between two searches

struct Event {  // no upload is left in flight when a call returns early
    cudaEvent_t e = nullptr;
    cudaStream_t stream = nullptr;
    ~Event() {
        if (!e) return;
        cudaStreamSynchronize(stream);
        cudaEventDestroy(e);
    }
};

}  // namespace
}  // namespace rcmvs

using namespace rcmvs;

extern "C" {

void rcmvs_matches_free(rcmvs_matches* m) {
    if (!m) return;
    std::free(m->offsets);
    std::free(m->a);
    std::free(m->b);
    m->offsets = nullptr;
    m->a = m->b = nullptr;
    m->n_pairs = 0;
}

int rcmvs_diag_match_distances(rcmvs_ctx* ctx, const float* q, int32_t n_q, const float* t, int32_t n_t, float* approx,
                               float* bound) {
    if (!ctx || !q || !t || n_q <= 0 || n_t <= 0 || n_q > (1 << 20) || n_t > (1 << 20) || !approx || !bound)
        return mfail(ctx, RCMVS_E_ARG, "rcmvs_diag_match_distances: bad argument");
    MCK(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    DeviceArena& A = ctx->arena;
    const int qb = (n_q + QB - 1) / QB, tb = (n_t + QB - 1) / QB;
    const size_t n = (size_t)n_q + n_t, nb = (size_t)qb + tb, row = sizeof(float) * DESC_LEN;
    const Frame frames[2] = {{0, 0, n_q}, {n_q, qb, n_t}};
    const int32_t blk[3] = {0, qb, qb + tb};
    PairJob job{};
    job.na = n_q;
    job.nb = n_t;
    job.fb = 1;
    void *p_desc, *p_frames, *p_pack, *p_norm, *p_maxn, *p_two, *p_st, *p_jobs, *p_out;
    MCK(A.get(M_DESC, row * n, &p_desc));
    MCK(A.get(M_FRAMES, sizeof(frames) + sizeof(blk), &p_frames));
    MCK(A.get(M_PACK, nb * QB_BYTES, &p_pack));
    MCK(A.get(M_NORM, nb * QB * sizeof(float), &p_norm));
    MCK(A.get(M_MAXN, sizeof(int) * 2, &p_maxn));
    MCK(A.get(M_TWO, sizeof(Two) * n, &p_two));
    MCK(A.get(M_STATUS, sizeof(MatchStatus), &p_st));
    MCK(A.get(M_JOBS, sizeof(PairJob), &p_jobs));
    MCK(A.get(M_FWD, sizeof(float) * 2 * (size_t)n_q, &p_out));
    Frame* df = (Frame*)p_frames;
    const int32_t* d_blk = (const int32_t*)(df + 2);
    MCK(cudaMemcpyAsync(p_desc, q, row * n_q, cudaMemcpyHostToDevice, st));
    MCK(cudaMemcpyAsync((float*)p_desc + (size_t)n_q * DESC_LEN, t, row * n_t, cudaMemcpyHostToDevice, st));
    MCK(cudaMemcpyAsync(df, frames, sizeof(frames), cudaMemcpyHostToDevice, st));
    MCK(cudaMemcpyAsync(df + 2, blk, sizeof(blk), cudaMemcpyHostToDevice, st));
    MCK(cudaMemcpyAsync(p_jobs, &job, sizeof(job), cudaMemcpyHostToDevice, st));
    MCK(cudaMemsetAsync(p_maxn, 0, sizeof(int) * 2, st));
    MCK(cudaMemsetAsync(p_st, 0, sizeof(MatchStatus), st));
    MCK(cudaFuncSetAttribute(nearest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kNearestSmem));
    pack_kernel<<<(unsigned)nb, 256, 0, st>>>((const float*)p_desc, df, d_blk, 2, 0, (unsigned char*)p_pack,
                                              (float*)p_norm, (int*)p_maxn, (MatchStatus*)p_st);
    MCK(cudaGetLastError());
    nearest_kernel<<<dim3(std::max(qb, tb), 2), kNearestThreads, kNearestSmem, st>>>(
        (const PairJob*)p_jobs, df, (const unsigned char*)p_pack, (const float*)p_norm, 1, (Two*)p_two, (Two*)p_two + n_q,
        ctx->d_fault);
    MCK(cudaGetLastError());
    distances_kernel<<<(n_q + 255) / 256, 256, 0, st>>>((const Two*)p_two, (const float*)p_norm, (const int*)p_maxn, n_q,
                                                        (float*)p_out, (float*)p_out + n_q);
    MCK(cudaGetLastError());
    MatchStatus status{};
    int fault = 0;
    MCK(cudaMemcpyAsync(&status, p_st, sizeof(status), cudaMemcpyDeviceToHost, st));
    MCK(cudaMemcpyAsync(&fault, ctx->d_fault, sizeof(int), cudaMemcpyDeviceToHost, st));
    MCK(cudaMemcpyAsync(approx, p_out, sizeof(float) * n_q, cudaMemcpyDeviceToHost, st));
    MCK(cudaMemcpyAsync(bound, (float*)p_out + n_q, sizeof(float) * n_q, cudaMemcpyDeviceToHost, st));
    MCK(cudaStreamSynchronize(st));
    if (fault) return report_fault(ctx);
    if (status.wild) return mfail(ctx, RCMVS_E_LIMIT, "rcmvs_diag_match_distances: a component past the packed range");
    return RCMVS_OK;
}

static int match_pairs_impl(rcmvs_ctx* ctx, const float* const* desc, const int32_t* n_desc, int32_t n_frames,
                            const int32_t* pairs, int32_t n_pairs, double ratio, rcmvs_matches* out);

int rcmvs_match_pairs(rcmvs_ctx* ctx, const float* const* desc, const int32_t* n_desc, int32_t n_frames,
                      const int32_t* pairs, int32_t n_pairs, double ratio, rcmvs_matches* out) {
    if (!ctx || !out || n_frames < 0 || n_pairs < 0 || (n_frames > 0 && (!desc || !n_desc)) ||
        (n_pairs > 0 && !pairs))
        return mfail(ctx, RCMVS_E_ARG, "rcmvs_match_pairs: bad argument");
    std::memset(out, 0, sizeof(*out));
    const int rc = match_pairs_impl(ctx, desc, n_desc, n_frames, pairs, n_pairs, ratio, out);
    if (rc) rcmvs_matches_free(out);  // nothing half-built reaches the caller
    return rc;
}

static int match_pairs_impl(rcmvs_ctx* ctx, const float* const* desc, const int32_t* n_desc, int32_t n_frames,
                            const int32_t* pairs, int32_t n_pairs, double ratio, rcmvs_matches* out) {
    std::vector<int64_t> foff(n_frames + 1, 0);
    for (int f = 0; f < n_frames; ++f) {
        if (n_desc[f] < 0 || (n_desc[f] > 0 && !desc[f])) return mfail(ctx, RCMVS_E_ARG, "bad descriptor set");
        foff[f + 1] = foff[f] + n_desc[f];
    }
    for (int p = 0; p < n_pairs; ++p)
        if (pairs[2 * p] < 0 || pairs[2 * p] >= n_frames || pairs[2 * p + 1] < 0 || pairs[2 * p + 1] >= n_frames)
            return mfail(ctx, RCMVS_E_ARG, "pair names a frame out of range");
    out->n_pairs = (uint64_t)n_pairs;
    out->offsets = (uint64_t*)std::calloc((size_t)n_pairs + 1, sizeof(uint64_t));
    if (!out->offsets) return mfail(ctx, RCMVS_E_NOMEM, "host allocation failed");
    std::vector<uint32_t> ra, rb;
    MCK(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    DeviceArena& A = ctx->arena;
    // tensor: no frame was found out of range (and a ratio the bound's tests
    // take), and the search's buffers fit
    const float r32 = (float)ratio;
    bool packed = false, tensor = r32 > 0.0f && r32 < 1e6f;
    // What the FP32 kernels need; the search's packed frames (as large as the
    // descriptors), this call's or an earlier one's, go where they take its room.
    auto need = [&](int slot, size_t bytes, void** p) -> cudaError_t {
        cudaError_t e = A.get(slot, bytes, p);
        if (e != cudaErrorMemoryAllocation) return e;
        cudaGetLastError();
        for (int s : {(int)M_PACK, (int)M_NORM, (int)M_TWO}) A.drop(s);
        packed = tensor = false;
        return A.get(slot, bytes, p);
    };
    // What they do without.
    auto room = [&](int slot, size_t bytes, void** p) {
        if (A.get(slot, bytes, p) == cudaSuccess) return true;
        cudaGetLastError();
        return false;
    };
    void* p_desc;
    MCK(need(M_DESC, sizeof(float) * DESC_LEN * (size_t)std::max<int64_t>(foff[n_frames], 1), &p_desc));
    auto upload = [&](int f, cudaStream_t on) -> cudaError_t {
        if (n_desc[f] == 0) return cudaSuccess;
        return cudaMemcpyAsync((float*)p_desc + foff[f] * DESC_LEN, desc[f], sizeof(float) * DESC_LEN * n_desc[f],
                               cudaMemcpyHostToDevice, on);
    };
    // the tensor-core search's packed frames (made with the first chunk that uses it)
    std::vector<Frame> frames(n_frames);
    std::vector<int32_t> blk(n_frames + 1, 0);
    for (int f = 0; f < n_frames; ++f) {
        frames[f] = Frame{foff[f], blk[f], n_desc[f]};
        if (blk[f] > INT32_MAX / 2) return mfail(ctx, RCMVS_E_LIMIT, "too many descriptors");
        blk[f + 1] = blk[f] + (n_desc[f] + QB - 1) / QB;
    }
    void *p_frames = nullptr, *p_blk = nullptr, *p_pack = nullptr, *p_norm = nullptr, *p_maxn = nullptr, *p_st = nullptr,
         *p_two = nullptr, *p_list = nullptr;
    void *p_jobs, *p_fwd, *p_bwd, *p_mb;
    auto chunk_room = [&](size_t n_jobs, int64_t rows, int64_t cols) -> cudaError_t {
        cudaError_t e = need(M_JOBS, sizeof(PairJob) * n_jobs, &p_jobs);
        if (!e) e = need(M_FWD, sizeof(Nearest) * (size_t)rows, &p_fwd);
        if (!e) e = need(M_BWD, sizeof(Nearest) * (size_t)cols, &p_bwd);
        if (!e) e = need(M_MB, sizeof(uint32_t) * (size_t)rows, &p_mb);
        return e;
    };
    auto tensor_room = [&](int64_t rows, int64_t cols) {
        const size_t nb = (size_t)std::max(blk[n_frames], 1);
        tensor = room(M_FRAMES, (sizeof(Frame) + sizeof(int32_t)) * n_frames, &p_frames) &&
                 room(M_PACK, nb * QB_BYTES, &p_pack) && room(M_NORM, nb * QB * sizeof(float), &p_norm) &&
                 room(M_MAXN, sizeof(int) * n_frames, &p_maxn) &&
                 room(M_TWO, sizeof(Two) * (size_t)(rows + cols), &p_two) &&
                 room(M_LIST, sizeof(int2) * RESCAN_MAX, &p_list) && room(M_STATUS, sizeof(MatchStatus), &p_st);
        if (tensor) p_blk = (Frame*)p_frames + n_frames;
        return tensor;
    };
    // Where all pairs make one chunk for the tensor-core search, the frames go
    // up on the context's second stream in groups, and a group is packed and
    // its pairs with the frames before it are searched while the next is
    // copied.  66 pairs of 12 frames of 2048, with the packed matches: 1760 -> 1315 us.
    bool overlap = false;
    if (tensor && n_pairs <= 32767 && foff[n_frames] * (int64_t)sizeof(float) * DESC_LEN >= 2 * GROUP_BYTES) {
        int64_t dists = 0, partials = 0, rows = 0, cols = 0;
        for (int p = 0; p < n_pairs && rows <= INT32_MAX / 2 && cols <= INT32_MAX / 2; ++p) {
            const int64_t na = n_desc[pairs[2 * p]], nb = n_desc[pairs[2 * p + 1]];
            partials += (nb + TILE - 1) / TILE * na + (na + TILE - 1) / TILE * nb;
            dists += na * nb;
            rows += na;
            cols += nb;
        }
        overlap = dists >= TENSOR_MIN && (size_t)partials * sizeof(Nearest) <= P_BUDGET && rows <= INT32_MAX / 2 &&
                  cols <= INT32_MAX / 2 && chunk_room((size_t)n_pairs, rows, cols) == cudaSuccess && tensor_room(rows, cols);
        if (!overlap) cudaGetLastError();
    }
    Event uploaded;
    if (overlap) {
        if (!ctx->upload) MCK(cudaStreamCreateWithFlags(&ctx->upload, cudaStreamNonBlocking));
        MCK(cudaEventCreateWithFlags(&uploaded.e, cudaEventDisableTiming));
        uploaded.stream = ctx->upload;
    } else {
        for (int f = 0; f < n_frames; ++f) MCK(upload(f, st));
    }
    int p = 0;
    while (p < n_pairs) {
        // a chunk of pairs whose distance matrices fit the budget (at least one)
        std::vector<PairJob> jobs;
        int64_t prow = 0, pcol = 0, rows = 0, cols = 0, dists = 0;
        int max_na = 0, max_nb = 0;
        while (p < n_pairs && jobs.size() < 32767) {
            const int fa = pairs[2 * p], fb = pairs[2 * p + 1];
            const int na = n_desc[fa], nb = n_desc[fb];
            const int64_t pr = (int64_t)((nb + TILE - 1) / TILE) * na, pc = (int64_t)((na + TILE - 1) / TILE) * nb;
            if (!jobs.empty() && (size_t)(prow + pr + pcol + pc) * sizeof(Nearest) > P_BUDGET) break;
            jobs.push_back(PairJob{foff[fa], foff[fb], prow, pcol, na, nb, (int32_t)rows, (int32_t)cols, fa, fb,
                                   (int32_t)jobs.size()});
            dists += (int64_t)na * nb;
            prow += pr;
            pcol += pc;
            rows += na;
            cols += nb;
            max_na = std::max(max_na, na);
            max_nb = std::max(max_nb, nb);
            ++p;
            if (rows > INT32_MAX / 2 || cols > INT32_MAX / 2) break;
        }
        const int first = p - (int)jobs.size();
        if (max_na > 0 && max_nb > 0) {
            void *p_rowp, *p_colp;
            MCK(chunk_room(jobs.size(), rows, cols));
            // on the device in the order in which their frames arrive
            std::vector<PairJob> queue(jobs);
            if (overlap)
                std::stable_sort(queue.begin(), queue.end(), [](const PairJob& x, const PairJob& y) {
                    return std::max(x.fa, x.fb) < std::max(y.fa, y.fb);
                });
            MCK(cudaMemcpyAsync(p_jobs, queue.data(), sizeof(PairJob) * jobs.size(), cudaMemcpyHostToDevice, st));
            const unsigned nj = (unsigned)jobs.size();
            const SpanHook& hook = ctx->hook();
            void *p_begin = nullptr, *p_ab = nullptr;
            const bool compact = rows >= COMPACT_MIN && room(M_BEGIN, sizeof(uint32_t) * (2 * jobs.size() + 1), &p_begin) &&
                                 room(M_AB, sizeof(uint32_t) * 2 * (size_t)rows, &p_ab);
            std::vector<uint32_t> mb(compact ? 0 : (size_t)rows), begin(compact ? jobs.size() + 1 : 0);
            // the answers' counts, or the answers, to the host
            auto collect = [&]() -> cudaError_t {
                if (!compact)
                    return cudaMemcpyAsync(mb.data(), p_mb, sizeof(uint32_t) * rows, cudaMemcpyDeviceToHost, st);
                uint32_t* d_begin = (uint32_t*)p_begin;
                uint32_t* d_count = d_begin + jobs.size() + 1;
                count_kernel<<<nj, 256, 0, st>>>((const PairJob*)p_jobs, (const uint32_t*)p_mb, d_count);
                begin_kernel<<<1, 1024, 0, st>>>(d_count, (int)nj, d_begin);
                compact_kernel<<<nj, 256, 0, st>>>((const PairJob*)p_jobs, (const uint32_t*)p_mb, d_begin, (uint32_t*)p_ab,
                                                   (uint32_t*)p_ab + rows);
                const cudaError_t e = cudaGetLastError();
                return e != cudaSuccess ? e
                                        : cudaMemcpyAsync(begin.data(), p_begin, sizeof(uint32_t) * begin.size(),
                                                          cudaMemcpyDeviceToHost, st);
            };
            bool on_tensor = tensor && dists >= TENSOR_MIN && tensor_room(rows, cols);
            if (on_tensor) {
                Two *f2 = (Two*)p_two, *b2 = f2 + rows;
                // the answers share the nearest entries' buffers (larger)
                uint32_t *fo = (uint32_t*)p_fwd, *bo = (uint32_t*)p_bwd;
                if (!packed) {
                    MCK(cudaMemcpyAsync(p_frames, frames.data(), sizeof(Frame) * n_frames, cudaMemcpyHostToDevice, st));
                    MCK(cudaMemcpyAsync(p_blk, blk.data(), sizeof(int32_t) * n_frames, cudaMemcpyHostToDevice, st));
                    MCK(cudaMemsetAsync(p_maxn, 0, sizeof(int) * n_frames, st));
                    MCK(cudaFuncSetAttribute(nearest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kNearestSmem));
                }
                MCK(cudaMemsetAsync(p_st, 0, sizeof(MatchStatus), st));
                const PairJob* dj = (const PairJob*)p_jobs;
                const Frame* df = (const Frame*)p_frames;
                MatchStatus* ds = (MatchStatus*)p_st;
                hook.begin("match_dist");
                auto pack = [&](int f0, int f1) -> cudaError_t {
                    if (blk[f1] == blk[f0]) return cudaSuccess;
                    pack_kernel<<<blk[f1] - blk[f0], 256, 0, st>>>((const float*)p_desc, df, (const int32_t*)p_blk,
                                                                   n_frames, blk[f0], (unsigned char*)p_pack,
                                                                   (float*)p_norm, (int*)p_maxn, ds);
                    return cudaGetLastError();
                };
                auto nearest = [&](size_t j0, size_t j1) -> cudaError_t {
                    // two query blocks per CTA share each target block's load; one when
                    // that would leave SMs without a CTA
                    int64_t qblocks = 0;
                    int most = 0;
                    for (size_t k = j0; k < j1; ++k) {
                        const int qa = (queue[k].na + QB - 1) / QB, qb = (queue[k].nb + QB - 1) / QB;
                        qblocks += qa + qb;
                        most = std::max(most, std::max(qa, qb));
                    }
                    if (qblocks == 0) return cudaSuccess;
                    const int per = qblocks >= 2 * 148 ? 2 : 1;
                    nearest_kernel<<<dim3((most + per - 1) / per, 2 * (unsigned)(j1 - j0)), kNearestThreads, kNearestSmem,
                                     st>>>(dj + j0, df, (const unsigned char*)p_pack, (const float*)p_norm, per, f2, b2,
                                           ctx->d_fault);
                    return cudaGetLastError();
                };
                const int max_n = std::max(max_na, max_nb);
                if (overlap) {
                    // earlier work on the descriptors' buffer ends before they are written
                    MCK(cudaEventRecord(uploaded.e, st));
                    MCK(cudaStreamWaitEvent(ctx->upload, uploaded.e, 0));
                    size_t j0 = 0;
                    for (int f0 = 0, f1; f0 < n_frames; f0 = f1) {
                        int64_t bytes = 0;
                        for (f1 = f0; f1 < n_frames && bytes < GROUP_BYTES; ++f1) {
                            MCK(upload(f1, ctx->upload));
                            bytes += (int64_t)sizeof(float) * DESC_LEN * n_desc[f1];
                        }
                        MCK(cudaEventRecord(uploaded.e, ctx->upload));
                        MCK(cudaStreamWaitEvent(st, uploaded.e, 0));
                        MCK(pack(f0, f1));
                        size_t j1 = j0;
                        while (j1 < queue.size() && std::max(queue[j1].fa, queue[j1].fb) < f1) ++j1;
                        MCK(nearest(j0, j1));
                        j0 = j1;
                    }
                } else {
                    if (!packed) MCK(pack(0, n_frames));
                    MCK(nearest(0, queue.size()));
                }
                packed = true;
                hook.end("match_dist");
                hook.begin("match_select");
                outcome_kernel<<<dim3((max_n + 255) / 256, 2 * nj), 256, 0, st>>>(
                    dj, df, (const float*)p_desc, (const float*)p_norm, (const int*)p_maxn, f2, b2, r32, fo, bo,
                    (int2*)p_list, ds, ctx->d_fault);
                MCK(cudaGetLastError());
                rescan_kernel<<<296, 256, 0, st>>>(dj, df, (const float*)p_desc, r32, fo, bo, (const int2*)p_list, ds,
                                                   ctx->d_fault);
                MCK(cudaGetLastError());
                mutual_kernel<<<dim3((max_na + 255) / 256, nj), 256, 0, st>>>(dj, fo, bo, (uint32_t*)p_mb, ctx->d_fault);
                MCK(cudaGetLastError());
                hook.end("match_select");
                MatchStatus status{};
                MCK(cudaMemcpyAsync(&status, p_st, sizeof(status), cudaMemcpyDeviceToHost, st));
                MCK(collect());
                MCK(cudaStreamSynchronize(st));
                if (status.fault) return report_fault(ctx);
                if (status.wild) tensor = false;
                on_tensor = !status.wild && status.listed <= RESCAN_MAX;
            }
            if (!on_tensor) {
                MCK(need(M_ROWP, sizeof(Nearest) * (size_t)std::max<int64_t>(prow, 1), &p_rowp));
                MCK(need(M_COLP, sizeof(Nearest) * (size_t)std::max<int64_t>(pcol, 1), &p_colp));
                hook.begin("match_dist");
                dist_kernel<<<dim3((max_nb + TILE - 1) / TILE, (max_na + TILE - 1) / TILE, nj), 256, 0, st>>>(
                    (const float*)p_desc, (const PairJob*)p_jobs, (Nearest*)p_rowp, (Nearest*)p_colp);
                MCK(cudaGetLastError());
                hook.end("match_dist");
                hook.begin("match_select");
                rows_kernel<<<dim3((max_na + 255) / 256, nj), 256, 0, st>>>((const PairJob*)p_jobs,
                                                                           (const Nearest*)p_rowp, (Nearest*)p_fwd);
                MCK(cudaGetLastError());
                cols_kernel<<<dim3((max_nb + 255) / 256, nj), 256, 0, st>>>((const PairJob*)p_jobs,
                                                                           (const Nearest*)p_colp, (Nearest*)p_bwd);
                MCK(cudaGetLastError());
                decide_kernel<<<dim3((max_na + 255) / 256, nj), 256, 0, st>>>(
                    (const PairJob*)p_jobs, (const Nearest*)p_fwd, (const Nearest*)p_bwd, r32, (uint32_t*)p_mb);
                MCK(cudaGetLastError());
                hook.end("match_select");
                MCK(collect());
                MCK(cudaStreamSynchronize(st));
            }
            if (compact) {
                const size_t had = ra.size(), n = begin.back();
                ra.resize(had + n);
                rb.resize(had + n);
                if (n) {
                    MCK(cudaMemcpyAsync(ra.data() + had, p_ab, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, st));
                    MCK(cudaMemcpyAsync(rb.data() + had, (uint32_t*)p_ab + rows, sizeof(uint32_t) * n,
                                        cudaMemcpyDeviceToHost, st));
                    MCK(cudaStreamSynchronize(st));
                }
                for (size_t c = 0; c < jobs.size(); ++c) out->offsets[first + c + 1] = had + begin[c + 1];
                continue;
            }
            for (size_t c = 0; c < jobs.size(); ++c) {
                for (int ia = 0; ia < jobs[c].na; ++ia) {
                    const uint32_t b = mb[(size_t)jobs[c].row_off + ia];
                    if (b != UINT32_MAX) {
                        ra.push_back((uint32_t)ia);
                        rb.push_back(b);
                    }
                }
                out->offsets[first + c + 1] = ra.size();
            }
        } else {
            for (size_t c = 0; c < jobs.size(); ++c) out->offsets[first + c + 1] = ra.size();
        }
    }
    const size_t n = ra.size();
    out->a = (uint32_t*)std::malloc(sizeof(uint32_t) * std::max<size_t>(n, 1));
    out->b = (uint32_t*)std::malloc(sizeof(uint32_t) * std::max<size_t>(n, 1));
    if (!out->a || !out->b) {
        rcmvs_matches_free(out);
        return mfail(ctx, RCMVS_E_NOMEM, "host allocation failed");
    }
    if (n) {
        std::memcpy(out->a, ra.data(), sizeof(uint32_t) * n);
        std::memcpy(out->b, rb.data(), sizeof(uint32_t) * n);
    }
    return RCMVS_OK;
}

}  // extern "C"
