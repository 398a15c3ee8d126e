// mappers.cu — numeric bin bounds on the device (dataset.rs:683-750).
//
// One block per numeric feature: the feature's sampled values (rows of the
// feature-major input picked by the ascending row sample, or every row) are
// filtered to the finite ones, sorted by a block-wide stable LSD radix sort
// of order-preserving 32-bit keys, reduced to their distinct values (+0.0 and
// -0.0 compare equal and are one value, as in the reference's dedup), and the
// bounds are the midpoints, in f64, between consecutive distinct values, or
// between the distinct values at the quantile positions
// floor(i / nb * (u - 1)) when there are more than nb of them, each kept only
// when it exceeds the previous bound. f64 arithmetic is the same IEEE
// sequence as the reference's (this file is compiled without contraction).
#include <float.h>
#include <math.h>

#include "kernels.h"

namespace bst {

namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr int MAP_THREADS = 512;
constexpr int MAP_WARPS = MAP_THREADS / 32;
constexpr int MAP_ITEMS = 16;                                 // keys per thread and tile
constexpr uint32_t MAP_WARP_KEYS = 32u * MAP_ITEMS;           // keys per warp and tile
constexpr uint32_t MAP_TILE = MAP_THREADS * MAP_ITEMS;        // keys per tile
constexpr int MAP_PARTS = MAP_THREADS / 256;                  // cross-warp scan: 2 x 8 warps
constexpr int MAP_PWARPS = MAP_WARPS / MAP_PARTS;
constexpr int MAP_COPIES = 8;                                 // of a digit's count while the keys are gathered

// Sign bit flipped for non-negative floats, all bits for negative ones:
// unsigned order of the keys is the numeric order of the floats (-0.0 just
// below +0.0).
__device__ __forceinline__ uint32_t float_key(float v) {
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    return __uint_as_float(u);
}

// Exclusive prefix sum of v over the block (blockDim.x = MAP_THREADS);
// *total = the block's sum. sh: MAP_WARPS + 1 words.
__device__ uint32_t map_block_scan(uint32_t v, uint32_t* sh, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, x, d);
        if (lane >= (uint32_t)d) x += t;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t y = lane < MAP_WARPS ? sh[lane] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, y, d);
            if (lane >= (uint32_t)d) y += t;
        }
        if (lane < MAP_WARPS) sh[lane] = y;
    }
    __syncthreads();
    const uint32_t r = (warp ? sh[warp - 1] : 0u) + x - v;
    *total = sh[MAP_WARPS - 1];
    __syncthreads();
    return r;
}

struct MapShared {
    union {
        struct {
            uint32_t wcnt[MAP_WARPS][256];  // per-warp digit counts, then the warps' exclusive prefixes
            uint32_t mask[MAP_WARPS][256];  // the lanes of a round with each digit
        };
        uint32_t tile[MAP_TILE];              // then the tile's keys in digit order
        uint32_t gcnt[4][256][MAP_COPIES];    // before: the gathered keys' digit counts
    };
    uint32_t qpre[MAP_PARTS][256];       // part sums, then places in the tile of the parts' first keys
    uint32_t base[256];                  // digit offsets of the next tile
    uint32_t goff[256];                  // place in the output less place in the tile, per digit
    uint32_t dcnt[4][256];               // the keys' counts of each digit value, per digit position
    uint32_t scan[MAP_WARPS + 1];
    uint32_t w;                          // finite keys
};
static_assert(sizeof(MapShared) <= 48 * 1024, "static shared memory");

// One stable pass of the LSD radix sort: the w keys of `in` by their digit
// at `shift` into `out`. Within a tile, key order is (warp, round, lane),
// which is index order; a key's place is the digit's offset + the keys of
// that digit in earlier tiles, earlier warps, earlier rounds and lower lanes.
// The tile is put in order in shared memory first, so that a warp's stores
// are a few runs of consecutive words instead of 32 sectors. Lanes of one digit find
// one another through a mask in shared memory: a vote takes the SM four cycles,
// and nine of them a key, or a match, were two thirds of a pass.
__device__ void radix_pass(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t w, uint32_t shift,
                           MapShared& s) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    for (uint32_t t0 = 0; t0 < w; t0 += MAP_TILE) {
        for (uint32_t d = lane; d < 256u; d += 32u) s.wcnt[warp][d] = s.mask[warp][d] = 0;
        __syncwarp();
        uint32_t key[MAP_ITEMS], dig[MAP_ITEMS], rank[MAP_ITEMS];
        const uint32_t wb = t0 + warp * MAP_WARP_KEYS;
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            const uint32_t i = wb + (uint32_t)r * 32u + lane;
            key[r] = i < w ? in[i] : 0u;
            dig[r] = i < w ? ((key[r] >> shift) & 255u) : 256u;  // 256: no digit
        }
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            const bool valid = dig[r] < 256u;
            if (valid) atomicOr(&s.mask[warp][dig[r]], 1u << lane);
            __syncwarp();
            const uint32_t peers = valid ? s.mask[warp][dig[r]] : 0u, c = valid ? s.wcnt[warp][dig[r]] : 0u;
            rank[r] = c + (uint32_t)__popc(peers & lt);
            __syncwarp();
            if (valid && (peers & lt) == 0u) {  // the first of the digit's lanes
                s.wcnt[warp][dig[r]] = c + (uint32_t)__popc(peers);
                s.mask[warp][dig[r]] = 0u;
            }
            __syncwarp();
        }
        __syncthreads();
        {  // exclusive prefixes over the warps of each part; part sums
            const uint32_t d = threadIdx.x & 255u, q = threadIdx.x >> 8;
            uint32_t c[MAP_PWARPS], run = 0;
#pragma unroll
            for (int k = 0; k < MAP_PWARPS; ++k) c[k] = s.wcnt[q * MAP_PWARPS + (uint32_t)k][d];
#pragma unroll
            for (int k = 0; k < MAP_PWARPS; ++k) {
                s.wcnt[q * MAP_PWARPS + (uint32_t)k][d] = run;
                run += c[k];
            }
            s.qpre[q][d] = run;
        }
        __syncthreads();
        uint32_t qs[MAP_PARTS], cnt = 0, incl = 0;
        if (threadIdx.x < 256u) {  // the digit's keys in the tile, summed over the lower digits of the warp
#pragma unroll
            for (int q = 0; q < MAP_PARTS; ++q) {
                qs[q] = s.qpre[q][threadIdx.x];
                cnt += qs[q];
            }
            incl = cnt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, incl, d);
                if (lane >= (uint32_t)d) incl += t;
            }
            if (lane == 31u) s.scan[warp] = incl;
        }
        __syncthreads();
        if (threadIdx.x < 256u) {
            uint32_t start = incl - cnt;
            for (uint32_t q = 0; q < warp; ++q) start += s.scan[q];
            s.goff[threadIdx.x] = s.base[threadIdx.x] - start;  // (wraps; the place added back is >= start)
            s.base[threadIdx.x] += cnt;
#pragma unroll
            for (int q = 0; q < MAP_PARTS; ++q) {
                s.qpre[q][threadIdx.x] = start;
                start += qs[q];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r)
            if (dig[r] < 256u) rank[r] += s.qpre[warp / MAP_PWARPS][dig[r]] + s.wcnt[warp][dig[r]];
        __syncthreads();  // the counts are read: their words become the tile
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r)
            if (dig[r] < 256u) s.tile[rank[r]] = key[r];
        __syncthreads();
        const uint32_t n = min(MAP_TILE, w - t0);
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            const uint32_t p = (uint32_t)r * MAP_THREADS + threadIdx.x;
            if (p < n) {
                const uint32_t k = s.tile[p];
                out[s.goff[(k >> shift) & 255u] + p] = k;
            }
        }
        __syncthreads();
    }
}

// Bound by one block's chain of phases a feature, so the phases are kept short
// (16 gathered values and 16 keys in flight a thread, plain shared atomics for
// the digit counts, one block scan a tile for the distinct values) and two
// blocks share an SM. 200,000 sampled values: 100 features 2049 -> 845 us, 200
// features 3952 -> 1336 us (one wave instead of two); 60,000: 585 -> 235 us.
__global__ void __launch_bounds__(MAP_THREADS, 2)
k_numeric_bounds(const float* __restrict__ x, uint64_t col_stride, const uint32_t* __restrict__ rows, uint32_t k,
                 const MapJob* __restrict__ jobs, uint32_t max_bins, uint32_t* __restrict__ scratch,
                 double* __restrict__ cand, double* __restrict__ bounds, uint32_t* __restrict__ n_bounds) {
    __shared__ MapShared s;
    const uint32_t j = blockIdx.x;
    const MapJob job = jobs[j];
    const float* col = x + (uint64_t)job.col * col_stride;
    uint32_t* A = scratch + (size_t)j * 2u * k;
    uint32_t* B = A + k;
    double* bj = bounds + (size_t)j * (max_bins + 2u);
    double* cj = cand + (size_t)j * max_bins;
    const uint32_t lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) s.w = 0;
    for (uint32_t i = threadIdx.x; i < 4u * 256u * MAP_COPIES; i += MAP_THREADS) (&s.gcnt[0][0][0])[i] = 0;
    __syncthreads();
    // finite sampled values as keys, in any order (the sort fixes it)
    for (uint32_t i0 = 0; i0 < k; i0 += MAP_TILE) {
        uint32_t at[MAP_ITEMS];
        float v[MAP_ITEMS];
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            const uint32_t i = i0 + (uint32_t)r * MAP_THREADS + threadIdx.x;
            at[r] = i < k ? (rows ? rows[i] : i) : 0u;
        }
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            const uint32_t i = i0 + (uint32_t)r * MAP_THREADS + threadIdx.x;
            v[r] = i < k ? col[at[r]] : INFINITY;
        }
        uint32_t m[MAP_ITEMS], tot = 0;
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            m[r] = __ballot_sync(FULL, isfinite(v[r]));
            tot += (uint32_t)__popc(m[r]);
        }
        uint32_t wbase = 0;
        if (lane == 0 && tot) wbase = atomicAdd(&s.w, tot);
        wbase = __shfl_sync(FULL, wbase, 0);
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            const bool fin = (m[r] >> lane) & 1u;
            const uint32_t key = float_key(v[r]);
            if (fin) A[wbase + (uint32_t)__popc(m[r] & ((1u << lane) - 1u))] = key;
            wbase += (uint32_t)__popc(m[r]);
            // the four digits' counts (the same for every pass: they depend
            // only on the keys), in copies for the lanes of a skewed digit
            if (fin)
#pragma unroll
                for (int dp = 0; dp < 4; ++dp) atomicAdd(&s.gcnt[dp][(key >> (8 * dp)) & 255u][lane % MAP_COPIES], 1u);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < 4u * 256u; i += MAP_THREADS) {
        uint32_t c = 0;
        for (uint32_t q = 0; q < MAP_COPIES; ++q) c += s.gcnt[i >> 8][i & 255u][q];
        s.dcnt[i >> 8][i & 255u] = c;
    }
    __syncthreads();
    const uint32_t w = s.w;
    if (w == 0) {
        if (threadIdx.x == 0) {
            bj[0] = DBL_MAX;
            n_bounds[j] = 1;
        }
        return;
    }
    // stable LSD radix sort, 8-bit digits; a pass whose digit is the same
    // for every key is skipped
    const uint32_t key0 = A[0];  // any one key: the digit counts do not depend on order
    uint32_t* in = A;
    uint32_t* out = B;
    for (uint32_t shift = 0; shift < 32u; shift += 8u) {
        const uint32_t* dc = s.dcnt[shift / 8u];
        if (dc[(key0 >> shift) & 255u] == w) continue;
        if (threadIdx.x < 32u) {  // exclusive scan of the 256 counts: 8 per lane
            uint32_t c[8], sum = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                c[q] = dc[lane * 8u + (uint32_t)q];
                sum += c[q];
            }
            uint32_t x = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, x, d);
                if (lane >= (uint32_t)d) x += t;
            }
            uint32_t run = x - sum;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                s.base[lane * 8u + (uint32_t)q] = run;
                run += c[q];
            }
        }
        __syncthreads();
        radix_pass(in, out, w, shift, s);
        uint32_t* t = in;
        in = out;
        out = t;
    }
    // distinct values (float equality), in order, into `out`
    uint32_t u = 0;
    for (uint32_t i0 = 0; i0 < w; i0 += MAP_TILE) {
        const uint32_t wb = i0 + (threadIdx.x >> 5) * MAP_WARP_KEYS + lane;
        uint32_t key[MAP_ITEMS], prev[MAP_ITEMS], m[MAP_ITEMS], tot = 0;
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            const uint32_t i = wb + (uint32_t)r * 32u;
            key[r] = i < w ? in[i] : 0u;
            prev[r] = i < w && i > 0 ? in[i - 1] : 0u;
        }
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            const uint32_t i = wb + (uint32_t)r * 32u;
            m[r] = __ballot_sync(FULL, i < w && (i == 0 || key_float(key[r]) != key_float(prev[r])));
            tot += (uint32_t)__popc(m[r]);
        }
        uint32_t all;  // the warp's place: its total counted once
        uint32_t pos = u + __shfl_sync(FULL, map_block_scan(lane == 0 ? tot : 0u, s.scan, &all), 0);
#pragma unroll
        for (int r = 0; r < MAP_ITEMS; ++r) {
            if ((m[r] >> lane) & 1u) out[pos + (uint32_t)__popc(m[r] & ((1u << lane) - 1u))] = key[r];
            pos += (uint32_t)__popc(m[r]);
        }
        u += all;
    }
    __syncthreads();
    if (u <= 1u) {  // one finite value (lo >= hi): a single bin, no NaN bin
        if (threadIdx.x == 0) {
            bj[0] = DBL_MAX;
            n_bounds[j] = 1;
        }
        return;
    }
    const uint32_t nb = w < max_bins ? w : max_bins;
    const uint32_t extra = job.has_nan ? 2u : 1u;  // the last bound (+ the NaN bin's)
    if (u <= nb) {
        for (uint32_t i = threadIdx.x; i + 1u < u; i += MAP_THREADS)
            bj[i] = ((double)key_float(out[i]) + (double)key_float(out[i + 1])) / 2.0;
        if (threadIdx.x == 0) {
            bj[u - 1] = DBL_MAX;
            if (job.has_nan) bj[u] = DBL_MAX;
            n_bounds[j] = u - 1 + extra;
        }
        return;
    }
    // quantile midpoints i = 1 .. nb - 1 (non-decreasing in i), kept when
    // above the previous one
    for (uint32_t i = 1u + threadIdx.x; i < nb; i += MAP_THREADS) {
        const double q = (double)i / (double)nb;
        uint64_t idx = (uint64_t)floor(q * (double)(u - 1u));
        if (idx > (uint64_t)(u - 2u)) idx = u - 2u;
        cj[i] = ((double)key_float(out[idx]) + (double)key_float(out[idx + 1])) / 2.0;
    }
    __syncthreads();
    uint32_t kept = 0;
    for (uint32_t i0 = 1; i0 < nb; i0 += MAP_THREADS) {
        const uint32_t i = i0 + threadIdx.x;
        const bool keep = i < nb && (i == 1u || cj[i] > cj[i - 1]);
        uint32_t tot;
        const uint32_t pos = map_block_scan(keep ? 1u : 0u, s.scan, &tot);
        if (keep) bj[kept + pos] = cj[i];
        kept += tot;
    }
    if (threadIdx.x == 0) {
        bj[kept] = DBL_MAX;
        if (job.has_nan) bj[kept + 1] = DBL_MAX;
        n_bounds[j] = kept + extra;
    }
}

}  // namespace

void launch_numeric_bounds(const float* x, uint64_t col_stride, const uint32_t* rows, uint32_t k, const MapJob* jobs,
                           uint32_t n_jobs, uint32_t max_bins, uint32_t* scratch, double* cand, double* bounds,
                           uint32_t* n_bounds, cudaStream_t st) {
    if (n_jobs == 0 || k == 0) return;
    k_numeric_bounds<<<n_jobs, MAP_THREADS, 0, st>>>(x, col_stride, rows, k, jobs, max_bins, scratch, cand, bounds,
                                                     n_bounds);
}

}  // namespace bst
