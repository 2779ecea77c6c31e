// cr_synth.cu -- synthetic LAS clouds, Morton ordering and the GPU build of
// the LAS-derived batched layout (include/cr_synth.h).
//
// The generator is a pure function of (seed, point index) built from 64-bit
// integer hashing and IEEE double + - * / floor; the host and device paths
// share the __host__ __device__ code below and compile without contraction
// (-ffp-contract=off / -fmad=false), so they write identical records.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <thread>
#include <utility>
#include <vector>

#include "../../include/cr_synth.h"
#include "cr_internal.h"
#include "cr_quant.h"

namespace {

constexpr int kRecBytes = CR_LAS_FORMAT2_BYTES;

// splitmix64 output function (Steele, Lea, Flood, "Fast splittable
// pseudorandom number generators", OOPSLA 2014).
__host__ __device__ inline uint64_t mix64(uint64_t z) {
    z ^= z >> 30;
    z *= 0xbf58476d1ce4e5b9ull;
    z ^= z >> 27;
    z *= 0x94d049bb133111ebull;
    z ^= z >> 31;
    return z;
}

__host__ __device__ inline uint64_t hash3(uint64_t seed, uint64_t a, uint64_t b) {
    return mix64(seed ^ mix64(a * 0x9E3779B97F4A7C15ull + b * 0xD6E8FEB86659FD93ull +
                              0x632BE59BD9B4E019ull));
}

__host__ __device__ inline double u53(uint64_t h) { return (double)(h >> 11) * (1.0 / 9007199254740992.0); }

// Value noise on the integer lattice with smoothstep interpolation.
__host__ __device__ inline double vnoise(double px, double py, uint64_t s) {
    const double fx = floor(px), fy = floor(py);
    const uint64_t ix = (uint64_t)(int64_t)fx, iy = (uint64_t)(int64_t)fy;
    const double tx = px - fx, ty = py - fy;
    const double v00 = u53(hash3(s, ix, iy)), v10 = u53(hash3(s, ix + 1, iy));
    const double v01 = u53(hash3(s, ix, iy + 1)), v11 = u53(hash3(s, ix + 1, iy + 1));
    const double sx = tx * tx * (3.0 - 2.0 * tx);
    const double sy = ty * ty * (3.0 - 2.0 * ty);
    const double a = v00 + sx * (v10 - v00);
    const double b = v01 + sx * (v11 - v01);
    return a + sy * (b - a);
}

// Fractional Brownian motion: octaves of halving amplitude, doubling frequency.
__host__ __device__ inline double fbm(double px, double py, uint64_t seed, int octaves) {
    double sum = 0.0, amp = 0.5, f = 1.0;
    for (int o = 0; o < octaves; o++) {
        sum = sum + amp * vnoise(px * f, py * f, seed + 0x1000ull * (uint64_t)(o + 1));
        amp = amp * 0.5;
        f = f * 2.0;
    }
    return sum;
}

// N(0, 1) by the Irwin-Hall sum of 12 uniforms.
__host__ __device__ inline double gauss(uint64_t seed, uint64_t i) {
    double s = 0.0;
    for (int k = 0; k < 3; k++) {
        const uint64_t h = hash3(seed, i, 10 + k);
        for (int j = 0; j < 4; j++)
            s = s + ((double)((h >> (16 * j)) & 0xFFFFu) * (1.0 / 65536.0) + (1.0 / 131072.0));
    }
    return s - 6.0;
}

__host__ __device__ inline int clamp255(int v) { return v < 0 ? 0 : (v > 255 ? 255 : v); }

struct GenPoint {
    double x, y, z;
    int r, g, b;
};

__host__ __device__ inline void terrain_color(const cr_synth_params& p, uint64_t i, double z, GenPoint& o) {
    double t = z / p.height;
    t = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
    const double c0[3] = {70.0, 110.0, 50.0}, c1[3] = {150.0, 120.0, 80.0}, c2[3] = {235.0, 235.0, 235.0};
    const uint64_t h = hash3(p.seed, i, 5);
    int c[3];
    for (int k = 0; k < 3; k++) {
        double v = t < 0.5 ? c0[k] + (c1[k] - c0[k]) * (2.0 * t) : c1[k] + (c2[k] - c1[k]) * (2.0 * t - 1.0);
        c[k] = clamp255((int)v + (int)((h >> (8 * k)) & 31u) - 16);
    }
    o.r = c[0];
    o.g = c[1];
    o.b = c[2];
}

__host__ __device__ inline void gen_point(const cr_synth_params& p, int64_t n, uint64_t i, GenPoint& o) {
    const int64_t box_total = (int64_t)p.num_boxes * p.points_per_box;
    const int64_t nbox_pts = p.kind == CR_SYNTH_TERRAIN_BOXES ? (box_total < n ? box_total : n) : 0;
    const int64_t nterrain = n - nbox_pts;
    const double inv_wl = 1.0 / p.wavelength;
    if ((int64_t)i < nterrain) {
        o.x = p.origin[0] + u53(hash3(p.seed, i, 0)) * p.extent;
        o.y = p.origin[1] + u53(hash3(p.seed, i, 1)) * p.extent;
        o.z = p.height * fbm(o.x * inv_wl, o.y * inv_wl, p.seed, p.octaves) + p.sigma * gauss(p.seed, i);
        terrain_color(p, i, o.z, o);
        return;
    }
    // points on the faces of axis-aligned boxes standing on the terrain
    const uint64_t k = i - (uint64_t)nterrain;
    const uint64_t bi = k / (uint64_t)p.points_per_box;
    const double cx = p.origin[0] + u53(hash3(p.seed ^ 0xB0C5ull, bi, 0)) * p.extent;
    const double cy = p.origin[1] + u53(hash3(p.seed ^ 0xB0C5ull, bi, 1)) * p.extent;
    const double wx = 10.0 + 30.0 * u53(hash3(p.seed ^ 0xB0C5ull, bi, 2));
    const double wy = 10.0 + 30.0 * u53(hash3(p.seed ^ 0xB0C5ull, bi, 3));
    const double h = p.box_min_height + (p.box_max_height - p.box_min_height) * u53(hash3(p.seed ^ 0xB0C5ull, bi, 4));
    const double z0 = p.height * fbm(cx * inv_wl, cy * inv_wl, p.seed, p.octaves);
    const double a_top = wx * wy, a_x = wy * h, a_y = wx * h;
    const double total = a_top + 2.0 * a_x + 2.0 * a_y;
    const double sel = u53(hash3(p.seed, i, 20)) * total;
    const double u = u53(hash3(p.seed, i, 21)), v = u53(hash3(p.seed, i, 22));
    const double x0 = cx - 0.5 * wx, y0 = cy - 0.5 * wy;
    if (sel < a_top) {
        o.x = x0 + u * wx; o.y = y0 + v * wy; o.z = z0 + h;
    } else if (sel < a_top + a_x) {
        o.x = x0; o.y = y0 + u * wy; o.z = z0 + v * h;
    } else if (sel < a_top + 2.0 * a_x) {
        o.x = x0 + wx; o.y = y0 + u * wy; o.z = z0 + v * h;
    } else if (sel < a_top + 2.0 * a_x + a_y) {
        o.x = x0 + u * wx; o.y = y0; o.z = z0 + v * h;
    } else {
        o.x = x0 + u * wx; o.y = y0 + wy; o.z = z0 + v * h;
    }
    const uint64_t hc = hash3(p.seed, i, 23);
    o.r = (int)(hc & 0xFFu);
    o.g = (int)((hc >> 8) & 0xFFu);
    o.b = (int)((hc >> 16) & 0xFFu);
}

__host__ __device__ inline void put_i32(uint8_t* d, int32_t v) {
    const uint32_t u = (uint32_t)v;
    for (int k = 0; k < 4; k++) d[k] = (uint8_t)(u >> (8 * k));
}
__host__ __device__ inline void put_u16(uint8_t* d, uint32_t v) {
    d[0] = (uint8_t)v;
    d[1] = (uint8_t)(v >> 8);
}
__host__ __device__ inline int32_t get_i32(const uint8_t* d) {
    return (int32_t)((uint32_t)d[0] | ((uint32_t)d[1] << 8) | ((uint32_t)d[2] << 16) | ((uint32_t)d[3] << 24));
}
__host__ __device__ inline uint32_t get_u16(const uint8_t* d) { return (uint32_t)d[0] | ((uint32_t)d[1] << 8); }

// floor(x / s + 0.5) (the LAS integer of a coordinate), bit for bit, with the
// division replaced by a multiplication with inv = RN(1/s) where that cannot
// change the result: x * inv lies within 3 ulps of RN(x / s) and
// r -> floor(RN(r + 0.5)) is monotone, so when both ends of a margin of 8
// ulps around the product give the same integer, so does RN(x / s).  Near a
// half-integer the division is done.  (Double division runs at a small
// fraction of the FP64 rate on this part.)
__host__ __device__ inline int32_t las_int(double x, double s, double inv) {
    const double r1 = x * inv;
    const double e = fabs(r1) * 0x1p-49;
    const double lo = floor((r1 - e) + 0.5), hi = floor((r1 + e) + 0.5);
    return (int32_t)(lo == hi ? lo : floor(x / s + 0.5));
}

// One LAS point-format-2 record (26 B).  Colors are stored as 16-bit values
// (c * 256) for 7 of 8 points and as plain 8-bit values for the rest, so both
// branches of the loader's `v < 256 ? v : v / 256` are exercised.
// inv_scale = 1 / p.las_scale.
__host__ __device__ inline void write_record(const cr_synth_params& p, double inv_scale, int64_t n,
                                             uint64_t i, uint8_t* d) {
    GenPoint g;
    gen_point(p, n, i, g);
    const int32_t X = las_int(g.x, p.las_scale, inv_scale);
    const int32_t Y = las_int(g.y, p.las_scale, inv_scale);
    const int32_t Z = las_int(g.z, p.las_scale, inv_scale);
    put_i32(d + 0, X);
    put_i32(d + 4, Y);
    put_i32(d + 8, Z);
    for (int k = 12; k < 20; k++) d[k] = 0;
    const bool wide = (hash3(p.seed, i, 6) & 7u) != 0u;
    const uint32_t m = wide ? 256u : 1u;
    put_u16(d + 20, (uint32_t)g.r * m);
    put_u16(d + 22, (uint32_t)g.g * m);
    put_u16(d + 24, (uint32_t)g.b * m);
}

// Sort_Frugal/src/main.cpp:58-77: 21 bits per axis, x at bit 0, y bit 1, z bit 2.
__host__ __device__ inline uint64_t spread3(uint32_t a) {
    uint64_t x = a & 0x1FFFFFu;
    x = (x | x << 32) & 0x1F00000000FFFFull;
    x = (x | x << 16) & 0x1F0000FF0000FFull;
    x = (x | x << 8) & 0x100F00F00F00F00Full;
    x = (x | x << 4) & 0x10C30C30C30C30C3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

// The same for 10 and 11 bits.
__host__ __device__ inline uint32_t spread10(uint32_t x) {
    x = (x | x << 16) & 0x030000FFu;
    x = (x | x << 8) & 0x0300F00Fu;
    x = (x | x << 4) & 0x030C30C3u;
    return (x | x << 2) & 0x09249249u;
}
__host__ __device__ inline uint32_t spread11(uint32_t x) { return spread10(x & 1023u) | (x >> 10) << 30; }

struct MortonFrame {
    double min[3];
    double cube, inv;  // inv = RN(1 / cube)
    double scale[3];
    double offset[3];
    // the GPU keys' integer form of morton_axis (cr_quant.h): decides all but about
    // one point in 10^5 per axis for LAS scales and extents; the host sort keeps the
    // double chain, so every GPU/host comparison checks it
    cr::QuantFx fx[3];
    cr::QuantQuick qq[3];
};

// Sort_Frugal/src/main.cpp:82-105: normalise by the largest header extent.
// The tool passes 2^21 for a point on the cube's far face to a 21-bit mask,
// which wraps it to 0 and sorts it to the front; it is clamped to 2^21 - 1 here.
// uint32(((v - min) / cube) * 2^21) as one product with the reciprocal: d *
// inv lies within a few ulps of RN(d / cube), so when no integer lies within
// 16 ulps of t1 = d * inv * 2^21 both truncate to the same integer; otherwise
// (rarely) the division is done.  Same rule as the encoder's quantize30.
__host__ __device__ inline uint32_t morton_axis(const MortonFrame& f, int k, int32_t X) {
    const double v = (double)X * f.scale[k] + f.offset[k];
    const double d = v - f.min[k];
    const double t1 = (d * f.inv) * 2097152.0;
    const double e = t1 * 0x1p-49;
    double t = t1;
    if (!(floor(t1 - e) == floor(t1 + e))) t = (d / f.cube) * 2097152.0;
    const uint32_t u = (t >= 0.0) ? (t < 4294967295.0 ? (uint32_t)t : 0xFFFFFFFFu) : 0u;
    return u < 2097151u ? u : 2097151u;
}

__host__ __device__ inline uint64_t morton_of(const MortonFrame& f, const uint8_t* rec) {
    uint32_t q[3];
    for (int k = 0; k < 3; k++) q[k] = morton_axis(f, k, get_i32(rec + 4 * k));
    return spread3(q[0]) | (spread3(q[1]) << 1) | (spread3(q[2]) << 2);
}

MortonFrame morton_frame(const cr_las_header* h) {
    MortonFrame f;
    double size[3];
    for (int k = 0; k < 3; k++) {
        f.min[k] = h->min[k];
        size[k] = h->max[k] - h->min[k];
        f.scale[k] = h->scale[k];
        f.offset[k] = h->offset[k];
    }
    f.cube = std::max(std::max(size[0], size[1]), size[2]);
    if (!(f.cube > 0.0)) f.cube = 1.0;
    f.inv = 1.0 / f.cube;
    for (int k = 0; k < 3; k++) {
        f.fx[k] = cr::quant_setup(f.scale[k], f.offset[k], f.min[k], 0.0, false, f.cube, 21, INT32_MIN, INT32_MAX);
        f.qq[k] = cr::quant_quick_setup(f.fx[k]);
    }
    return f;
}

void fill_header(const cr_synth_params* p, int64_t n, const int32_t mn[3], const int32_t mx[3],
                 cr_las_header* h) {
    h->num_points = n;
    h->point_format = 2;
    h->bytes_per_point = kRecBytes;
    for (int k = 0; k < 3; k++) {
        h->scale[k] = p->las_scale;
        h->offset[k] = 0.0;
        h->min[k] = (double)mn[k] * p->las_scale + 0.0;
        h->max[k] = (double)mx[k] * p->las_scale + 0.0;
    }
}

bool valid_params(const cr_synth_params* p) {
    return p && p->extent > 0.0 && p->height > 0.0 && p->wavelength > 0.0 && p->las_scale > 0.0 &&
           p->octaves >= 1 && p->octaves <= 16 &&
           (p->kind == CR_SYNTH_TERRAIN ||
            (p->kind == CR_SYNTH_TERRAIN_BOXES && p->num_boxes >= 0 && p->points_per_box > 0));
}

// ---- device kernels ------------------------------------------------------------

__global__ void k_gen(cr_synth_params p, double inv_scale, int64_t n, uint8_t* rec) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        write_record(p, inv_scale, n, (uint64_t)i, rec + i * kRecBytes);
}

__global__ void k_bounds(const uint8_t* rec, int64_t n, int32_t bpp, int32_t* mnmx) {
    int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        for (int k = 0; k < 3; k++) {
            int32_t v = get_i32(rec + i * bpp + 4 * k);
            mn[k] = min(mn[k], v);
            mx[k] = max(mx[k], v);
        }
    }
    for (int k = 0; k < 3; k++) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[k] = min(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
            mx[k] = max(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
        }
    }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 3; k++) {
            atomicMin(&mnmx[k], mn[k]);
            atomicMax(&mnmx[3 + k], mx[k]);
        }
}

// ---- record tiles in shared memory ----------------------------------------------
//
// LAS records are packed (26 bytes in format 2), so a thread that reads its own
// record issues a load per byte or half word and a warp's loads share sectors:
// the encoder and the keys were bound by those loads.  Here a CTA copies whole
// tiles of records with 16-byte cp.async, one tile ahead of the one it works on,
// and takes the fields from shared memory.

constexpr int kTileBytes = 53248;  // the keys': two tiles per CTA, two CTAs per SM

// Records per tile of `bytes`: whole 16-byte vectors, so every tile starts on one.
inline int tile_records(int32_t bpp, int bytes) { return std::min(2048, bytes / bpp) & ~15; }

// The int32 / uint16 at byte p of a tile; EVEN: every field starts on a half word.
template <bool EVEN>
__device__ __forceinline__ int32_t tile_i32(const uint8_t* p) {
    if (!EVEN) return get_i32(p);
    const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
    return (int32_t)((uint32_t)h[0] | ((uint32_t)h[1] << 16));
}
template <bool EVEN>
__device__ __forceinline__ uint32_t tile_u16(const uint8_t* p) {
    return EVEN ? *reinterpret_cast<const uint16_t*>(p) : get_u16(p);
}

// Starts the copy of `bytes` from the 16-byte aligned `src` to `dst` by the CTA.
__device__ __forceinline__ void copy_tile(uint8_t* dst, const uint8_t* src, int bytes) {
    const int vecs = bytes >> 4;
    for (int k = threadIdx.x; k < vecs; k += blockDim.x) {
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + 16 * k);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + 16 * (int64_t)k) : "memory");
    }
    for (int k = (vecs << 4) + threadIdx.x; k < bytes; k += blockDim.x) dst[k] = src[k];
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// Waits for all but the newest `PENDING` copies.
template <int PENDING>
__device__ __forceinline__ void wait_tile() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
    __syncthreads();
}

// A tile kernel's dynamic shared memory, allowed on the current device.
template <typename K>
bool allow_shared(K kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

// Morton keys and identity permutation of records [0, n), and a copy of the
// records for the gather to read: tiles go out again from shared memory, which
// saves the copy of the sorted records back a read of its own.
// (bpp even; copy null: none)
__global__ void __launch_bounds__(512, 2) k_morton_keys(MortonFrame f, const uint8_t* __restrict__ rec, int64_t n,
                                                        int32_t bpp, int tile_recs, unsigned long long* keys,
                                                        uint32_t* idx, uint8_t* __restrict__ copy) {
    extern __shared__ __align__(16) uint8_t s_tiles[];
    const int64_t ntiles = (n + tile_recs - 1) / tile_recs;
    auto recs = [&](int64_t t) { return (int)min((int64_t)tile_recs, n - t * tile_recs); };
    int64_t t = blockIdx.x;
    if (t < ntiles) copy_tile(s_tiles, rec + t * tile_recs * bpp, recs(t) * bpp);
    for (int buf = 0; t < ntiles; t += gridDim.x, buf ^= 1) {
        const int64_t next = t + gridDim.x;
        if (next < ntiles) {
            copy_tile(s_tiles + (buf ^ 1) * kTileBytes, rec + next * tile_recs * bpp, recs(next) * bpp);
            wait_tile<1>();
        } else {
            wait_tile<0>();
        }
        const uint8_t* tile = s_tiles + buf * kTileBytes;
        const int cnt = recs(t);
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
            uint32_t q[3];
            for (int k = 0; k < 3; k++) {
                const int32_t X = tile_i32<true>(tile + i * bpp + 4 * k);
                if (!cr::quant_quick(f.qq[k], X, 2097151u, &q[k]) &&
                    !cr::quant_fast(f.fx[k], X, 2097151u, &q[k]))
                    q[k] = morton_axis(f, k, X);
            }
            // spread3 of the low 10 and the high 11 bits of each axis, in 32 bits
            const uint32_t lo = spread10(q[0] & 1023u) | spread10(q[1] & 1023u) << 1 | spread10(q[2] & 1023u) << 2;
            const uint32_t hx = spread11(q[0] >> 10), hy = spread11(q[1] >> 10), hz = spread11(q[2] >> 10);
            const uint64_t hi = (uint64_t)hx | (uint64_t)hy << 1 | (uint64_t)hz << 2;
            keys[t * tile_recs + i] = hi << 30 | lo;
            idx[t * tile_recs + i] = (uint32_t)(t * tile_recs + i);
        }
        if (copy) {
            uint8_t* out = copy + t * tile_recs * bpp;
            const int bytes = cnt * bpp, vecs = bytes >> 4;
            for (int k = threadIdx.x; k < vecs; k += blockDim.x)
                reinterpret_cast<uint4*>(out)[k] = reinterpret_cast<const uint4*>(tile)[k];
            for (int k = (vecs << 4) + threadIdx.x; k < bytes; k += blockDim.x) out[k] = tile[k];
        }
        __syncthreads();  // the tile is free for the copy after next
    }
}

// Finishes a radix sort that left out the keys' lowest `low` bits: each run of
// equal upper bits, in index order so far, is sorted by the whole key (stable, so
// ties keep the index order).  A run of kMaxRun keys raises *flag, and the rest of the
// work is left, for the caller then sorts by all bits.  The keys of a
// tile, the key before and kMaxRun after it come to shared memory; each key finds
// its place by counting, in its run, the larger ones before it and the smaller ones
// after it, so a run is the work of as many threads as it has keys (an insertion
// sort by one thread per run was as fast on runs of one or two keys, but a sort of
// 5M points whose header spans 30 times their extent took 1712 us, now 1171, and
// one of 40M at 10 times 13.3 ms, now 6.6; 1.2 and 6.8 with passes over all bits).
// A run belongs to the CTA of its first key, which writes the keys that moved; the
// neighbouring CTA, which has its last keys too, takes only their upper bits, which
// no move changes (loads and stores are relaxed accesses, since they may meet).
constexpr int kMaxRun = 64, kRunTile = 1024;
__global__ void __launch_bounds__(256) k_sort_runs(unsigned long long* keys, uint32_t* idx, int64_t n, int low,
                                                   uint32_t* flag) {
    __shared__ unsigned long long s_key[1 + kRunTile + kMaxRun];
    __shared__ uint32_t s_idx[1 + kRunTile + kMaxRun];
    for (int64_t base = (int64_t)blockIdx.x * kRunTile; base < n; base += (int64_t)gridDim.x * kRunTile) {
        // (also the barrier between one tile's last reads and the next one's copy)
        if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile uint32_t*>(flag))) return;
        const int cnt = (int)min((int64_t)(kRunTile + kMaxRun), n - base);  // keys from base on
        const int before = base > 0 ? 1 : 0;
        for (int k = (int)threadIdx.x - before; k < cnt; k += 256) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(s_key[1 + k]) : "l"(keys + base + k) : "memory");
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(s_idx[1 + k]) : "l"(idx + base + k) : "memory");
        }
        __syncthreads();
        for (int i = 1 + threadIdx.x; i <= cnt; i += 256) {
            const unsigned long long key = s_key[i], head = key >> low;
            // first..last: the run, as far as the copy and kMaxRun keys each way go
            int first = i, last = i, at = i;
            while (first > 1 - before && i - first < kMaxRun && s_key[first - 1] >> low == head)
                at -= s_key[--first] > key;
            // begins before or after the tile, or is too long
            if (first < 1 || first > kRunTile || i - first >= kMaxRun) continue;
            while (last < cnt && last - first < kMaxRun && s_key[last + 1] >> low == head)
                at += s_key[++last] < key;
            if (last - first + 1 >= kMaxRun) {  // (may go on past the copy)
                if (i == first) *reinterpret_cast<volatile uint32_t*>(flag) = 1u;
                continue;
            }
            if (at == i) continue;
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(keys + base + at - 1), "l"(key) : "memory");
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(idx + base + at - 1), "r"(s_idx[i]) : "memory");
        }
    }
}

// dst[i] = src[perm[i]] for records of `bpp` bytes (even, <= kGatherMaxBpp).
// A warp gathers 32 records: each lane reads its source record as 16-bit
// words (records start on 2-byte boundaries), writes them into the warp's
// slice of shared memory at their destination offsets, and the warp stores the
// 32 * bpp contiguous destination bytes as 16-byte vectors (bpp is even, so
// 32 * bpp is a multiple of 16 and the warp's first byte is 16-byte aligned
// when dst is: `vec`).  The tail warp (fewer than 32 records) stores 16-bit words.
constexpr int kGatherMaxBpp = 64;
constexpr int kGatherWarps = 8;
__global__ void __launch_bounds__(32 * kGatherWarps) k_gather(const uint8_t* __restrict__ src,
                                                              uint8_t* __restrict__ dst,
                                                              const uint32_t* __restrict__ perm,
                                                              int64_t n, int32_t bpp, bool vec) {
    __shared__ __align__(16) uint16_t s_buf[kGatherWarps][32 * kGatherMaxBpp / 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint16_t* buf = s_buf[warp];
    const int words = bpp >> 1;
    const int64_t nwarps = (int64_t)gridDim.x * kGatherWarps;
    for (int64_t w0 = ((int64_t)blockIdx.x * kGatherWarps + warp) * 32; w0 < n; w0 += nwarps * 32) {
        const int64_t i = w0 + lane;
        const int cnt = (int)min((int64_t)32, n - w0);
        if (lane < cnt) {
            const uint16_t* s = reinterpret_cast<const uint16_t*>(src + (int64_t)perm[i] * bpp);
            for (int k = 0; k < words; k++) buf[lane * words + k] = __ldg(s + k);
        }
        __syncwarp();
        uint8_t* d = dst + w0 * bpp;
        if (cnt == 32 && vec) {
            const int vecs = (32 * bpp) >> 4;
            for (int k = lane; k < vecs; k += 32)
                reinterpret_cast<uint4*>(d)[k] = reinterpret_cast<const uint4*>(buf)[k];
        } else {
            for (int k = lane; k < cnt * words; k += 32) reinterpret_cast<uint16_t*>(d)[k] = buf[k];
        }
        __syncwarp();
    }
}

struct EncodeArgs {
    double scale[3], offset[3], box_min[3];
    int64_t n, sparse_offset;
    int32_t bpp, rgb, file_index;
};

// LasLoaderSparse.cpp:146-148: min(uint32(((v - min) / size) * 2^30), 2^30 - 1)
// (NaN -> 0), bit for bit, with one multiplication by inv = RN(1/size) in
// place of the division where that cannot change the result: d * inv lies
// within 3 ulps of RN(d / size), so when no integer lies within 8 ulps of
// t1 = d * inv * 2^30 both truncate to the same integer.  Otherwise (a point
// on the box's far face, about one in 2^20 others, a zero or subnormal size)
// the division is done.
__device__ __forceinline__ uint32_t quantize30(double d, double size, double inv) {
    const double t1 = (d * inv) * 1073741824.0;
    const double e = t1 * 0x1p-49;
    double t = t1;
    if (!(floor(t1 - e) == floor(t1 + e))) t = (d / size) * 1073741824.0;
    const uint32_t u = (t != t) ? 0u : (uint32_t)t;
    return u < 1073741823u ? u : 1073741823u;
}

// One batch's box and quantisation from the integer extremes, in shared memory.
struct EncodeBox {
    double box[6], size[3], inv[3];  // min and max; max - min; 1 / size
    cr::QuantFx fx[3];
    cr::QuantQuick qq[3];
};

// Writes a batch's record and the shared box from each thread's extremes.
// The batch AABB of v = double(X) * scale + offset - boxMin
// (LasLoaderSparse.cpp:93-105): every step rounds monotonically, so v is
// monotone in the integer X and the box is v at the integer extremes.
template <bool QUICK>
__device__ __forceinline__ void encode_box(const EncodeArgs& a, int32_t mn[3], int32_t mx[3], int64_t first,
                                           int cnt, cr_batch* batches, EncodeBox& s_b) {
    __shared__ int32_t s_red[6][32];
    for (int o = 16; o > 0; o >>= 1)
        for (int k = 0; k < 3; k++) {
            mn[k] = min(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
            mx[k] = max(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
        }
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 3; k++) {
            s_red[k][warp] = mn[k];
            s_red[3 + k][warp] = mx[k];
        }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        int32_t lo = s_red[k][0], hi = s_red[3 + k][0];
        for (int w = 1; w < nwarps; w++) {
            lo = min(lo, s_red[k][w]);
            hi = max(hi, s_red[3 + k][w]);
        }
        const double vlo = (double)lo * a.scale[k] + a.offset[k] - a.box_min[k];
        const double vhi = (double)hi * a.scale[k] + a.offset[k] - a.box_min[k];
        const double b0 = a.scale[k] < 0.0 ? vhi : vlo, b1 = a.scale[k] < 0.0 ? vlo : vhi;
        s_b.box[k] = b0;
        s_b.box[3 + k] = b1;
        s_b.size[k] = b1 - b0;
        s_b.inv[k] = 1.0 / (b1 - b0);
        s_b.fx[k] = cr::quant_setup(a.scale[k], a.offset[k], a.box_min[k], b0, true, b1 - b0, 30, lo, hi);
        if (QUICK) s_b.qq[k] = cr::quant_quick_setup(s_b.fx[k]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        cr_batch b;
        memset(&b, 0, sizeof(b));
        b.min_x = (float)s_b.box[0]; b.min_y = (float)s_b.box[1]; b.min_z = (float)s_b.box[2];
        b.max_x = (float)s_b.box[3]; b.max_y = (float)s_b.box[4]; b.max_z = (float)s_b.box[5];
        b.num_points = cnt;
        b.first_point = (int32_t)(a.sparse_offset + first);
        b.file_index = a.file_index;
        batches[blockIdx.x] = b;
    }
}

// The cell of a point that quant_quick left undecided, out of line: it would cost the
// common path registers.  quant_fast still decides those whose two cells clamp to one.
// The rest lie on a cell border or next to it, where quantize30's short cut would not
// hold either: the division is done at once.  (A batch whose range is a power of two
// times a small number has a whole axis of them, and the FP64 unit holds its CTA: 870k
// records with such a batch 98.6 -> 72.6 us, 40M 457 -> 431.)
__device__ __noinline__ uint32_t encode_exact(const EncodeArgs& a, const EncodeBox& s_b, int k, int32_t x) {
    uint32_t q;
    if (cr::quant_fast(s_b.fx[k], x, 1073741823u, &q)) return q;
    const double v = (double)x * a.scale[k] + a.offset[k] - a.box_min[k] - s_b.box[k];
    if (!s_b.fx[k].ok) return quantize30(v, s_b.size[k], s_b.inv[k]);  // any point
    const uint32_t u = (uint32_t)((v / s_b.size[k]) * 1073741824.0);
    return u < 1073741823u ? u : 1073741823u;
}

// One point to word `pi` of the streams, from its integer coordinates X (a
// callable of the axis) and its color word.  Each coordinate's 30-bit cell in
// integer arithmetic where the error bound decides it (cr_quant.h), else the
// double chain: the same integer either way.
// QUICK false: quant_quick's setup was left out.
template <bool QUICK, typename F>
__device__ __forceinline__ void encode_point(const EncodeArgs& a, const EncodeBox& s_b, F X, uint32_t color,
                                             int64_t pi, uint32_t* lo, uint32_t* md, uint32_t* hi, uint32_t* rgba) {
    uint32_t l = 0, m = 0, h = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int32_t x = X(k);
        uint32_t q;
        const bool done = QUICK ? cr::quant_quick(s_b.qq[k], x, 1073741823u, &q)
                                : cr::quant_fast(s_b.fx[k], x, 1073741823u, &q);
        if (!done) q = encode_exact(a, s_b, k, x);
        l |= ((q >> 20) & 1023u) << (10 * k);
        m |= ((q >> 10) & 1023u) << (10 * k);
        h |= (q & 1023u) << (10 * k);
    }
    lo[pi] = l;
    md[pi] = m;
    hi[pi] = h;
    rgba[pi] = color;
}

// The color word of a record (LasLoaderSparse.cpp:133-144).
template <bool EVEN>
__device__ __forceinline__ uint32_t encode_color(const EncodeArgs& a, const uint8_t* r) {
    if (a.rgb < 0) return 0u;
    uint32_t R = tile_u16<EVEN>(r + a.rgb), G = tile_u16<EVEN>(r + a.rgb + 2), B = tile_u16<EVEN>(r + a.rgb + 4);
    R = R < 256u ? R : R / 256u;
    G = G < 256u ? G : G / 256u;
    B = B < 256u ? B : B / 256u;
    return R | (G << 8) | (B << 16);
}

// LasLoaderSparse.cpp:84-199, one CTA per batch: its extremes, then its points,
// over a ring of STAGES tiles in shared memory.  The second walk runs backwards
// from the tiles that are still there.
//
// Reading each field from global memory (12 byte loads per record and walk) and
// quantising in 421 warp instructions per 32 points held it at 2.4 TB/s; tiles and
// quant_quick (one third of the instructions) leave the barriers and the box's
// serial double chain, which four small CTAs per SM cover: 40M records 1109 -> 523
// us, 200M 5329 -> 2288 (3.7 TB/s).  With few batches nothing covers them, and
// fewer, wider CTAs whose rings hold more of their batch are faster: at most one
// per SM (a load task of the LAS loader is 100) 1.0M records 65.5 -> 61 and 300k
// 52.8 -> 38, at most two 2M 108 -> 103 (EncodeMany 115).
template <int THREADS, int CTAS, int STAGES, int TILE_BYTES>
struct EncodeShape {
    static constexpr int kThreads = THREADS, kCtas = CTAS, kStages = STAGES, kBytes = TILE_BYTES;
    static constexpr int kShared = STAGES * TILE_BYTES;
};
using EncodeMany = EncodeShape<256, 4, 2, 26624>;
using EncodeTwo = EncodeShape<512, 2, 2, 53248>;
using EncodeFew = EncodeShape<1024, 1, 4, 53248>;

template <bool EVEN, typename S>
__global__ void __launch_bounds__(S::kThreads, S::kCtas) k_encode(EncodeArgs a, const uint8_t* __restrict__ rec,
                                                                  int tile_recs, cr_batch* batches, uint32_t* lo,
                                                                  uint32_t* md, uint32_t* hi, uint32_t* rgba) {
    extern __shared__ __align__(16) uint8_t s_tiles[];
    __shared__ EncodeBox s_b;
    const int64_t first = (int64_t)blockIdx.x * cr::kPointsPerBatch;
    const int cnt = (int)min((int64_t)cr::kPointsPerBatch, a.n - first);
    const uint8_t* src = rec + first * a.bpp;
    const int ntiles = (cnt + tile_recs - 1) / tile_recs;
    auto recs = [&](int t) { return min(tile_recs, cnt - t * tile_recs); };
    auto tile = [&](int t) { return s_tiles + (t % S::kStages) * S::kBytes; };
    // one copy group per call, empty outside the batch, so the waits count alike
    auto fetch = [&](int t) {
        copy_tile(tile(max(t, 0)), src + (int64_t)t * tile_recs * a.bpp, t >= 0 && t < ntiles ? recs(t) * a.bpp : 0);
    };
    int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    for (int t = 0; t < S::kStages - 1; t++) fetch(t);
    for (int t = 0; t < ntiles; t++) {
        fetch(t + S::kStages - 1);
        wait_tile<S::kStages - 1>();
        const uint8_t* r = tile(t);
        const int m = recs(t);
        for (int i = threadIdx.x; i < m; i += S::kThreads)
            for (int k = 0; k < 3; k++) {
                const int32_t X = tile_i32<EVEN>(r + i * a.bpp + 4 * k);
                mn[k] = min(mn[k], X);
                mx[k] = max(mx[k], X);
            }
        __syncthreads();
    }
    encode_box<true>(a, mn, mx, first, cnt, batches, s_b);
    for (int t = ntiles - 1; t >= 0; t--) {
        if (t < ntiles - S::kStages) wait_tile<S::kStages - 1>();
        const int m = recs(t);
        for (int i = threadIdx.x; i < m; i += S::kThreads) {
            const uint8_t* r = tile(t) + i * a.bpp;
            encode_point<true>(a, s_b, [&](int k) { return tile_i32<EVEN>(r + 4 * k); }, encode_color<EVEN>(a, r),
                               first + (int64_t)t * tile_recs + i, lo, md, hi, rgba);
        }
        __syncthreads();
        fetch(t - S::kStages);
    }
}

template <typename S>
cudaError_t launch_encode(const EncodeArgs& a, const uint8_t* rec, cr_batch* batches, uint32_t* lo, uint32_t* md,
                          uint32_t* hi, uint32_t* rgba, unsigned nb, cudaStream_t s) {
    const int tile = tile_records(a.bpp, S::kBytes);
    const bool even = (a.bpp & 1) == 0 && (a.rgb < 0 || (a.rgb & 1) == 0);
    const auto kernel = even ? k_encode<true, S> : k_encode<false, S>;
    if (!allow_shared(kernel, S::kShared)) return cudaErrorInvalidConfiguration;
    kernel<<<nb, S::kThreads, S::kShared, s>>>(a, rec, tile, batches, lo, md, hi, rgba);
    return cudaGetLastError();
}

// The same straight from global memory, a load per byte: records that do not start
// on a 16-byte boundary, that are long (a tile fetches all of a record, this the 18
// bytes it needs), or few.  QUICK false: without quant_quick, whose setup costs a CTA
// more than its few points gain.
template <bool QUICK>
__global__ void __launch_bounds__(256) k_encode_bytes(EncodeArgs a, const uint8_t* __restrict__ rec,
                                                      cr_batch* batches, uint32_t* lo, uint32_t* md, uint32_t* hi,
                                                      uint32_t* rgba) {
    __shared__ EncodeBox s_b;
    const int64_t first = (int64_t)blockIdx.x * cr::kPointsPerBatch;
    const int cnt = (int)min((int64_t)cr::kPointsPerBatch, a.n - first);
    int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    for (int i = threadIdx.x; i < cnt; i += blockDim.x)
        for (int k = 0; k < 3; k++) {
            const int32_t X = get_i32(rec + (first + i) * a.bpp + 4 * k);
            mn[k] = min(mn[k], X);
            mx[k] = max(mx[k], X);
        }
    encode_box<QUICK>(a, mn, mx, first, cnt, batches, s_b);
    for (int i = threadIdx.x; i < cnt; i += blockDim.x)
        encode_point<QUICK>(a, s_b, [&](int k) { return get_i32(rec + (first + i) * a.bpp + 4 * k); },
                            encode_color<false>(a, rec + (first + i) * a.bpp), first + i, lo, md, hi, rgba);
}

__host__ __device__ inline cr_vertex uniform_vertex(uint64_t seed, uint64_t i, float size) {
    const uint64_t h0 = hash3(seed, i, 0), h1 = hash3(seed, i, 1), h2 = hash3(seed, i, 2);
    const float k = 1.0f / 16777216.0f;
    cr_vertex v;
    v.x = ((float)(uint32_t)(h0 >> 40) * k) * size;
    v.y = ((float)(uint32_t)((h0 >> 16) & 0xFFFFFFu) * k) * size;
    v.z = ((float)(uint32_t)(h1 >> 40) * k) * size;
    v.color = (uint32_t)(h2 >> 32);
    return v;
}

__global__ void k_uniform(uint64_t seed, int64_t n, float size, cr_vertex* out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = uniform_vertex(seed, (uint64_t)i, size);
}

int grid_for(int64_t n) {
    int64_t g = (n + 255) / 256;
    return (int)std::min<int64_t>(std::max<int64_t>(g, 1), 65535);
}

template <typename F>
void parallel_for(int64_t n, F f) {
    unsigned t = std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
    if (n < 65536) t = 1;
    std::vector<std::thread> th;
    for (unsigned k = 0; k < t; k++)
        th.emplace_back([=] { f(n * k / t, n * (k + 1) / t); });
    for (auto& x : th) x.join();
}

cr_status cuda_status(cudaError_t e) {
    return e == cudaSuccess ? CR_OK : (e == cudaErrorMemoryAllocation ? CR_ERR_OUT_OF_MEMORY : CR_ERR_CUDA);
}

}  // namespace

cr_status cr::encode_records_device(const uint8_t* d_rec, int64_t n, int32_t bpp, int32_t rgb,
                                   const double scale[3], const double offset[3], const double box_min[3],
                                   int64_t sparse_offset, int32_t file_index, cr_batch* d_batches,
                                   uint32_t* d_lo, uint32_t* d_md, uint32_t* d_hi, uint32_t* d_rgba,
                                   void* stream) {
    if (n < 0 || (n > 0 && !d_rec) || bpp < 12 || !scale || !offset || !box_min || !d_batches || !d_lo ||
        !d_md || !d_hi || !d_rgba || sparse_offset < 0 || sparse_offset + n >= ((int64_t)1 << 31))
        return CR_ERR_INVALID_ARG;
    for (int k = 0; k < 3; k++)
        if (!std::isfinite(scale[k]) || !std::isfinite(offset[k]) || !std::isfinite(box_min[k]))
            return CR_ERR_INVALID_ARG;
    if (rgb >= 0 && rgb + 6 > bpp) return CR_ERR_INVALID_ARG;
    const int64_t nb = cr_num_batches(n);
    if (nb == 0) return CR_OK;
    EncodeArgs a;
    for (int k = 0; k < 3; k++) {
        a.scale[k] = scale[k];
        a.offset[k] = offset[k];
        a.box_min[k] = box_min[k];
    }
    a.n = n;
    a.sparse_offset = sparse_offset;
    a.bpp = bpp;
    a.rgb = rgb < 0 ? -1 : rgb;
    a.file_index = file_index;
    cudaStream_t s = (cudaStream_t)stream;
    // Where neither tiles nor the quick form pay.  us by the bytes / by tiles (before there
    // were tiles): 1,000 points 15.5 / 18.5 (15.5), 2,000 19.1 / 19.7 (19.4), 4,500 25.6 /
    // 23.7 (27.4); 10M points of 300 bytes 549 / 912 (710), 100k 71 / 126 (83), 6M of 200
    // bytes 324 / 386 (380), of 140 300 / 292 (384), of 100 238 / 225 (288).
    constexpr int64_t kFewPoints = 2048;
    constexpr int32_t kTileMaxBpp = 140;
    if (n <= kFewPoints) {
        k_encode_bytes<false><<<(unsigned)nb, 256, 0, s>>>(a, d_rec, d_batches, d_lo, d_md, d_hi, d_rgba);
        return cuda_status(cudaGetLastError());
    }
    if (bpp > kTileMaxBpp || (reinterpret_cast<uintptr_t>(d_rec) & 15) != 0) {
        k_encode_bytes<true><<<(unsigned)nb, 256, 0, s>>>(a, d_rec, d_batches, d_lo, d_md, d_hi, d_rgba);
        return cuda_status(cudaGetLastError());
    }
    int device = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) {
        // (the ring of EncodeFew holds most of a batch of 28-byte records; of 34 bytes, 600k
        // points took 44.1 us with it, 42.1 in EncodeTwo)
        const auto launch = nb <= sms && bpp <= 28 ? launch_encode<EncodeFew>
                            : nb <= 2 * sms        ? launch_encode<EncodeTwo>
                                                   : launch_encode<EncodeMany>;
        e = launch(a, d_rec, d_batches, d_lo, d_md, d_hi, d_rgba, (unsigned)nb, s);
    }
    return cuda_status(e);
}

extern "C" {

void cr_synth_params_default(int32_t kind, double extent, uint64_t seed, cr_synth_params* out) {
    if (!out) return;
    std::memset(out, 0, sizeof(*out));
    out->kind = kind;
    out->octaves = 6;
    out->seed = seed;
    out->extent = extent;
    out->height = 20.0;
    out->sigma = 0.05;
    out->wavelength = extent / 4.0;
    out->las_scale = 0.001;
    out->num_boxes = 2000;
    out->points_per_box = 20000;
    out->box_min_height = 10.0;
    out->box_max_height = 60.0;
}

cr_status cr_synth_points_host(const cr_synth_params* p, int64_t n, uint8_t* rec, cr_las_header* hdr) {
    if (!valid_params(p) || n < 0 || (n > 0 && !rec) || !hdr) return CR_ERR_INVALID_ARG;
    const cr_synth_params pp = *p;
    const double inv = 1.0 / pp.las_scale;
    parallel_for(n, [&](int64_t a, int64_t b) {
        for (int64_t i = a; i < b; i++) write_record(pp, inv, n, (uint64_t)i, rec + i * kRecBytes);
    });
    int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    for (int64_t i = 0; i < n; i++)
        for (int k = 0; k < 3; k++) {
            const int32_t v = get_i32(rec + i * kRecBytes + 4 * k);
            mn[k] = std::min(mn[k], v);
            mx[k] = std::max(mx[k], v);
        }
    if (n == 0)
        for (int k = 0; k < 3; k++) mn[k] = mx[k] = 0;
    fill_header(p, n, mn, mx, hdr);
    return CR_OK;
}

cr_status cr_morton_sort_host(uint8_t* rec, int64_t n, int32_t bpp, const cr_las_header* hdr) {
    if (n < 0 || (n > 0 && !rec) || bpp < 12 || !hdr || n >= ((int64_t)1 << 32)) return CR_ERR_INVALID_ARG;
    const MortonFrame f = morton_frame(hdr);
    std::vector<std::pair<uint64_t, uint32_t>> keys((size_t)n);
    parallel_for(n, [&](int64_t a, int64_t b) {
        for (int64_t i = a; i < b; i++) keys[i] = {morton_of(f, rec + i * bpp), (uint32_t)i};
    });
    std::sort(keys.begin(), keys.end());
    std::vector<uint8_t> tmp((size_t)n * bpp);
    parallel_for(n, [&](int64_t a, int64_t b) {
        for (int64_t i = a; i < b; i++)
            std::memcpy(&tmp[(size_t)i * bpp], rec + (int64_t)keys[i].second * bpp, bpp);
    });
    std::memcpy(rec, tmp.data(), tmp.size());
    return CR_OK;
}

cr_status cr_synth_points_device(cr_ctx* ctx, const cr_synth_params* p, int64_t n, uint8_t* d_rec,
                                 cr_las_header* hdr, void* stream) {
    if (!ctx || !valid_params(p) || n < 0 || (n > 0 && !d_rec) || !hdr) return CR_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    int32_t init[6] = {INT32_MAX, INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN, INT32_MIN};
    int32_t* d_mm = nullptr;
    cudaError_t e = cr::ctx_alloc(ctx, &d_mm, sizeof(init));
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_mm, init, sizeof(init), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && n > 0) {
        k_gen<<<grid_for(n) * 4 > 65535 ? 65535 : grid_for(n) * 4, 256, 0, s>>>(*p, 1.0 / p->las_scale,
                                                                                 n, d_rec);
        k_bounds<<<grid_for(n) > 2048 ? 2048 : grid_for(n), 256, 0, s>>>(d_rec, n, kRecBytes, d_mm);
        e = cudaGetLastError();
    }
    int32_t mm[6];
    if (e == cudaSuccess) e = cudaMemcpyAsync(mm, d_mm, sizeof(mm), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (d_mm) cudaFree(d_mm);
    if (e != cudaSuccess) return cuda_status(e);
    if (n == 0)
        for (int k = 0; k < 6; k++) mm[k] = 0;
    fill_header(p, n, mm, mm + 3, hdr);
    return CR_OK;
}

cr_status cr_morton_sort_device(cr_ctx* ctx, uint8_t* d_rec, int64_t n, int32_t bpp,
                                const cr_las_header* hdr, void* stream) {
    if (!ctx || n < 0 || (n > 0 && !d_rec) || bpp < 12 || (bpp & 1) || bpp > kGatherMaxBpp || !hdr ||
        n >= ((int64_t)1 << 31))
        return CR_ERR_INVALID_ARG;
    if (n == 0) cr::release_work(ctx);
    if (n <= 1) return CR_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const MortonFrame f = morton_frame(hdr);
    // The sort's buffers in one piece (six allocations of their own took 2 ms of a
    // 40M-point sort in the driver): keys and indices twice, the radix sort's own, a
    // copy of the records (the gather reads it and writes d_rec in place), a flag.
    cub::DoubleBuffer<unsigned long long> keys;
    cub::DoubleBuffer<uint32_t> vals;
    size_t cub_bytes = 0;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, keys, vals, (int)n, 0, 63, s);
    if (e != cudaSuccess) return cuda_status(e);
    const auto padded = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    const size_t key_bytes = padded((size_t)n * 8), val_bytes = padded((size_t)n * 4);
    cr::WorkBuffer buf(ctx, 2 * key_bytes + 2 * val_bytes + padded(cub_bytes) + padded((size_t)n * bpp) + 256);
    if (buf.status != cudaSuccess) return cuda_status(buf.status);
    uint8_t* at = buf.data;
    const auto take = [&at](size_t bytes) {
        uint8_t* p = at;
        at += bytes;
        return p;
    };
    for (auto& k : keys.d_buffers) k = reinterpret_cast<unsigned long long*>(take(key_bytes));
    for (auto& v : vals.d_buffers) v = reinterpret_cast<uint32_t*>(take(val_bytes));
    void* cub_tmp = take(padded(cub_bytes));
    uint32_t* flag = reinterpret_cast<uint32_t*>(take(256));
    uint8_t* copy = at;
    // tiles start on 16 bytes: records that do not are copied to where they do first
    const bool aligned = (reinterpret_cast<uintptr_t>(d_rec) & 15) == 0;
    if (!aligned) e = cudaMemcpyAsync(copy, d_rec, (size_t)n * bpp, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess && !allow_shared(k_morton_keys, 2 * kTileBytes)) e = cudaErrorInvalidConfiguration;
    if (e == cudaSuccess) {
        // bpp <= kGatherMaxBpp: at least 832; less for few points, so that every SM has
        // some (its FP64 unit is slow where a cube's cells put points on their borders:
        // 10,000 points in a cube of 2^21 units 169 -> 134 us per sort)
        const int ctas = 2 * cr_ctx_num_sms(ctx);
        const int tile = (int)std::min<int64_t>(tile_records(bpp, kTileBytes), std::max<int64_t>((n / ctas + 16) & ~15, 128));
        const int grid = (int)std::min<int64_t>((n + tile - 1) / tile, ctas);
        k_morton_keys<<<grid, 512, 2 * kTileBytes, s>>>(f, aligned ? d_rec : copy, n, bpp, tile, keys.Current(),
                                                        vals.Current(), aligned ? copy : nullptr);
        e = cudaGetLastError();
    }
    // Radix passes over the upper 40 bits, 5 in place of 8 at 0.3 ms each for 40M
    // points; k_sort_runs (0.2 ms) finishes the runs they leave equal.  A surface scan
    // fills about two bits of three, so 40 bits are 2^26 cells and runs stay short;
    // points so clustered that a run reaches kMaxRun (a far outlier stretches the
    // header's cube, or duplicates) get the passes over all bits after all.  The sort
    // then takes, against all bits at once with allocations of its own: 40M points
    // 6.1-6.6 ms (6.7-6.9), 5M 0.99-1.17 (1.2), 300k 302 us (495).  Where a clustered
    // cloud would lose, all bits come first and only:
    //   up to kFullKeys points (10,000 by both sorts 335 us, 80,000 280, against 145 and
    //   245): 131 us at 10,000 points, 166 at 65,536 (115 and 145 by the short passes,
    //   where no run is long);
    //   above 2^26, whose cells take 48 bits, 6 passes (200M by both 37.6-38.9 ms
    //   against 33.0-33.7, 600M 112-116 against 96-99): 29.9-30.6 and 90-92 ms; 31.2 and
    //   93.7 where no run is long (28.7 and 86.6 by the short passes, 34.3 and 100 with
    //   allocations of its own).
    constexpr int64_t kFullKeys = 8 * cr::kPointsPerBatch;
    const int low = n <= kFullKeys || n > ((int64_t)1 << 26) ? 0 : 23;
    if (e == cudaSuccess)
        e = cub::DeviceRadixSort::SortPairs(cub_tmp, cub_bytes, keys, vals, (int)n, low, 63, s);
    if (low > 0) {
        uint32_t long_runs = 0;
        if (e == cudaSuccess) e = cudaMemsetAsync(flag, 0, 4, s);
        if (e == cudaSuccess) {
            k_sort_runs<<<(unsigned)std::min<int64_t>((n + kRunTile - 1) / kRunTile, 65535), 256, 0, s>>>(
                keys.Current(), vals.Current(), n, low, flag);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(&long_runs, flag, 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess && long_runs)
            e = cub::DeviceRadixSort::SortPairs(cub_tmp, cub_bytes, keys, vals, (int)n, 0, 63, s);
    }
    if (e == cudaSuccess) {
        const int64_t warps = (n + 31) / 32;
        const int grid = (int)std::min<int64_t>((warps + kGatherWarps - 1) / kGatherWarps, 65535);
        k_gather<<<grid, 32 * kGatherWarps, 0, s>>>(copy, d_rec, vals.Current(), n, bpp, aligned);
        e = cudaGetLastError();
    }
    // idle before the buffer is given back, after an error too
    const cudaError_t done = cudaStreamSynchronize(s);
    return cuda_status(e == cudaSuccess ? done : e);
}

cr_status cr_encode_las_device(cr_ctx* ctx, const uint8_t* d_rec, int64_t n, int32_t bpp, int32_t fmt,
                               const double scale[3], const double offset[3], const double box_min[3],
                               int64_t sparse_offset, int32_t file_index, cr_batch* d_batches,
                               uint32_t* d_lo, uint32_t* d_md, uint32_t* d_hi, uint32_t* d_rgba,
                               void* stream) {
    if (!ctx) return CR_ERR_INVALID_ARG;
    // LasLoaderSparse.cpp:123-131: formats without RGB read their colour at byte 0
    const int rgb = fmt == 2 ? 20 : (fmt == 3 ? 28 : ((fmt == 7 || fmt == 8) ? 30 : 0));
    return cr::encode_records_device(d_rec, n, bpp, rgb, scale, offset, box_min, sparse_offset, file_index,
                                     d_batches, d_lo, d_md, d_hi, d_rgba, stream);
}

cr_status cr_synth_cloud_device(cr_ctx* ctx, const cr_synth_params* p, int64_t n, cr_cloud* cloud,
                                cr_las_header* hdr, void* stream) {
    if (!ctx || !valid_params(p) || !cloud || !hdr || n <= 0) return CR_ERR_INVALID_ARG;
    if (cr_cloud_num_points(cloud) != n || cr_cloud_num_batches(cloud) != cr_num_batches(n))
        return CR_ERR_INVALID_ARG;
    cr_batch* db;
    uint32_t *lo, *md, *hi, *rgba;
    cr_status st = cr_cloud_device(cloud, &db, &lo, &md, &hi, &rgba);
    if (st != CR_OK || !lo || !md || !hi || !rgba) return CR_ERR_INVALID_ARG;
    uint8_t* rec = nullptr;
    cudaError_t e = cr::ctx_alloc(ctx, &rec, (size_t)n * kRecBytes);
    if (e != cudaSuccess) return cuda_status(e);
    st = cr_synth_points_device(ctx, p, n, rec, hdr, stream);
    if (st == CR_OK) st = cr_morton_sort_device(ctx, rec, n, kRecBytes, hdr, stream);
    if (st == CR_OK)
        st = cr_encode_las_device(ctx, rec, n, kRecBytes, 2, hdr->scale, hdr->offset, hdr->min, 0, 0, db,
                                  lo, md, hi, rgba, stream);
    if (st == CR_OK) st = cuda_status(cudaStreamSynchronize((cudaStream_t)stream));
    cudaFree(rec);
    if (st == CR_OK) st = cr_cloud_set_files(ctx, cloud, hdr->min);
    return st;
}

cr_status cr_synth_uniform_host(uint64_t seed, int64_t n, float size, cr_vertex* out) {
    if (n < 0 || (n > 0 && !out)) return CR_ERR_INVALID_ARG;
    parallel_for(n, [&](int64_t a, int64_t b) {
        for (int64_t i = a; i < b; i++) out[i] = uniform_vertex(seed, (uint64_t)i, size);
    });
    return CR_OK;
}

cr_status cr_synth_uniform_device(cr_ctx* ctx, uint64_t seed, int64_t n, float size, cr_vertex* d_out,
                                  void* stream) {
    if (!ctx || n < 0 || (n > 0 && !d_out)) return CR_ERR_INVALID_ARG;
    if (n == 0) return CR_OK;
    k_uniform<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(seed, n, size, d_out);
    return cuda_status(cudaGetLastError());
}

}  // extern "C"
