// rrb_fills.cu — the reference's two GPU coverage operators behind their own
// parameter layouts: record_aa_fill (64-sample Halton-jittered coverage) and
// record_tile_fill (analytic signed-area coverage over 16x16 tiles), the
// GpuBackend entry points of crates/gpu/src/backend/mod.rs with AaFillParams /
// TileFillParams (backend/params.rs:90-103,170-185). Both write a u8 coverage
// buffer of width x height; neither composites.
//
// aa_fill. The reference launches one 64-thread block per pixel and tests
// every segment at every sample: O(pixels x 64 x segments). Here a CTA owns a
// band of 4 pixel rows and a thread one of its sample lines: all 64 samples of
// a pixel row share one y per sample index, so a line's crossings (x and
// winding sign) are found once, each as the number of pixels whose sample lies
// at or left of it; sorted, they give the runs of pixels inside, added up in
// a difference array per row. The set of crossings that a sample counts is
// that of the per-sample test, so the result is bit-identical to aa_fill_cpu
// (crates/gpu/src/fill.rs:346-421): IEEE division and the fma of its mul_add,
// evaluated once per (line, segment) instead of per pixel.
//
// tile_fill. Same decomposition as the reference (one 16x16 tile per CTA,
// one pixel per thread), with the tile's records staged through shared
// memory 256 at a time and every operation of tile_fill.cu rounded on its
// own (products via __fmul_rn so that none is contracted into an fma).
// A tile whose [start, start + count) runs past the records buffer is
// treated as empty instead of being read out of bounds.
//
// record_tile_fill_segs takes the same segments as aa_fill: where that is the
// faster way (tile_scan_pays by the sizes, tile_look by the contents) they go
// straight to coverage (k_tile_fill_segs); otherwise the records are built on the
// device (build_tile_records, fill.rs:82-264: count, write in segment order,
// stable radix sort by tile key, per-tile ranges by binary search), then run
// tile_fill. Neither builds or uploads records on the host.

#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>

#include "../../include/rrb.h"
#include "rrb_device_scope.h"

int rrb_ctx_device(const rrb_ctx* c);
bool rrb_ctx_page_open(const rrb_ctx* c);
int rrb_ctx_fail(rrb_ctx* c, int code, const char* msg);
int rrb_ctx_sm_count(const rrb_ctx* c);
int rrb_ctx_fill_scratch(rrb_ctx* c, int k, size_t bytes, void** out);
int rrb_ctx_read(rrb_ctx* c, const void* dev, size_t bytes, void* out);

namespace {

// ---- sample offsets ----------------------------------------------------------
// x: Halton base 2 of n = 1..64 (exact binary fractions). y: Halton base 3 of
// n = 1..64 as the reference writes it, rounded to 6 decimals, then to f32.
struct AaJitter {
    float x[64];
    float y[64];
};

double radical_inverse(uint32_t n, uint32_t base) {
    const double inv = 1.0 / base;
    double f = inv, r = 0.0;
    while (n) {
        r += f * static_cast<double>(n % base);
        n /= base;
        f *= inv;
    }
    return r;
}

const AaJitter& jitter() {
    static const AaJitter j = [] {
        AaJitter t;
        for (uint32_t i = 0; i < 64; ++i) {
            t.x[i] = static_cast<float>(radical_inverse(i + 1, 2));
            t.y[i] = static_cast<float>(std::nearbyint(radical_inverse(i + 1, 3) * 1e6) / 1e6);
        }
        return t;
    }();
    return j;
}

// The same offsets in ascending order of y: the kernel's sample lines. Hits
// are a sum over the 64 samples, so their order is free.
const AaJitter& jitter_by_y() {
    static const AaJitter j = [] {
        const AaJitter& a = jitter();
        int at[64];
        for (int i = 0; i < 64; ++i) at[i] = i;
        std::sort(at, at + 64, [&](int p, int q) { return a.y[p] < a.y[q]; });
        AaJitter t;
        for (int i = 0; i < 64; ++i) {
            t.x[i] = a.x[at[i]];
            t.y[i] = a.y[at[i]];
        }
        return t;
    }();
    return j;
}

// ---- aa_fill -------------------------------------------------------------------
// A CTA owns AA_ROWS pixel rows x up to AA_CW columns, 64 sample lines a row.
// The row's coverage is a sum of 64 step functions of the pixel, one per
// sample line, so nothing is evaluated per pixel and sample: a crossing at x
// with winding sign d counts for the pixels whose sample lies at or left of
// x, a prefix [0, p) of the row (sample x grows with the pixel), and p is
// found once per crossing. Three phases, each over all threads:
//   tasks: (segment, row, quarter of the row's lines in order of y) triples
//     that overlap; a thread takes one and finds its crossings on 16 lines;
//   lines: a thread takes an eighth of a line (the winding right of it comes
//     from the sums of the parts there), sorts its few crossings by p, walks
//     them from the right and adds +1 / -1 to the row's difference array at
//     both ends of each run of pixels inside;
//   rows: a warp's prefix sum over the differences gives the hits.
// Work per row: 64 x crossings + width, instead of 64 x width x
// log(crossings). Crossings right of the chunk only shift its winding, those
// left of it count for no pixel: neither is stored.
// Two CTAs an SM: AaShared is 81,184 bytes (three, which 40 registers with 28
// bytes of spills were compiled for, never fitted: calls 41.9 -> 41.1 and 50.8 ->
// 49.0 us).
// Measured: 48 glyph outlines (13,844 segments) in a 1,024 x 1,024 window 616
// -> 36 us; 6 outlines (1,344 segments) in 2,047 x 2,050, even-odd, 960 -> 44
// us (1 byte a pixel is 95 GB/s there). What is left is latency and barriers
// between short phases (a sixth to a third of the issue slots used). With a
// thread per line sorting up to 64 crossings, 70 and 46; with a warp per line
// and a bitonic network, 54 and 93.
constexpr int AA_ROWS = 4;                 // pixel rows per CTA
constexpr int AA_LINES = AA_ROWS * 64;     // sample lines per CTA
constexpr int AA_NT = 512;                 // threads per CTA
constexpr int AA_CW = 1024;                // columns per chunk
constexpr int AA_SEG_CAP = 448;            // band segments kept in shared memory
constexpr int AA_TASKS = 16 * AA_SEG_CAP;  // (segment, row, quarter) of each
constexpr int AA_PARTS = 8;                // column parts of a chunk, a list of crossings each
constexpr int AA_K = 16;                   // crossings per line and part kept in shared memory
constexpr int AA_BCW = 32;                 // columns per bucket sub-chunk (lines of more crossings)
constexpr int AA_DENSE = 4 * AA_K;         // crossings of a part that an eighth of its columns is not expected to hold
static_assert(AA_PARTS * AA_K == sizeof(int) * AA_BCW, "the buckets take the lists' place");
static_assert(AA_NT / 32 == 4 * AA_ROWS, "a warp per quarter row");
static_assert(AA_CW / AA_PARTS <= 128 && 2 * AA_TASKS <= 65536, "list entries in 8 bits, tasks in 16");

struct AaShared {
    float4 seg[AA_SEG_CAP];                        // oriented: y <= w
    int diff[AA_ROWS][AA_CW];
    union {
        uint8_t list[AA_PARTS][AA_K][AA_LINES];    // 2 (p mod the part's width) + (d > 0)
        int bucket[AA_BCW][AA_LINES];              // winding change at pixel p
    };
    uint32_t cnt[AA_PARTS][AA_LINES];              // crossings of a part (low half), sum of their signs (high)
    int wind[AA_LINES];                            // winding of the chunk's last pixels
    uint16_t task[AA_TASKS];                       // (segment << 4 | row << 2 | quarter) << 1 | (d > 0)
    float sy[AA_LINES], jx[64];
    uint32_t n_seg, n_task, over;
    uint32_t plan, plan_c;  // see k_aa_fill
};

static_assert(2 * (sizeof(AaShared) + 1024) <= 228 * 1024, "two CTAs an SM");

// Sample x of pixel px for sample offset jx, rounded as aa_fill_cpu does.
__host__ __device__ __forceinline__ float aa_sample_x(uint32_t px, float jx) {
    return (static_cast<float>(px) + 0.5f + jx) - 0.5f;
}

// The number of pixels of [c, c + cw) whose sample lies at or left of xi (the
// pixels the crossing counts for): a guess from the real sum, then exact steps
// over the rounded sample positions, which never decrease with the pixel.
__host__ __device__ __forceinline__ uint32_t aa_pixels_left(float xi, float jx, uint32_t c, uint32_t cw) {
    const float g = fminf(fmaxf(xi - jx - static_cast<float>(c), -4.0f), static_cast<float>(cw) + 4.0f);
    const int guess = static_cast<int>(floorf(g)) + 1;
    uint32_t p = guess < 0 ? 0u : (static_cast<uint32_t>(guess) > cw ? cw : static_cast<uint32_t>(guess));
    while (p < cw && aa_sample_x(c + p, jx) <= xi) ++p;
    while (p > 0 && aa_sample_x(c + p - 1, jx) > xi) --p;
    return p;
}

__global__ void __launch_bounds__(AA_NT, 2) k_aa_fill(const float4* __restrict__ segs, uint32_t n_segs,
                                                      uint32_t width, uint32_t height, int eo,
                                                      const __grid_constant__ AaJitter J,
                                                      uint8_t* __restrict__ coverage) {
    extern __shared__ __align__(16) unsigned char aa_smem[];
    AaShared& S = *reinterpret_cast<AaShared*>(aa_smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid < 64) S.jx[tid] = J.x[tid];
    const uint32_t bands = (height + AA_ROWS - 1) / AA_ROWS, chunks = (width + AA_CW - 1) / AA_CW;
    for (uint64_t item = blockIdx.x; item < static_cast<uint64_t>(bands) * chunks; item += gridDim.x) {
        const uint32_t r0 = static_cast<uint32_t>(item / chunks) * AA_ROWS, r1 = min(height, r0 + AA_ROWS) - 1;
        const uint32_t c0 = static_cast<uint32_t>(item % chunks) * AA_CW;
        const uint32_t c1 = width - c0 < AA_CW ? width : c0 + AA_CW;
        __syncthreads();  // the previous item's readers are done
        if (tid < AA_LINES) S.sy[tid] = (static_cast<float>(r0 + (tid >> 6)) + 0.5f + J.y[tid & 63]) - 0.5f;
        if (tid == 0) S.n_seg = S.n_task = S.plan = 0;
        __syncthreads();
        // The band's first and last sample lines: lines ascend in y (each
        // rounding step is monotone), so these are exact extremes.
        const float lo = S.sy[0], hi = S.sy[(r1 - r0) * 64 + 63];
        auto keep = [&](const float4& g) {
            // A crossing of aa_fill_cpu_sample (fill.rs:400-421) is y0 <= sy < y1 going
            // up (d = 1), y1 <= sy < y0 going down (d = -1, interpolated from the
            // other end): one form over the segment from its lower end.
            const bool up = g.y < g.w;
            const float4 s = up ? g : make_float4(g.z, g.w, g.x, g.y);
            if (!(s.y <= hi && s.w > lo)) return;
            uint32_t m = 0;  // quarters of rows with a line in [s.y, s.w)
            for (uint32_t q = 0; q < 4 * (r1 - r0 + 1); ++q)
                if (s.y <= S.sy[16 * q + 15] && s.w > S.sy[16 * q]) m |= 1u << q;
            const uint32_t at = atomicAdd(&S.n_seg, 1u);
            if (at >= AA_SEG_CAP) return;
            S.seg[at] = s;
            uint32_t t = atomicAdd(&S.n_task, static_cast<uint32_t>(__popc(m)));
            while (m) {
                S.task[t++] = static_cast<uint16_t>((at << 4 | static_cast<uint32_t>(__ffs(m) - 1)) << 1 | (up ? 1u : 0u));
                m &= m - 1;
            }
        };
        // Segments [b, e): the y of eight per thread in flight, then the few that stay.
        auto scan = [&](uint32_t b, uint32_t e) {
            for (uint32_t k0 = b + tid; k0 < e; k0 += 8 * AA_NT) {
                uint32_t m = 0;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t k = k0 + u * AA_NT;
                    float y0 = INFINITY, y1 = INFINITY;
                    if (k < e) {
                        y0 = segs[k].y;
                        y1 = segs[k].w;
                    }
                    if (fminf(y0, y1) <= hi && fmaxf(y0, y1) > lo) m |= 1u << u;
                }
                for (; m; m &= m - 1) keep(segs[k0 + (__ffs(m) - 1) * AA_NT]);
            }
        };
        // The band's segments, once for every sub-chunk when they fit.
        scan(0, n_segs);
        __syncthreads();
        const uint32_t n_band = S.n_seg;
        // Parts with a line of more crossings than a list holds are done again by
        // themselves, in parts of an eighth of their columns, and by pixel buckets
        // where that is too many still (or far too many at once: dense). The
        // columns between them stay whole. Buckets for all columns from the
        // first such line on (32 gathers of a 1,024-column chunk) took 234 us
        // for 48 outlines (15,897 segments) at the left edge of 1,024 x 1,024;
        // this way 44.
        // S.plan: masks of such parts (bits 0-7) and of the dense ones (8-15) and
        // log2 of their columns (16 on); S.plan_c: where the first part begins.
        auto inside = [eo](int wind) { return eo ? (wind & 1) != 0 : wind != 0; };
        for (uint32_t c = c0; c < c1;) {
            uint32_t cw = c1 - c;
            bool buckets = false;
            if (S.plan) {
                const uint32_t mps = S.plan >> 16, part = (c - S.plan_c) >> mps, rest = (S.plan & 0xffu) >> part;
                buckets = (S.plan >> (8 + part)) & 1u;
                if (buckets) cw = min(min(cw, static_cast<uint32_t>(AA_BCW)), S.plan_c + ((part + 1) << mps) - c);
                else if (rest) cw = min(cw, max(static_cast<uint32_t>(__ffs(rest)) - 1u, 1u) << mps);
            }
            for (uint32_t i = tid; i < AA_ROWS * AA_CW / 4; i += AA_NT)
                if (4 * i % AA_CW < cw) reinterpret_cast<int4*>(&S.diff[0][0])[i] = make_int4(0, 0, 0, 0);
            if (buckets)
                for (uint32_t i = tid; i < cw * AA_LINES; i += AA_NT) (&S.bucket[0][0])[i] = 0;
            for (uint32_t i = tid; i < AA_PARTS * AA_LINES; i += AA_NT) (&S.cnt[0][0])[i] = 0;
            if (tid < AA_LINES) S.wind[tid] = 0;
            // Parts of 2^ps columns: as few as hold the chunk in AA_PARTS of them.
            uint32_t ps = 0;
            while ((AA_PARTS << ps) < cw) ++ps;
            if (tid == 0) S.over = 0;
            auto gather = [&]() {
                // Four threads a task, four lines each: a thread's chains overlap.
                for (uint32_t t = tid; t < 4 * S.n_task; t += AA_NT) {
                    const uint32_t k = S.task[t >> 2];
                    const uint32_t l0 = 16 * ((k >> 1) & 15) + 4 * (t & 3);
                    const int d = (k & 1) ? 1 : -1;
                    const float4 s = S.seg[k >> 5];
                    const float dy = s.w - s.y, dx = s.z - s.x;
                    // p is the floor of xi - jx - c plus one unless that is within
                    // rounding of a whole number, so a reciprocal in place of the
                    // division does for most: its error and that of the samples'
                    // positions are under 2^-20 of the magnitudes in eps. Nearer
                    // than that (or not finite) p comes from the exact crossing.
                    const float inv = dy < 1e30f ? __frcp_rn(dy) : __int_as_float(0x7fc00000);
                    const float eps = (fabsf(dx) + fabsf(s.x) + static_cast<float>(c + cw) + 4.0f) * 0x1p-20f;
                    uint32_t ln[4], p[4], at[4];
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u) {
                        ln[u] = l0 + ((u + (t >> 2)) & 3);  // lanes of one quarter start apart
                        const float sy = S.sy[ln[u]], jx = S.jx[ln[u] & 63];
                        const float g = (fmaf((sy - s.y) * inv, dx, s.x) - jx) - static_cast<float>(c);
                        const float fl = floorf(g), f = g - fl;
                        p[u] = fl < 0.0f ? 0u : (fl >= static_cast<float>(cw) ? cw : static_cast<uint32_t>(fl) + 1u);
                        const bool on = s.y <= sy && sy < s.w;
                        if (on && !(f > eps && f < 1.0f - eps)) {
                            const float xi = fmaf((sy - s.y) / dy, dx, s.x);
                            // A NaN x never passes `xi >= sx`.
                            p[u] = isnan(xi) ? 0u : aa_pixels_left(xi, jx, c, cw);
                        }
                        if (!on) p[u] = 0;
                    }
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u) {
                        at[u] = AA_K;
                        if (p[u] == cw) atomicAdd(&S.wind[ln[u]], d);
                        else if (p[u] > 0 && buckets) atomicAdd(&S.bucket[p[u]][ln[u]], d);
                        else if (p[u] > 0) at[u] = atomicAdd(&S.cnt[p[u] >> ps][ln[u]], (static_cast<uint32_t>(d) << 16) + 1u) & 0xffffu;
                    }
                    if (!buckets) {
#pragma unroll
                        for (uint32_t u = 0; u < 4; ++u) {
                            if (p[u] == 0 || p[u] == cw) continue;
                            const uint32_t q = p[u] & ((1u << ps) - 1u);
                            if (at[u] < AA_K) S.list[p[u] >> ps][at[u]][ln[u]] = static_cast<uint8_t>(2 * q + (d > 0));
                            else atomicOr(&S.over, (at[u] < AA_DENSE ? 1u : 257u) << (p[u] >> ps));
                        }
                    }
                }
            };
            __syncthreads();
            if (n_band <= AA_SEG_CAP) {
                gather();
            } else {
                // More segments than the list holds: AA_SEG_CAP of them at a time.
                for (uint32_t b = 0; b < n_segs; b += AA_SEG_CAP) {
                    __syncthreads();
                    if (tid == 0) S.n_seg = S.n_task = 0;
                    __syncthreads();
                    const uint32_t e = n_segs - b < AA_SEG_CAP ? n_segs : b + AA_SEG_CAP;
                    scan(b, e);
                    __syncthreads();
                    gather();
                }
            }
            __syncthreads();
            if (S.over) {  // some line has more crossings than its list
                if (tid == 0) {
                    if (S.plan) {
                        S.plan |= 257u << ((c - S.plan_c) >> (S.plan >> 16));
                    } else {
                        S.plan = S.over | ps << 16;
                        S.plan_c = c;
                    }
                }
                __syncthreads();
                continue;
            }
            if (buckets) {
                if (tid < AA_LINES) {
                    int wind = S.wind[tid];
                    bool in = inside(wind);
                    for (uint32_t p = cw - 1; p > 0; --p) {
                        const int d = S.bucket[p][tid];
                        if (!d) continue;
                        wind += d;
                        const bool now = inside(wind);  // the state left of pixel p
                        if (now != in) atomicAdd(&S.diff[tid >> 6][p], now ? -1 : 1);
                        in = now;
                    }
                    if (in) atomicAdd(&S.diff[tid >> 6][0], 1);
                }
            } else {
                // A part of a line by a thread, from the right: its few
                // entries sorted descending, then walked.
                for (uint32_t i = tid; i < AA_PARTS * AA_LINES; i += AA_NT) {
                    const uint32_t part = i / AA_LINES, ln = i % AA_LINES;
                    const uint32_t n = S.cnt[part][ln] & 0xffffu;
                    if (n == 0 && part) continue;
                    int wind = S.wind[ln];
                    for (uint32_t q = part + 1; q < AA_PARTS; ++q) wind += static_cast<int16_t>(S.cnt[q][ln] >> 16);
                    uint8_t(*L)[AA_LINES] = S.list[part];
                    int* drow = S.diff[ln >> 6];
                    bool in = inside(wind);
                    for (uint32_t a = 1; a < n; ++a) {
                        const uint8_t v = L[a][ln];
                        uint32_t b = a;
                        while (b > 0) {
                            const uint8_t u = L[b - 1][ln];
                            if (u >= v) break;
                            L[b][ln] = u;
                            --b;
                        }
                        L[b][ln] = v;
                    }
                    for (uint32_t k = 0; k < n; ++k) {
                        const uint32_t v = L[k][ln];
                        wind += (v & 1u) ? 1 : -1;
                        const bool now = inside(wind);  // the state left of the entry's pixel
                        if (now != in) atomicAdd(&drow[(part << ps) + (v >> 1)], now ? -1 : 1);
                        in = now;
                    }
                    if (part == 0 && in) atomicAdd(&drow[0], 1);
                }
            }
            __syncthreads();
            // Hits of a quarter of a row by a warp, four pixels per lane and step.
            const uint32_t hr = w & (AA_ROWS - 1), quarter = ((cw + 511) / 512) * 128;
            const uint32_t b0 = (w / AA_ROWS) * quarter, b1 = min(cw, b0 + quarter);
            if (r0 + hr < height && b0 < b1) {
                const int* d = S.diff[hr];
                uint8_t* out = coverage + static_cast<size_t>(r0 + hr) * width + c;
                const bool words = (reinterpret_cast<uintptr_t>(out) & 3u) == 0;
                int carry = 0;  // the sum of the differences left of the quarter
                for (uint32_t i = 4 * lane; i < b0; i += 128) {
                    const int4 v = *reinterpret_cast<const int4*>(d + i);
                    carry += v.x + v.y + v.z + v.w;
                }
                for (int o = 16; o; o >>= 1) carry += __shfl_xor_sync(0xffffffffu, carry, o);
                for (uint32_t b = b0; b < b1; b += 128) {
                    const uint32_t i = b + 4 * lane;
                    int4 v = make_int4(0, 0, 0, 0);
                    if (i < cw) v = *reinterpret_cast<const int4*>(d + i);  // zero past cw up to a multiple of 4
                    v.y += v.x;
                    v.z += v.y;
                    v.w += v.z;
                    int incl = v.w;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, incl, o);
                        if (static_cast<int>(lane) >= o) incl += t;
                    }
                    const int before = carry + incl - v.w;
                    carry += __shfl_sync(0xffffffffu, incl, 31);
                    const uint32_t q[4] = {static_cast<uint32_t>(before + v.x), static_cast<uint32_t>(before + v.y),
                                           static_cast<uint32_t>(before + v.z), static_cast<uint32_t>(before + v.w)};
                    uint32_t packed = 0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) packed |= ((q[j] * 255u + 32u) >> 6) << (8 * j);
                    if (words && i + 4 <= cw) {
                        *reinterpret_cast<uint32_t*>(out + i) = packed;
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j)
                            if (i + j < cw) out[i + j] = static_cast<uint8_t>(packed >> (8 * j));
                    }
                }
            }
            __syncthreads();  // the next sub-chunk clears the differences
            c += cw;
        }
    }
}

// ---- tile_fill -----------------------------------------------------------------
constexpr uint32_t TILE = 16;
constexpr int TF_THREADS = TILE * TILE;

struct __align__(16) TileRec {
    uint32_t key;
    float x_enter, dxdy, y0_tile, y1_tile, sign;
    uint32_t pad, pad2;
};
static_assert(sizeof(TileRec) == 32 && sizeof(TileRec) == sizeof(rrb_tile_record), "TileRecord is 32 bytes");

// segment_pixel_area of tile_fill.cu:64-115, every operation rounded on its own.
__device__ __forceinline__ float segment_pixel_area(float x_enter, float dxdy, float iy0, float iy1, float sign,
                                                    float px) {
    const float y_len = iy1 - iy0;
    if (y_len <= 0.0f) return 0.0f;
    const float x0 = x_enter;
    const float x1 = __fadd_rn(x_enter, __fmul_rn(dxdy, y_len));
    const float xl = fminf(x0, x1), xr = fmaxf(x0, x1);
    float cover;
    if (xr <= px) {
        cover = 0.0f;
    } else if (xl >= px + 1.0f) {
        cover = y_len;
    } else {
        const float dx = xr - xl;
        if (dx < 1e-6f) {
            const float xmid = __fmul_rn(0.5f, x0 + x1);
            cover = (xmid >= px + 0.5f) ? y_len : 0.0f;
        } else {
            const float left = fmaxf(xl, px);
            const float right = fminf(xr, px + 1.0f);
            const float yf_left = __fmul_rn(__fdiv_rn(left - xl, dx), y_len);
            const float yf_right = __fmul_rn(__fdiv_rn(right - xl, dx), y_len);
            const float above = y_len - yf_right;
            cover = (yf_right - yf_left) + above;
        }
    }
    return __fmul_rn(sign, cover);
}

// Rust / PTX float -> int conversion: truncate, saturate, NaN -> 0.
__device__ __forceinline__ int32_t sat_i32(float v) {
    if (isnan(v)) return 0;
    if (v <= -2147483648.0f) return INT32_MIN;
    if (v >= 2147483648.0f) return INT32_MAX;
    return static_cast<int32_t>(v);
}

// ---- tile records on the device (build_tile_records, fill.rs:82-264) ----------
__device__ __forceinline__ uint32_t sat_u32(float v) {
    if (isnan(v) || v <= 0.0f) return 0;
    if (v >= 4294967296.0f) return UINT32_MAX;
    return static_cast<uint32_t>(v);
}

// A segment as build_tile_records sees it: downward, with the slope and its
// clip to the raster's rows; on == false where it gives no records.
struct TileSeg {
    float sx0, sy0, dxdy, sign, ey0, ey1;
    uint32_t ty0, ty_end;
    bool on;
};
__device__ __forceinline__ TileSeg tile_segment(const float4 sg, uint32_t height, uint32_t grid_h) {
    TileSeg t;
    t.on = false;
    float sx0 = sg.x, sy0 = sg.y, sx1 = sg.z, sy1 = sg.w;
    const float dy = fabsf(sy1 - sy0);
    if (!isfinite(dy) || dy < 1e-6f || !isfinite(sx0) || !isfinite(sx1)) return t;
    t.sign = 1.0f;
    if (sy0 > sy1) {
        float v = sx0;
        sx0 = sx1;
        sx1 = v;
        v = sy0;
        sy0 = sy1;
        sy1 = v;
        t.sign = -1.0f;
    }
    t.sx0 = sx0;
    t.sy0 = sy0;
    t.dxdy = __fdiv_rn(sx1 - sx0, sy1 - sy0);
    t.ey0 = fmaxf(sy0, 0.0f);
    t.ey1 = fminf(sy1, static_cast<float>(height));
    if (t.ey0 >= t.ey1) return t;
    const float th = static_cast<float>(TILE);
    t.ty0 = sat_u32(floorf(__fdiv_rn(t.ey0, th)));
    t.ty_end = min(sat_u32(floorf(__fdiv_rn(fmaxf(t.ey1 - 1e-6f, 0.0f), th))), grid_h - 1);
    t.on = true;
    return t;
}

// Its part in tile row ty: the record of tile tx in [tx0, tx1] has x_enter =
// x - 16 tx; false where the row has none.
struct TileRow {
    float x, y0, y1;
    uint32_t tx0, tx1;
};
__device__ __forceinline__ bool tile_row(const TileSeg& t, uint32_t ty, uint32_t grid_w, TileRow& r) {
    const float tw = static_cast<float>(TILE);
    const float tile_top = static_cast<float>(ty * TILE);
    const float tile_bot = tile_top + static_cast<float>(TILE);
    r.y0 = fmaxf(t.ey0, tile_top) - tile_top;
    r.y1 = fminf(t.ey1, tile_bot) - tile_top;
    if (r.y0 >= r.y1) return false;
    r.x = fmaf(t.dxdy, fmaxf(t.ey0, tile_top) - t.sy0, t.sx0);
    const float x_at_exit = fmaf(t.dxdy, r.y1 - r.y0, r.x);
    const int32_t tx0_i = sat_i32(floorf(__fdiv_rn(fminf(r.x, x_at_exit), tw)));
    const int32_t tx1_i = sat_i32(floorf(__fdiv_rn(fmaxf(r.x, x_at_exit), tw)));
    if (tx1_i < 0) return false;
    r.tx0 = static_cast<uint32_t>(max(tx0_i, 0));
    r.tx1 = min(static_cast<uint32_t>(tx1_i), grid_w - 1);
    return r.tx0 <= r.tx1;
}

// Records of a segment in the reference's order (tile rows, then columns);
// with out == nullptr only counts them.
__device__ uint32_t segment_records(const float4 sg, uint32_t height, uint32_t grid_w, uint32_t grid_h, TileRec* out,
                                    uint32_t* keys) {
    const TileSeg t = tile_segment(sg, height, grid_h);
    if (!t.on) return 0;
    uint32_t n = 0;
    for (uint64_t ty = t.ty0; ty <= t.ty_end; ++ty) {
        TileRow w;
        if (!tile_row(t, static_cast<uint32_t>(ty), grid_w, w)) continue;
        if (out) {
            for (uint32_t tx = w.tx0; tx <= w.tx1; ++tx) {
                TileRec r;
                r.key = (static_cast<uint32_t>(ty) << 16) | tx;
                r.x_enter = w.x - static_cast<float>(tx * TILE);
                r.dxdy = t.dxdy;
                r.y0_tile = w.y0;
                r.y1_tile = w.y1;
                r.sign = t.sign;
                r.pad = r.pad2 = 0;
                out[n + (tx - w.tx0)] = r;
                keys[n + (tx - w.tx0)] = r.key;
            }
        }
        n += w.tx1 - w.tx0 + 1;
    }
    return n;
}

// Area that a record adds to a pixel of its tile (tile_fill.cu:117-150); false where it adds none.
__device__ __forceinline__ bool record_area(float x_enter, float dxdy, float y0, float y1, float sign, float px_f,
                                            float py_f, float& a) {
    const float iy0 = fmaxf(y0, py_f);
    const float iy1 = fminf(y1, py_f + 1.0f);
    const float x_at_iy0 = __fadd_rn(x_enter, __fmul_rn(dxdy, iy0 - y0));
    a = segment_pixel_area(x_at_iy0, dxdy, iy0, iy1, sign, px_f);
    return iy0 < iy1;
}

__device__ __forceinline__ uint8_t area_coverage(float area, int eo) {
    int32_t cov;
    if (eo) {
        float a = fabsf(area);
        a = a - floorf(a);
        if (a > 0.5f) a = 1.0f - a;
        cov = sat_i32(__fmul_rn(__fmul_rn(a, 2.0f), 255.5f));
    } else {
        cov = sat_i32(__fmul_rn(fminf(fabsf(area), 1.0f), 255.5f));
    }
    return static_cast<uint8_t>(min(cov, 255));
}

__global__ void __launch_bounds__(TF_THREADS) k_tile_fill(const TileRec* __restrict__ recs, uint64_t n_recs,
                                                          const uint32_t* __restrict__ starts,
                                                          const uint32_t* __restrict__ counts, uint32_t grid_w,
                                                          uint32_t grid_h, uint32_t width, uint32_t height, int eo,
                                                          uint8_t* __restrict__ coverage) {
    __shared__ TileRec srec[TF_THREADS];
    const uint32_t tid = threadIdx.x, pxl = tid % TILE, pyl = tid / TILE;
    const float px_f = static_cast<float>(pxl), py_f = static_cast<float>(pyl);
    const uint64_t n_tiles = static_cast<uint64_t>(grid_w) * grid_h;
    for (uint64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t tx = static_cast<uint32_t>(tile % grid_w), ty = static_cast<uint32_t>(tile / grid_w);
        const uint64_t start = starts[tile];
        uint64_t cnt = counts[tile];
        if (start + cnt > n_recs) cnt = 0;
        float area = 0.0f;
        for (uint64_t base = 0; base < cnt; base += TF_THREADS) {
            const uint32_t m = cnt - base < TF_THREADS ? static_cast<uint32_t>(cnt - base) : TF_THREADS;
            __syncthreads();
            if (tid < m) srec[tid] = recs[start + base + tid];
            __syncthreads();
            for (uint32_t r = 0; r < m; ++r) {
                const TileRec rec = srec[r];
                float a;
                if (record_area(rec.x_enter, rec.dxdy, rec.y0_tile, rec.y1_tile, rec.sign, px_f, py_f, a))
                    area = __fadd_rn(area, a);
            }
        }
        const uint32_t px = tx * TILE + pxl, py = ty * TILE + pyl;
        if (px < width && py < height) coverage[static_cast<size_t>(py) * width + px] = area_coverage(area, eo);
    }
}

// tile_fill straight from the segments: a segment gives a tile at most one
// record, so a tile's records in their sorted order are its segments in index
// order, and the sort only sorts what an ordered scan finds in order. A CTA
// owns a row of up to TSF_TILES tiles: 1,024 segments at a time, those that reach the tile row are packed in order
// into shared memory (a scan of the warps' counts) and become its records,
// and each warp walks the records that reach its two pixel rows, 32 at a time
// by ballot, a pixel a lane.
// Against count, scan, write, radix sort, gather, ranges and fill (12
// launches, most of them on two or fewer CTAs, and a wait in the middle), whole
// calls: 14,752 segments in 1,024 x 1,024 189 -> 64 us (the kernel 50), in
// 200 x 200 249 -> 99, 384 in 64 x 64 116 -> 50. What bounds it is the scan of
// all segments by every CTA (20,000 cycles of the 14,752) and the chain of the
// areas in the busiest tile row.
constexpr int TSF_NT = 256, TSF_TILES = 16, TSF_CAP = 1024;
static_assert(TSF_NT == TF_THREADS && TSF_CAP == 4 * TSF_NT, "a pixel of a tile per thread, four segments at a time");
struct TsfWork {
    unsigned long long records;  // of all tile rows
    uint32_t leave, pad;         // the sorted records are the faster way (tile_look): what is written does not count
};

struct __align__(8) RowPart {
    float x, dxdy, y0, y1;  // before convert(): the segment
    float sign;
    uint32_t tx;            // first tile | last tile << 16
};

// Whether the contents are for the scan. Where a tile row, or a part of one, has
// many records the chain of its CTA is the scan's time, and many records in all cost
// it more of the whole chip than the sort. So a sample of the segments is added up by
// the CTAs that they would load: tile rows x groups of tiles in `cells`, with the
// rows' listed segments behind them.
// In ns, fitted to 792 contents of 400 to 32,000 segments (short, long, upright, flat,
// crowded in rows, in columns, in both) in windows from 64 x 64 to 5,000 x 6,000:
//   scan: 320 for a hit of the busiest warp's two pixel rows and 176 for each further
//   tile of it, 7 for a listed segment; or 0.88 for each record of all;
//   sorted records: sort_call (what the call costs more than the scan's) and 46,000
//   beyond 5,000 records, 2 a segment, 0.45 a tile, 920 for each record of the mean
//   segment (a thread writes them one after another), 0.8 of the scan's chain in the
//   fullest tile; or 0.6 for each record of all.
// The records are asked for beyond `margin` times their estimate.
// Whole calls, scan / sorted records / as chosen, in us: 917 x 1,341, 4,096 segments
// around 14 pixel rows 521 / 151 / 201, 2,000 269 / 131 / 179; 3,000 x 100, a tenth of
// both sides full, 6,000 741 / 196 / 215, 12,000 1,394 / 341 / 332; 1,024 x 1,024, long
// ones, 4,096 447 / 292 / 359, 8,192 854 / 433 / 467, 32,768 3,311 / 1,139 / 1,165; all
// in 28 pixel rows of it, 9,000 356 / 142 / 165; short ones all over it, 14,752 50 /
// 135 / 54, 3,000 32 / 77 / 32.
constexpr uint32_t TL_MIN = 512;     // segments from which it is worth asking (511 in 14 pixel rows: 85 / 69)
constexpr uint32_t TL_CTAS = 1000;   // CTAs of a scan up to which it is asked beside it
constexpr uint32_t TL_ROWS = 6;      // tile rows looked at per segment
constexpr uint32_t TL_CELLS = TSF_TILES * TSF_NT;
template <uint32_t NT, uint32_t PICKS>  // threads of the block, segments looked at
__device__ __forceinline__ void tile_look(const float4* __restrict__ segs, uint32_t n_segs, uint32_t grid_w,
                                          uint32_t grid_h, uint32_t height, uint32_t group_tiles, uint32_t* cells,
                                          float sort_call, float margin, TsfWork* __restrict__ work) {
    __shared__ float all_of[NT / 32];
    __shared__ uint32_t peaks[NT / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t groups = (grid_w + group_tiles - 1) / group_tiles;
    // Large windows: 2^rs rows and 2^gs groups a cell, and their mean.
    uint32_t rs = 0, gs = 0;
    while (static_cast<uint64_t>(((groups - 1) >> gs) + 2) * (((grid_h - 1) >> rs) + 1) > TL_CELLS) {
        if ((grid_h >> rs) >= (groups >> gs)) ++rs;
        else ++gs;
    }
    const uint32_t cols = ((groups - 1) >> gs) + 2;  // the last: listed segments
    const uint32_t wide = group_tiles << gs;
    const uint32_t n_cells = cols * (((grid_h - 1) >> rs) + 1);
    for (uint32_t i = tid; i < n_cells; i += NT) cells[i] = 0;
    __syncthreads();
    const uint32_t per = (n_segs + PICKS - 1) / PICKS, picks = n_segs / per;
    float recs = 0.0f;
    const float bottom = static_cast<float>(height);
#pragma unroll 1
    for (uint32_t i = tid; i < picks; i += NT) {
        // One out of `per` consecutive segments stands for them all.
        const uint32_t hash = i * 2654435761u;
        const float4 q = segs[i * per + __umulhi(hash, per)];
        const bool up = q.y > q.w;
        const float x0 = up ? q.z : q.x, y0 = up ? q.w : q.y;
        const float e0 = fmaxf(y0, 0.0f), e1 = fminf(up ? q.y : q.w, bottom);
        const float slope = __fdividef(q.z - q.x, q.w - q.y);
        if (!(e0 < e1) || !(fabsf(slope) < 1e30f)) continue;
        const uint32_t r0 = min(static_cast<uint32_t>(e0) / TILE, grid_h - 1);
        const uint32_t r1 = min(static_cast<uint32_t>(e1) / TILE, grid_h - 1);
        // One out of `step` rows, from a row of its own on: else those of long
        // segments that start in the same rows would meet in the same cells.
        const uint32_t step = (r1 - r0) / TL_ROWS + 1;
        for (uint32_t r = r0 + __umulhi(hash, step); r <= r1; r += step) {
            const float a = fmaxf(e0, static_cast<float>(r * TILE)), b = fminf(e1, static_cast<float>(r * TILE + TILE));
            if (!(a < b)) continue;
            uint32_t* row = cells + (r >> rs) * cols;
            atomicAdd(&row[cols - 1], step);
            const float xa = x0 + slope * (a - y0), xb = x0 + slope * (b - y0);
            const float lo = fminf(xa, xb) / TILE, hi = fmaxf(xa, xb) / TILE;
            if (!(hi >= 0.0f && lo < static_cast<float>(grid_w))) continue;
            const uint32_t ta = static_cast<uint32_t>(fmaxf(lo, 0.0f));
            const uint32_t tb = static_cast<uint32_t>(fminf(hi, static_cast<float>(grid_w - 1)));
            recs += static_cast<float>((tb - ta + 1) * step);
            // Warps of the busiest row among those that it touches, in eighths.
            const uint32_t pairs = static_cast<uint32_t>(ceilf(0.5f * b)) - static_cast<uint32_t>(0.5f * a);
            const uint32_t load = step * min(8u, (8 * pairs + 2) / 5);
            for (uint32_t g = ta / wide; g <= tb / wide; ++g) {
                const uint32_t more = min(tb, g * wide + wide - 1) - max(ta, g * wide);
                atomicAdd(&row[g], load * (20 + 11 * more));  // of 16 ns
            }
        }
    }
    __syncthreads();
    uint32_t peak = 0;
    for (uint32_t i = tid; i < n_cells; i += NT)
        if (i % cols != cols - 1) peak = max(peak, 2 * cells[i] + 7 * cells[i - i % cols + cols - 1]);
    peak = __reduce_max_sync(0xffffffffu, peak);
    for (int o = 16; o; o >>= 1) recs += __shfl_xor_sync(0xffffffffu, recs, o);
    if (lane == 0) {
        all_of[w] = recs;
        peaks[w] = peak;
    }
    __syncthreads();
    if (tid) return;
    for (uint32_t k = 1; k < NT / 32; ++k) {
        recs += all_of[k];
        peak = max(peak, peaks[k]);
    }
    const float n = static_cast<float>(n_segs), of = n / static_cast<float>(picks);
    const float chain = of * static_cast<float>(peak) / static_cast<float>(1u << (rs + gs)), all = of * recs;
    const float scan = fmaxf(chain, 0.88f * all);
    const float tiles = static_cast<float>(grid_w) * static_cast<float>(grid_h);
    const float sorted = sort_call + (all > 5000.0f ? 4.6e4f : 0.0f) + 2.0f * n + 0.45f * tiles + 920.0f * all / n +
                         fmaxf(0.8f * chain / static_cast<float>(wide), 0.6f * all);
    if (scan > margin * sorted) *const_cast<volatile uint32_t*>(&work->leave) = 1;
}

// The look by itself, before the scan.
constexpr uint32_t TL_THREADS = 512;  // a segment each
__global__ void __launch_bounds__(TL_THREADS) k_tile_look(const float4* __restrict__ segs, uint32_t n_segs, uint32_t grid_w,
                                                      uint32_t grid_h, uint32_t height, uint32_t group_tiles,
                                                      TsfWork* __restrict__ work) {
    __shared__ uint32_t cells[TL_CELLS];
    if (threadIdx.x == 0) *work = TsfWork{};
    tile_look<TL_THREADS, TL_THREADS>(segs, n_segs, grid_w, grid_h, height, group_tiles, cells, 5.5e4f, 1.1f, work);
}

// LOOK: block 0 looks, the others scan meanwhile.
template <bool LOOK>
__global__ void __launch_bounds__(TSF_NT, 3) k_tile_fill_segs(const float4* __restrict__ segs, uint32_t n_segs,
                                                              uint32_t grid_w, uint32_t grid_h, uint32_t width,
                                                              uint32_t height, int eo, uint8_t* __restrict__ coverage,
                                                              uint32_t group_tiles, TsfWork* __restrict__ work) {
    __shared__ RowPart part[TSF_CAP];
    __shared__ float area[TSF_TILES][TSF_NT];  // a warp's two pixel rows are its own
    if (LOOK && blockIdx.x == 0) {
        tile_look<TSF_NT, 4 * TSF_NT>(segs, n_segs, grid_w, grid_h, height, group_tiles,
                                      reinterpret_cast<uint32_t*>(&area[0][0]), 7.5e4f, 1.4f, work);
        return;
    }
    if (!LOOK && work && work->leave) return;  // as k_tile_look left it
    // LOOK: what block 0 has found by now.
    auto left = [&]() { return LOOK && *const_cast<const volatile uint32_t*>(&work->leave) != 0; };
    __shared__ uint32_t counts[4 * TSF_NT / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t groups = (grid_w + group_tiles - 1) / group_tiles;
    const uint32_t cta = blockIdx.x - (LOOK ? 1 : 0), ty = cta / groups, g = cta % groups;
    const uint32_t t0 = g * group_tiles, t1 = min(grid_w, t0 + group_tiles);  // tiles of this CTA
    const float px_f = static_cast<float>(tid % TILE), py_f = static_cast<float>(tid / TILE);
    const float wy0 = 2.0f * static_cast<float>(w), wy1 = wy0 + 2.0f;     // this warp's rows
#pragma unroll
    for (int k = 0; k < TSF_TILES; ++k) area[k][tid] = 0.0f;
    const float top = static_cast<float>(ty * TILE), bot = top + static_cast<float>(TILE);
    uint32_t n = 0;                   // parts in the list
    unsigned long long records = 0;   // of this tile row (counted by the first group)
    auto walk = [&]() {
        uint32_t since = 0;  // hits since the flag was last read
        for (uint32_t b = 0; b < n; b += 32) {
            const bool hit = b + lane < n && part[b + lane].y0 < wy1 && part[b + lane].y1 > wy0;
            uint32_t m = __ballot_sync(0xffffffffu, hit);
            if (LOOK && (since += __popc(m)) >= 32) {  // some 10 us
                if (__any_sync(0xffffffffu, left())) return;
                since = 0;
            }
            // Four records' areas at a time (their chains overlap), added in order.
            while (m) {
                float add[4];
                bool on[4];
                uint32_t at[4], t[4], e[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    on[k] = false;
                    t[k] = 1;
                    e[k] = 0;
                    if (!m) continue;
                    at[k] = b + __ffs(m) - 1;
                    m &= m - 1;
                    const RowPart r = part[at[k]];
                    t[k] = max(t0, r.tx & 0xffffu);
                    e[k] = min(t1 - 1, r.tx >> 16);
                    on[k] = record_area(r.x - static_cast<float>(t[k] * TILE), r.dxdy, r.y0, r.y1, r.sign, px_f, py_f, add[k]);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (on[k]) area[t[k] - t0][tid] = __fadd_rn(area[t[k] - t0][tid], add[k]);
                    for (uint32_t u = t[k] + 1; u <= e[k]; ++u) {  // the record's further tiles
                        const RowPart r = part[at[k]];
                        float a;
                        if (record_area(r.x - static_cast<float>(u * TILE), r.dxdy, r.y0, r.y1, r.sign, px_f, py_f, a))
                            area[u - t0][tid] = __fadd_rn(area[u - t0][tid], a);
                    }
                }
            }
        }
    };
    // The listed segments' parts in this tile row, a segment a thread: packed
    // first, so that no warp runs this for a lane or two. True where the sorted
    // records are asked for: the block leaves as one.
    auto convert = [&]() -> bool {
        const bool gone = tid == 0 && left();
        for (uint32_t i = tid; i < n; i += TSF_NT) {
            const RowPart s = part[i];
            RowPart r{0.0f, 0.0f, 1.0f, 0.0f, 0.0f, 0u};  // reaches no row
            const TileSeg t = tile_segment(make_float4(s.x, s.dxdy, s.y0, s.y1), height, grid_h);
            TileRow q;
            if (t.on && t.ty0 <= ty && ty <= t.ty_end && tile_row(t, ty, grid_w, q)) {
                records += q.tx1 - q.tx0 + 1;
                if (q.tx0 < t1 && q.tx1 >= t0) r = RowPart{q.x, t.dxdy, q.y0, q.y1, t.sign, q.tx0 | q.tx1 << 16};
            }
            part[i] = r;
        }
        return __syncthreads_or(gone);
    };
    for (uint32_t base = 0; base < n_segs; base += TSF_CAP) {
        float4 s[4];
        uint32_t m[4];  // segments base + 256 u + (this warp's 32) that reach the tile row
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t k = base + u * TSF_NT + tid;
            if (k < n_segs) s[u] = segs[k];
        }
        const bool gone = base == 0 && tid == 0 && left();  // with the loads above
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            // Off the tile row for certain (a NaN stays; convert() drops it).
            const bool off = base + u * TSF_NT + tid >= n_segs || fmaxf(s[u].y, s[u].w) < top ||
                             fminf(s[u].y, s[u].w) > bot;
            m[u] = __ballot_sync(0xffffffffu, !off);
            if (lane == 0) counts[u * (TSF_NT / 32) + w] = __popc(m[u]);
        }
        if (__syncthreads_or(gone)) return;
        const uint32_t mine_n = counts[lane];  // four steps x eight warps
        uint32_t incl = mine_n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (static_cast<int>(lane) >= o) incl += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        if (n + total > TSF_CAP) {  // the same for every thread
            if (convert()) return;
            walk();
            n = 0;
            __syncthreads();
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t at = n + __shfl_sync(0xffffffffu, incl - mine_n, u * (TSF_NT / 32) + w) +
                                __popc(m[u] & ((1u << lane) - 1u));
            if (m[u] >> lane & 1u) part[at] = RowPart{s[u].x, s[u].y, s[u].z, s[u].w, 0.0f, 0u};
        }
        n += total;
        __syncthreads();
    }
    if (convert()) return;
    walk();
    const uint32_t py = ty * TILE + tid / TILE;
    for (uint32_t t = t0; t < t1; ++t) {
        const uint32_t px = t * TILE + tid % TILE;
        if (px < width && py < height) coverage[static_cast<size_t>(py) * width + px] = area_coverage(area[t - t0][tid], eo);
    }
    if (g == 0 && work) {
        for (int o = 16; o; o >>= 1) records += __shfl_xor_sync(0xffffffffu, records, o);
        if (lane == 0 && records) atomicAdd(&work->records, records);
    }
}

__global__ void k_tile_count(const float4* __restrict__ segs, uint32_t n_segs, uint32_t height, uint32_t grid_w,
                             uint32_t grid_h, unsigned long long* __restrict__ counts) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_segs; k += gridDim.x * blockDim.x)
        counts[k] = segment_records(segs[k], height, grid_w, grid_h, nullptr, nullptr);
}

// Exclusive scan of n u64 counts in place (one CTA; the offsets of each
// segment's records in segment order); out[n] = total.
__global__ void __launch_bounds__(1024) k_scan_u64(unsigned long long* __restrict__ v, uint32_t n) {
    __shared__ unsigned long long part[1024];
    const uint32_t t = threadIdx.x, per = (n + 1023) / 1024;
    const uint32_t b = min(n, t * per), e = min(n, b + per);
    unsigned long long s = 0;
    for (uint32_t i = b; i < e; ++i) s += v[i];
    part[t] = s;
    __syncthreads();
    for (uint32_t o = 1; o < 1024; o <<= 1) {
        const unsigned long long x = t >= o ? part[t - o] : 0ull;
        __syncthreads();
        part[t] += x;
        __syncthreads();
    }
    unsigned long long run = part[t] - s;
    for (uint32_t i = b; i < e; ++i) {
        const unsigned long long c = v[i];
        v[i] = run;
        run += c;
    }
    if (t == 1023) v[n] = part[1023];
}

__global__ void k_tile_write(const float4* __restrict__ segs, uint32_t n_segs, uint32_t height, uint32_t grid_w,
                             uint32_t grid_h, const unsigned long long* __restrict__ off, TileRec* __restrict__ recs,
                             uint32_t* __restrict__ keys, uint32_t* __restrict__ idx) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_segs; k += gridDim.x * blockDim.x) {
        const unsigned long long o = off[k];
        const uint32_t n = segment_records(segs[k], height, grid_w, grid_h, recs + o, keys + o);
        for (uint32_t i = 0; i < n; ++i) idx[o + i] = static_cast<uint32_t>(o + i);
    }
}

// Sorted records and, per tile, the range of its key in the sorted keys.
__global__ void k_tile_gather(const TileRec* __restrict__ recs, const uint32_t* __restrict__ order, uint32_t n,
                              TileRec* __restrict__ sorted) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        sorted[i] = recs[order[i]];
}

__global__ void k_tile_ranges(const uint32_t* __restrict__ keys, uint32_t n, uint32_t grid_w, uint32_t grid_h,
                              uint32_t* __restrict__ starts, uint32_t* __restrict__ counts) {
    const uint64_t n_tiles = static_cast<uint64_t>(grid_w) * grid_h;
    for (uint64_t t = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; t < n_tiles;
         t += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t key = (static_cast<uint32_t>(t / grid_w) << 16) | static_cast<uint32_t>(t % grid_w);
        auto lower = [&](uint32_t k) {
            uint32_t a = 0, z = n;
            while (a < z) {
                const uint32_t m = (a + z) >> 1;
                if (keys[m] < k) a = m + 1;
                else z = m;
            }
            return a;
        };
        const uint32_t s = lower(key);
        starts[t] = s;
        counts[t] = lower(key + 1) - s;
    }
}

#define FILL_CUDA(ctx, call)                                                                             \
    do {                                                                                                 \
        cudaError_t e__ = (call);                                                                        \
        if (e__ != cudaSuccess) {                                                                        \
            cudaGetLastError();                                                                          \
            return rrb_ctx_fail(ctx, RRB_ERR_DEVICE, (std::string(#call ": ") + cudaGetErrorString(e__)).c_str()); \
        }                                                                                                \
    } while (0)

// Checks shared by the coverage operators; `dev` is the status of the
// caller's DeviceScope (the context's device made current for the call).
int begin(rrb_ctx* c, cudaError_t dev) {
    if (!rrb_ctx_page_open(c)) return rrb_ctx_fail(c, RRB_ERR_STATE, "record_* outside begin_page/submit_page");
    FILL_CUDA(c, dev);
    return RRB_OK;
}

int check_cov(rrb_ctx* c, const rrb_buf* cov, uint32_t w, uint32_t h) {
    if (!cov) return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "coverage buffer is null");
    if (static_cast<uint64_t>(w) * h > rrb_device_buffer_len(cov))
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "coverage buffer is smaller than width * height");
    return RRB_OK;
}

int check_segs(rrb_ctx* c, const rrb_buf* segs, uint32_t n) {
    if (n && !segs) return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "segs buffer is null");
    if (n && 16ull * n > rrb_device_buffer_len(segs))
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "segs buffer is smaller than 16 * n_segs bytes");
    if (n && (reinterpret_cast<uintptr_t>(rrb_device_ptr(segs)) & 15))
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "segs buffer is not 16-byte aligned");
    return RRB_OK;
}

// Whether every CTA scanning all segments beats sorting their records, from
// the sizes alone. The scan costs 2.1 ps per segment and CTA and 0.5 ns per
// tile, the sort some 100 us and 1 ns per tile. Whole calls of short segments
// spread over the window, scan / sorted records in us: 1,024 x 1,024 and 14,752
// segments 70 / 143, 32,768 98 / 200; 2,048 x 2,048, 32,768 170 / 230; 4,096 x
// 4,096, 14,752 221 / 234, 32,768 411 / 395; 8,192 x 8,192, 2,048 198 / 414, 8,192
// 417 / 421, 32,768 1,304 / 617; 16,384 x 16,384, 2,048 681 / 1,221, 8,192 1,465 /
// 1,242. Windows of a few tiles leave a CTA or two with everything in either
// form, and the fill's chain per record is the shorter one: 18,432 segments in 17
// x 17 5,535 / 5,096, 5,760 in 40 x 30 357 / 453.
constexpr uint32_t kTileScanSegs = 1u << 15;
// Beyond this many segments the contents are looked at before the scan (3.5 us, and a
// call that leaves has lost only that and a wait). Up to there the look runs beside
// the scan's CTAs, which ask for its answer as they go: 2% or less with 256 CTAs,
// 14% with 7,500 (hence TL_CTAS), and a call that leaves has lost some 45 us; and
// only where the call waits for the count in any case.
constexpr uint32_t kTileLook = 4096;
constexpr bool tile_scan_pays(uint32_t n, uint64_t row_ctas, uint64_t tiles) {
    return n <= kTileScanSegs && n <= 4096 * tiles && n * row_ctas <= (48ull << 20) + 300 * tiles;
}

int launch_tile_fill(rrb_ctx* c, const TileRec* recs, uint64_t n_recs, const uint32_t* starts,
                     const uint32_t* counts, uint32_t w, uint32_t h, int eo, uint8_t* cov) {
    const uint32_t gw = (w + TILE - 1) / TILE, gh = (h + TILE - 1) / TILE;
    const uint64_t tiles = static_cast<uint64_t>(gw) * gh;
    const int grid = static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>(tiles, 8ull * rrb_ctx_sm_count(c))));
    cudaStream_t s = static_cast<cudaStream_t>(rrb_stream(c));
    k_tile_fill<<<grid, TF_THREADS, 0, s>>>(recs, n_recs, starts, counts, gw, gh, w, h, eo, cov);
    FILL_CUDA(c, cudaGetLastError());
    return RRB_OK;
}

// record_scan's phases (ScanPhase, crates/gpu/src/backend/params.rs:221-289).
// A block of SCAN_THREADS threads owns a tile of 2 * SCAN_THREADS u32; thread
// t holds elements 2t and 2t + 1. The exclusive scan of the pair sums is a
// warp shuffle scan, then a scan of the warp totals by warp 0; u32 sums wrap.
constexpr int SCAN_THREADS = static_cast<int>(RRB_SCAN_WORKGROUP_SIZE);
constexpr uint32_t SCAN_TILE = 2u * RRB_SCAN_WORKGROUP_SIZE;

// Exclusive scan of v over the block; *total receives the block's sum.
__device__ __forceinline__ uint32_t scan_block_excl(uint32_t v, uint32_t* warp_sums, uint32_t* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[w] = incl;
    __syncthreads();
    if (w == 0) {
        constexpr int NW = SCAN_THREADS / 32;
        uint32_t x = lane < NW ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += t;
        }
        if (lane < NW) warp_sums[lane] = x;  // inclusive over the warps
    }
    __syncthreads();
    *total = warp_sums[SCAN_THREADS / 32 - 1];
    return (w ? warp_sums[w - 1] : 0u) + incl - v;
}

// Phase 0 (and phase 1 with tile_sums == nullptr over the block sums): each
// block scans its tile of data[0, n) in place; tile_sums[block] = its total.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(uint32_t* __restrict__ data, uint32_t n,
                                                             uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t warp_sums[SCAN_THREADS / 32];
    const uint64_t i0 = static_cast<uint64_t>(blockIdx.x) * SCAN_TILE + 2u * threadIdx.x;
    const uint32_t a = i0 < n ? data[i0] : 0u, b = i0 + 1 < n ? data[i0 + 1] : 0u;
    uint32_t total;
    const uint32_t excl = scan_block_excl(a + b, warp_sums, &total);
    if (i0 < n) data[i0] = excl;
    if (i0 + 1 < n) data[i0 + 1] = excl + a;
    if (tile_sums && threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Phase 2: block b adds the scanned tile_sums[b] to its tile.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_scatter(uint32_t* __restrict__ data, uint32_t n,
                                                               const uint32_t* __restrict__ tile_sums) {
    const uint32_t add = tile_sums[blockIdx.x];
    const uint64_t i0 = static_cast<uint64_t>(blockIdx.x) * SCAN_TILE + threadIdx.x;
    if (i0 < n) data[i0] += add;
    if (i0 + SCAN_THREADS < n) data[i0 + SCAN_THREADS] += add;
}

}  // namespace

extern "C" {

int rrb_record_scan(rrb_ctx* c, const rrb_scan_params* p) {
    if (!c || !p) return RRB_ERR_INVARIANT;
    const rrb_host::DeviceScope dev_scope(rrb_ctx_device(c));
    int rc;
    if ((rc = begin(c, dev_scope.status()))) return rc;
    // ScanParams::validate (crates/gpu/src/backend/params.rs:338-372).
    if (p->len_elems == 0) return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "len_elems must be > 0");
    if (!p->data || 4ull * p->len_elems > rrb_device_buffer_len(p->data))
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "data buffer is smaller than len_elems * 4 bytes");
    const uint32_t blocks = (p->len_elems + SCAN_TILE - 1) / SCAN_TILE;
    if (blocks > RRB_SCAN_MAX_BLOCKS)
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "block_count exceeds SCAN_MAX_BLOCKS (1024)");
    if (!p->block_sums || 4ull * blocks > rrb_device_buffer_len(p->block_sums))
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "block_sums buffer is smaller than block_count * 4 bytes");
    if (p->phase > RRB_SCAN_SCATTER_BLOCK_SUMS) return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "unknown scan phase");
    if (reinterpret_cast<uintptr_t>(rrb_device_ptr(p->data)) & 3 ||
        reinterpret_cast<uintptr_t>(rrb_device_ptr(p->block_sums)) & 3)
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "scan buffers must be 4-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(rrb_stream(c));
    uint32_t* data = static_cast<uint32_t*>(rrb_device_ptr(p->data));
    uint32_t* sums = static_cast<uint32_t*>(rrb_device_ptr(p->block_sums));
    if (p->phase == RRB_SCAN_PER_WORKGROUP) k_scan_tiles<<<blocks, SCAN_THREADS, 0, s>>>(data, p->len_elems, sums);
    else if (p->phase == RRB_SCAN_BLOCK_SUMS) k_scan_tiles<<<1, SCAN_THREADS, 0, s>>>(sums, blocks, nullptr);
    else k_scan_scatter<<<blocks, SCAN_THREADS, 0, s>>>(data, p->len_elems, sums);
    FILL_CUDA(c, cudaGetLastError());
    return RRB_OK;
}

void rrb_aa_fill_jitter(float* x, float* y) {
    if (x) std::memcpy(x, jitter().x, sizeof jitter().x);
    if (y) std::memcpy(y, jitter().y, sizeof jitter().y);
}

int rrb_record_aa_fill(rrb_ctx* c, const rrb_aa_fill_params* p) {
    if (!c || !p) return RRB_ERR_INVARIANT;
    const rrb_host::DeviceScope dev_scope(rrb_ctx_device(c));
    int rc;
    if ((rc = begin(c, dev_scope.status())) || (rc = check_cov(c, p->coverage, p->width, p->height)) ||
        (rc = check_segs(c, p->segs, p->n_segs)))
        return rc;
    if (!p->width || !p->height) return RRB_OK;
    cudaStream_t s = static_cast<cudaStream_t>(rrb_stream(c));
    uint8_t* cov = static_cast<uint8_t*>(rrb_device_ptr(p->coverage));
    if (!p->n_segs) {
        FILL_CUDA(c, cudaMemsetAsync(cov, 0, static_cast<size_t>(p->width) * p->height, s));
        return RRB_OK;
    }
    const uint64_t items = static_cast<uint64_t>((p->height + AA_ROWS - 1) / AA_ROWS) * ((p->width + AA_CW - 1) / AA_CW);
    const int grid = static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>(items, 16ull * rrb_ctx_sm_count(c))));
    FILL_CUDA(c, cudaFuncSetAttribute(k_aa_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(AaShared))));
    k_aa_fill<<<grid, AA_NT, sizeof(AaShared), s>>>(static_cast<const float4*>(rrb_device_ptr(p->segs)), p->n_segs,
                                           p->width, p->height, p->fill_rule != 0, jitter_by_y(), cov);
    FILL_CUDA(c, cudaGetLastError());
    return RRB_OK;
}

int rrb_record_tile_fill(rrb_ctx* c, const rrb_tile_fill_params* p) {
    if (!c || !p) return RRB_ERR_INVARIANT;
    const rrb_host::DeviceScope dev_scope(rrb_ctx_device(c));
    int rc;
    if ((rc = begin(c, dev_scope.status())) || (rc = check_cov(c, p->coverage, p->width, p->height))) return rc;
    if (!p->width || !p->height) return RRB_OK;
    const uint32_t gw = (p->width + TILE - 1) / TILE, gh = (p->height + TILE - 1) / TILE;
    const uint64_t tiles = static_cast<uint64_t>(gw) * gh;
    if (!p->records || !p->tile_starts || !p->tile_counts)
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "records / tile_starts / tile_counts buffer is null");
    if (rrb_device_buffer_len(p->tile_starts) < 4 * tiles || rrb_device_buffer_len(p->tile_counts) < 4 * tiles)
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "tile_starts / tile_counts hold fewer than grid_w * grid_h entries");
    if (reinterpret_cast<uintptr_t>(rrb_device_ptr(p->records)) & 15)
        return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "records buffer is not 16-byte aligned");
    return launch_tile_fill(c, static_cast<const TileRec*>(rrb_device_ptr(p->records)),
                            rrb_device_buffer_len(p->records) / sizeof(TileRec),
                            static_cast<const uint32_t*>(rrb_device_ptr(p->tile_starts)),
                            static_cast<const uint32_t*>(rrb_device_ptr(p->tile_counts)), p->width, p->height,
                            p->fill_rule != 0, static_cast<uint8_t*>(rrb_device_ptr(p->coverage)));
}

int rrb_record_tile_fill_segs(rrb_ctx* c, const rrb_aa_fill_params* p, uint64_t* n_records) {
    if (!c || !p) return RRB_ERR_INVARIANT;
    const rrb_host::DeviceScope dev_scope(rrb_ctx_device(c));
    int rc;
    if ((rc = begin(c, dev_scope.status())) || (rc = check_cov(c, p->coverage, p->width, p->height)) ||
        (rc = check_segs(c, p->segs, p->n_segs)))
        return rc;
    if (n_records) *n_records = 0;
    if (!p->width || !p->height) return RRB_OK;
    const uint32_t gw = (p->width + TILE - 1) / TILE, gh = (p->height + TILE - 1) / TILE;
    if (gw > 0xFFFF || gh > 0xFFFF) return rrb_ctx_fail(c, RRB_ERR_INVARIANT, "raster exceeds the 16-bit tile key range");
    const uint64_t tiles = static_cast<uint64_t>(gw) * gh;
    cudaStream_t s = static_cast<cudaStream_t>(rrb_stream(c));
    const int sm = rrb_ctx_sm_count(c);
    const uint32_t n = p->n_segs;
    const float4* segs = static_cast<const float4*>(rrb_device_ptr(p->segs));
    void *v_off, *v_rec, *v_key, *v_idx, *v_key2, *v_idx2, *v_sorted, *v_ranges;
    // Few enough segments for every CTA to scan them all: one kernel, no records.
    // (A segment has at most 2 grid_h + grid_w records: those taken here cannot pass the limit below.)
    // A CTA owns 16 tiles of a row; fewer where that leaves the chip idle.
    uint32_t group_tiles = TSF_TILES;
    auto ctas = [&](uint32_t t) { return static_cast<uint64_t>(gh) * ((gw + t - 1) / t); };
    while (group_tiles > 1 && ctas(group_tiles) < static_cast<uint64_t>(sm)) group_tiles /= 2;
    const uint64_t row_ctas = ctas(group_tiles);
    if (tile_scan_pays(n, row_ctas, tiles) && row_ctas < 0x7FFFFFFFull && n * (2ull * gh + gw) < (1ull << 31)) {
        const bool look = n > kTileLook, beside = !look && n_records && n >= TL_MIN && row_ctas <= TL_CTAS;
        TsfWork* work = nullptr;
        if (look || n_records) {
            if ((rc = rrb_ctx_fill_scratch(c, 0, sizeof(TsfWork), &v_off))) return rc;
            work = static_cast<TsfWork*>(v_off);
            if (!look) FILL_CUDA(c, cudaMemsetAsync(work, 0, sizeof(TsfWork), s));
            else k_tile_look<<<1, TL_THREADS, 0, s>>>(segs, n, gw, gh, p->height, group_tiles, work);
        }
        const auto fill = beside ? k_tile_fill_segs<true> : k_tile_fill_segs<false>;
        fill<<<static_cast<unsigned>(row_ctas) + (beside ? 1 : 0), TSF_NT, 0, s>>>(
            segs, n, gw, gh, p->width, p->height, p->fill_rule != 0,
            static_cast<uint8_t*>(rrb_device_ptr(p->coverage)), group_tiles, work);
        FILL_CUDA(c, cudaGetLastError());
        TsfWork done{};
        if (work && (rc = rrb_ctx_read(c, work, sizeof done, &done))) return rc;
        if (!done.leave) {
            if (n_records) *n_records = done.records;
            return RRB_OK;
        }
    }
    if ((rc = rrb_ctx_fill_scratch(c, 0, 8ull * (n + 1), &v_off))) return rc;
    auto* off = static_cast<unsigned long long*>(v_off);
    uint64_t total = 0;
    if (n) {
        const int g = static_cast<int>(std::max<uint32_t>(1, std::min<uint32_t>((n + 255) / 256, 8u * sm)));
        k_tile_count<<<g, 256, 0, s>>>(segs, n, p->height, gw, gh, off);
        k_scan_u64<<<1, 1024, 0, s>>>(off, n);
        FILL_CUDA(c, cudaGetLastError());
        FILL_CUDA(c, cudaMemcpyAsync(&total, off + n, 8, cudaMemcpyDeviceToHost, s));
        FILL_CUDA(c, cudaStreamSynchronize(s));
    }
    if (total >= (1ull << 31)) return rrb_ctx_fail(c, RRB_ERR_POOL_EXHAUSTED, "more than 2^31 tile records");
    const uint32_t nr = static_cast<uint32_t>(total);
    if (n_records) *n_records = nr;
    const size_t nr1 = std::max<uint32_t>(1, nr);
    if ((rc = rrb_ctx_fill_scratch(c, 1, nr1 * sizeof(TileRec), &v_rec)) ||
        (rc = rrb_ctx_fill_scratch(c, 2, nr1 * 4, &v_key)) || (rc = rrb_ctx_fill_scratch(c, 3, nr1 * 4, &v_idx)) ||
        (rc = rrb_ctx_fill_scratch(c, 4, nr1 * 4, &v_key2)) || (rc = rrb_ctx_fill_scratch(c, 5, nr1 * 4, &v_idx2)) ||
        (rc = rrb_ctx_fill_scratch(c, 6, nr1 * sizeof(TileRec), &v_sorted)) ||
        (rc = rrb_ctx_fill_scratch(c, 7, 8 * tiles, &v_ranges)))
        return rc;
    auto* starts = static_cast<uint32_t*>(v_ranges);
    auto* counts = starts + tiles;
    if (nr) {
        const int g = static_cast<int>(std::max<uint32_t>(1, std::min<uint32_t>((n + 255) / 256, 8u * sm)));
        k_tile_write<<<g, 256, 0, s>>>(segs, n, p->height, gw, gh, off, static_cast<TileRec*>(v_rec),
                                       static_cast<uint32_t*>(v_key), static_cast<uint32_t*>(v_idx));
        size_t temp = 0;
        FILL_CUDA(c, cub::DeviceRadixSort::SortPairs(nullptr, temp, static_cast<uint32_t*>(v_key),
                                                     static_cast<uint32_t*>(v_key2), static_cast<uint32_t*>(v_idx),
                                                     static_cast<uint32_t*>(v_idx2), static_cast<int>(nr), 0, 32, s));
        // The sort's temporary storage reuses the offsets slot (no longer needed).
        if ((rc = rrb_ctx_fill_scratch(c, 0, std::max<size_t>(temp, 8ull * (n + 1)), &v_off))) return rc;
        FILL_CUDA(c, cub::DeviceRadixSort::SortPairs(v_off, temp, static_cast<uint32_t*>(v_key),
                                                     static_cast<uint32_t*>(v_key2), static_cast<uint32_t*>(v_idx),
                                                     static_cast<uint32_t*>(v_idx2), static_cast<int>(nr), 0, 32, s));
        const int g2 = static_cast<int>(std::max<uint32_t>(1, std::min<uint32_t>((nr + 255) / 256, 8u * sm)));
        k_tile_gather<<<g2, 256, 0, s>>>(static_cast<const TileRec*>(v_rec), static_cast<const uint32_t*>(v_idx2), nr,
                                         static_cast<TileRec*>(v_sorted));
    }
    const int g3 = static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>((tiles + 255) / 256, 8ull * sm)));
    k_tile_ranges<<<g3, 256, 0, s>>>(static_cast<const uint32_t*>(v_key2), nr, gw, gh, starts, counts);
    FILL_CUDA(c, cudaGetLastError());
    return launch_tile_fill(c, static_cast<const TileRec*>(v_sorted), nr, starts, counts, p->width, p->height,
                            p->fill_rule != 0, static_cast<uint8_t*>(rrb_device_ptr(p->coverage)));
}

}  // extern "C"
