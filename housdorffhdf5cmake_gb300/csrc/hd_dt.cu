// hd_dt.cu -- 6-neighbour element: the dilation counts from an exact
// city-block distance transform (sm_103a).
//
// The step at which the 6-neighbour dilation of a source first reaches a
// voxel (forBench/HausdorffDistance.cu:24-42, 96) is the voxel's city-block
// distance to the source: every path of face steps has at least
// |dx| + |dy| + |dz| steps, and the box between two voxels of the volume lies
// in the volume.  That distance separates by axis, so two kernels after the
// packing give every voxel's count whatever the number of steps, with no
// grid barrier and no queue:
//
//   dt_plane_kernel  per plane z: distances along x from the bits, then along
//                    y; stored as bytes
//   dt_depth_kernel  per column of voxels: distances along z at the target
//                    voxels, histogram per direction, result
//
// Distances are 16-bit pairs in one register; one step of a sweep,
// d[i] = min(d[i], d[i - 1] + 1), is one add-min instruction for both.
// A plane's values differ by at most one between face neighbours, so
// within a tile of 32 columns x 64 rows they lie within 94 of each other: a
// byte per voxel over a base per tile holds them exactly.
//
// Both kernels together, against the dilation loop with its set-up: 512^3
// with 445 steps 0.072 against 3.5 ms, 512x512x256 with 19 and 28 steps 0.045
// against 0.10 to 0.13 ms, 64^3 0.019 against 0.08 ms.  Their time follows the
// domain, not the steps: for masks that fill a large volume and differ by a few
// steps the loop is the faster one (whole calls, us, transform / loop: 512x512x256
// filled at random with 1 in 1000, 33 and 2 voxels, HD 22, 8 and 3: 282 / 345,
// 355 / 166, 363 / 107; a box against itself moved by one voxel, HD 3: 216 / 93;
// the same at 117x131x75 and below: the transform throughout).  Neither the
// domain nor the number of steps is known before the launches; the options and
// the autotuner choose the loop.
//
// Several pairs share launches (dt_planes_kernel, dt_list_kernel,
// dt_columns_kernel): their planes and their columns with targets are claimed
// from one list each, as their domains, which only the device knows, differ a
// lot (CTAs dealt to pairs by volume: 1.4 against 0.8 ms for 256 ragged
// pairs).  There the work fills the GPU, so a column is one warp's and no
// warp waits for another.  256 ragged pairs of 64 to 384 voxels a side: 0.74
// to 0.91 against 1.18 to 1.54 ms of the dilation loop.
#include <algorithm>
#include <atomic>
#include <cuda_runtime.h>
#include <stdint.h>

#include "hd/hd.h"
#include "hd_device.cuh"
#include "hd_kernels.h"
#include "hd_solve.cuh"

namespace hdk {

namespace {

constexpr unsigned kInf = 0x4000u;           // above any distance: W + H + D <= kDtMaxSum
constexpr unsigned kInf2 = kInf * 0x10001u;
constexpr int kSpread = 94;                  // largest difference of two voxels of a tile: 31 + 63
static_assert(kDtMaxSum < (int)kInf && 2 * kSpread < 256, "distances fit");

__device__ __forceinline__ uint32_t addmin2(uint32_t a, uint32_t b, uint32_t c) { return __viaddmin_u16x2(a, b, c); }
__device__ __forceinline__ constexpr uint32_t two(unsigned v) { return v * 0x10001u; }
// Bytes of the result, each the sign of a chosen byte of a (0x00 or 0xff).
template <unsigned kSel>
__device__ __forceinline__ uint32_t byte_signs(uint32_t a) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(d) : "r"(a), "n"(kSel));
    return d;
}

// Adds 1 to a counter in shared memory if `in`; predicated, no branch.
__device__ __forceinline__ void red_shared_inc(uint32_t at, unsigned in) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %1, 0;\n @q red.shared.add.u32 [%0], 1;\n}" ::"r"(at), "r"(in)
                 : "memory");
}

// Counts a plane's four rows of one column (a lane's distances v, target words
// t4); found(row, distance) at each target.
template <class F>
__device__ __forceinline__ void count_rows(uint2 v, uint4 t4, int lane, uint32_t hist_at, unsigned& dm, F found) {
    const uint32_t tw[4] = {t4.x, t4.y, t4.z, t4.w};
    const unsigned dd[4] = {v.x & 0xffffu, v.x >> 16, v.y & 0xffffu, v.y >> 16};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const unsigned in = (tw[r] >> lane) & 1u;
        red_shared_inc(hist_at + 4u * dd[r], in);
        dm = max(dm, in ? dd[r] : 0u);
        if (in) found(r, dd[r]);
    }
}

// A pair's domain: the bounding box of A u B, x in whole words.
struct Geom {
    int wx0, w1;             // first and last word column
    int oy, h, oz, d;        // rows, planes
    int wx, nq, ntile, nyq;  // words, 4-word groups they touch, 64-row tiles, 4-row groups
};
__device__ __forceinline__ Geom dt_geom(const PairInfo& I) {
    Geom g;
    g.wx0 = I.bb[0];
    g.w1 = I.bb[1];
    g.oy = I.bb[2];
    g.h = I.bb[3] - I.bb[2] + 1;
    g.oz = I.bb[4];
    g.d = I.bb[5] - I.bb[4] + 1;
    g.wx = g.w1 - g.wx0 + 1;
    g.nq = (g.w1 >> 2) - (g.wx0 >> 2) + 1;
    g.ntile = (g.h + 63) >> 6;
    g.nyq = (g.h + 3) >> 2;
    return g;
}

// Directions with target voxels (none of a pair with an empty mask).
__device__ __forceinline__ int dt_directions(const PairInfo& I) {
    return I.n_a == 0 || I.n_b == 0 ? 0 : (I.n_b > I.n_ab) + (I.n_a > I.n_ab);
}

// Nearest set voxel before (after) the end (start) of a word, carried over
// the words of a row: distance at the word's last (first) voxel.
__device__ __forceinline__ unsigned carry_left(unsigned c, uint32_t w) { return w ? __clz(w) : min(c + 32u, kInf); }
__device__ __forceinline__ unsigned carry_right(unsigned c, uint32_t w) {
    return w ? __ffs(w) - 1 : min(c + 32u, kInf);
}

constexpr int kPlaneWarps = 8;
constexpr int kTr = 32 * 33;  // transpose tile of a warp: 32 columns, padded
constexpr int kPlaneEnds = 2 * kPlaneWarps * 2 * 32;

}  // namespace

// Barrier `id` of `threads` threads of the CTA.
__device__ __forceinline__ void plane_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Planes: a warp takes a tile of 64 rows x 32 columns (one word column), the
// warps of a CTA the tiles of one or several planes; the CTA walks the word
// columns from left to right.
//   x: lane = rows (r, r + 32) in the halves of a register, 32 registers =
//      the word's voxels; the carries from the words on either side come from
//      whole words (clz / ffs), the left one kept, the right ones collected
//      beforehand per group of four words
//   y: after a transpose through shared memory, lane = column, registers =
//      rows; segments of 32 rows (the two halves) sweep on their own, then
//      take the carry over the segments above and below from shared memory
// About 400 warp instructions per 2048 voxels; issue slots 40 % busy (the
// barrier per word column and the sweeps' chains): 19 and 31 us for 512x512x256
// pairs with 19 and 28 steps (cold caches).  A CTA whose planes have no source
// voxel skips them, and rows are scanned once, from the right (the words come one
// at a time after that, from L1): 3 us less for a 512x512x256 pair than with the
// words in groups of four registers, 512^3 with small blobs (both directions) half
// (51 to 65 against 97 to 114 us).  The barrier
// per word column is among the plane's warps only (256 ragged pairs' planes and
// columns 0.767 against 0.791 ms).

// Plane z of a direction: this warp's tile t (a warp without one: act false).
// claimed() is called once, before the first barrier.
template <class F>
__device__ __forceinline__ void plane_unit(const DtPair& p, const Geom& g, int j, int z, int t, bool act, uint32_t* sm,
                                           F claimed) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t* const tr = sm + warp * kTr;
    uint32_t* const s_end = sm + kPlaneWarps * kTr;  // [2][warps][2][32]
    uint32_t* const s_r = s_end + kPlaneEnds;        // [words][warps][32]
    const int q0 = g.wx0 >> 2;
    const size_t vrow = (size_t)g.wx * 32;
    const int ya = t * 64 + lane, yb = ya + 32;
    // rows ya, yb of the plane's columns of 4 words, p.H apart
    const uint4* const src = (const uint4*)(p.packed[j] + (size_t)(g.oz + (act ? z : 0)) * p.H * p.pitch) + g.oy;
    const uint4* const ra = src + (ya < g.h ? ya : 0);
    const uint4* const rb = src + (yb < g.h ? yb : 0);
    const ptrdiff_t other = (const uint4*)p.packed[1 - j] - (const uint4*)p.packed[j];
    const bool va = act && ya < g.h, vb = act && yb < g.h;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    // One scan of the rows from the right: the carries at each word, the
    // rows with target voxels, and whether the plane has a source at all
    unsigned ca = kInf, cb = kInf;
    const int tz = t * g.d + (act ? z : 0);
    if (act) {
#pragma unroll 1
        for (int q = g.nq - 1; q >= 0; --q) {
            const ptrdiff_t o = (ptrdiff_t)(q0 + q) * p.H;
            const uint4 a = va ? __ldg(ra + o) : zero, b = vb ? __ldg(rb + o) : zero;
            const uint4 c = va ? __ldg(ra + other + o) : zero, d = vb ? __ldg(rb + other + o) : zero;
            const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
            const uint32_t ta[4] = {c.x & ~a.x, c.y & ~a.y, c.z & ~a.z, c.w & ~a.w};
            const uint32_t tb[4] = {d.x & ~b.x, d.y & ~b.y, d.z & ~b.z, d.w & ~b.w};
            unsigned fa = 0, fb = 0;
#pragma unroll
            for (int k = 3; k >= 0; --k) {
                s_r[((4 * q + k) * kPlaneWarps + warp) * 32 + lane] = ca | (cb << 16);
                ca = carry_right(ca, wa[k]);
                cb = carry_right(cb, wb[k]);
                const unsigned ba = __ballot_sync(kFull, ta[k] != 0u), bb = __ballot_sync(kFull, tb[k] != 0u);
                if (lane == k) {
                    fa = ba;
                    fb = bb;
                }
            }
            const int w = 4 * (q0 + q) + lane;
            if (lane < 4 && w >= g.wx0 && w <= g.w1) {
                uint32_t* const f = p.rows[j] + (size_t)(w - g.wx0) * 2 * g.ntile * g.d + t * g.d + tz;
                f[0] = fa;
                f[g.d] = fb;
                uint32_t* const c = p.cols + j * p.ncols + (w - g.wx0) * 2 * g.ntile + 2 * t;
                if (fa) atomicOr(c, fa);
                if (fb) atomicOr(c + 1, fb);
            }
        }
    }
    claimed();
    if (!__syncthreads_or(act && (ca < kInf || cb < kInf))) {  // nothing to measure from
        if (act)
            for (int w = lane; w < g.wx; w += 32) p.base[j][(size_t)w * g.ntile * g.d + tz] = (uint16_t)kInf;
        return;
    }
    unsigned la = kInf, lb = kInf;
    uint32_t* const vol = p.vol[j] + (size_t)(act ? z : 0) * g.nyq * vrow;
    const uint32_t* const pa = (const uint32_t*)ra;
    const uint32_t* const pb = (const uint32_t*)rb;
    auto word = [&](int w) { return (ptrdiff_t)(w & ~3) * p.H + (w & 3); };
    uint32_t na = va ? __ldg(pa + word(g.wx0)) : 0u, nb = vb ? __ldg(pb + word(g.wx0)) : 0u;
#pragma unroll 1
    for (int w = g.wx0; w <= g.w1; ++w) {
        const uint32_t ua = na, ub = nb;
        if (w < g.w1) {  // the next word's
            na = va ? __ldg(pa + word(w + 1)) : 0u;
            nb = vb ? __ldg(pb + word(w + 1)) : 0u;
        }
        {
            const uint32_t rcw = act ? s_r[((w - 4 * q0) * kPlaneWarps + warp) * 32 + lane] : 0u;
            uint32_t V[32];
            uint32_t* const end = s_end + ((w & 1) * kPlaneWarps) * 64;
            if (act) {
                // x: a seed is 0 on a set voxel, else 0xffff
                const uint32_t n0 = ~__byte_perm(ua, ub, 0x5410), n1 = ~__byte_perm(ua, ub, 0x7632);
                uint32_t f = la | (lb << 16);
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const uint32_t s = (i < 16 ? n0 : n1) << (7 - (i & 7));
                    const uint32_t seed = (i & 8) ? byte_signs<0xBB99>(s) : byte_signs<0xAA88>(s);
                    f = addmin2(f, two(1), seed);
                    V[i] = f;
                }
                f = rcw;
#pragma unroll
                for (int i = 31; i >= 0; --i) {
                    f = addmin2(f, two(1), V[i]);
                    tr[i * 33 + lane] = f;
                }
                la = carry_left(la, ua);
                lb = carry_left(lb, ub);
                __syncwarp();
                // y: the two segments on their own
#pragma unroll
                for (int i = 0; i < 32; ++i) V[i] = tr[lane * 33 + i];
                __syncwarp();
#pragma unroll
                for (int i = 1; i < 32; ++i) V[i] = addmin2(V[i - 1], two(1), V[i]);
#pragma unroll
                for (int i = 30; i >= 0; --i) V[i] = addmin2(V[i + 1], two(1), V[i]);
                end[warp * 64 + lane] = V[0];
                end[warp * 64 + 32 + lane] = V[31];
            }
            // ends are double-buffered by word: one barrier per word, of the plane's warps
            if (act) plane_sync(1 + warp / g.ntile, 32 * g.ntile);
            if (act) {
                // carries over the segments above (value at the row before
                // the segment) and below
                const uint32_t* const e0 = end + (warp - t) * 64 + lane;
                unsigned cf = kInf, cb = kInf;
#pragma unroll 1
                for (int s = 0; s < t; ++s) {
                    const uint32_t e = e0[s * 64 + 32];
                    cf = min(e & 0xffffu, cf + 32u);
                    cf = min(e >> 16, cf + 32u);
                }
#pragma unroll 1
                for (int s = g.ntile - 1; s > t; --s) {
                    const uint32_t e = e0[s * 64];
                    cb = min(e >> 16, cb + 32u);
                    cb = min(e & 0xffffu, cb + 32u);
                }
                const uint32_t CF = cf | (min(V[31] & 0xffffu, cf + 32u) << 16);
                const uint32_t CB = min(V[0] >> 16, cb + 32u) | (cb << 16);
                // a carry that does not lower its first row lowers none
                if (__any_sync(kFull, addmin2(CF, two(1), V[0]) != V[0])) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) V[i] = addmin2(CF, two(i + 1), V[i]);
                }
                if (__any_sync(kFull, addmin2(CB, two(1), V[31]) != V[31])) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) V[i] = addmin2(CB, two(32 - i), V[i]);
                }
                // bytes over the tile's base; an empty plane stores its base alone
                const unsigned v0 = __shfl_sync(kFull, V[0] & 0xffffu, 0);
                const unsigned b = v0 >= kInf ? kInf : (v0 > kSpread ? v0 - kSpread : 0u);
                if (lane == 0) p.base[j][(size_t)(w - g.wx0) * g.ntile * g.d + tz] = (uint16_t)b;
                if (b < kInf) {
                    uint32_t* const o = vol + (size_t)(w - g.wx0) * 32 + lane;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint32_t p01 = __byte_perm(V[4 * i] - two(b), V[4 * i + 1] - two(b), 0x6240);
                        const uint32_t p23 = __byte_perm(V[4 * i + 2] - two(b), V[4 * i + 3] - two(b), 0x6240);
                        const int yl = t * 16 + i, yh = yl + 8;
                        if (yl < g.nyq) o[yl * vrow] = __byte_perm(p01, p23, 0x5410);
                        if (yh < g.nyq) o[yh * vrow] = __byte_perm(p01, p23, 0x7632);
                    }
                }
            }
        }
    }
    __syncthreads();  // the ends' buffers start over with the next planes
}

// Planes per CTA: as many as its warps have tiles for, but no fewer CTAs than
// are resident (most: planes per resident CTA).
__device__ __forceinline__ int planes_per_cta(const Geom& g, int most) { return max(1, min(kPlaneWarps / g.ntile, most)); }

// One pair: a CTA per group of planes, so that the next group goes to whichever
// SM is free (planes without a source, or with few words, end early; 512^3 160
// to 154 us a call against one wave of CTAs that take every n-th).  kCtas per
// SM: plane_ctas.
template <int kCtas>
__global__ void __launch_bounds__(kPlaneWarps * 32, kCtas) dt_plane_kernel(const __grid_constant__ DtPair p, int sms) {
    extern __shared__ uint4 sm4[];
    cudaGridDependencySynchronize();  // placed as the packing ends
    const PairInfo I = *p.info;
    // histograms and counters of the depth kernel
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t <= p.kmax; t += gridDim.x * blockDim.x)
        p.hist[0][t] = p.hist[1][t] = 0ull;
    if (blockIdx.x == 0 && threadIdx.x == 0) *p.state = DtState{};
    const int nact = dt_directions(I);
    if (nact == 0) return;
    const Geom g = dt_geom(I);
    const int G = planes_per_cta(g, nact * g.d / (kCtas * sms));
    const int groups = (g.d + G - 1) / G, warp = threadIdx.x >> 5;
    const int pl = warp / g.ntile, t = warp - pl * g.ntile;
    const int u = blockIdx.x;
    if (u >= nact * groups) return;
    const int j = nact == 2 ? (u >= groups) : !(I.n_b > I.n_ab);
    const int z = (nact == 2 && j ? u - groups : u) * G + pl;
    plane_unit(p, g, j, z, t, pl < G && z < g.d, (uint32_t*)sm4, [] {});
}

// Several pairs: their units in one list, claimed from a counter one ahead;
// every CTA holds all the pairs' descriptors and counts.  Issue slots 55 %
// busy while it runs, the barriers per word column most of the rest.
__global__ void __launch_bounds__(kPlaneWarps * 32, 3) dt_planes_kernel(const DtPair* __restrict__ many, int n, int quads,
                                                                        DtGroup* group) {
    extern __shared__ uint4 sm4[];
    __shared__ int s_next[2], s_total, s_most;
    cudaGridDependencySynchronize();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    DtPair* const s_pair = (DtPair*)((uint32_t*)sm4 + kPlaneWarps * kTr + kPlaneEnds + quads * 4 * kPlaneWarps * 32);
    PairInfo* const s_info = (PairInfo*)(s_pair + n);
    int* const s_begin = (int*)(s_info + n);  // [kDtMaxGroup]: first unit
    // histograms and counters of the columns' kernel
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const DtPair& p = many[i];
        for (int t = threadIdx.x; t <= p.kmax; t += blockDim.x) p.hist[0][t] = p.hist[1][t] = 0ull;
        if (threadIdx.x == 0) *p.state = DtState{};
    }
    static_assert(sizeof(DtPair) % 16 == 0 && sizeof(PairInfo) % 8 == 0 && kDtMaxGroup == 64, "copied in vectors");
    constexpr int kV = sizeof(DtPair) / 16, kI = sizeof(PairInfo) / 8;
    for (int t = threadIdx.x; t < n * kV; t += blockDim.x) ((uint4*)s_pair)[t] = __ldg((const uint4*)many + t);
    __syncthreads();
    for (int t = threadIdx.x; t < n * kI; t += blockDim.x)
        ((uint2*)s_info)[t] = __ldcg((const uint2*)s_pair[t / kI].info + t % kI);
    __syncthreads();
    if (warp == 0) {
        int planes = 0, before = 0;
        for (int i = lane; i < n; i += 32) planes += dt_directions(s_info[i]) * dt_geom(s_info[i]).d;
        const int most = __reduce_add_sync(kFull, planes) / (int)gridDim.x;
#pragma unroll 1
        for (int i = lane; i < kDtMaxGroup; i += 32) {
            const int nact = i < n ? dt_directions(s_info[i]) : 0;
            int units = 0;
            if (nact) {
                const Geom g = dt_geom(s_info[i]);
                const int G = planes_per_cta(g, most);
                units = nact * ((g.d + G - 1) / G);
            }
            int x = units;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(kFull, x, o);
                if (lane >= o) x += v;
            }
            s_begin[i] = i < n ? before + x - units : 0x7fffffff;
            before += __shfl_sync(kFull, x, 31);
        }
        if (lane == 0) {
            s_total = before;
            s_most = most;
        }
    }
    __syncthreads();
    const int total = s_total, most = s_most;
    int slot = 0;
#pragma unroll 1
    for (int u = blockIdx.x; u < total; slot ^= 1) {
        int next = 0;
        if (threadIdx.x == 0) next = atomicAdd(&group->next_plane, 1) + gridDim.x;
        const int i = __popc(__ballot_sync(kFull, s_begin[lane] <= u)) + __popc(__ballot_sync(kFull, s_begin[32 + lane] <= u)) - 1;
        const PairInfo& I = s_info[i];
        const Geom g = dt_geom(I);
        const int G = planes_per_cta(g, most), groups = (g.d + G - 1) / G, v = u - s_begin[i];
        const int pl = warp / g.ntile, t = warp - pl * g.ntile;
        const bool both = dt_directions(I) == 2;
        const int j = both ? v >= groups : !(I.n_b > I.n_ab);
        const int z = (both && j ? v - groups : v) * G + pl;
        // the slots alternate: a claim is read between this barrier and the next
        plane_unit(s_pair[i], g, j, z, t, pl < G && z < g.d, (uint32_t*)sm4, [&] {
            if (threadIdx.x == 0) s_next[slot] = next;
        });
        u = s_next[slot];
    }
}

// One warp: the pair's result from the counts and the two histograms, with
// the rules of decode_pair_warp (statuses, exact sums, one double division,
// robust HD).  One pass over the bins, 32 of both directions at a time, until
// every target is counted.
__device__ __forceinline__ void dt_decode(const DtPair& p, const PairInfo& I) {
    const int lane = threadIdx.x & 31;
    const unsigned long long n_ab = I.n_a - I.n_ab, n_ba = I.n_b - I.n_ab;  // A's, B's voxels outside the other
    unsigned long long sum[2] = {0ull, 0ull}, cov[2] = {0ull, 0ull};
    int hd[2] = {0, 0}, rk[2] = {-1, -1};
    const bool empty = I.n_a == 0 || I.n_b == 0;
    if (!empty) {
        const float tf[2] = {(float)n_ba * p.pct, (float)n_ab * p.pct};  // job 0 measures B's voxels
        const unsigned long long total[2] = {n_ba, n_ab};
#pragma unroll 1
        for (int k0 = 0; k0 <= p.kmax && (cov[0] < total[0] || cov[1] < total[1]); k0 += 32) {
            const int k = k0 + lane;
            unsigned long long c2[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) c2[j] = k <= p.kmax ? __ldcg(p.hist[j] + k) : 0ull;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                unsigned long long c = c2[j];
                sum[j] += (unsigned long long)k * c;
                if (c) hd[j] = k;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned long long x = __shfl_up_sync(kFull, c, o);
                    if (lane >= o) c += x;
                }
                // hello.cu:1751-1758: first step whose covered count no longer lies under the percentile
                const unsigned m = __ballot_sync(kFull, !(tf[j] > (float)(cov[j] + c)));
                if (m && rk[j] < 0) rk[j] = k0 + __ffs(m) - 1;
                cov[j] += __shfl_sync(kFull, c, 31);
            }
        }
        // (no targets at all: stops at step 0)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            hd[j] = __reduce_max_sync(kFull, hd[j]);
            if (total[j] == 0ull && rk[j] < 0) rk[j] = 0;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sum[0] += __shfl_xor_sync(kFull, sum[0], o);
            sum[1] += __shfl_xor_sync(kFull, sum[1], o);
        }
    }
    if (lane != 0) return;
    hd_result r;
    memset(&r, 0, sizeof r);
    r.n_a = I.n_a;
    r.n_b = I.n_b;
    r.n_a_not_b = n_ab;
    r.n_b_not_a = n_ba;
    if (I.n_a == 0 && I.n_b == 0) {
        r.status = HD_OK;
    } else if (empty) {
        r.status = HD_EMPTY_MASK;
        r.hd = r.hd_ab = r.hd_ba = r.hd_robust = -1;
        r.avg_hd = __longlong_as_double(0x7ff8000000000000LL);  // quiet NaN
    } else {
        r.status = HD_OK;
        r.hd_ba = hd[0];
        r.sum_ba = sum[0];
        r.hd_ab = hd[1];
        r.sum_ab = sum[1];
        r.hd = max(hd[0], hd[1]);
        r.avg_hd = (double)(sum[0] + sum[1]) / (double)(I.n_a + I.n_b);
        r.hd_robust = max(rk[0] < 0 ? p.kmax : rk[0], rk[1] < 0 ? p.kmax : rk[1]);
    }
    *p.out = r;
    *p.info = pair_info_start();  // for the next packing
}

namespace {
constexpr int kDepthMaxWarps = 8;
constexpr int kSeg = 16;  // planes of a segment
constexpr int kHalf = 8;  // planes of a segment staged for counting at a time
// Dynamic shared memory of a CTA: staged distances per warp, the column's end
// planes per segment, the distances' counters of both directions, the masks
// of a segment's planes with targets, and the list of columns with targets.
__host__ __device__ constexpr size_t depth_smem(int warps, int nseg, int bins, int ncols) {
    return (size_t)warps * kHalf * 32 * 8 + (size_t)nseg * (32 * 16 + 4) + ((size_t)bins * 8 + 16) + (size_t)ncols * 8;
}
}  // namespace

// Columns: a unit is one direction's four rows x one word column that hold a
// target in some plane, all planes; its tasks are segments of 16 planes (a
// warp: lane = column, two registers of 16-bit pairs per plane = the four
// rows).
//   1. first pass: every segment is swept and leaves its two end planes in
//      shared memory
//   2. second pass: the segments with targets (few: targets are a shell) are
//      swept again, now with the carry over the segments before and after
//      from the end planes, and count the distances at their targets
// Every CTA lists the units itself, from the plane kernel's masks of rows with
// targets per word column, and takes every gridDim-th: about half of a
// domain's columns have no target.
// Sweeping twice costs less than holding a segment over the barrier: the
// warps that have no targets would wait there for those that have.  The two
// passes share one piece of code, and the targets of a task are visited in a
// rolled loop: a CTA runs a few tasks only, so instruction fetches count.
// Bound by the chain of loads, barriers and counters of one unit: a
// 512x512x256 pair has 400 to 530 units for 608 CTAs.  512x512x256 pairs with 19
// and 28 steps 17 and 28 us (cold caches).  When it was written, 512x512x256 pair /
// 512^3 / 64^3: 17 to 22 / 29 to 34 / 12.5 us; with every column visited and its
// segments' masks read behind a barrier 25-29 / 40-44 / 14; units claimed from a
// counter 28-35 at 512x512x256 (the claim waits once per unit); 16 warps per CTA
// holding their segments over the barrier likewise.
template <bool kMap>
__global__ void __launch_bounds__(kDepthMaxWarps * 32, 4) dt_depth_kernel(const __grid_constant__ DtPair p) {
    extern __shared__ uint4 sm4[];
    __shared__ int s_max[2], s_last, s_warp[kDepthMaxWarps], s_first[2];
    __shared__ uint4 s_tgt[kDepthMaxWarps][kSeg];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    cudaGridDependencySynchronize();  // launched while the plane kernel ends
    const PairInfo I = *p.info;
    const bool act0 = I.n_b > I.n_ab, act1 = I.n_a > I.n_ab;  // directions with targets
    const int nact = (I.n_a == 0 || I.n_b == 0) ? 0 : act0 + act1;
    const Geom g = dt_geom(I);
    const int nseg = nact ? (g.d + kSeg - 1) / kSeg : 0;
    const int bins = nact ? min(32 * g.wx, p.W) + g.h + g.d : 0;     // above any distance in the domain
    const int per = g.wx * 2 * g.ntile;                              // masks of 32 rows, per direction
    uint2* const s_v = (uint2*)sm4 + warp * kHalf * 32;
    uint4* const s_end = sm4 + nwarps * kHalf * 16;          // [nseg][32]: first and last plane
    uint4* const s_hist4 = s_end + nseg * 32;                // [direction][bins]
    unsigned* const s_hist = (unsigned*)s_hist4;
    unsigned* const s_list = (unsigned*)(s_hist4 + (2 * bins + 3) / 4);  // per mask: four-row groups with targets, units before
    unsigned* const s_zm = s_list + nact * per;              // [nseg]: planes with targets
    for (int t = threadIdx.x; t < (2 * bins + 3) / 4; t += blockDim.x) s_hist4[t] = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0;
    int units = 0;
#pragma unroll 1
    for (int i0 = 0; i0 < nact * per; i0 += blockDim.x) {
        const int i = i0 + threadIdx.x, jj = i >= per;
        unsigned m = i < nact * per ? __ldcg(p.cols + (act0 ? jj : 1) * p.ncols + (i - jj * per)) : 0u;
        m |= m >> 2;
        m = (m | (m >> 1)) & 0x11111111u;  // one bit per four rows
        const int c = __popc(m);
        int x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += v;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        int before = units;
        for (int v = 0; v < nwarps; ++v) {
            if (v < warp) before += s_warp[v];
            units += s_warp[v];
        }
        before += x - c;
        if ((int)blockIdx.x >= before && (int)blockIdx.x < before + c) {  // the CTA's first unit
            unsigned g1 = m;
            for (int k = blockIdx.x - before; k > 0; --k) g1 &= g1 - 1u;
            s_first[0] = i;
            s_first[1] = (__ffs(g1) - 1) >> 2;
        }
        // bits 0, 4, .. 28 -> bits 24 .. 31
        m = (m | (m >> 3)) & 0x03030303u;
        m = (m | (m >> 6)) & 0x000f000fu;
        m = (m | (m >> 12)) << 24;
        if (i < nact * per) s_list[i] = m | (unsigned)before;
        __syncthreads();
    }
    const size_t vrow = (size_t)g.wx * 32, vplane = vrow * g.nyq;
    const uint32_t s_hist_at = (uint32_t)__cvta_generic_to_shared(s_hist);
    int dmax[2] = {0, 0};
#pragma unroll 1
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        int lo = s_first[0], group = s_first[1];
        if (u != (int)blockIdx.x) {
            // the last mask with at most u units before it that has any
            int hi = nact * per - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((int)(s_list[mid] & 0xffffffu) <= u) lo = mid;
                else hi = mid - 1;
            }
            const unsigned le = s_list[lo];
            unsigned gm = le >> 24;
            for (int k = u - (int)(le & 0xffffffu); k > 0; --k) gm &= gm - 1u;
            group = __ffs(gm) - 1;
        }
        const int jj = lo >= per, j = act0 ? jj : 1, wh = lo - jj * per;
        const int w = wh / (2 * g.ntile), half = wh - w * 2 * g.ntile;
        const int yq = 8 * half + group;
        const uint32_t* const rows = p.rows[j] + (size_t)wh * g.d;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            // Second pass: the segments with targets; if they are few, one
            // task per half of a segment's planes (counting takes longer than
            // loading and sweeping again, and other warps would wait).
            unsigned long long lower = 0ull, upper = 0ull;
            int ntasks = nseg, nlower = 0;
            if (pass) {
                for (int i0 = 0; i0 < nseg; i0 += 32) {
                    const unsigned v = i0 + lane < nseg ? s_zm[i0 + lane] : 0u;
                    lower |= (unsigned long long)__ballot_sync(kFull, (v & 0x00ffu) != 0u) << i0;
                    upper |= (unsigned long long)__ballot_sync(kFull, (v & 0xff00u) != 0u) << i0;
                }
                if (2 * __popcll(lower | upper) > nwarps) {
                    lower |= upper;
                    upper = 0ull;
                }
                nlower = __popcll(lower);
                ntasks = nlower + __popcll(upper);
            }
#pragma unroll 1
            for (int task = warp; task < ntasks; task += nwarps) {
                int sg = task;
                unsigned zm = 0u;
                if (pass) {
                    const bool up = task >= nlower;
                    unsigned long long m = up ? upper : lower;
#pragma unroll 1
                    for (int k = up ? task - nlower : task; k > 0; --k) m &= m - 1ull;
                    sg = __ffsll(m) - 1;
                    zm = s_zm[sg];
                    if (upper) zm &= up ? 0xff00u : 0x00ffu;
                }
                // the segment's planes: distances within their planes
                const int z0 = sg * kSeg;
                unsigned b = kInf, r = 0u;
                if (pass == 0 && lane < kSeg && z0 + lane < g.d) r = __ldg(rows + z0 + lane);
                if (lane < kSeg && z0 + lane < g.d)
                    b = __ldg(p.base[j] + ((size_t)w * g.ntile + (yq >> 4)) * g.d + z0 + lane);
                const uint32_t* const vp = p.vol[j] + (size_t)z0 * vplane + (size_t)yq * vrow + (size_t)w * 32 + lane;
                uint32_t V[kSeg][2];
#pragma unroll
                for (int i = 0; i < kSeg; ++i)  // (an empty plane's bytes are not written: read, not used)
                    V[i][0] = z0 + i < g.d ? __ldcg(vp + i * vplane) : 0u;
                // target words: lane = (plane, two of the four rows)
                uint32_t tw0 = 0u, tw1 = 0u;
                uint32_t f0 = kInf2, f1 = kInf2, c0 = kInf2, c1 = kInf2;
                if (pass) {
                    const int z = z0 + (lane & 15), y = 4 * yq + 2 * (lane >> 4);
                    if (z < g.d && y < g.h) {
                        const int wf = g.wx0 + w;
                        const size_t o = ((size_t)(g.oz + z) * p.pitch + (wf & ~3)) * p.H + 4 * (g.oy + y) + (wf & 3);
                        tw0 = __ldg(p.packed[1 - j] + o) & ~__ldg(p.packed[j] + o);
                        if (y + 1 < g.h) tw1 = __ldg(p.packed[1 - j] + o + 4) & ~__ldg(p.packed[j] + o + 4);
                    }
#pragma unroll 4
                    for (int s = 0; s < sg; ++s) {
                        const uint4 e = s_end[s * 32 + lane];
                        f0 = addmin2(f0, two(kSeg), e.z);
                        f1 = addmin2(f1, two(kSeg), e.w);
                    }
#pragma unroll 4
                    for (int s = nseg - 1; s > sg; --s) {
                        const uint4 e = s_end[s * 32 + lane];
                        c0 = addmin2(c0, two(kSeg), e.x);
                        c1 = addmin2(c1, two(kSeg), e.y);
                    }
                }
#pragma unroll
                for (int i = 0; i < kSeg; ++i) {
                    const uint32_t x = V[i][0], bb = two(__shfl_sync(kFull, b, i));
                    const bool in = bb < kInf2;
                    V[i][0] = f0 = addmin2(f0, two(1), in ? __byte_perm(x, 0u, 0x4140) + bb : kInf2);
                    V[i][1] = f1 = addmin2(f1, two(1), in ? __byte_perm(x, 0u, 0x4342) + bb : kInf2);
                }
#pragma unroll
                for (int i = kSeg - 1; i >= 0; --i) {
                    V[i][0] = c0 = addmin2(c0, two(1), V[i][0]);
                    V[i][1] = c1 = addmin2(c1, two(1), V[i][1]);
                }
                if (pass == 0) {
                    s_end[sg * 32 + lane] = make_uint4(c0, c1, f0, f1);
                    zm = __ballot_sync(kFull, ((r >> (4 * (yq & 7))) & 0xfu) != 0u);
                    if (lane == 0) s_zm[sg] = zm;
                    continue;
                }
                ((uint2*)s_tgt[warp])[(lane & 15) * 2 + (lane >> 4)] = make_uint2(tw0, tw1);
                const uint32_t hist = s_hist_at + 4u * (unsigned)(j * bins);
                unsigned dm = 0u;
                auto count = [&](int i, int h) {  // the targets of plane h + i of the segment
                    count_rows(s_v[i * 32 + lane], s_tgt[warp][h + i], lane, hist, dm, [&](int r, unsigned d) {
                        if constexpr (kMap) {
                            const size_t row = (size_t)(g.oz + z0 + h + i) * p.H + g.oy + 4 * yq + r;
                            p.map[j][row * p.W + 32 * (g.wx0 + w) + lane] = (int32_t)d;
                        }
                    });
                };
#pragma unroll
                for (int h = 0; h < kSeg; h += kHalf) {
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < kHalf; ++i) s_v[i * 32 + lane] = make_uint2(V[h + i][0], V[h + i][1]);
                    __syncwarp();
                    // two planes at a time: their loads overlap
#pragma unroll 1
                    for (unsigned m = (zm >> h) & ((1u << kHalf) - 1u); m;) {
                        const int i0 = __ffs(m) - 1;
                        m &= m - 1u;
                        count(i0, h);
                        if (m) {
                            count(__ffs(m) - 1, h);
                            m &= m - 1u;
                        }
                    }
                }
                if (j) dmax[1] = max(dmax[1], (int)dm);
                else dmax[0] = max(dmax[0], (int)dm);
            }
            __syncthreads();  // end planes complete; after the second pass the shared data are free
        }
    }
    // this CTA's counts
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int m = __reduce_max_sync(kFull, dmax[j]);
        if (lane == 0 && m) atomicMax(&s_max[j], m);
    }
    __syncthreads();
#pragma unroll 1
    for (int j = 0; j < 2; ++j)
        for (int t = threadIdx.x; t <= s_max[j] && t < bins; t += blockDim.x)
            if (const unsigned v = s_hist[j * bins + t]) atomicAdd(p.hist[j] + t, (unsigned long long)v);
    __threadfence();
    __syncthreads();
    // the last CTA to finish decodes the result
    if (threadIdx.x == 0) {
        s_last = atomicAdd(&p.state->done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (s_last && warp == 0) {
        __threadfence();
        dt_decode(p, I);
    }
}

// Several pairs: lists the columns with targets, a CTA per pair: bits 0-2 the
// four-row group within its mask of 32 rows, 3-13 the mask (word column, 32
// rows), 14 the direction, 15- the pair.
constexpr int kListThreads = 128;
__global__ void __launch_bounds__(kListThreads) dt_list_kernel(const DtPair* many, uint32_t* list, DtGroup* group) {
    __shared__ unsigned s_units;
    cudaGridDependencySynchronize();
    const DtPair& p = many[blockIdx.x];
    const int lane = threadIdx.x & 31;
    const PairInfo I = *p.info;
    const int nact = dt_directions(I);
    __syncthreads();  // every thread has its copy: the decode puts *p.info back to the start values
    if (nact == 0) {
        if (threadIdx.x < 32) dt_decode(p, I);
        return;
    }
    const Geom g = dt_geom(I);
    const int per = g.wx * 2 * g.ntile, first = I.n_b > I.n_ab ? 0 : 1;
    if (threadIdx.x == 0) s_units = 0u;
    __syncthreads();
    for (int i0 = threadIdx.x - lane; i0 < nact * per; i0 += kListThreads) {
        const int i = i0 + lane, jj = i >= per, j = first + jj;
        unsigned m = i < nact * per ? __ldcg(p.cols + j * p.ncols + (i - jj * per)) : 0u;
        m |= m >> 2;
        m = (m | (m >> 1)) & 0x11111111u;  // one bit per four rows
        const int c = __popc(m);
        int x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += v;
        }
        unsigned at = 0u;
        if (lane == 31 && x) {
            at = atomicAdd(&group->units, (unsigned)x);
            atomicAdd(&s_units, (unsigned)x);
        }
        at = __shfl_sync(kFull, at, 31) + x - c;
        for (; m; m &= m - 1u)
            list[at++] = (unsigned)blockIdx.x << 15 | (unsigned)j << 14 | (unsigned)(i - jj * per) << 3 |
                         (unsigned)(__ffs(m) - 1) >> 2;
    }
    __syncthreads();
    if (threadIdx.x == 0) p.state->units = s_units;
}

// Several pairs: a column per warp at a time, claimed one ahead.  From the
// last plane down to the first segment with targets each segment leaves the
// carry from the planes after it in shared memory; then up to the last with
// targets, counting where there are any.  No barrier, and every warp has a
// histogram of its own, added to the pair's after each column.
// Bound by latency (a third of the issue slots, 10 warps per SM: the
// histograms and carries take the shared memory).  256 ragged pairs, planes
// and columns: 0.74 to 0.91 ms; 4 warps per CTA and one plane counted at a time
// 0.77 to 0.94 ms; the next segment loaded ahead (110 registers) or 64 registers:
// the same, 4 % more; histograms of 256 bins: 6 % less, but distances have no
// such limit.
constexpr int kManyWarps = 2, kManyCtas = 12;
__host__ __device__ constexpr size_t many_warp_smem(int nseg, int bins) {
    return (size_t)kHalf * 32 * 8 + (size_t)nseg * (32 * 8) + ((size_t)nseg * 2 + 31) / 16 * 16 +
           ((size_t)bins * 4 + 15) / 16 * 16;
}
__global__ void __launch_bounds__(kManyWarps * 32, kManyCtas)
    dt_columns_kernel(const DtPair* many, const uint32_t* list, DtGroup* group, int max_seg, int bins) {
    extern __shared__ uint4 sm4[];
    __shared__ uint4 s_tgt[kManyWarps][kSeg];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    char* const sm = (char*)sm4 + warp * many_warp_smem(max_seg, bins);
    uint2* const s_v = (uint2*)sm;
    uint2* const s_carry = s_v + kHalf * 32;            // [max_seg][32]
    unsigned* const s_hist = (unsigned*)(s_carry + max_seg * 32);  // [bins]
    uint16_t* const s_zm = (uint16_t*)(s_hist + (bins + 3) / 4 * 4);  // [max_seg]: planes with targets
    const uint32_t hist_at = (uint32_t)__cvta_generic_to_shared(s_hist);
    for (int t = lane; t < bins; t += 32) s_hist[t] = 0u;
    cudaGridDependencySynchronize();
    const int total = (int)__ldcg(&group->units);
#pragma unroll 1
    for (int u = blockIdx.x * kManyWarps + warp; u < total;) {
        int next = 0;
        if (lane == 0) next = atomicAdd(&group->next_column, 1) + gridDim.x * kManyWarps;
        const unsigned rec = __ldcg(list + u);
        const DtPair& p = many[rec >> 15];
        const int j = (rec >> 14) & 1u, wh = (rec >> 3) & 0x7ffu;
        const Geom g = dt_geom(*p.info);
        const int nseg = (g.d + kSeg - 1) / kSeg;
        const int w = wh / (2 * g.ntile), half = wh - w * 2 * g.ntile, yq = 8 * half + (int)(rec & 7u);
        const size_t vrow = (size_t)g.wx * 32, vplane = vrow * g.nyq;
        const uint32_t* const vol = p.vol[j] + (size_t)yq * vrow + (size_t)w * 32 + lane;
        const uint16_t* const base = p.base[j] + ((size_t)w * g.ntile + (yq >> 4)) * g.d;
        // planes with targets
        const uint32_t* const rows = p.rows[j] + (size_t)wh * g.d;
        int first = nseg, last = -1;
        __syncwarp();
        for (int z = 0; z < g.d; z += 32) {
            const unsigned r = z + lane < g.d ? __ldcg(rows + z + lane) : 0u;
            const unsigned zm = __ballot_sync(kFull, ((r >> (4 * (yq & 7))) & 0xfu) != 0u);
            if (lane < 2) s_zm[(z >> 4) + lane] = (uint16_t)(zm >> (16 * lane));
            if (zm) {
                first = min(first, (z >> 4) + ((zm & 0xffffu) == 0u));
                last = (z >> 4) + ((zm >> 16) != 0u);
            }
        }
        uint32_t V[kSeg][2];
        // A segment's in-plane distances (an empty plane's bytes are not
        // written; over its base they are no distance whatever they are)
        auto load = [&](int sg) {
            const int z0 = sg * kSeg;
            const unsigned b = lane < kSeg && z0 + lane < g.d ? (unsigned)__ldcg(base + z0 + lane) : kInf;
#pragma unroll
            for (int i = 0; i < kSeg; ++i) V[i][0] = z0 + i < g.d ? __ldcg(vol + (z0 + i) * vplane) : 0u;
#pragma unroll
            for (int i = 0; i < kSeg; ++i) {
                const uint32_t x = V[i][0], bb = two(__shfl_sync(kFull, b, i));
                V[i][0] = __byte_perm(x, 0u, 0x4140) + bb;
                V[i][1] = __byte_perm(x, 0u, 0x4342) + bb;
            }
        };
        uint32_t c0 = kInf2, c1 = kInf2;
#pragma unroll 1
        for (int sg = nseg - 1;; --sg) {
            s_carry[sg * 32 + lane] = make_uint2(c0, c1);
            if (sg <= first) break;
            load(sg);
#pragma unroll
            for (int i = kSeg - 1; i >= 0; --i) {
                c0 = addmin2(c0, two(1), V[i][0]);
                c1 = addmin2(c1, two(1), V[i][1]);
            }
        }
        __syncwarp();  // s_zm
        uint32_t f0 = kInf2, f1 = kInf2;
        unsigned dm = 0u;
#pragma unroll 1
        for (int sg = 0; sg <= last; ++sg) {
            const unsigned zm = s_zm[sg];
            const int z0 = sg * kSeg;
            uint32_t tw0 = 0u, tw1 = 0u;  // lane = (plane, two of the four rows)
            if (zm) {
                const int z = z0 + (lane & 15), y = 4 * yq + 2 * (lane >> 4);
                if (z < g.d && y < g.h) {
                    const int wf = g.wx0 + w;
                    const size_t o = ((size_t)(g.oz + z) * p.pitch + (wf & ~3)) * p.H + 4 * (g.oy + y) + (wf & 3);
                    tw0 = __ldg(p.packed[1 - j] + o) & ~__ldg(p.packed[j] + o);
                    if (y + 1 < g.h) tw1 = __ldg(p.packed[1 - j] + o + 4) & ~__ldg(p.packed[j] + o + 4);
                }
            }
            load(sg);
#pragma unroll
            for (int i = 0; i < kSeg; ++i) {
                V[i][0] = f0 = addmin2(f0, two(1), V[i][0]);
                V[i][1] = f1 = addmin2(f1, two(1), V[i][1]);
            }
            if (!zm) continue;
            const uint2 c = s_carry[sg * 32 + lane];
            c0 = c.x;
            c1 = c.y;
#pragma unroll
            for (int i = kSeg - 1; i >= 0; --i) {
                V[i][0] = c0 = addmin2(c0, two(1), V[i][0]);
                V[i][1] = c1 = addmin2(c1, two(1), V[i][1]);
            }
            ((uint2*)s_tgt[warp])[(lane & 15) * 2 + (lane >> 4)] = make_uint2(tw0, tw1);
#pragma unroll
            for (int h = 0; h < kSeg; h += kHalf) {
                __syncwarp();
#pragma unroll
                for (int i = 0; i < kHalf; ++i) s_v[i * 32 + lane] = make_uint2(V[h + i][0], V[h + i][1]);
                __syncwarp();
                // two planes at a time: their loads overlap
#pragma unroll 1
                for (unsigned m = (zm >> h) & ((1u << kHalf) - 1u); m;) {
                    const int i = __ffs(m) - 1;
                    m &= m - 1u;
                    const int i2 = m ? __ffs(m) - 1 : i;
                    const uint2 v = s_v[i * 32 + lane], v2 = s_v[i2 * 32 + lane];
                    const uint4 t = s_tgt[warp][h + i], t2 = m ? s_tgt[warp][h + i2] : make_uint4(0u, 0u, 0u, 0u);
                    m &= m - 1u;
                    count_rows(v, t, lane, hist_at, dm, [](int, unsigned) {});
                    count_rows(v2, t2, lane, hist_at, dm, [](int, unsigned) {});
                }
            }
            __syncwarp();
        }
        // to the pair's counts; the pair's last column decodes its result
        dm = __reduce_max_sync(kFull, dm);
        __syncwarp();
        for (int t = lane; t <= (int)dm; t += 32)
            if (const unsigned v = s_hist[t]) {
                atomicAdd(p.hist[j] + t, (unsigned long long)v);
                s_hist[t] = 0u;
            }
        __threadfence();
        __syncwarp();
        bool done = false;
        if (lane == 0) done = atomicAdd(&p.state->done, 1u) + 1u == __ldcg(&p.state->units);
        if (__shfl_sync(kFull, (int)done, 0)) {
            __threadfence();
            const PairInfo I = *p.info;
            dt_decode(p, I);
        }
        u = __shfl_sync(kFull, next, 0);
    }
}

// ---- launch wrappers --------------------------------------------------------
bool dt_fits(int W, int H, int D) {
    return W <= kDtMaxW && H <= kDtMaxH && D <= kDtMaxD && W + H + D <= kDtMaxSum;
}

namespace {

constexpr int kPlaneCtas = 3;  // resident CTAs per SM (several pairs)

// Resident CTAs per SM of one pair's planes: 3 (80 registers) or 2 (122), by the
// depth alone, as the host knows neither the domain nor the planes with a source.
// On a group of 48 SMs there are always more planes than CTAs: 3 (eight
// 512x512x256 pairs 396 against 401 us).  On the whole GPU 3 where the planes of
// both directions, taken as 3/4 of all, are more than 2 per SM but not much more
// than 3.  Both kernels, 2 / 3 per SM, us, mean of 24 CT-like pairs (a single one
// is 20 % either way, as its last round of CTAs fills up): 301x287x173 25.9 /
// 25.6, 512x512 at D 210 / 256 / 300 / 340 / 440 30.1 / 29.6, 33.2 / 32.2, 35.9 /
// 33.9, 38.9 / 36.6, 47.2 / 45.5, 256^3 30.0 / 28.7.  Domains of the whole volume: 1
// % for 2 at 512x512, 2 to 5 % for 3 at 256x256 and 301x287 from D 173 on.  Few
// planes with a source (far blobs) want 2: 512x512 at D 256 / 370 / 512 57.9 /
// 70.2, 64.0 / 76.1, 74.0 / 82.2, hence the upper end.
int plane_ctas(int D, int sms) {
    const double planes = 1.5 * D;
    return sms < 100 || (planes > 2 * sms && planes <= 3.5 * sms) ? 3 : 2;
}

size_t plane_smem(int quads, int pairs) {
    return sizeof(uint32_t) * (kPlaneWarps * kTr + kPlaneEnds + (size_t)quads * 4 * kPlaneWarps * 32) +
           (pairs ? pairs * (sizeof(DtPair) + sizeof(PairInfo)) + sizeof(int) * kDtMaxGroup : 0);
}
int quads_of(const DtPair& p) { return ((p.W + 31) / 32 + 3) / 4; }
int segs_of(const DtPair& p) { return (p.D + kSeg - 1) / kSeg; }

// Raises the kernels' limit of dynamic shared memory, once per device, for the
// largest size (calls of other sizes may run on other threads).
cudaError_t raise_limits() {
    static std::atomic<bool> raised[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || (dev < 64 && raised[dev].load(std::memory_order_acquire))) return e;
    const int lim = 200 * 1024;  // above any size taken (dt_fits), with the static part below 227 KB
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    e = cudaFuncSetAttribute(&dt_plane_kernel<2>, attr, lim);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(&dt_plane_kernel<3>, attr, lim);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(&dt_planes_kernel, attr, lim);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(&dt_depth_kernel<false>, attr, lim);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(&dt_depth_kernel<true>, attr, lim);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(&dt_columns_kernel, attr, lim);
    if (e == cudaSuccess && dev < 64) raised[dev].store(true, std::memory_order_release);
    return e;
}

// A launch whose CTAs are placed as the kernel before it ends (they wait for
// that kernel's results themselves): 3 us less per call at 64^3 and 301x287x173
// than after it.  Not before: CTAs that wait beside a running packing take
// its SMs' L1 (512^3 197 against 160 us a call, 301x287x173 212 against 202).
template <class... P, class... A>
cudaError_t launch_early(void (*kernel)(P...), long long grid, int threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    return cudaLaunchKernelEx(&c, kernel, args...);
}

}  // namespace

cudaError_t launch_dt(const DtPair& p, int sms, cudaStream_t s) {
    cudaError_t e = raise_limits();
    if (e != cudaSuccess) return e;
    const int nseg = segs_of(p), dwarps = nseg > 2 ? kDepthMaxWarps : 4;
    e = launch_early(plane_ctas(p.D, sms) == 3 ? dt_plane_kernel<3> : dt_plane_kernel<2>, 2ll * p.D, kPlaneWarps * 32,
                     plane_smem(quads_of(p), 0), s, p, sms);
    if (e != cudaSuccess) return e;
    // one resident wave, or fewer CTAs than that for small volumes
    const long long dg = std::min<long long>(dt_list(p.W, p.H), 4ll * kDepthMaxWarps / dwarps * sms);
    return launch_early(p.map[0] ? dt_depth_kernel<true> : dt_depth_kernel<false>, dg, dwarps * 32,
                        depth_smem(dwarps, nseg, p.W + p.H + p.D, p.ncols), s, p);
}

cudaError_t launch_dt_group(const DtPair* pairs, const DtPair* d_pairs, int n, uint32_t* d_list, DtGroup* d_group, int sms,
                            cudaStream_t s) {
    cudaError_t e = raise_limits();
    int quads = 0, nseg = 0, bins = 0;
    long long planes = 0, columns = 0;
    for (int i = 0; i < n; ++i) {
        const DtPair& p = pairs[i];
        quads = std::max(quads, quads_of(p));
        nseg = std::max(nseg, segs_of(p));
        bins = std::max(bins, p.W + p.H + p.D);
        planes += 2ll * p.D;
        columns += dt_list(p.W, p.H);
    }
    if (e == cudaSuccess)
        e = launch_early(dt_planes_kernel, std::min<long long>(planes, (long long)kPlaneCtas * sms), kPlaneWarps * 32,
                         plane_smem(quads, n), s, d_pairs, n, quads, d_group);
    if (e == cudaSuccess) e = launch_early(dt_list_kernel, n, kListThreads, 0, s, d_pairs, d_list, d_group);
    if (e == cudaSuccess)
        e = launch_early(dt_columns_kernel, std::min<long long>((columns + kManyWarps - 1) / kManyWarps, (long long)kManyCtas * sms),
                         kManyWarps * 32, kManyWarps * many_warp_smem(nseg, bins), s, d_pairs, (const uint32_t*)d_list, d_group, nseg,
                         bins);
    return e;
}

}  // namespace hdk
