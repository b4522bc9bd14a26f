// hd_pack.cu -- packing and set-up kernels (sm_103a).
//
// pack_kernel   replaces boolPrepareKernel (hello.cu:539-748) and the bounding
//               box of getMinMaxes (hello.cu:398-526): uint8 masks -> 32 voxels
//               per uint32 along x (the prototype packs along z, :598-631),
//               with |A|, |B|, |A n B| and the bounding box of A u B (x in
//               whole words).  One pass over the bytes, 128-bit streaming
//               loads; words stored in columns of 4 (see hd_device.cuh).
// setup_kernel  replaces firstMetaPrepareKernel (hello.cu:763-877): writes
//               the job descriptors and queues every brick of each job for
//               its first step; for the one-step kernel it also crops the
//               packed masks to each job's domain and builds the
//               uncovered-target words.
// map_init_kernel  -1 / 0 initialisation of the optional per-voxel maps.
#include <algorithm>
#include <climits>
#include <cuda_runtime.h>
#include <stdint.h>

#include "hd/hd.h"
#include "hd_device.cuh"
#include "hd_kernels.h"

namespace hdk {

// Foreground bytes of a 32-bit word as flags at bits 28..31 (byte i -> bit
// 28 + i).  Foreground = nonzero, or (kLabel) equal to the label, whose
// byte `pat` repeats four times: the XOR turns those bytes into zeros and
// the zero-byte flags are the complement of the nonzero ones.  The
// normalised word has bits only at 7, 15, 23, 31; times 2^0 + 2^7 + 2^14 +
// 2^21 its partial products land on distinct bits (7, 14, 15, 21, 22, 23
// below 28, the flags at 28..31), so nothing carries.
template <bool kLabel>
__device__ __forceinline__ uint32_t fg4_top(uint32_t w, uint32_t pat) {
    if constexpr (kLabel) w ^= pat;
    uint32_t t = (((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) & 0x80808080u;
    if constexpr (kLabel) t ^= 0x80808080u;
    return t * 0x00204081u;
}

// Foreground bytes of 16 bytes -> 16 bits (byte i -> bit i).  The partial
// products below bit 24 vanish in the two larger shifts and are masked off in
// the two smaller ones.
template <bool kLabel>
__device__ __forceinline__ uint32_t fg16(uint4 v, uint32_t pat) {
    return (fg4_top<kLabel>(v.x, pat) >> 28) | (fg4_top<kLabel>(v.y, pat) >> 24) |
           ((fg4_top<kLabel>(v.z, pat) >> 20) & 0xF00u) | ((fg4_top<kLabel>(v.w, pat) >> 16) & 0xF000u);
}

// The same for 16 bytes that are all 0 or 1: each dot product weighs four
// bytes with their bits.
__device__ __forceinline__ uint32_t bits16(uint4 v) {
    const uint32_t lo = __dp4a(v.y, 0x80402010u, __dp4a(v.x, 0x08040201u, 0u));
    const uint32_t hi = __dp4a(v.w, 0x80402010u, __dp4a(v.z, 0x08040201u, 0u));
    return lo | (hi << 8);
}

// The pair that owns work tile `tile` (first tiles increase with the pair
// index; setup = false: packing tiles, true: set-up tiles).
__device__ __forceinline__ int pair_of_tile(const PairDesc* __restrict__ descs, int npairs, long long tile,
                                            bool setup) {
    int lo = 0, hi = npairs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((setup ? descs[mid].stile0 : descs[mid].tile0) <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Counts and bounding box of the packed words a thread has seen in one pair.
// 32-bit counts: a thread packs at most 2^31 / 256 words of a pair.  The
// box is kept as word columns (x), rows (y) and row indices r = y + H z (z
// follows at the flush: r -> r / H is monotone).
struct PackAcc {
    uint32_t na = 0, nb = 0, nab = 0;
    int wmin = INT_MAX, wmax = -1, ymin = INT_MAX, ymax = -1, rmin = INT_MAX, rmax = -1;
    __device__ __forceinline__ void add(uint32_t wa, uint32_t wb, int r, int y, int w) {
        na += __popc(wa);
        nb += __popc(wb);
        nab += __popc(wa & wb);
        if (wa | wb) {
            wmin = min(wmin, w);
            wmax = max(wmax, w);
            ymin = min(ymin, y);
            ymax = max(ymax, y);
            rmin = min(rmin, r);
            rmax = max(rmax, r);
        }
    }
};

constexpr int kPackWarps = 8;  // (flush_acc's scratch holds this many)
constexpr int kPackThreads = 32 * kPackWarps;

// Block-wide reduction of the accumulators, then one set of atomics per CTA
// (many CTAs update one PairInfo: per-warp atomics serialise on its lines).
// Called by all threads of the CTA.  A warp's counts fit in 32 bits: a volume
// has fewer than 2^36 voxels, spread over hundreds of warps.
__device__ __forceinline__ void flush_acc(PairInfo* const I, int H, const PackAcc& acc) {
    __shared__ unsigned s_cnt[3][kPackWarps];
    __shared__ int s_bb[6][kPackWarps];
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const unsigned na = __reduce_add_sync(0xffffffffu, acc.na), nb = __reduce_add_sync(0xffffffffu, acc.nb),
                   nab = __reduce_add_sync(0xffffffffu, acc.nab);
    const int bb[6] = {__reduce_min_sync(0xffffffffu, acc.wmin), __reduce_max_sync(0xffffffffu, acc.wmax),
                       __reduce_min_sync(0xffffffffu, acc.ymin), __reduce_max_sync(0xffffffffu, acc.ymax),
                       __reduce_min_sync(0xffffffffu, acc.rmin), __reduce_max_sync(0xffffffffu, acc.rmax)};
    __syncthreads();  // earlier readers of the scratch are done
    if ((threadIdx.x & 31) == 0) {
        s_cnt[0][warp] = na;
        s_cnt[1][warp] = nb;
        s_cnt[2][warp] = nab;
#pragma unroll
        for (int i = 0; i < 6; ++i) s_bb[i][warp] = bb[i];
    }
    __syncthreads();
    // one thread per value
    if (threadIdx.x < 3) {
        unsigned long long n = 0;
        for (int w = 0; w < nwarps; ++w) n += s_cnt[threadIdx.x][w];
        if (n) atomicAdd(threadIdx.x == 0 ? &I->n_a : (threadIdx.x == 1 ? &I->n_b : &I->n_ab), n);
    } else if (threadIdx.x >= 32 && threadIdx.x < 38) {
        const int i = threadIdx.x - 32;
        int v = s_bb[i][0];
        bool any = s_bb[1][0] >= 0;
        for (int w = 1; w < nwarps; ++w) {
            v = (i & 1) ? max(v, s_bb[i][w]) : min(v, s_bb[i][w]);
            any = any || s_bb[1][w] >= 0;
        }
        if (i >= 4) v = v / H;
        if (any) {
            if (i & 1) atomicMax(&I->bb[i], v);
            else atomicMin(&I->bb[i], v);
        }
    }
}

constexpr int kPackCtas = 2;            // resident CTAs per SM
constexpr int kWords = 4;               // words per lane and span
constexpr int kSpan = 32 * kWords;      // words a warp packs at a time
constexpr int kRounds = 2 * kWords;     // 16-byte chunks per lane and mask
constexpr int kSpanChunks = 2 * kSpan;  // chunks of a span (one more when unaligned)
constexpr int kBitWords = kSpan + 4;    // words of a span's bit stream
static_assert(kPackTileWords == kPackWarps * kSpan, "one tile = one span per warp");

// Constants of one pair's packing walk (taken when a CTA's run of tiles
// enters the pair).
struct PackWalk {
    const uint8_t* src[2];
    uint32_t* dst[2];           // packed masks
    size_t nbytes;              // bytes of a mask
    unsigned wxf, W, H, total;  // words per row, bytes per row, rows per plane, words of the pair
    unsigned pitch;             // packed row pitch (words): wxf rounded up to 4, zero words in between
    unsigned dq, dr;            // 32 words = dq rows + dr words
    unsigned tq, tr;            // from a span's end to the warp's next span = tq rows + tr words
    // (row, word, y) 32 words on, and from a span's end to the next span
    __device__ __forceinline__ void step(unsigned& r, unsigned& w, unsigned& y, unsigned q, unsigned m) const {
        w += m;
        const unsigned d = q + (w >= wxf ? 1u : 0u);
        if (w >= wxf) w -= wxf;
        r += d;
        y += d;
        if (y >= H) y %= H;
    }
    // word w of row r = y + H z in the packed volume
    __device__ __forceinline__ size_t at(unsigned r, unsigned w, unsigned y) const {
        return (size_t)(r - y) * pitch + ((size_t)(w >> 2) * H + y) * 4u + (w & 3u);
    }
    __device__ __forceinline__ void next_words(unsigned& r, unsigned& w, unsigned& y) const { step(r, w, y, dq, dr); }
    __device__ __forceinline__ void next_span(unsigned& r, unsigned& w, unsigned& y) const { step(r, w, y, tq, tr); }
};

// One warp's span of a pair: words t0 .. t0 + kSpan - 1 of both masks (word t =
// row r, word w of the row, stored at PackWalk::at), the bytes that hold them
// and the 16-byte chunks that cover these.
struct PackSpan {
    unsigned cnt;            // words of the span
    size_t lo;               // first byte
    unsigned sh[2], nch[2];  // per mask: bytes of the first chunk before it, chunks
};

__device__ __forceinline__ PackWalk make_walk(const PairDesc& P) {
    PackWalk k;
    k.src[0] = P.a;
    k.src[1] = P.b;
    k.dst[0] = P.pa;
    k.dst[1] = P.pb;
    k.nbytes = (size_t)P.W * P.H * P.D;
    k.wxf = (unsigned)P.wxf;
    k.pitch = (unsigned)packed_pitch(P.W);
    k.W = (unsigned)P.W;
    k.H = (unsigned)P.H;
    k.total = (unsigned)((long long)P.wxf * P.H * P.D);  // < 2^31 words
    k.dq = 32u / k.wxf;
    k.dr = 32u - k.dq * k.wxf;
    k.tq = ((unsigned)kPackTileWords - kSpan) / k.wxf;
    k.tr = ((unsigned)kPackTileWords - kSpan) - k.tq * k.wxf;
    return k;
}

// Locates the span of words t0 ..: row r and word w are its first word's.
__device__ __forceinline__ PackSpan locate(const PackWalk& k, unsigned t0, unsigned r, unsigned w) {
    PackSpan n;
    n.cnt = min((unsigned)kSpan, k.total - t0);
    n.lo = (size_t)r * k.W + 32u * w;
    // the last word: cnt - 1 words on
    const unsigned lw = w + n.cnt - 1u, q = lw / k.wxf, x = lw - q * k.wxf;
    const unsigned len = q * k.W + 32u * x - 32u * w + min(32u, k.W - 32u * x);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        n.sh[m] = (unsigned)((uintptr_t)(k.src[m] + n.lo) & 15u);
        n.nch[m] = (n.sh[m] + len + 15u) >> 4;
    }
    return n;
}

// Issues the loads of a span's chunks of mask m (streaming).  Lanes past the
// last chunk, and chunks that stick out of the mask (the first or last of a
// pair), repeat a neighbouring one: those bits are not used, or written by
// put_bits byte by byte.  x: a lane's byte of the one chunk more that an unaligned span may have.
__device__ __forceinline__ void load_chunks(const PackWalk& k, const PackSpan& n, int m, uint4 (&c)[kRounds], unsigned& x) {
    const int lane = threadIdx.x & 31;
    const uint8_t* const q = k.src[m] + n.lo - n.sh[m];
    const bool head = n.lo < n.sh[m], tail = n.lo - n.sh[m] + 16ull * n.nch[m] > k.nbytes && !(head && n.nch[m] == 1u);
    const int c_lo = head ? 1 : 0, c_hi = (int)n.nch[m] - (tail ? 2 : 1);  // first and last chunk inside
    if (c_hi >= c_lo) {  // uniform
#pragma unroll
        for (int i = 0; i < kRounds; ++i)
            c[i] = __ldcs(reinterpret_cast<const uint4*>(q) + max(min(32 * i + lane, c_hi), c_lo));
    }
    x = 0u;
    if (n.nch[m] > kSpanChunks) {  // uniform
        const size_t o = n.lo - n.sh[m] + 16u * kSpanChunks + lane;
        if (lane < 16 && o < k.nbytes) x = __ldg(k.src[m] + o);
    }
}

// Foreground flags of the span's chunks of mask m, as a stream of bits.
template <bool kLabel>
__device__ __forceinline__ void put_bits(const PackWalk& k, const PackSpan& n, int m, const uint4 (&c)[kRounds], unsigned x,
                                         unsigned label, uint32_t* s_bits) {
    const int lane = threadIdx.x & 31;
    const uint32_t pat = label * 0x01010101u;
    uint16_t* const s = reinterpret_cast<uint16_t*>(s_bits);
    bool general = kLabel;
    if constexpr (!kLabel) {
        uint32_t any = 0u;
#pragma unroll
        for (int i = 0; i < kRounds; ++i) any |= c[i].x | c[i].y | c[i].z | c[i].w;
        general = __any_sync(0xffffffffu, (any & 0xfefefefeu) != 0u);
    }
    if (general) {
#pragma unroll
        for (int i = 0; i < kRounds; ++i) s[32 * i + lane] = (uint16_t)fg16<kLabel>(c[i], pat);
    } else {
#pragma unroll
        for (int i = 0; i < kRounds; ++i) s[32 * i + lane] = (uint16_t)bits16(c[i]);
    }
    if (n.nch[m] > kSpanChunks) {  // uniform
        const unsigned bits = __ballot_sync(0xffffffffu, lane < 16 && (kLabel ? x == label : x != 0u));
        if (lane == 0) s[kSpanChunks] = (uint16_t)bits;
    }
    const bool head = n.lo < n.sh[m], tail = n.lo - n.sh[m] + 16ull * n.nch[m] > k.nbytes;
    if (head || tail) {  // uniform: a chunk sticks out of the mask
#pragma unroll 1
        for (int e = 0; e < 2; ++e) {
            __syncwarp();
            if (!(e ? tail : head)) continue;
            const unsigned ch = e ? n.nch[m] - 1u : 0u;
            const size_t o = n.lo + 16u * ch + lane;  // byte of the mask, plus sh
            const bool in = lane < 16 && o >= n.sh[m] && o - n.sh[m] < k.nbytes;
            const unsigned v = in ? __ldg(k.src[m] + (o - n.sh[m])) : 0u;
            const unsigned bits = __ballot_sync(0xffffffffu, in && (kLabel ? v == label : v != 0u));
            if (lane == 0) s[ch] = (uint16_t)bits;
        }
    }
}

// Cuts the span's words out of the bit streams (a row starts at any bit).
// (r, w, y): this lane's first word, advanced past the span.
__device__ __forceinline__ void put_words(const PackWalk& k, const PackSpan& n, unsigned& r,
                                          unsigned& w, unsigned& y, PackAcc& acc, const uint32_t (*s_bits)[kBitWords]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
        if (32u * i + lane < n.cnt) {
            const bool last = w + 1u == k.wxf;
            const unsigned nbits = last ? k.W - 32u * w : 32u;
            const uint32_t mask = 0xffffffffu >> (32u - nbits);
            const unsigned d = (unsigned)((size_t)r * k.W + 32u * w - n.lo);
            uint32_t out[2];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const unsigned o = d + n.sh[m];
                out[m] = __funnelshift_r(s_bits[m][o >> 5], s_bits[m][(o >> 5) + 1], o & 31u) & mask;
            }
            const size_t o = k.at(r, w, y);
            k.dst[0][o] = out[0];
            k.dst[1][o] = out[1];
            if (last)  // the row's last word also writes its padding (up to 3 words)
#pragma unroll 1
                for (unsigned x = 1u; x <= k.pitch - k.wxf; ++x) k.dst[0][o + x] = k.dst[1][o + x] = 0u;
            acc.add(out[0], out[1], (int)r, (int)y, (int)w);
        }
        k.next_words(r, w, y);
    }
}

// Asks for the bytes of a span of aligned words of both masks (from byte lo
// on), a line per lane, in L2.  Taken on part of the SMs, where the packing is bound
// by the latency of its loads (eight pipelined 512x512x256 pairs 395 -> 363 us;
// two spans ahead 366, bulk prefetches that leave L2 first the same; pairs whose
// distances take the longer part 1 % slower); on all of them HBM is the bound
// (512^3 141 against 143 us), and the kernel for other words waits for its
// instructions (509x511x250 60.5 against 60.8 us a pair).
__device__ __forceinline__ void fetch_ahead(const PackWalk& k, size_t lo) {
    const size_t o = lo + 128u * (threadIdx.x & 31);
#pragma unroll
    for (int m = 0; m < 2; ++m)
        if (o < k.nbytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(k.src[m] + o));
}

// 32 mask bytes at p (32-byte aligned), read once: one 256-bit load, first to
// leave L2 (without that hint 512x512x256 takes 32 instead of 27 us: the
// masks push the packed words and the next kernels' data out).
__device__ __forceinline__ void load32(const uint8_t* p, uint32_t (&v)[8]) {
    asm volatile("ld.global.L1::evict_first.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
}

// A warp's spans of a pair whose words are 32 aligned bytes each (rows of a
// multiple of 32 voxels, 32-byte aligned masks): word t is bytes 32 t .. of
// the mask, so a lane loads, converts and stores its words without the bit
// stream, at less than half the instructions.  On every SM it is as fast as
// the other kernel (27 us at 512x512x256, 51 at 512^3: HBM), on the 56 SMs of
// the pipelined entry, where instructions count, 44 against 58 us.
template <bool kLabel, bool kAhead>
__device__ __forceinline__ void pack_aligned(const PackWalk& k, unsigned t0, unsigned t1, unsigned r, unsigned w,
                                             unsigned y, PackAcc& acc, unsigned label) {
    const int lane = threadIdx.x & 31;
    const uint32_t pat = label * 0x01010101u;
#pragma unroll 1
    for (; t0 < t1; t0 += (unsigned)kPackTileWords) {
        uint32_t v[2][kWords][8], out[2][kWords];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < kWords; ++i)
                load32(k.src[m] + 32 * (size_t)min(t0 + 32u * i + lane, k.total - 1u), v[m][i]);
        if (kAhead && t0 + (unsigned)kPackTileWords < t1) fetch_ahead(k, 32 * (size_t)(t0 + (unsigned)kPackTileWords));
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            bool general = kLabel;
            if constexpr (!kLabel) {
                uint32_t any = 0u;
#pragma unroll
                for (int i = 0; i < kWords; ++i)
#pragma unroll
                    for (int b = 0; b < 8; ++b) any |= v[m][i][b];
                general = __any_sync(0xffffffffu, (any & 0xfefefefeu) != 0u);
            }
#pragma unroll
            for (int i = 0; i < kWords; ++i) {
                const uint4 lo = make_uint4(v[m][i][0], v[m][i][1], v[m][i][2], v[m][i][3]);
                const uint4 hi = make_uint4(v[m][i][4], v[m][i][5], v[m][i][6], v[m][i][7]);
                if (general) out[m][i] = fg16<kLabel>(lo, pat) | (fg16<kLabel>(hi, pat) << 16);
                else out[m][i] = bits16(lo) | (bits16(hi) << 16);
            }
        }
#pragma unroll
        for (int i = 0; i < kWords; ++i) {
            if (t0 + 32u * i + lane < k.total) {
                const size_t o = k.at(r, w, y);
                k.dst[0][o] = out[0][i];
                k.dst[1][o] = out[1][i];
                if (w + 1u == k.wxf)
#pragma unroll 1
                    for (unsigned x = 1u; x <= k.pitch - k.wxf; ++x) k.dst[0][o + x] = k.dst[1][o + x] = 0u;
                acc.add(out[0][i], out[1][i], (int)r, (int)y, (int)w);
            }
            k.next_words(r, w, y);
        }
        k.next_span(r, w, y);
    }
}

// Packing launch: one wave of resident CTAs, each over a contiguous run of
// tiles (a run crosses few pairs, so the pair lookup and the accumulator
// flush are rare); a tile is one span per warp, of any width, alignment or
// memory kind (device or host-mapped).  Rows are contiguous in the mask, so a
// span is one run of bytes: it is read in the 16-byte chunks that cover it,
// each once and coalesced, their foreground flags go to shared memory as a
// stream of bits (masks of zeros and ones, by a vote over the span, with one
// dot product per four bytes), and the words are cut out of that stream.
// Bound by HBM for large volumes (8 KB in flight per warp, 128 KB per SM) and
// by its own start for small ones, where short code counts.  Between events,
// against one 16-byte chunk pair per word with shuffles for the third chunk
// (80 KB of code): 512^3 52 against 55.5 us, 512x512x256 27 against 29.5 us,
// 301x287x173 with a label 15 against 19 us, 64^3 8.7 against 14.7 us, 48
// patches 18 against 27 us, 256 ragged pairs 1.025 against 1.040 ms (with each
// warp on a contiguous share of the CTA's run 1.043 ms).  64-word spans at 3
// CTAs per SM were 14 % slower at 512^3, with the next span's loads issued
// between the two masks' 37 %.
template <bool kLabel, bool kAligned, bool kAhead = false>
__global__ void __launch_bounds__(kPackThreads, kPackCtas) pack_kernel(const PairDesc* __restrict__ descs, int npairs,
                                                               long long ntiles, int label,
                                                               const __grid_constant__ PairDesc one, Ctl* ctl, uint32_t* zero, int nzero,
                                                               bool queued) {
    __shared__ uint32_t s_bits_all[kPackWarps][2][kBitWords];
    if (queued) cudaGridDependencySynchronize();  // placed as the kernel before it ends
    // nobody uses these before the next kernel
    if (ctl && blockIdx.x == 0 && threadIdx.x == 0) *ctl = Ctl{};
    for (int t = blockIdx.x * kPackThreads + threadIdx.x; t < nzero; t += gridDim.x * kPackThreads) zero[t] = 0u;
    const long long per = (ntiles + gridDim.x - 1) / gridDim.x;
    long long tile = (long long)blockIdx.x * per;
    const long long t_hi = min(ntiles, tile + per);
    if (tile >= t_hi) return;
    int pi = npairs == 1 ? 0 : pair_of_tile(descs, npairs, tile, false);
    uint32_t (*const s_bits)[kBitWords] = s_bits_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (;;) {  // the pairs of this CTA's run
        const PairDesc& P = descs ? descs[pi] : one;
        const PackWalk k = make_walk(P);
        const long long first = P.tile0;
        const long long end = pi + 1 < npairs ? min(t_hi, descs[pi + 1].tile0) : t_hi;
        PackAcc acc;
        unsigned t0 = (unsigned)((tile - first) * kPackTileWords) + (threadIdx.x >> 5) * kSpan;
        const unsigned t1 = min((unsigned)((end - first) * kPackTileWords), k.total);
        unsigned r = (t0 + lane) / k.wxf;
        unsigned w = t0 + lane - r * k.wxf;
        unsigned y = r % k.H;
        if constexpr (kAligned) pack_aligned<kLabel, kAhead>(k, t0, t1, r, w, y, acc, (unsigned)label);
#pragma unroll 1
        for (; !kAligned && t0 < t1; t0 += (unsigned)kPackTileWords) {
            const PackSpan n = locate(k, t0, __shfl_sync(0xffffffffu, r, 0), __shfl_sync(0xffffffffu, w, 0));
            uint4 c[2][kRounds];
            unsigned x[2];
#pragma unroll
            for (int m = 0; m < 2; ++m) load_chunks(k, n, m, c[m], x[m]);
            __syncwarp();  // the last span's bits have been read
#pragma unroll
            for (int m = 0; m < 2; ++m) put_bits<kLabel>(k, n, m, c[m], x[m], (unsigned)label, s_bits[m]);
            __syncwarp();
            put_words(k, n, r, w, y, acc, s_bits);
            k.next_span(r, w, y);  // this warp's span of the next tile
        }
        flush_acc(P.info, P.H, acc);
        tile = end;
        if (tile >= t_hi) break;
        ++pi;
    }
}

struct Domain {
    int ox, oy, oz, wv, h, d, wx0, wx, pitch;
};

// Bounding box of the domain, before any rounding of its first word: the
// 6-neighbour element uses the bounding box of A u B (x in whole words), the
// 18-neighbour element that box widened by one word in x and one row and
// plane in y and z, clipped to the volume.  Exactness: a shortest
// 6-neighbour path between two voxels of a box is monotone and stays in it.
// An 18-neighbour step (the 6 face neighbours, the 4 in-plane diagonals and
// the 8 corners) changes z by at most 1 and x and y together through the
// corners; between two voxels at offsets (a, b, c) a shortest path takes c
// z steps whose corners' x and y moves alternate around the needed offset,
// plus king moves in the plane, so it leaves the box of the two voxels by
// at most one voxel in x or y and never in z (where it would need two more
// z steps).  Where the widened box is clipped by the volume, the whole
// volume offers no detour on that side either.  (Without the margin the
// results differ: offset (0, 2, 2) takes the corners (1, 1, 1) and
// (-1, 1, 1), 2 steps, against 4 inside a box one voxel wide in x.)
struct DomainBox {
    int w0, w1, y0, y1, z0, z1;  // inclusive: word columns, rows, planes
};
__device__ __forceinline__ DomainBox domain_box(const PairDesc& P, const PairInfo& I) {
    DomainBox b{I.bb[0], I.bb[1], I.bb[2], I.bb[3], I.bb[4], I.bb[5]};
    if (P.se != 0) {
        const int wxf = (P.W + 31) >> 5;
        b.w0 = max(0, b.w0 - 1);
        b.w1 = min(wxf - 1, b.w1 + 1);
        b.y0 = max(0, b.y0 - 1);
        b.y1 = min(P.H - 1, b.y1 + 1);
        b.z0 = max(0, b.z0 - 1);
        b.z1 = min(P.D - 1, b.z1 + 1);
    }
    return b;
}

// The domain of a pair (quad: its first word rounded down to a multiple of
// 4, so that its rows start on 16-byte boundaries of the packed masks; any
// box inside the volume that contains the one above is as exact).
__device__ __forceinline__ Domain make_domain(const PairDesc& P, const PairInfo& I, bool quad) {
    const DomainBox b = domain_box(P, I);
    Domain m;
    m.wx0 = quad ? (b.w0 & ~3) : b.w0;  // word columns
    m.ox = 32 * m.wx0;
    m.wv = min(P.W, 32 * (b.w1 + 1)) - m.ox;
    m.oy = b.y0;
    m.h = b.y1 - b.y0 + 1;
    m.oz = b.z0;
    m.d = b.z1 - b.z0 + 1;
    m.wx = (m.wv + 31) >> 5;
    m.pitch = (m.wx + 3) & ~3;
    return m;
}

// Blocked kernel: can the domain start on a multiple of 4 words (its rows
// then start on 16-byte boundaries of the packed masks, which the kernel
// reads in place) without adding a brick column?
__device__ __forceinline__ bool blocked_in_place(const PairDesc& P, const PairInfo& I) {
    const DomainBox b = domain_box(P, I);
    const int w1 = b.w1 + 1;  // the domain's words end here (inside the volume)
    return (w1 - b.w0 + 3) / 4 == (w1 - (b.w0 & ~3) + 3) / 4;
}

__device__ __forceinline__ long long setup_tile(const PairDesc& P, long long tile_in_pair, Job* jobs,
                                                JobState* states, unsigned long long* queue0, Ctl* ctl, int g0,
                                                int bxw, int by, int bz, int mode, unsigned* s_base);

// 1D grid, block 256: CTAs stride over the tiles of all pairs
// (setup_tiles_of per pair); tile 0 of a pair also writes its job
// descriptors.  Modes:
//   kSetupOneStep         crop the packed masks into both ping-pong buffers
//                         and the uncovered-target array of each job
//   kSetupBlocked         the blocked kernel reads the packed masks in place
//                         when blocked_in_place, else crops of A and B (one
//                         pair: an extra brick column costs a whole
//                         latency-bound first iteration more than the copy)
//   kSetupBlockedCrop     crops of A and B (the packed masks are freed after
//                         set-up)
//   kSetupBlockedInPlace  the packed masks in place (batches: the copy costs
//                         more than the extra bricks)
__global__ void __launch_bounds__(256) setup_kernel(const PairDesc* __restrict__ descs, int npairs, long long ntiles,
                                                    Job* jobs, JobState* states, unsigned long long* queue0,
                                                    Ctl* ctl, int g0, int bxw, int by, int bz, int mode,
                                                    unsigned long long* zq1, unsigned long long* zq2, int nz,
                                                    const __grid_constant__ PairDesc one, PairDesc* desc_out) {
    __shared__ unsigned s_base;
    cudaGridDependencySynchronize();  // placed as the packing ends
    if (desc_out && blockIdx.x == 0 && threadIdx.x == 0) *desc_out = one;  // for the result decode
    int pi = -1;
    const long long G = gridDim.x;
    // the first nz slots of the two queues the first step does not read
    // (the dilation kernel reads a warp's next first entry early where a
    // slot is non-zero)
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nz; t += G * blockDim.x) {
        zq1[t] = 0ull;
        zq2[t] = 0ull;
    }
    // CTAs stride over the tiles: a pair's domain fills only the first of
    // its tiles, so contiguous runs would leave some CTAs without work
    for (long long tile = blockIdx.x; tile < ntiles; tile += G) {
        int np = pi < 0 ? pair_of_tile(descs, npairs, tile, true) : pi;
        while (np + 1 < npairs && descs[np + 1].stile0 <= tile) ++np;  // tiles only increase
        pi = np;
        const PairDesc& P = descs ? descs[pi] : one;
        const long long t0 = P.stile0;
        const long long need = setup_tile(P, tile - t0, jobs, states, queue0, ctl, g0, bxw, by, bz, mode,
                                          &s_base);
        // The pair's tiles from `need` on have nothing to do (the host sizes
        // the tiles for the largest domain and for copies that reading the
        // packed masks in place makes unnecessary): continue at this CTA's
        // first tile of the next pair.  CTA-uniform.
        if (tile - t0 + G >= need) {
            const long long next0 = pi + 1 < npairs ? descs[pi + 1].stile0 : ntiles;
            const long long first = next0 + ((((long long)blockIdx.x - next0) % G) + G) % G;  // >= tile + G
            tile = first - G;
        }
    }
}

// Returns the number of tiles of the pair that have work (descriptors,
// copies or queue entries): later tiles return at once.
__device__ __forceinline__ long long setup_tile(const PairDesc& P, long long tile_in_pair, Job* jobs,
                                                JobState* states, unsigned long long* queue0, Ctl* ctl, int g0,
                                                int bxw, int by, int bz, int mode, unsigned* s_base) {
    const PairInfo I = *P.info;
    const bool empty_a = I.n_a == 0, empty_b = I.n_b == 0;
    const unsigned long long rem[2] = {I.n_b - I.n_ab, I.n_a - I.n_ab};
    const long long cap = domain_cap_words(P.W, P.H, P.D);  // copying modes: the tiles cover [0, cap) words
    const long long ntiles_pair = setup_tiles_of(P.W, P.H, P.D, mode, bxw, by, bz);
    const long long w_lo = tile_in_pair * kTileWords, w_hi = min(cap, w_lo + kTileWords);
    const long long tid0 = threadIdx.x;
    const long long nthr = blockDim.x;
    const bool first = tile_in_pair == 0;
    const int kmax = P.kmax;
    // histograms are zeroed for every pair
    if (first)
        for (int j = 0; j < 2; ++j)
            for (int t = (int)tid0; t <= kmax; t += (int)nthr) P.hist[j][t] = 0ull;
    if (empty_a || empty_b) {
        if (first && tid0 == 0) {
            for (int j = 0; j < 2; ++j) {
                JobState& s = states[P.job0 + j];
                s.sum = 0; s.remaining = 0; s.bricks = 0; s.hd = 0; s.last_k = 0;
                s.status = (empty_a && empty_b) ? 0 : 1;  // HD_EMPTY_MASK
                s.active = 0;
                Job& J = jobs[P.job0 + j];
                J.nbx = J.nby = J.nbz = 0;
                J.epoch = P.epoch;
            }
        }
        return 1;
    }
    const bool one_step = mode == kSetupOneStep;
    const bool in_place = mode == kSetupBlockedInPlace || (mode == kSetupBlocked && blocked_in_place(P, I));
    const Domain m = make_domain(P, I, in_place);
    const int nbx = (m.wx + bxw - 1) / bxw, nby = (m.h + by - 1) / by, nbz = (m.d + bz - 1) / bz;
    const long long nbricks = (long long)nbx * nby * nbz;
    // crops of A and B (blocked kernel) live in the two jobs' U slots
    uint32_t* const crop[2] = {P.jb[0][2], P.jb[1][2]};
    if (first && tid0 == 0) {
        for (int j = 0; j < 2; ++j) {
            Job& J = jobs[P.job0 + j];
            J.buf[0] = P.jb[j][0];
            J.buf[1] = P.jb[j][1];
            J.U = one_step ? P.jb[j][2] : nullptr;
            if (in_place) {
                J.vol[0] = j == 0 ? P.pa : P.pb;
                J.vol[1] = j == 0 ? P.pb : P.pa;
                J.vpitch = packed_pitch(P.W);
                J.vh = P.H;
                J.vx0 = m.wx0;
                J.vy0 = m.oy;
                J.vz0 = m.oz;
            } else {
                J.vol[0] = crop[j];
                J.vol[1] = crop[1 - j];
                J.vpitch = m.pitch;
                J.vh = m.h;
                J.vx0 = J.vy0 = J.vz0 = 0;
            }
            J.hist = P.hist[j];
            J.wv = m.wv; J.h = m.h; J.d = m.d;
            J.wx = m.wx; J.pitch = m.pitch;
            const int tb = m.wv - 32 * (m.wx - 1);
            J.tailmask = tb >= 32 ? 0xffffffffu : ((1u << tb) - 1u);
            J.nbx = nbx; J.nby = nby; J.nbz = nbz;
            J.k0 = g0;
            J.kmax = kmax;
            J.ox = m.ox; J.oy = m.oy; J.oz = m.oz;
            J.tw = (P.W + 31) >> 5; J.th = (P.H + 31) >> 5;
            J.brick0 = P.brick0[j];
            J.tstamp = P.tstamp[j];
            J.tcount = P.tcount[j];
            J.epoch = P.epoch;
            JobState& s = states[P.job0 + j];
            s.sum = 0; s.remaining = rem[j]; s.bricks = 0; s.hd = 0; s.last_k = 0; s.status = 0;
            s.active = rem[j] > 0 ? 1 : 0;
            if (rem[j] > 0) atomicAdd(&ctl->jobs_active, 1);
        }
    }
    // Crop copy.  Job 0 dilates A and must cover B; job 1 dilates B and covers A.
    const bool act0 = rem[0] > 0, act1 = rem[1] > 0;
    const long long words_all = (one_step || !in_place) ? (long long)m.pitch * m.h * m.d : 0;
    const long long words = min(words_all, w_hi);
    const int vpitch = packed_pitch(P.W);
    for (long long t = w_lo + tid0; t < words; t += nthr) {
        // domain word index < 2^31: 32-bit divisions.  Rows of pitch words
        // for the one-step kernel, columns of 4 words for the blocked one
        const unsigned tu = (unsigned)t;
        unsigned r;
        int w, yl, zl;
        if (one_step) {
            r = tu / (unsigned)m.pitch;
            w = (int)(tu - r * (unsigned)m.pitch);
            zl = (int)(r / (unsigned)m.h);
            yl = (int)(r - (unsigned)zl * (unsigned)m.h);
        } else {
            r = tu >> 2;
            const unsigned c = r / (unsigned)m.h, nq = (unsigned)m.pitch >> 2;
            yl = (int)(r - c * (unsigned)m.h);
            zl = (int)(c / nq);
            w = (int)(4u * (c - (unsigned)zl * nq) + (tu & 3u));
        }
        uint32_t a = 0, b = 0;
        if (w < m.wx) {
            const int wf = m.wx0 + w;
            const long long src = ((long long)(m.oz + zl) * vpitch + (wf & ~3)) * P.H + 4ll * (m.oy + yl) + (wf & 3);
            a = __ldg(P.pa + src);
            b = __ldg(P.pb + src);
        }
        if (one_step) {
            if (act0) {
                P.jb[0][0][t] = a;
                P.jb[0][1][t] = a;
                P.jb[0][2][t] = b & ~a;
            }
            if (act1) {
                P.jb[1][0][t] = b;
                P.jb[1][1][t] = b;
                P.jb[1][2][t] = a & ~b;
            }
        } else {  // source and target of both jobs
            crop[0][t] = a;
            crop[1][t] = b;
        }
    }
    // First step of each active job: every brick of its domain.  The
    // bricks go to the pair's first tiles, at least 256 per tile, and each
    // such tile reserves its queue entries with one atomic per job.
    const long long b_even = (long long)(((unsigned)nbricks + (unsigned)ntiles_pair - 1u) / (unsigned)ntiles_pair);
    const long long b_per = mode == kSetupBlockedInPlace ? kSetupBricks
                                                          : (b_even > 256 ? b_even : 256);  // < 2^31 bricks, tiles
    const long long b_lo = tile_in_pair * b_per, b_hi = min(nbricks, b_lo + b_per);
    const long long need = max(max((words_all + kTileWords - 1) / kTileWords, (nbricks + b_per - 1) / b_per), 1ll);
    if (b_lo >= b_hi) return need;  // CTA-uniform
    for (int j = 0; j < 2; ++j) {
        if (!(j == 0 ? act0 : act1)) continue;
        if (tid0 == 0) *s_base = atomicAdd(&ctl->qcount[g0 % 3], (unsigned)(b_hi - b_lo));
        __syncthreads();
        const unsigned base = *s_base;
        for (long long t = b_lo + tid0; t < b_hi; t += nthr)
            queue0[base + (unsigned)(t - b_lo)] = make_entry(P.epoch, (uint32_t)(P.job0 + j), (uint32_t)t);
        __syncthreads();  // s_base is written again next
    }
    return need;
}

// Start values of each pair's counts and bounding box (one thread per pair).
__global__ void info_init_kernel(const PairDesc* __restrict__ descs, int npairs, PairDesc* __restrict__ slot_descs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npairs) return;
    if (slot_descs) slot_descs[descs[i].job0 / 2] = descs[i];  // serving: the slot's copy for the result decode
    *descs[i].info = pair_info_start();
}

// Serving: retire finished pairs' slots.  list holds (slot, epoch) pairs: the
// slot's jobs take the new epoch (queue entries still listed for them are
// dropped) and the slot's descriptor copy is marked unused (info = null).
__global__ void retire_kernel(Job* __restrict__ jobs, PairDesc* __restrict__ slot_descs,
                              const uint32_t* __restrict__ list, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t slot = list[2 * i], ep = list[2 * i + 1];
    jobs[2 * slot].epoch = ep;
    jobs[2 * slot + 1].epoch = ep;
    slot_descs[slot].info = nullptr;
}

// Instrumented runs: zero the per-tile stamps and per-step tile counters.
__global__ void zero_i32_kernel(int32_t* p, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x)
        p[t] = 0;
}

// Per-voxel maps: -1 outside the mask, 0 on the overlap, and (filled later by
// the dilation) the distance on voxels of one mask outside the other.
// Four voxels per thread and round, kMapRounds rounds in flight; kVec: masks
// aligned to 4 bytes, maps to 16 (any others, and the last voxels: one by one).
// Bound by the maps' writes (the masks come from L2): 256^3 20 us (6.7 TB/s)
// against 33.5 us with one voxel per thread and round; 1, 2, 8 rounds or 4 CTAs
// per SM the same.
constexpr int kMapThreads = 256, kMapRounds = 4, kMapGrid = 8 * 152;  // 8 CTAs per SM of GB300
template <bool kVec>
__global__ void __launch_bounds__(kMapThreads) map_init_kernel(const __grid_constant__ PairDesc P, int32_t* __restrict__ map_a,
                                                               int32_t* __restrict__ map_b, int label) {
    const long long n = (long long)P.W * P.H * P.D, quads = kVec ? n / 4 : 0;
    const uint32_t pat = (uint32_t)label * 0x01010101u;
    const long long step = (long long)gridDim.x * kMapThreads, first = (long long)blockIdx.x * kMapThreads + threadIdx.x;
    auto quad = [](uint32_t v) {  // four signed bytes
        return make_int4((int8_t)v, (int8_t)(v >> 8), (int8_t)(v >> 16), (int8_t)(v >> 24));
    };
    for (long long t = first; t < quads; t += kMapRounds * step) {
        uint32_t a[kMapRounds], b[kMapRounds];
#pragma unroll
        for (int r = 0; r < kMapRounds; ++r) {
            const bool in = t + r * step < quads;
            a[r] = in ? __ldg((const uint32_t*)P.a + t + r * step) : 0u;
            b[r] = in ? __ldg((const uint32_t*)P.b + t + r * step) : 0u;
        }
#pragma unroll
        for (int r = 0; r < kMapRounds; ++r) {
            if (t + r * step >= quads) break;
            const uint32_t fa = label ? __vcmpeq4(a[r], pat) : __vcmpne4(a[r], 0u);
            const uint32_t fb = label ? __vcmpeq4(b[r], pat) : __vcmpne4(b[r], 0u);
            // -2: to be filled by the dilation
            ((int4*)map_a)[t + r * step] = quad(~fa | (~fb & 0xfefefefeu));
            ((int4*)map_b)[t + r * step] = quad(~fb | (~fa & 0xfefefefeu));
        }
    }
    for (long long t = 4 * quads + first; t < n; t += step) {
        const bool a = label ? P.a[t] == label : P.a[t] != 0, b = label ? P.b[t] == label : P.b[t] != 0;
        map_a[t] = a ? (b ? 0 : -2) : -1;
        map_b[t] = b ? (a ? 0 : -2) : -1;
    }
}

}  // namespace hdk

// ---- launch wrappers (called from the host orchestration) -----------------
namespace hdk {

namespace {
// A launch whose CTAs may be placed as the stream's kernel before it ends;
// the kernel waits for that one's results itself.
template <class... P, class... A>
cudaError_t launch_early(void (*kernel)(P...), unsigned grid, int threads, cudaStream_t s, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    return cudaLaunchKernelEx(&c, kernel, args...);
}
}  // namespace

cudaError_t launch_pack(const PairDesc* d_descs, int npairs, long long ntiles, int grid, int label, int sms,
                        cudaStream_t s, const PairDesc* one, Ctl* ctl, uint32_t* zero, int nzero, bool queued) {
    // a single pair of 32-byte aligned words takes the kernel without the bit stream
    const PairDesc P = one ? *one : PairDesc{};
    const bool aligned = one && (P.W & 31) == 0 && (((uintptr_t)P.a | (uintptr_t)P.b) & 31) == 0;
    const int v = (label ? 1 : 0) + (aligned ? (sms > 0 ? 4 : 2) : 0);
    using Kernel = void (*)(const PairDesc*, int, long long, int, PairDesc, Ctl*, uint32_t*, int, bool);
    static const Kernel kernels[6] = {pack_kernel<false, false>,      pack_kernel<true, false>,
                                      pack_kernel<false, true>,       pack_kernel<true, true>,
                                      pack_kernel<false, true, true>, pack_kernel<true, true, true>};
    const Kernel fn = kernels[v];
    // one wave of resident CTAs (per device and variant, from the occupancy calculator)
    static int resident[6][64] = {{0}};
    static int per_sm_of[6][64] = {{0}};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && resident[v][dev] == 0) {
        int per_sm = 0, sms_dev = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kPackThreads, 0);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms_dev, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        per_sm_of[v][dev] = std::max(1, per_sm);
        resident[v][dev] = std::max(1, per_sm) * std::max(1, sms_dev);
    }
    if (dev < 64) grid = sms > 0 ? per_sm_of[v][dev] * sms : resident[v][dev];
    if (grid > ntiles) grid = (int)ntiles;
    if (grid < 1) grid = 1;
    // Asynchronous calls on one stream: the CTAs are placed as the kernel before
    // ends (six 301x287x173 pairs 202 -> 189 us).  A blocking call's stream is
    // idle, and this form of launch takes the host 1 us longer.
    if (!queued) {
        fn<<<grid, kPackThreads, 0, s>>>(d_descs, npairs, ntiles, label, P, ctl, zero, nzero, queued);
        return cudaGetLastError();
    }
    return launch_early(fn, (unsigned)grid, kPackThreads, s, d_descs, npairs, ntiles, label, P, ctl, zero, nzero, queued);
}

cudaError_t launch_setup(const PairDesc* d_descs, int npairs, long long ntiles, int sms, Job* jobs,
                         JobState* states, unsigned long long* queue0, Ctl* ctl, int g0, int bxw, int by, int bz,
                         int mode, cudaStream_t s, unsigned long long* zq1, unsigned long long* zq2, int nz,
                         const PairDesc* one, PairDesc* desc_out, bool early) {
    // one wave of resident CTAs (per device, from the occupancy calculator):
    // CTAs whose tiles have nothing to do leave at once, later waves would
    // only add their scheduling
    static int per_sm_of[64] = {0};
    static int sms_of[64] = {0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int per_sm = 8, nsm = sms > 0 ? sms : 1;
    if (dev < 64) {
        if (per_sm_of[dev] == 0) {
            int occ = 0, sms_dev = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, reinterpret_cast<const void*>(&setup_kernel), 256,
                                                              0);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms_dev, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return e;
            per_sm_of[dev] = std::max(1, occ);
            sms_of[dev] = std::max(1, sms_dev);
        }
        per_sm = per_sm_of[dev];
        if (sms <= 0) nsm = sms_of[dev];
    }
    long long grid = std::min<long long>((long long)per_sm * nsm, ntiles);
    if (grid < 1) grid = 1;
    const PairDesc P = one ? *one : PairDesc{};
    if (!zq1 || !zq2) nz = 0;
    if (!early) {
        setup_kernel<<<(unsigned)grid, 256, 0, s>>>(d_descs, npairs, ntiles, jobs, states, queue0, ctl, g0, bxw, by, bz, mode,
                                                    zq1, zq2, nz, P, desc_out);
        return cudaGetLastError();
    }
    // (117x131x75 63.5 -> 62 us a call)
    return launch_early(setup_kernel, (unsigned)grid, 256, s, d_descs, npairs, ntiles, jobs, states, queue0, ctl, g0, bxw, by,
                        bz, mode, zq1, zq2, nz, P, desc_out);
}

cudaError_t launch_info_init(const PairDesc* d_descs, int npairs, cudaStream_t s, PairDesc* slot_descs) {
    if (npairs <= 0) return cudaSuccess;
    info_init_kernel<<<(npairs + 255) / 256, 256, 0, s>>>(d_descs, npairs, slot_descs);
    return cudaGetLastError();
}

cudaError_t launch_retire(Job* jobs, PairDesc* slot_descs, const uint32_t* list, int n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    retire_kernel<<<(n + 127) / 128, 128, 0, s>>>(jobs, slot_descs, list, n);
    return cudaGetLastError();
}

cudaError_t launch_zero_i32(int32_t* p, long long n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    long long blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    zero_i32_kernel<<<(int)blocks, 256, 0, s>>>(p, n);
    return cudaGetLastError();
}

cudaError_t launch_map_init(const PairDesc& one, int32_t* map_a, int32_t* map_b, int label, cudaStream_t s) {
    const long long n = (long long)one.W * one.H * one.D;
    const bool vec = (((uintptr_t)one.a | (uintptr_t)one.b) & 3) == 0 && (((uintptr_t)map_a | (uintptr_t)map_b) & 15) == 0;
    const long long blocks = std::min<long long>((n + 4 * kMapThreads - 1) / (4 * kMapThreads), kMapGrid);
    if (vec) map_init_kernel<true><<<(int)blocks, kMapThreads, 0, s>>>(one, map_a, map_b, label);
    else map_init_kernel<false><<<(int)blocks, kMapThreads, 0, s>>>(one, map_a, map_b, label);
    return cudaGetLastError();
}

}  // namespace hdk
