// prim.cuh -- device-wide primitives of the build path: prefix sums, stable
// LSD radix sort of (key, payload) pairs, stream compaction, segmented
// sums and the per-row column sort of a CSR block.
//
// They replace the library sorts and scans used before, with two choices
// made for this workload:
//   * the radix sort visits only the bits a key can use: a determinant
//     word holds n_orb bits, so a (alpha, beta) key of a 13-orbital system
//     takes 4 passes of 8 bits instead of 16, and a 30-orbital one 8;
//   * the row sort keeps a block per row in shared memory (bitonic network)
//     and sends only rows longer than a block holds through the global sort.
//
// Radix sort: LSD passes of 8 bits over (one key word, position) pairs; keys of
// several words are packed into one when their significant bits fit 64, else
// sorted word by word through the positions, and the keys and payloads are
// gathered once at the end.
//   * Up to kSmallSort keys: one block sorts them in shared memory, one launch
//     for all passes (a pass is about 1 us there; through the grid its three
//     launches alone take longer).
//   * More: per pass k_radix_hist counts the digits of each tile of 4096 keys
//     (warp-aggregated with __match_any_sync), k_radix_rows prefix-sums every
//     digit's row of tile counts, and k_radix_scatter ranks every key inside
//     its tile -- each warp walks its keys in rounds of 32 in input order, a
//     key's rank is the count of its digit in earlier rounds plus its lanes
//     before it in the round, and warps are offset per digit --, orders the
//     tile in shared memory and writes every digit's run with neighbouring
//     lanes (a pass moves 2 (key + 4) bytes per key; unordered stores cost it
//     twice that in partial sectors).
// Equal digits keep their input order, so the passes compose into a stable
// sort.  Measured: a pass over 4.35e6 (u64, u32)
// pairs 78 us before, 61 now (the scatter 45 -> 38); 2,241 keys of 26 bits 90 us
// in 30 launches before, 13.5 in one now; 4.2e6 keys of 256 bits, 200 of them
// significant, 3.3 ms before, 1.9 now.
//
// Scan: three phases over tiles of 2048 items (tile sums, one-block scan of
// the tile sums, tile scans from their offsets), or one block that carries its
// sum from tile to tile when there are at most kScanTiles.  Every phase reads
// its items before it writes, so in == out is allowed.
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace dnq {
namespace prim {
// Internal linkage: every translation unit that includes this header gets
// its own instances of the kernels.
namespace {

constexpr int kThreads = 256;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;   // 2048
constexpr int kWarps = kThreads / 32;

__device__ __forceinline__ unsigned lt_mask() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---------------------------------------------------------------------------
// Block-wide exclusive scan of one value per thread (256 threads); returns
// the exclusive prefix and writes the block total to *total.
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ T block_exclusive(T v, T* total) {
    __shared__ T warp_tot[kWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (w == 0) {
        T t = lane < kWarps ? warp_tot[lane] : T(0);
        T ti = t;
#pragma unroll
        for (int o = 1; o < kWarps; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += y;
        }
        if (lane < kWarps) warp_tot[lane] = ti - t;   // exclusive per warp
        if (lane == kWarps - 1) *total = ti;
    }
    __syncthreads();
    const T r = warp_tot[w] + incl - v;
    __syncthreads();
    return r;
}

template <class Tin, class Tout>
__global__ void __launch_bounds__(kThreads) k_tile_sums(const Tin* in, i64 n, Tout* sums) {
    const i64 base = (i64)blockIdx.x * kTile;
    Tout v = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const i64 p = base + (i64)i * kThreads + threadIdx.x;
        if (p < n) v += (Tout)in[p];
    }
    __shared__ Tout tot;
    block_exclusive<Tout>(v, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// One block: exclusive scan of m tile sums in place, chunk by chunk.
template <class T>
__global__ void __launch_bounds__(kThreads) k_scan_sums(T* sums, i64 m) {
    __shared__ T tot;
    T carry = 0;
    for (i64 c0 = 0; c0 < m; c0 += kThreads) {
        const i64 p = c0 + threadIdx.x;
        const T v = p < m ? sums[p] : T(0);
        const T e = block_exclusive<T>(v, &tot);
        if (p < m) sums[p] = carry + e;
        carry += tot;
        __syncthreads();
    }
}

// Each thread scans kItems consecutive items of its tile.
template <class Tin, class Tout, bool Inclusive>
__global__ void __launch_bounds__(kThreads) k_scan_tiles(const Tin* in, Tout* out, i64 n,
                                                         const Tout* tile_off) {
    const i64 base = (i64)blockIdx.x * kTile + (i64)threadIdx.x * kItems;
    Tout v[kItems];
    Tout sum = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const i64 p = base + i;
        v[i] = p < n ? (Tout)in[p] : Tout(0);
        sum += v[i];
    }
    __shared__ Tout tot;
    Tout run = tile_off[blockIdx.x] + block_exclusive<Tout>(sum, &tot);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const i64 p = base + i;
        if (Inclusive) run += v[i];
        if (p < n) out[p] = run;
        if (!Inclusive) run += v[i];
    }
}

inline i64 tiles_of(i64 n) { return (n + kTile - 1) / kTile; }

// A few tiles by one block: three launches take longer than its tile after
// tile (about 1.2 us each) up to there.
constexpr i64 kScanTiles = 4;
template <class Tin, class Tout, bool Inclusive>
__global__ void __launch_bounds__(kThreads) k_scan_few(const Tin* in, Tout* out, i64 n) {
    __shared__ Tout tot;
    Tout carry = 0;
    for (i64 b = 0; b < n; b += kTile) {
        const i64 base = b + (i64)threadIdx.x * kItems;
        Tout v[kItems];
        Tout sum = 0;
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            const i64 p = base + i;
            v[i] = p < n ? (Tout)in[p] : Tout(0);
            sum += v[i];
        }
        Tout run = carry + block_exclusive<Tout>(sum, &tot);
        carry += tot;
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            const i64 p = base + i;
            if (Inclusive) run += v[i];
            if (p < n) out[p] = run;
            if (!Inclusive) run += v[i];
        }
        __syncthreads();   // tot is read before the next tile writes it
    }
}

// Temporary bytes of a scan of n items with Tout sums.
template <class Tout>
inline size_t scan_tmp_bytes(i64 n) {
    return (size_t)std::max<i64>(1, tiles_of(n)) * sizeof(Tout);
}

// out[i] = sum of in[0..i) (exclusive) or in[0..i] (inclusive).  tmp: at
// least scan_tmp_bytes<Tout>(n) bytes, or null to allocate it on s.
template <class Tin, class Tout, bool Inclusive = false>
void scan(const Tin* in, Tout* out, i64 n, cudaStream_t s, void* tmp = nullptr) {
    if (n <= 0) return;
    const i64 nt = tiles_of(n);
    if (nt <= kScanTiles) {
        k_scan_few<Tin, Tout, Inclusive><<<1, kThreads, 0, s>>>(in, out, n);
        DNQ_CHECK_LAUNCH();
        return;
    }
    DBuf<Tout> own;
    Tout* sums = static_cast<Tout*>(tmp);
    if (!sums) {
        own.alloc(nt, s);
        sums = own.p;
    }
    k_tile_sums<Tin, Tout><<<(unsigned)nt, kThreads, 0, s>>>(in, n, sums);
    DNQ_CHECK_LAUNCH();
    k_scan_sums<Tout><<<1, kThreads, 0, s>>>(sums, nt);
    DNQ_CHECK_LAUNCH();
    k_scan_tiles<Tin, Tout, Inclusive><<<(unsigned)nt, kThreads, 0, s>>>(in, out, n, sums);
    DNQ_CHECK_LAUNCH();
}

template <class Tin, class Tout>
void scan_inclusive(const Tin* in, Tout* out, i64 n, cudaStream_t s, void* tmp = nullptr) {
    scan<Tin, Tout, true>(in, out, n, s, tmp);
}

// ---------------------------------------------------------------------------
// Radix sort
// ---------------------------------------------------------------------------

// Words of a key, most significant first.
template <class K>
struct RadixKey;

template <>
struct RadixKey<u32> {
    static constexpr int W = 1;
    __device__ __forceinline__ static u64 word(const u32& k, int) { return k; }
};
template <>
struct RadixKey<u64> {
    static constexpr int W = 1;
    __device__ __forceinline__ static u64 word(const u64& k, int) { return k; }
};
// (alpha, beta) determinant keys: alpha word first.
template <>
struct RadixKey<ulonglong2> {
    static constexpr int W = 2;
    __device__ __forceinline__ static u64 word(const ulonglong2& k, int i) {
        return i == 0 ? k.x : k.y;
    }
};

// The digits of a sort: (word, shift) of every pass, least significant first.
constexpr int kMaxPasses = 40;
struct RadixPasses {
    int n = 0;
    unsigned char word[kMaxPasses], shift[kMaxPasses];
    // 8-bit windows over the set bits of `mask` in word w
    void add(int w, u64 mask) {
        while (mask) {
            const int sh = __builtin_ctzll(mask);
            require(n < kMaxPasses, DNQ_ERR_INVALID, "too many radix passes");
            word[n] = (unsigned char)w;
            shift[n] = (unsigned char)sh;
            ++n;
            mask &= sh + 8 >= 64 ? 0ull : ~0ull << (sh + 8);
        }
    }
};

// Word i of key p, narrowed to the word type of its passes.
template <class K>
__device__ __forceinline__ u64 key_word(const K* k, i64 p, int w) {
    return RadixKey<K>::word(k[p], w);
}

constexpr int kSmallThreads = 512;
constexpr int kSmallItems = 7;
constexpr int kSmallSort = kSmallThreads * kSmallItems;   // 3584 keys: 45 KB shared
constexpr int kSmallWarps = kSmallThreads / 32;

// All passes of up to kSmallSort keys.  The current word of every key stays
// at its input place in shared memory; the passes permute the places.
template <class K, class P>
__global__ void __launch_bounds__(kSmallThreads)
k_radix_small(const K* kin, const P* pin, K* kout, P* pout, int n, RadixPasses R) {
    __shared__ u64 sk[kSmallSort];
    __shared__ u16 si[kSmallSort];
    __shared__ u16 wh[kSmallWarps][256];
    __shared__ u32 dsum[8];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int base = w * (kSmallItems * 32) + lane;
    u16 at[kSmallItems];   // input place of this thread's items
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) at[i] = (u16)(base + 32 * i);
    int cur = -1;
    for (int q = 0; q < R.n; ++q) {
        const int word = R.word[q], shift = R.shift[q];
        if (word != cur) {
            cur = word;
            for (int p = tid; p < n; p += kSmallThreads) sk[p] = key_word(kin, p, word);
        }
        for (int t = tid; t < kSmallWarps * 128; t += kSmallThreads)
            reinterpret_cast<u32*>(&wh[0][0])[t] = 0u;
        __syncthreads();
        u32 dg[kSmallItems], rk[kSmallItems];
#pragma unroll
        for (int i = 0; i < kSmallItems; ++i) {
            const bool ok = base + 32 * i < n;
            dg[i] = ok ? (u32)(sk[at[i]] >> shift) & 0xffu : 256u;
            const unsigned m = __match_any_sync(0xffffffffu, dg[i]);
            const u32 before = ok ? wh[w][dg[i]] : 0u;
            rk[i] = before + __popc(m & lt_mask());
            __syncwarp();
            if (ok && (m & lt_mask()) == 0) wh[w][dg[i]] = (u16)(before + __popc(m));
            __syncwarp();
        }
        __syncthreads();
        u32 tot = 0, incl = 0;
        if (tid < 256) {   // per digit: warps' counts -> offsets in the digit
#pragma unroll
            for (int k = 0; k < kSmallWarps; ++k) {
                const u32 t = wh[k][tid];
                wh[k][tid] = (u16)tot;
                tot += t;
            }
            incl = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u32 y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) dsum[w] = incl;
        }
        __syncthreads();
        if (tid < 256) {   // start of the digit
            u32 st = incl - tot;
            for (int k = 0; k < w; ++k) st += dsum[k];
#pragma unroll
            for (int k = 0; k < kSmallWarps; ++k) wh[k][tid] = (u16)(wh[k][tid] + st);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSmallItems; ++i)
            if (dg[i] < 256u) si[wh[w][dg[i]] + rk[i]] = at[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSmallItems; ++i)
            if (base + 32 * i < n) at[i] = si[base + 32 * i];
    }
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) {
        const int p = base + 32 * i;
        if (p >= n) continue;
        if (kout) kout[p] = kin[at[i]];
        if (pout) pout[p] = pin ? pin[at[i]] : (P)at[i];
    }
}

constexpr int kRadixItems = 16;
constexpr int kRadixTile = kThreads * kRadixItems;   // 4096

template <class T>
__global__ void __launch_bounds__(kThreads) k_radix_hist(const T* keys, i64 n, int shift,
                                                         u32* hist, i64 ntiles) {
    __shared__ u32 h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const i64 base = (i64)blockIdx.x * kRadixTile;
    T k[kRadixItems];
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i) {
        const i64 p = base + (i64)i * kThreads + threadIdx.x;
        k[i] = p < n ? keys[p] : T(0);
    }
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i) {
        const bool ok = base + (i64)i * kThreads + threadIdx.x < n;
        const u32 d = ok ? (u32)(k[i] >> shift) & 0xffu : 256u;
        const unsigned m = __match_any_sync(0xffffffffu, d);
        if (ok && (m & lt_mask()) == 0) atomicAdd(&h[d], (u32)__popc(m));
    }
    __syncthreads();
    hist[(i64)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Block d: exclusive prefix sums of digit d's tile counts, in place, and
// their total.
__global__ void __launch_bounds__(kThreads) k_radix_rows(u32* hist, i64 ntiles, u32* total) {
    __shared__ u32 tot;
    u32* row = hist + (i64)blockIdx.x * ntiles;
    u32 carry = 0;
    for (i64 c0 = 0; c0 < ntiles; c0 += kThreads * 4) {
        u32 v[4], sum = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const i64 p = c0 + (i64)threadIdx.x * 4 + i;
            v[i] = p < ntiles ? row[p] : 0u;
            sum += v[i];
        }
        u32 run = carry + block_exclusive<u32>(sum, &tot);
        carry += tot;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const i64 p = c0 + (i64)threadIdx.x * 4 + i;
            if (p < ntiles) row[p] = run;
            run += v[i];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

// One pass.  pin == null gives each key's place; pout == null moves keys only.
template <class T>
__global__ void __launch_bounds__(kThreads)
k_radix_scatter(const T* kin, const u32* pin, T* kout, u32* pout, i64 n, int shift,
                const u32* offs, const u32* total, i64 ntiles) {
    __shared__ T stage[kRadixTile];
    __shared__ u16 wh[kWarps][256];
    __shared__ u32 dst[256];   // global place of the digit's first key, less its place in the tile
    __shared__ u32 tot;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int t = threadIdx.x; t < kWarps * 128; t += kThreads)
        reinterpret_cast<u32*>(&wh[0][0])[t] = 0u;
    const i64 tile0 = (i64)blockIdx.x * kRadixTile;
    const int m_tile = (int)min((i64)kRadixTile, n - tile0);
    const int base = w * (kRadixItems * 32) + lane;
    T k[kRadixItems];
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i)
        k[i] = base + 32 * i < m_tile ? kin[tile0 + base + 32 * i] : T(0);
    __syncthreads();
    u16 rk[kRadixItems];
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i) {
        const bool ok = base + 32 * i < m_tile;
        const u32 d = ok ? (u32)(k[i] >> shift) & 0xffu : 256u;
        const unsigned m = __match_any_sync(0xffffffffu, d);
        const u32 before = ok ? wh[w][d] : 0u;
        rk[i] = (u16)(before + __popc(m & lt_mask()));
        __syncwarp();
        if (ok && (m & lt_mask()) == 0) wh[w][d] = (u16)(before + __popc(m));
        __syncwarp();
    }
    __syncthreads();
    {   // per digit: warps' counts -> places in the tile, and where it goes
        const int d = threadIdx.x;
        u32 acc = 0;
#pragma unroll
        for (int q = 0; q < kWarps; ++q) {
            const u32 t = wh[q][d];
            wh[q][d] = (u16)acc;
            acc += t;
        }
        const u32 start = block_exclusive<u32>(acc, &tot);       // in the tile
        const u32 below = block_exclusive<u32>(total[d], &tot);  // keys of lower digits
#pragma unroll
        for (int q = 0; q < kWarps; ++q) wh[q][d] = (u16)(wh[q][d] + start);
        dst[d] = below + offs[(i64)d * ntiles + blockIdx.x] - start;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i) {
        if (base + 32 * i >= m_tile) continue;
        rk[i] = (u16)(rk[i] + wh[w][(u32)(k[i] >> shift) & 0xffu]);   // place in the tile
        stage[rk[i]] = k[i];
    }
    __syncthreads();
    u32 to[kRadixItems];
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i) {
        const int l = i * kThreads + threadIdx.x;
        if (l >= m_tile) continue;
        const T key = stage[l];
        to[i] = dst[(u32)(key >> shift) & 0xffu] + (u32)l;
        kout[to[i]] = key;
    }
    if (!pout) return;
    u32 pl[kRadixItems];
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i) {
        const i64 p = tile0 + base + 32 * i;
        if (base + 32 * i < m_tile) pl[i] = pin ? pin[p] : (u32)p;
    }
    __syncthreads();
    u32* sp = reinterpret_cast<u32*>(stage);
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i)
        if (base + 32 * i < m_tile) sp[rk[i]] = pl[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kRadixItems; ++i) {
        const int l = i * kThreads + threadIdx.x;
        if (l < m_tile) pout[to[i]] = sp[l];
    }
}

template <class K, class P>
__global__ void k_copy_pairs(const K* kin, const P* pin, K* kout, P* pout, i64 n) {
    for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < n;
         t += (i64)gridDim.x * blockDim.x) {
        kout[t] = kin[t];
        if (pout) pout[t] = pin ? pin[t] : (P)t;
    }
}

// out[t] = word w of key at[t] (at == null: key t); with w < 0 all words of a
// two-word key packed as word 0 << lo_bits | word 1, both masked.
template <class K>
__global__ void k_radix_word(const K* k, const u32* at, i64 n, int w, int hi_bits, int lo_bits,
                             u64* out) {
    for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < n;
         t += (i64)gridDim.x * blockDim.x) {
        const i64 p = at ? (i64)at[t] : t;
        out[t] = w >= 0 ? key_word(k, p, w)
                        : ((key_word(k, p, 0) & low_mask(hi_bits)) << lo_bits) |
                              (key_word(k, p, 1) & low_mask(lo_bits));
    }
}

template <class K, class P>
__global__ void k_radix_gather(const K* kin, const P* pin, const u32* at, i64 n, K* kout,
                               P* pout) {
    for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < n;
         t += (i64)gridDim.x * blockDim.x) {
        const u32 p = at[t];
        kout[t] = kin[p];
        if (pout) pout[t] = pin ? pin[p] : (P)p;
    }
}

// The passes of R (one word) over n (key, u32) pairs; the result ends in
// kout / pout (pout null: keys only).
template <class T>
void radix_passes(const T* kin, const u32* pin, T* kout, u32* pout, i64 n, const RadixPasses& R,
                  cudaStream_t s) {
    const i64 nt = (n + kRadixTile - 1) / kRadixTile;
    DBuf<T> kt(R.n > 1 ? n : 0, s);
    DBuf<u32> pt((R.n > 1 && pout) ? n : 0, s);
    DBuf<u32> hist(256 * nt, s), total(256, s);
    const T* ksrc = kin;
    const u32* psrc = pin;
    for (int q = 0; q < R.n; ++q) {
        const bool to_out = ((R.n - 1 - q) & 1) == 0;
        T* kdst = to_out ? kout : kt.p;
        u32* pdst = pout ? (to_out ? pout : pt.p) : nullptr;
        k_radix_hist<T><<<(unsigned)nt, kThreads, 0, s>>>(ksrc, n, R.shift[q], hist.p, nt);
        DNQ_CHECK_LAUNCH();
        k_radix_rows<<<256, kThreads, 0, s>>>(hist.p, nt, total.p);
        DNQ_CHECK_LAUNCH();
        k_radix_scatter<T><<<(unsigned)nt, kThreads, 0, s>>>(ksrc, psrc, kdst, pdst, n,
                                                             R.shift[q], hist.p, total.p, nt);
        DNQ_CHECK_LAUNCH();
        ksrc = kdst;
        psrc = pdst;
    }
}

// Stable sort of n (key, payload) pairs by key, ascending; n < 2^32.
// mask[i] = significant bits of key word i (most significant word first; the
// other bits of the word must be equal in all keys).  pout == null sorts keys
// only; pin == null with a payload output gives each key's input position.
// kin != kout.
template <class K, class P>
void radix_sort_masked(const K* kin, K* kout, const P* pin, P* pout, i64 n, const u64* mask,
                       cudaStream_t s) {
    if (n <= 0) return;
    require(n < (i64)0xffffffffll, DNQ_ERR_OVERFLOW, "radix sort of 2^32 or more keys");
    constexpr int W = RadixKey<K>::W;
    const unsigned grid = (unsigned)std::min<i64>((n + 255) / 256, 1 << 20);
    RadixPasses all;
    for (int i = W - 1; i >= 0; --i) all.add(i, mask[i]);   // least significant word first
    if (all.n == 0) {
        k_copy_pairs<K, P><<<grid, 256, 0, s>>>(kin, pin, kout, pout, n);
        DNQ_CHECK_LAUNCH();
        return;
    }
    if (n <= kSmallSort) {
        k_radix_small<K, P><<<1, kSmallThreads, 0, s>>>(kin, pin, kout, pout, (int)n, all);
        DNQ_CHECK_LAUNCH();
        return;
    }
    if constexpr (W == 1) {
        if constexpr (std::is_same<P, u32>::value) {
            radix_passes<K>(kin, pin, kout, pout, n, all, s);
            return;
        }
    }
    // several words, or another payload: positions by one word after the other
    DBuf<u32> at(n, s), at2(n, s);
    DBuf<u64> kw(n, s), kw2(n, s);
    u32 *cur = nullptr, *next = at.p;
    auto by_word = [&](int w, int hi_bits, int lo_bits, u64 m) {
        if (!m) return;
        RadixPasses R;
        R.add(0, m);
        k_radix_word<K><<<grid, 256, 0, s>>>(kin, cur, n, w, hi_bits, lo_bits, kw.p);
        DNQ_CHECK_LAUNCH();
        radix_passes<u64>(kw.p, cur, kw2.p, next, n, R, s);
        cur = next;
        next = cur == at.p ? at2.p : at.p;
    };
    int hb = 0, lb = 0;
    if constexpr (W == 2) {
        hb = mask[0] ? 64 - __builtin_clzll(mask[0]) : 0;
        lb = mask[1] ? 64 - __builtin_clzll(mask[1]) : 0;
    }
    if (W == 2 && hb && lb && hb + lb <= 64) {
        by_word(-1, hb, lb, low_mask(hb + lb));
    } else {
        for (int i = W - 1; i >= 0; --i) by_word(i, 0, 0, mask[i]);
    }
    kw.release();
    kw2.release();
    k_radix_gather<K, P><<<grid, 256, 0, s>>>(kin, pin, cur, n, kout, pout);
    DNQ_CHECK_LAUNCH();
}

// The same with bits[i] = significant low bits of key word i.
template <class K, class P>
void radix_sort(const K* kin, K* kout, const P* pin, P* pout, i64 n, const int* bits,
                cudaStream_t s) {
    u64 mask[RadixKey<K>::W];
    for (int i = 0; i < RadixKey<K>::W; ++i) mask[i] = low_mask(bits[i]);
    radix_sort_masked<K, P>(kin, kout, pin, pout, n, mask, s);
}

// ---------------------------------------------------------------------------
// Compaction and segmented sums
// ---------------------------------------------------------------------------

template <class F>
__global__ void k_flag_u32(const F* flag, i64 n, u32* f) {
    for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < n;
         t += (i64)gridDim.x * blockDim.x)
        f[t] = flag[t] != F(0) ? 1u : 0u;
}

template <class T>
__global__ void k_select_scatter(const T* in, const u32* flag, const u32* pos, i64 n, T* out) {
    for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < n;
         t += (i64)gridDim.x * blockDim.x)
        if (flag[t]) out[pos[t]] = in[t];
}

// out = the in[t] with flag[t] != 0, in order; returns their count.
template <class T, class F>
i64 select_flagged(const T* in, const F* flag, T* out, i64 n, cudaStream_t s) {
    if (n <= 0) return 0;
    DBuf<u32> f(n, s), pos(n, s);
    const unsigned g = (unsigned)std::min<i64>((n + 255) / 256, 4096);
    k_flag_u32<F><<<g, 256, 0, s>>>(flag, n, f.p);
    DNQ_CHECK_LAUNCH();
    scan<u32, u32, false>(f.p, pos.p, n, s);
    k_select_scatter<T><<<g, 256, 0, s>>>(in, f.p, pos.p, n, out);
    DNQ_CHECK_LAUNCH();
    u32 lp = 0, lf = 0;
    DNQ_CUDA(cudaMemcpyAsync(&lp, pos.p + n - 1, 4, cudaMemcpyDeviceToHost, s));
    DNQ_CUDA(cudaMemcpyAsync(&lf, f.p + n - 1, 4, cudaMemcpyDeviceToHost, s));
    DNQ_CUDA(cudaStreamSynchronize(s));
    return (i64)lp + lf;
}

// out[i] = sum of v[t] over segment i = [rp[i], rp[i+1]) for integer v
// (order-free sums).  One warp per segment, lanes strided, then a butterfly;
// a segment longer than kSegWarp is listed instead (its sum set to 0) and
// summed by the whole grid in k_segment_sums_long.
constexpr i64 kSegWarp = 1 << 16;

template <class T, class Tout>
__global__ void k_segment_sums(const T* v, const i64* rp, i64 nseg, Tout* out, u32* longs,
                               u32* nlong) {
    const i64 w = (blockIdx.x * (i64)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const i64 nw = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 i = w; i < nseg; i += nw) {
        const i64 b = rp[i], e = rp[i + 1];
        if (e - b > kSegWarp) {
            if (lane == 0) {
                out[i] = 0;
                longs[atomicAdd(nlong, 1u)] = (u32)i;
            }
            continue;
        }
        Tout a = 0;
        for (i64 t = b + lane; t < e; t += 32) a += (Tout)v[t];
#pragma unroll
        for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0) out[i] = a;
    }
}

template <class T, class Tout>
__global__ void k_segment_sums_long(const T* v, const i64* rp, const u32* longs,
                                    const u32* nlong, Tout* out) {
    static_assert(sizeof(Tout) == 8, "64-bit sums");
    const u32 n = *nlong;
    for (u32 q = 0; q < n; ++q) {
        const u32 i = longs[q];
        Tout a = 0;
        for (i64 t = rp[i] + blockIdx.x * (i64)blockDim.x + threadIdx.x; t < rp[i + 1];
             t += (i64)gridDim.x * blockDim.x)
            a += (Tout)v[t];
#pragma unroll
        for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if ((threadIdx.x & 31) == 0 && a)
            atomicAdd(reinterpret_cast<unsigned long long*>(&out[i]), (unsigned long long)a);
    }
}

// out[0..nseg) = the integer sums of v over the segments of rp (64-bit out).
template <class T, class Tout>
void segment_sums(const T* v, const i64* rp, i64 nseg, Tout* out, cudaStream_t s) {
    if (nseg <= 0) return;
    DBuf<u32> longs(nseg, s), nlong(1, s);
    DNQ_CUDA(cudaMemsetAsync(nlong.p, 0, 4, s));
    const unsigned g = (unsigned)std::min<i64>((nseg * 32 + 255) / 256, 8192);
    k_segment_sums<T, Tout><<<g, 256, 0, s>>>(v, rp, nseg, out, longs.p, nlong.p);
    DNQ_CHECK_LAUNCH();
    k_segment_sums_long<T, Tout><<<1184, 256, 0, s>>>(v, rp, longs.p, nlong.p, out);
    DNQ_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// Row of every entry of a CSR block
// ---------------------------------------------------------------------------

// Four consecutive entries per thread: one binary search of the row pointers
// for the first, the others walk on from its row, and one 16-byte store.  (A
// thread per row wrote the rows of a 13-million-entry block in 2.3 ms, a
// search per entry of 4.35e6 took 47 us.)
__global__ void k_rows_of(const i64* rowptr, i64 nr, i64 nnz, u32* rows) {
    for (i64 k = 4 * (blockIdx.x * (i64)blockDim.x + threadIdx.x); k < nnz;
         k += 4 * (i64)gridDim.x * blockDim.x) {
        i64 lo = 0, hi = nr;   // last r with rowptr[r] <= k
        while (hi - lo > 1) {
            const i64 mid = (lo + hi) >> 1;
            if (__ldg(&rowptr[mid]) <= k) lo = mid; else hi = mid;
        }
        u32 r[4];
        i64 end = __ldg(&rowptr[lo + 1]);
        const int m = (int)min((i64)4, nnz - k);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (q < m)
                while (k + q >= end) end = __ldg(&rowptr[++lo + 1]);   // empty rows too
            r[q] = (u32)lo;
        }
        if (m == 4) {   // rows starts an allocation and k is a multiple of 4
            *reinterpret_cast<uint4*>(rows + k) = make_uint4(r[0], r[1], r[2], r[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < m) rows[k + q] = r[q];
        }
    }
}

// rows[k] = the row of entry k < nnz; rows 16-byte aligned.
inline void rows_of(const i64* rowptr, i64 nr, i64 nnz, u32* rows, cudaStream_t s) {
    if (nnz <= 0) return;
    const unsigned g = (unsigned)std::min<i64>((nnz + 1023) / 1024, 1 << 20);
    k_rows_of<<<g, 256, 0, s>>>(rowptr, nr, nnz, rows);
    DNQ_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// Column sort of every row of a CSR block (columns of a row are distinct)
// ---------------------------------------------------------------------------

constexpr i64 kRowSortSmall = 256;     // one block of 256 threads, one entry each
constexpr i64 kRowSortMid = 4096;      // one block, 16 entries per thread
// Longer rows go through the global radix sort.

// Rows by length class: 0 = at most 1 entry (copied), 1 = small, 2 = mid,
// 3 = long.  lists: 4 x nr row ids; counts: 4.
__global__ void k_row_classes(const i64* rp, i64 nr, u32* lists, u32* counts) {
    for (i64 r = blockIdx.x * (i64)blockDim.x + threadIdx.x; r < nr;
         r += (i64)gridDim.x * blockDim.x) {
        const i64 len = rp[r + 1] - rp[r];
        const int c = len <= 1 ? 0 : len <= kRowSortSmall ? 1 : len <= kRowSortMid ? 2 : 3;
        const u32 at = atomicAdd(&counts[c], 1u);
        lists[(i64)c * nr + at] = (u32)r;
    }
}

__global__ void k_row_copy(const u32* rows, const u32* cnt, const i64* rp, const u32* cin,
                           const double* vin, u32* cout, double* vout) {
    const u32 n = *cnt;
    for (u32 t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const u32 r = rows[t];
        for (i64 k = rp[r]; k < rp[r + 1]; ++k) {
            cout[k] = cin[k];
            vout[k] = vin[k];
        }
    }
}

// One block per listed row: (column, position) pairs of the row sorted by a
// bitonic network over N = CAP slots in shared memory (padding: column
// 0xffffffff), then columns and the values they carry written in order.
template <int CAP>
__global__ void __launch_bounds__(256)
k_row_sort(const u32* rows, const u32* cnt, const i64* rp, const u32* cin, const double* vin,
           u32* cout, double* vout) {
    __shared__ u32 key[CAP];
    __shared__ u16 pos[CAP];
    const u32 n = *cnt;
    for (u32 b = blockIdx.x; b < n; b += gridDim.x) {
        const u32 r = rows[b];
        const i64 lo = rp[r];
        const int len = (int)(rp[r + 1] - lo);
        int N = 2;
        while (N < len) N <<= 1;
        for (int i = threadIdx.x; i < N; i += blockDim.x) {
            key[i] = i < len ? cin[lo + i] : 0xffffffffu;
            pos[i] = (u16)i;
        }
        __syncthreads();
        for (int k = 2; k <= N; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = threadIdx.x; i < N; i += blockDim.x) {
                    const int l = i ^ j;
                    if (l > i) {
                        const bool up = (i & k) == 0;
                        const u32 a = key[i], c = key[l];
                        if ((a > c) == up) {
                            key[i] = c;
                            key[l] = a;
                            const u16 t = pos[i];
                            pos[i] = pos[l];
                            pos[l] = t;
                        }
                    }
                }
                __syncthreads();
            }
        for (int i = threadIdx.x; i < len; i += blockDim.x) {
            cout[lo + i] = key[i];
            vout[lo + i] = vin[lo + pos[i]];
        }
        __syncthreads();
    }
}

// Long rows: key = (place of the row in the long list) << 32 | column.  The
// whole grid strides over each long row in turn (a row can hold millions of
// entries).
__global__ void k_long_row_keys(const u32* rows, u32 nlong, const i64* rp, const i64* base,
                                const u32* cin, u64* key, u32* src) {
    for (u32 q = 0; q < nlong; ++q) {
        const u32 r = rows[q];
        const i64 lo = rp[r], len = rp[r + 1] - lo, b = base[q];
        for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < len;
             t += (i64)gridDim.x * blockDim.x) {
            key[b + t] = ((u64)q << 32) | cin[lo + t];
            src[b + t] = (u32)(lo + t);
        }
    }
}

__global__ void k_long_row_put(const u32* rows, u32 nlong, const i64* rp, const i64* base,
                               const u64* skey, const u32* src, const double* vin, u32* cout,
                               double* vout) {
    for (u32 q = 0; q < nlong; ++q) {
        const u32 r = rows[q];
        const i64 lo = rp[r], len = rp[r + 1] - lo, b = base[q];
        for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < len;
             t += (i64)gridDim.x * blockDim.x) {
            cout[lo + t] = (u32)skey[b + t];
            vout[lo + t] = vin[src[b + t]];
        }
    }
}

__global__ void k_long_row_lens(const u32* rows, u32 nlong, const i64* rp, i64* len) {
    for (u32 q = blockIdx.x * blockDim.x + threadIdx.x; q < nlong; q += gridDim.x * blockDim.x)
        len[q] = rp[rows[q] + 1] - rp[rows[q]];
}

// cout/vout = every row of (rp, cin, vin) sorted by column.
inline void sort_row_columns(const i64* rp, i64 nr, const u32* cin, const double* vin, u32* cout,
                             double* vout, cudaStream_t s) {
    if (nr <= 0) return;
    require(nr < (i64)0xffffffffll, DNQ_ERR_OVERFLOW, "row sort of 2^32 or more rows");
    DBuf<u32> lists(4 * nr, s), counts(4, s);
    DNQ_CUDA(cudaMemsetAsync(counts.p, 0, 4 * sizeof(u32), s));
    const unsigned g = (unsigned)std::min<i64>((nr + 255) / 256, 4096);
    k_row_classes<<<g, 256, 0, s>>>(rp, nr, lists.p, counts.p);
    DNQ_CHECK_LAUNCH();
    u32 c[4];
    DNQ_CUDA(cudaMemcpyAsync(c, counts.p, sizeof(c), cudaMemcpyDeviceToHost, s));
    DNQ_CUDA(cudaStreamSynchronize(s));
    if (c[0]) {
        k_row_copy<<<(unsigned)std::min<u32>((c[0] + 255) / 256, 4096u), 256, 0, s>>>(
            lists.p, counts.p, rp, cin, vin, cout, vout);
        DNQ_CHECK_LAUNCH();
    }
    if (c[1]) {
        k_row_sort<(int)kRowSortSmall><<<(unsigned)std::min<u32>(c[1], 1u << 20), 256, 0, s>>>(
            lists.p + nr, counts.p + 1, rp, cin, vin, cout, vout);
        DNQ_CHECK_LAUNCH();
    }
    if (c[2]) {
        k_row_sort<(int)kRowSortMid><<<(unsigned)std::min<u32>(c[2], 1u << 20), 256, 0, s>>>(
            lists.p + 2 * nr, counts.p + 2, rp, cin, vin, cout, vout);
        DNQ_CHECK_LAUNCH();
    }
    if (c[3]) {
        const u32 nl = c[3];
        const u32* rows = lists.p + 3 * nr;
        DBuf<i64> len(nl + 1, s), base(nl + 1, s);
        k_long_row_lens<<<(unsigned)std::min<u32>((nl + 255) / 256, 4096u), 256, 0, s>>>(
            rows, nl, rp, len.p);
        DNQ_CHECK_LAUNCH();
        DNQ_CUDA(cudaMemsetAsync(len.p + nl, 0, sizeof(i64), s));
        scan<i64, i64, false>(len.p, base.p, nl + 1, s);
        i64 m = 0;
        DNQ_CUDA(cudaMemcpyAsync(&m, base.p + nl, sizeof(i64), cudaMemcpyDeviceToHost, s));
        DNQ_CUDA(cudaStreamSynchronize(s));
        DBuf<u64> key(m, s), skey(m, s);
        DBuf<u32> src(m, s), ssrc(m, s);
        const unsigned gl = (unsigned)std::min<i64>((m + 255) / 256, 4096);
        k_long_row_keys<<<gl, 256, 0, s>>>(rows, nl, rp, base.p, cin, key.p, src.p);
        DNQ_CHECK_LAUNCH();
        int hb = 32;
        while (hb < 64 && ((u64)1 << (hb - 32)) < (u64)nl) ++hb;
        const int bits[1] = {hb};
        radix_sort<u64, u32>(key.p, skey.p, src.p, ssrc.p, m, bits, s);
        k_long_row_put<<<gl, 256, 0, s>>>(rows, nl, rp, base.p, skey.p, ssrc.p, vin, cout,
                                          vout);
        DNQ_CHECK_LAUNCH();
    }
}

}  // namespace
}  // namespace prim
}  // namespace dnq
