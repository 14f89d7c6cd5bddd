// Determinant batch features for the neural models (the reference's
// prepare_det_batch, csrc/src/determinant/det_batch.cpp:184-318, bound as
// detnqs.core.prepare_det_batch in csrc/bridge/bridge.cpp:347-430).
//
// One thread per determinant: every field is a short loop over set bits (32
// bits wide for at most 32 orbitals), so a warp keeps 32 determinants in
// flight.  The bound is the result, 250 B per determinant at 30 orbitals: a
// warp's rows are one contiguous piece of each array, so its threads write them
// to shared memory and the warp copies the piece out, 16 bytes a lane side by
// side.  Rows written by their threads (16 bytes at a stride of the row) cost
// the L2 twice the sectors, half filled, and the loops' divergence most of the
// rest: 140 us for 1e6 determinants, 58 now (38 at the measured copy bandwidth).
// The sign is that of the reference's sequence -- holes removed highest first,
// particles added lowest first, each flipping it by the parity of the occupied
// orbitals below (det_batch.cpp:61-98) -- in closed form (excitation_parity).
//
// A determinant that fails a check records (index << 2 | code) with an
// atomic minimum, so the host reports the first failing determinant in
// batch order with the reference's message for its first failing check.
#include "common.cuh"

namespace dnq {

void keep_pool(int device);

namespace {

enum : int { kNeedK = 1, kNeedPhase = 2, kNeedHp = 4, kNeedPos = 8 };
enum : u64 { kBadBits = 1, kBadCount = 2, kBadHp = 3 };

// Strings as W: u32 for at most 32 orbitals, else u64.
template <class W> struct Bits;
template <> struct Bits<u32> {
    __device__ __forceinline__ static int low(u32 x) { return __ffs(x) - 1; }
    __device__ __forceinline__ static int high(u32 x) { return 31 - __clz(x); }
    __device__ __forceinline__ static int count(u32 x) { return __popc(x); }
};
template <> struct Bits<u64> {
    __device__ __forceinline__ static int low(u64 x) { return __ffsll((long long)x) - 1; }
    __device__ __forceinline__ static int high(u64 x) { return 63 - __clzll((long long)x); }
    __device__ __forceinline__ static int count(u64 x) { return __popcll(x); }
};
template <class W>
__device__ __forceinline__ W one_at(int q) { return (W)1 << q; }
template <class W>
__device__ __forceinline__ int count_below(W x, int q) {   // 0 <= q < bits of W
    return Bits<W>::count(x & (W)(one_at<W>(q) - 1));
}

// Parity of one spin's excitation from r to d (both masked).  The sequence
// "holes highest first, then particles lowest first" counts, at each, the
// occupied orbitals below: for a hole the common ones and the holes below it,
// for a particle the common ones and the particles below it.  With as many
// particles as holes, k, the two latter sums are k (k - 1) / 2 each and cancel
// mod 2; the common ones are the prefix parity of r & d at the bits of r ^ d.
template <class W>
__device__ __forceinline__ int excitation_parity(W r, W d) {
    W p = (W)((r & d) << 1);
#pragma unroll
    for (int s = 1; s < (int)sizeof(W) * 8; s <<= 1) p ^= (W)(p << s);
    return Bits<W>::count((r ^ d) & p) & 1;
}

struct BatchOut {
    int32_t* occ;
    int8_t* k;
    int8_t* phase;
    int32_t* holes;
    int32_t* parts;
    uint8_t* mask;
    int32_t* hpos;
    int32_t* ppos;
};

constexpr int kFeatWarps = 4;
constexpr int kListCols = 32;   // hole / particle columns staged at a time

// A staged piece: cnt <= 32 rows of len values at an odd stride (a column is
// then conflict-free), copied to rows of dst `pitch` values apart, 16 bytes a
// lane where they are contiguous and dst allows.
__device__ __forceinline__ void piece_out(int32_t* dst, int pitch, const int32_t* buf, int len,
                                          int cnt, int lane) {
    const int stride = len | 1, total = cnt * len;
    // f / len for f < 4096 by the rounded reciprocal: the product's error is
    // far inside the 1 / (2 len) distance of (f + 0.5) / len from an integer
    const float rcp = __frcp_rn((float)len);
    __syncwarp();
    int done = 0;
    if (pitch == len && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        done = total & ~3;
        for (int f = 4 * lane; f < done; f += 128) {
            int row = (int)(((float)f + 0.5f) * rcp), col = f - row * len, v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                v[q] = buf[row * stride + col];
                if (++col == len) {
                    col = 0;
                    ++row;
                }
            }
            __stcs(reinterpret_cast<int4*>(dst + f), make_int4(v[0], v[1], v[2], v[3]));
        }
    }
    for (int f = done + lane; f < total; f += 32) {
        const int row = (int)(((float)f + 0.5f) * rcp), col = f - row * len;
        dst[(i64)row * pitch + col] = buf[row * stride + col];
    }
    __syncwarp();
}

// Position of the next hole (highest first) of x, removed from it.
template <class W>
__device__ __forceinline__ int take_high(W& x) {
    const int q = Bits<W>::high(x);
    x ^= one_at<W>(q);
    return q;
}
template <class W>
__device__ __forceinline__ int take_low(W& x) {
    const int q = Bits<W>::low(x);
    x &= x - 1;
    return q;
}

template <class W>
__global__ void __launch_bounds__(kFeatWarps * 32)
k_det_batch(const u64* dets, i64 B, u64 ref_a, u64 ref_b, int n_orb, int na, int nb, int kmax,
            int flags, int piece_words, BatchOut o, unsigned long long* err) {
    extern __shared__ __align__(16) int32_t feat_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const u64 m = low_mask(n_orb);
    const int ne = na + nb;
    const W ra = (W)(ref_a & m), rb = (W)(ref_b & m);
    int32_t* buf = feat_smem + (size_t)w * piece_words;
    const bool pos = flags & kNeedPos;
    const int kw = 32 * (min(kmax, kListCols) | 1);   // words of a piece of lists
    for (i64 i0 = ((i64)blockIdx.x * kFeatWarps + w) * 32; i0 < B;
         i0 += (i64)gridDim.x * kFeatWarps * 32) {
        const int cnt = (int)min((i64)32, B - i0);
        const i64 i = i0 + lane;
        u64 a64 = 0, b64 = 0, bad = 0;
        if (lane < cnt) {
            const ulonglong2 d = reinterpret_cast<uintptr_t>(dets) & 15
                                     ? make_ulonglong2(dets[2 * i], dets[2 * i + 1])
                                     : reinterpret_cast<const ulonglong2*>(dets)[i];
            a64 = d.x;
            b64 = d.y;
            if ((a64 & ~m) || (b64 & ~m)) bad = kBadBits;
            else if (__popcll(a64) != na || __popcll(b64) != nb) bad = kBadCount;
            else if ((flags & kNeedPhase) &&
                     (Bits<W>::count(ra & ~(W)a64) != Bits<W>::count((W)a64 & ~ra) ||
                      Bits<W>::count(rb & ~(W)b64) != Bits<W>::count((W)b64 & ~rb)))
                bad = kBadHp;
            if (bad) atomicMin(err, ((unsigned long long)i << 2) | bad);
        }
        // a determinant that fails a check keeps its lane idle; its rows are
        // then whatever the piece holds (the call reports the error)
        const bool on = lane < cnt && !bad;
        const W a = (W)a64, b = (W)b64;
        if (on) {
            int32_t* p = buf + lane * (ne | 1);
            for (W x = a; x;) *p++ = take_low(x);
            for (W x = b; x;) *p++ = take_low(x) + n_orb;
        }
        if (ne && na <= n_orb && nb <= n_orb) piece_out(o.occ + i0 * ne, ne, buf, ne, cnt, lane);
        W ha = ra & ~a, hb = rb & ~b, pa = a & ~ra, pb = b & ~rb;
        const int kk = Bits<W>::count(ha) + Bits<W>::count(hb);
        if (on && (flags & (kNeedK | kNeedHp))) o.k[i] = (int8_t)min(kk, 127);
        if (on && (flags & kNeedPhase))
            o.phase[i] = excitation_parity<W>(ra, a) ^ excitation_parity<W>(rb, b) ? -1 : 1;
        if (!(flags & kNeedHp) || kmax == 0) continue;
        // holes: alpha then beta (+ n_orb), each highest first; position in the
        // reference's occupied list (alpha ascending, then beta).  Particles:
        // alpha then beta (+ n_orb), each lowest first; position in the
        // reference's virtual list (the other spin orbitals, ascending).  -1 past
        // the last.
        for (int j0 = 0; j0 < kmax; j0 += kListCols) {
            const int kc = min(kListCols, kmax - j0);
            int32_t* h = buf + lane * (kc | 1);
            for (int j = 0; on && j < kc; ++j) {
                int qh = -1, qp = -1, sh = -1, sp = -1;
                if (ha) {
                    qh = take_high(ha);
                    sh = count_below<W>(ra, qh);
                } else if (hb) {
                    const int q = take_high(hb);
                    qh = q + n_orb;
                    sh = na + count_below<W>(rb, q);
                }
                if (pa) {
                    qp = take_low(pa);
                    sp = qp - count_below<W>(ra, qp);
                } else if (pb) {
                    const int q = take_low(pb);
                    qp = q + n_orb;
                    sp = qp - na - count_below<W>(rb, q);
                }
                h[j] = qh;
                h[kw + j] = qp;
                if (pos) {
                    h[2 * kw + j] = sh;
                    h[3 * kw + j] = sp;
                }
            }
            const i64 to = i0 * kmax + j0;
            piece_out(o.holes + to, kmax, buf, kc, cnt, lane);
            piece_out(o.parts + to, kmax, buf + kw, kc, cnt, lane);
            if (pos) {
                piece_out(o.hpos + to, kmax, buf + 2 * kw, kc, cnt, lane);
                piece_out(o.ppos + to, kmax, buf + 3 * kw, kc, cnt, lane);
            }
        }
        // mask: the first min(k, kmax) bytes set, eight to a store when the
        // row starts on an 8-byte boundary and holds whole words
        if (on) {
            const int kcap = min(kk, kmax);
            uint8_t* mrow = o.mask + i * kmax;
            if ((reinterpret_cast<uintptr_t>(mrow) & 7) == 0 && (kmax & 7) == 0) {
                for (int q = 0; q < kmax; q += 8) {
                    const int set = min(max(kcap - q, 0), 8);
                    const u64 lo = set == 8 ? ~0ull : ((1ull << (8 * set)) - 1ull);
                    *reinterpret_cast<u64*>(mrow + q) = 0x0101010101010101ull & lo;
                }
            } else {
                for (int j = 0; j < kmax; ++j) mrow[j] = j < kcap;
            }
        }
    }
}

// Device target of one output: the caller's device buffer, or a staging
// buffer copied back to the caller's host buffer by finish().
template <class T>
struct DOut {
    T* user = nullptr;
    T* p = nullptr;
    size_t n = 0;
    DBuf<T> own;
    void set(T* dst, size_t count, cudaStream_t s) {
        user = dst;
        n = count;
        if (!dst || count == 0) return;
        if (is_device_ptr(dst)) {
            p = dst;
            return;
        }
        own.alloc(count, s);
        p = own.p;
    }
    void finish(cudaStream_t s) {
        if (own.p) copy_out(user, own.p, n, s);
    }
};

}  // namespace
}  // namespace dnq

using namespace dnq;

extern "C" {

int dnq_prepare_det_batch(const uint64_t* dets, int64_t B, const uint64_t* ref, int n_orb,
                          int n_alpha, int n_beta, int kmax, int flags, int32_t* occ,
                          int8_t* k, int8_t* phase, int32_t* holes, int32_t* parts,
                          uint8_t* hp_mask, int32_t* holes_pos, int32_t* parts_pos,
                          int device, void* stream) {
    DNQ_API_BEGIN
    // the reference's checks, in its order (det_batch.cpp:200-215, :104-124)
    require(n_orb >= 0 && n_orb <= 64, DNQ_ERR_INVALID, "n_orb out of range [0,64]");
    require(B >= 0, DNQ_ERR_INVALID, "negative size");
    require(ref != nullptr && (B == 0 || (dets && occ)), DNQ_ERR_INVALID,
            "null pointer in required outputs");
    require((flags & ~15) == 0, DNQ_ERR_INVALID, "unknown flags");
    const bool need_hp = flags & kNeedHp, need_pos = flags & kNeedPos;
    if (need_hp) flags |= kNeedK;
    require(!need_pos || need_hp, DNQ_ERR_INVALID, "need_hp_pos requires need_hp");
    require(!need_hp || kmax >= 0, DNQ_ERR_INVALID, "kmax must be non-negative");
    require(n_alpha >= 0 && n_beta >= 0, DNQ_ERR_INVALID, "electron count mismatch");
    const u64 m = low_mask(n_orb);
    const u64 ra = ref[0], rb = ref[1];
    if (need_pos)
        require(__builtin_popcountll(ra & m) == n_alpha && __builtin_popcountll(rb & m) == n_beta,
                DNQ_ERR_INVALID, "reference electron count mismatch");
    if (B == 0) return DNQ_OK;
    require(!(flags & kNeedK) || k, DNQ_ERR_INVALID, "k_out is null");
    require(!(flags & kNeedPhase) || phase, DNQ_ERR_INVALID, "phase_out is null");
    require(!need_hp || kmax == 0 || (holes && parts && hp_mask), DNQ_ERR_INVALID,
            "hp outputs are null");
    require(!need_pos || kmax == 0 || (holes_pos && parts_pos), DNQ_ERR_INVALID,
            "pos outputs are null");
    DeviceGuard g(device);
    keep_pool(device);   // the device pool keeps freed memory, as for every other entry point
    cudaStream_t s = (cudaStream_t)stream;
    const int ne = n_alpha + n_beta;
    const size_t nk = need_hp ? (size_t)B * (size_t)kmax : 0;
    DIn<u64> d(dets, 2 * (size_t)B, s);
    DOut<int32_t> o_occ, o_h, o_p, o_hp, o_pp;
    DOut<int8_t> o_k, o_ph;
    DOut<uint8_t> o_m;
    o_occ.set(occ, (size_t)B * ne, s);
    o_k.set((flags & kNeedK) ? k : nullptr, B, s);
    o_ph.set((flags & kNeedPhase) ? phase : nullptr, B, s);
    o_h.set(need_hp ? holes : nullptr, nk, s);
    o_p.set(need_hp ? parts : nullptr, nk, s);
    o_m.set(need_hp ? hp_mask : nullptr, nk, s);
    o_hp.set(need_pos ? holes_pos : nullptr, nk, s);
    o_pp.set(need_pos ? parts_pos : nullptr, nk, s);
    DBuf<unsigned long long> err(1, s);
    DNQ_CUDA(cudaMemsetAsync(err.p, 0xff, sizeof(unsigned long long), s));
    BatchOut bo{o_occ.p, o_k.p, o_ph.p, o_h.p, o_p.p, o_m.p, o_hp.p, o_pp.p};
    // words of a warp's pieces: at most 32 x 4 x 33, 66 KB a block.  With more
    // electrons of a spin than orbitals no determinant has a row to stage (the
    // kernel reports the first)
    const int kc = need_hp ? std::min(kmax, kListCols) : 0;
    const int row = n_alpha <= n_orb && n_beta <= n_orb ? ne : 0;
    const int piece_words = 32 * std::max(row | 1, (kc | 1) * (need_pos ? 4 : 2));
    const size_t smem = (size_t)kFeatWarps * piece_words * sizeof(int32_t);
    auto kern = n_orb <= 32 ? k_det_batch<u32> : k_det_batch<u64>;
    if (smem > 48 * 1024)
        DNQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    const i64 per = 32 * kFeatWarps;
    const int grid = (int)std::min<i64>((B + per - 1) / per, (i64)sm_count(device) * 64);
    kern<<<grid, kFeatWarps * 32, smem, s>>>(d.p, B, ra, rb, n_orb, n_alpha, n_beta, kmax, flags,
                                             piece_words, bo, err.p);
    DNQ_CHECK_LAUNCH();
    unsigned long long e = 0;
    DNQ_CUDA(cudaMemcpyAsync(&e, err.p, sizeof(e), cudaMemcpyDeviceToHost, s));
    o_occ.finish(s);
    o_k.finish(s);
    o_ph.finish(s);
    o_h.finish(s);
    o_p.finish(s);
    o_m.finish(s);
    o_hp.finish(s);
    o_pp.finish(s);
    DNQ_CUDA(cudaStreamSynchronize(s));
    if (e != ~0ull) {
        const u64 code = e & 3;
        require(code != kBadBits, DNQ_ERR_INVALID, "det bits outside n_orb range");
        require(code != kBadCount, DNQ_ERR_INVALID, "electron count mismatch");
        require(false, DNQ_ERR_INVALID, "holes != parts in spin channel");
    }
    DNQ_API_END
}

}  // extern "C"
