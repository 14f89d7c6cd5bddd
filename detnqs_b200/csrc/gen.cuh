// gen.cuh -- warp-per-determinant enumeration of connected determinants.
//
// One warp owns one bra row.  It walks the candidates in the reference's
// order -- singles alpha then beta, holes ascending outer and particles
// ascending inner (det_ops.hpp:123-159), then heat-bath doubles over the
// occupied spin-orbital pairs (p > q in the alpha-then-beta occupied list)
// with each pair's table prefix (ham_utils.hpp:280-313) -- 32 candidates per
// step, one per lane.  Every lane forms its ket with bit operations, the
// fermionic phase with popcounts (Scemama-Giner rules, det_ops.cpp:85-196)
// and the matrix element:
//   single h->p : h1[h,p] + sum over the other occupied orbitals of the
//                 precomputed same/opposite-spin terms, in the reference's
//                 summation order (ham_eval.cpp:88-115);
//   double      : +-v from the signed pair table (no ERI reads).
// A sink object (routing, screening, output) sees each step collectively,
// so it can compact survivors with __ballot_sync in candidate order.
#pragma once

#include <algorithm>

#include "context.cuh"
#include "detmap.cuh"

namespace dnq {

// Per-warp occupancy lists, in shared memory.
struct WarpRow {
    u64 a, b;                 // bra alpha / beta masks
    u64 fulla, fullb;         // no place for a particle: occupied, or not among the n_orb
    int na, nb, nva, nvb, ne;
    u8 occ[128];              // spin-orbitals: 2p (alpha asc) then 2p+1 (beta asc)
    u8 occa[64], occb[64], vira[64], virb[64];
};

// One lane per orbital: an orbital's place in its list is the count of the
// listed orbitals below it.
__device__ __forceinline__ void load_row(WarpRow& R, u64 a, u64 b, int n_orb) {
    const int lane = threadIdx.x & 31;
    const u64 all = low_mask(n_orb);
    const int na = __popcll(a), nb = __popcll(b);
    for (int o = lane; o < 64; o += 32) {
        const u64 below = (1ull << o) - 1ull;
        const int oa = __popcll(a & below), ob = __popcll(b & below);
        if ((a >> o) & 1ull) {
            R.occa[oa] = (u8)o;
            R.occ[oa] = (u8)(2 * o);
        } else if (o < n_orb) {
            R.vira[o - oa] = (u8)o;
        }
        if ((b >> o) & 1ull) {
            R.occb[ob] = (u8)o;
            R.occ[na + ob] = (u8)(2 * o + 1);
        } else if (o < n_orb) {
            R.virb[o - ob] = (u8)o;
        }
    }
    if (lane == 0) {
        R.a = a;
        R.b = b;
        R.fulla = a | ~all;
        R.fullb = b | ~all;
        R.na = na;
        R.nb = nb;
        R.ne = na + nb;
        R.nva = __popcll(~a & all);
        R.nvb = __popcll(~b & all);
    }
    __syncwarp();
}

// diag_elem for at most 32 orbitals, without the list of orbitals (which lies in
// local memory): strings with orbital 0 in the highest bit, so an orbital is one
// count of leading zeros.  Chosen at the launch, not here: a kernel that holds
// both forms has the registers of both (k_pt2_runs 794 us so, 871 with a branch,
// 1,010 with the list; k_diag at 1e6 dets of 30 orbitals 212 with the list, 176
// so).
__device__ __forceinline__ double diag_elem32(const CtxView& C, u32 a, u32 b) {
    const u32 ra = __brev(a), rb = __brev(b);
    auto sum = [](double e, const double* t, int stride, u32 x) {
        while (x) {
            const int o = __clz(x);
            x &= ~(0x80000000u >> o);
            e += __ldg(&t[o * stride]);
        }
        return e;
    };
    const double one = sum(sum(0.0, C.h1, C.n + 1, ra), C.h1, C.n + 1, rb);
    double two = 0.0;
    for (u32 x = ra; x;) {
        const int p = __clz(x);
        x &= ~(0x80000000u >> p);
        two = sum(two, C.dss + p * C.n, 1, ra & ~(0xffffffffu >> p));
    }
    for (u32 x = rb; x;) {
        const int p = __clz(x);
        x &= ~(0x80000000u >> p);
        two = sum(two, C.dos + p * C.n, 1, ra);
        two = sum(two, C.dss + p * C.n, 1, rb & ~(0xffffffffu >> p));
    }
    return one + two;
}

// <bra|H|bra> with the reference's order: one-body over alpha then beta
// occupied orbitals, then sum_{x>y} <occ_x occ_y||occ_x occ_y>
// (ham_eval.cpp:53-86).  Serial per thread so the rounding matches.
__device__ __forceinline__ double diag_elem(const CtxView& C, u64 a, u64 b) {
    const int n = C.n;
    u8 occ[128];
    int m = 0;
    for (u64 x = a; x; x &= x - 1) occ[m++] = (u8)(2 * (__ffsll(x) - 1));
    for (u64 x = b; x; x &= x - 1) occ[m++] = (u8)(2 * (__ffsll(x) - 1) + 1);
    double one = 0.0;
    for (int t = 0; t < m; ++t) {
        const int p = occ[t] >> 1;
        one += C.h1[p * n + p];
    }
    double two = 0.0;
    for (int x = 1; x < m; ++x) {
        const int P = occ[x];
        const double* dss = C.dss + (P >> 1) * n;
        const double* dos = C.dos + (P >> 1) * n;
        for (int y = 0; y < x; ++y) {
            const int Q = occ[y];
            two += ((P ^ Q) & 1) ? dos[Q >> 1] : dss[Q >> 1];
        }
    }
    return one + two;
}

// e + t[o] over the set bits o of x, ascending, one addition after the other;
// the loads of four bits are issued ahead of their additions (each is an L1 or
// L2 read that the next addition would wait for).  k_vv_singles at 1e6 rows of
// 30 orbitals: 568 us one load at a time, 314 so.
__device__ __forceinline__ double add_bits(double e, const double* t, u64 x) {
    while (x) {
        const int o0 = __ffsll(x) - 1;
        x &= x - 1;
        const int o1 = x ? __ffsll(x) - 1 : -1;
        x &= x - 1;
        const int o2 = x ? __ffsll(x) - 1 : -1;
        x &= x - 1;
        const int o3 = x ? __ffsll(x) - 1 : -1;
        x &= x - 1;
        const double v0 = __ldg(&t[o0]);
        const double v1 = o1 >= 0 ? __ldg(&t[o1]) : 0.0;
        const double v2 = o2 >= 0 ? __ldg(&t[o2]) : 0.0;
        const double v3 = o3 >= 0 ? __ldg(&t[o3]) : 0.0;
        e += v0;
        if (o1 >= 0) e += v1;
        if (o2 >= 0) e += v2;
        if (o3 >= 0) e += v3;
    }
    return e;
}

// The same without the look-ahead, for kernels short of registers.
__device__ __forceinline__ double add_bits_plain(double e, const double* t, u64 x) {
    for (; x; x &= x - 1) e += t[__ffsll(x) - 1];
    return e;
}

// Single excitation h -> p in spin `s` of the bra (a, b); returns the signed
// element <bra|H|ket>.
template <bool AHEAD = true>
__device__ __forceinline__ double single_elem(const CtxView& C, u64 a, u64 b, int s, int h,
                                              int p) {
    const int n = C.n;
    double e = C.h1[h * n + p];
    const size_t base = ((size_t)h * n + p) * n;
    const double* ss = C.sss + base;
    const double* os = C.sos + base;
    const u64 hole = 1ull << h;
    const double* first = s == 0 ? ss : os;
    const double* second = s == 0 ? os : ss;
    const u64 xa = s == 0 ? a & ~hole : a, xb = s == 0 ? b : b & ~hole;
    e = AHEAD ? add_bits(e, first, xa) : add_bits_plain(e, first, xa);
    e = AHEAD ? add_bits(e, second, xb) : add_bits_plain(e, second, xb);
    const int perm = occ_between(s ? b : a, h, p);
    return (perm & 1) ? -e : e;
}

// e + col[k * n] for the listed occupied orbitals k but `skip`, in order; four
// reads ahead of their additions.
__device__ __forceinline__ double add_col(double e, const double* col, int n, const u8* occ,
                                          int cnt, int skip) {
    int t = 0;
    for (; t + 4 <= cnt; t += 4) {
        double v[4];
        int o[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            o[q] = occ[t + q];
            v[q] = __ldg(&col[o[q] * n]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (o[q] != skip) e += v[q];
    }
    for (; t < cnt; ++t)
        if (occ[t] != skip) e += __ldg(&col[occ[t] * n]);
    return e;
}

// Unsigned single h -> p in spin s, for warps that evaluate the singles of
// one determinant from its occupied lists (ham_eval.cpp:88-115: h1, then
// alpha ascending, then beta ascending).  Lanes hold neighbouring p and share
// k, so a read of the [h][k][p] tables is a few sectors a warp; from the
// [h][p][k] tables each lane draws a line of its own, and the L1 serves one
// line a clock: the count pass of the two-word build (3.2e7 singles of 40
// terms) took 4.52 ms so, 3.15 from these, and 1.58 with the pairs looked up 32
// at a time (enumerate_pairs).
__device__ __forceinline__ double single_sum(const CtxView& C, const u8* occa, int na,
                                             const u8* occb, int nb, int s, int h, int p) {
    const int n = C.n;
    const size_t base = (size_t)h * n * n + p;
    double e = C.h1[h * n + p];
    e = add_col(e, (s ? C.sosT : C.sssT) + base, n, occa, na, s ? -1 : h);
    return add_col(e, (s ? C.sssT : C.sosT) + base, n, occb, nb, s ? h : -1);
}

// Double i,j -> a,b (spin-orbitals, i > j, a > b) of the bra from the
// signed table value v = <ij||ab>.
__device__ __forceinline__ double double_elem(u64 ba, u64 bb, int i, int j, int a, int b,
                                              double v) {
    const bool same = ((i ^ j) & 1) == 0;
    double raw = (same || ((a ^ i) & 1) == 0) ? v : -v;
    int perm;
    if (same) {
        const u64 occ = (i & 1) ? bb : ba;
        const int h0 = b >> 1, h1 = a >> 1;     // ket-only orbitals, ascending
        const int p0 = j >> 1, p1 = i >> 1;     // bra-only orbitals, ascending
        perm = occ_between(occ, h0, p0) + occ_between(occ, h1, p1);
        const int A = min(h0, p0), B = max(h0, p0), Cc = min(h1, p1), D = max(h1, p1);
        if ((Cc > A && Cc < B && D > B) || (A > Cc && A < D && B > D)) ++perm;
    } else {
        const int ha = ((a & 1) == 0 ? a : b) >> 1;
        const int hb = ((a & 1) == 1 ? a : b) >> 1;
        const int pa = ((i & 1) == 0 ? i : j) >> 1;
        const int pb = ((i & 1) == 1 ? i : j) >> 1;
        perm = occ_between(ba, ha, pa) + occ_between(bb, hb, pb);
    }
    return (perm & 1) ? -raw : raw;
}

// Candidate handed to a sink (per lane).
struct Cand {
    bool valid;
    bool single;
    u64 a, b;       // ket
    double h;       // <bra|H|ket>
};

// Walk all candidates of the bra in R.  `plen` (optional) holds the prefix
// length of every table row for a cut shared by all rows; otherwise the
// prefix is searched with `cut`.  Sink::step(const Cand&) is called by all
// 32 lanes together.
// Singles of the bra in R: alpha then beta, holes ascending outer and
// particles ascending inner (det_ops.hpp:123-159, :248-253).
template <class Sink>
__device__ __forceinline__ void enumerate_singles(const CtxView& C, const WarpRow& R,
                                                  Sink& sink) {
    const int lane = threadIdx.x & 31;
    const int nsa = R.na * R.nva;
    const int nst = nsa + R.nb * R.nvb;
    for (int t0 = 0; t0 < nst; t0 += 32) {
        Cand c;
        const int t = t0 + lane;
        c.valid = t < nst;
        c.single = true;
        c.a = R.a;
        c.b = R.b;
        c.h = 0.0;
        if (c.valid) {
            int s, h, p;
            if (t < nsa) {
                s = 0;
                h = R.occa[t / R.nva];
                p = R.vira[t % R.nva];
                c.a = R.a ^ (1ull << h) ^ (1ull << p);
            } else {
                const int u = t - nsa;
                s = 1;
                h = R.occb[u / R.nvb];
                p = R.virb[u % R.nvb];
                c.b = R.b ^ (1ull << h) ^ (1ull << p);
            }
            const double e = single_sum(C, R.occa, R.na, R.occb, R.nb, s, h, p);
            c.h = (occ_between(s ? R.b : R.a, h, p) & 1) ? -e : e;
        }
        sink.step(c);
    }
}

// Pair p = x (x - 1) / 2 + y of the occupied list, y < x.
__device__ __forceinline__ void pair_of(int p, int& x, int& y) {
    x = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)p)) * 0.5f);
    while (x * (x - 1) / 2 > p) --x;
    while ((x + 1) * x / 2 <= p) ++x;
    y = p - x * (x - 1) / 2;
}

// Doubles over the occupied pairs [p_lo, p_hi) (x ascending, y < x ascending).
// The table lists particles among all orbitals of the integrals; one past n_orb
// is no candidate (ham_utils.cpp:470-479).
// The table rows of 32 pairs are looked up at once, a pair per lane, and the
// prefixes of a cut of the row's own searched side by side: one pair after
// the other, a warp waits several L2 reads for each, most of them for an empty
// prefix under dynamic screening.
template <class Sink>
__device__ __forceinline__ void enumerate_pairs(const CtxView& C, const WarpRow& R,
                                                const i64* plen, double cut, Sink& sink, int p_lo,
                                                int p_hi) {
    const int lane = threadIdx.x & 31;
    for (int p0 = p_lo; p0 < p_hi; p0 += 32) {
        i64 lo_l = 0;
        u32 len_l = 0, ij_l = 0;
        if (p0 + lane < p_hi) {
            int x, y;
            pair_of(p0 + lane, x, y);
            const int i = R.occ[x], j = R.occ[y];
            const i64 row = pair_row(i, j);
            lo_l = __ldg(&C.tab.off[row]);
            ij_l = (u32)max(i, j) | (u32)min(i, j) << 8;
            if (plen) {
                len_l = (u32)__ldg(&plen[row]);
            } else {
                const u32 all = (u32)(__ldg(&C.tab.off[row + 1]) - lo_l);
                u32 L = 0, H = all;
                if (cut <= 0.0) {
                    L = all;
                } else if (all && fabs(__ldg(&C.tab.v[lo_l])) >= cut) {
                    L = 1;
                    while (L < H) {   // weights descend
                        const u32 mid = (L + H) >> 1;
                        if (fabs(__ldg(&C.tab.v[lo_l + mid])) >= cut) L = mid + 1; else H = mid;
                    }
                }
                len_l = L;
            }
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, len_l != 0); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const i64 lo = __shfl_sync(0xffffffffu, lo_l, src);
            const u32 len = __shfl_sync(0xffffffffu, len_l, src);
            const u32 ij = __shfl_sync(0xffffffffu, ij_l, src);
            const int ii = ij & 0xff, jj = ij >> 8;
            u64 ha = R.a, hb = R.b;   // the bra without the pair
            if (ii & 1) hb &= ~(1ull << (ii >> 1)); else ha &= ~(1ull << (ii >> 1));
            if (jj & 1) hb &= ~(1ull << (jj >> 1)); else ha &= ~(1ull << (jj >> 1));
            for (u32 e0 = 0; e0 < len; e0 += 32) {
                Cand c;
                const u32 e = e0 + lane;
                c.valid = e < len;
                c.single = false;
                c.a = R.a;
                c.b = R.b;
                c.h = 0.0;
                if (c.valid) {
                    const u16 ab = __ldg(&C.tab.ab[lo + e]);
                    const double v = __ldg(&C.tab.v[lo + e]);
                    const int A = ab & 0xff, B = ab >> 8;
                    const u64 ma = 1ull << (A >> 1), mb = 1ull << (B >> 1);
                    const bool noA = ((A & 1) ? R.fullb : R.fulla) & ma;
                    const bool noB = ((B & 1) ? R.fullb : R.fulla) & mb;
                    if (noA || noB) {
                        c.valid = false;
                    } else {
                        c.a = ha | ((A & 1) ? 0ull : ma) | ((B & 1) ? 0ull : mb);
                        c.b = hb | ((A & 1) ? ma : 0ull) | ((B & 1) ? mb : 0ull);
                        c.h = double_elem(R.a, R.b, ii, jj, A, B, v);
                    }
                }
                sink.step(c);
            }
        }
    }
}

// Part `part` of `parts` of a row, in candidate order over the parts: the
// singles, then equal shares of the occupied pairs (one part holds all).
// Spaces of fewer rows than the GPU has warps are cut so (row_parts).
template <class Sink>
__device__ __forceinline__ void enumerate_row(const CtxView& C, const WarpRow& R,
                                              const i64* plen, double cut, Sink& sink,
                                              int part = 0, int parts = 1) {
    if (part == 0) enumerate_singles(C, R, sink);
    const int np = R.ne * (R.ne - 1) / 2;
    if (parts == 1) enumerate_pairs(C, R, plen, cut, sink, 0, np);
    else if (part > 0)
        enumerate_pairs(C, R, plen, cut, sink, (int)((i64)np * (part - 1) / (parts - 1)),
                        (int)((i64)np * part / (parts - 1)));
}

// Parts per row: enough for four units of work per warp, at most one of eight
// pairs each (a unit sets its row up again, ~1 us).  At 403 rows of 24 orbitals
// a warp per row left nine in ten warps idle: a count and a fill pass 5.06 ms so,
// 0.48 cut (2,241 rows of 13 orbitals 0.65 -> 0.31, PT2 at 3,001 rows of 20
// orbitals 3.50 -> 1.49).
inline int row_parts(i64 n, i64 warps, int n_orb) {
    if (n <= 0 || n >= 2 * warps) return 1;
    const i64 want = (4 * warps + n - 1) / n;
    const i64 pairs = (i64)n_orb * (n_orb - 1) / 2;   // of a half-filled row
    const i64 parts = std::min<i64>(want, pairs / 8 + 1) + 1;
    return parts <= 2 ? 1 : (int)std::min<i64>(parts, 128);
}

// rowptr[r] = first offset of row r's parts, r <= n.
__global__ static void k_first_parts(const i64* off, int parts, i64 n, i64* rowptr) {
    for (i64 r = blockIdx.x * (i64)blockDim.x + threadIdx.x; r <= n;
         r += (i64)gridDim.x * blockDim.x)
        rowptr[r] = off[r * parts];
}

// All candidates of the bra in the order get_local_conn visits them without
// heat-bath screening (local_conn.cpp:69-91): the singles, then every double
// in det_ops::for_each_double's order -- alpha-alpha (hole pairs h1 < h2
// outer, particle pairs p1 < p2 inner; det_ops.hpp:161-187), beta-beta
// (:189-215), alpha-beta (alpha hole, alpha particle, beta hole, beta
// particle; :217-246).  A double's element comes from the ERIs through the
// same antisymmetrised value the pair table stores, so it has the same bits
// as on the table walk.
template <class Sink>
__device__ __forceinline__ void enumerate_row_full(const CtxView& C, const WarpRow& R,
                                                   Sink& sink) {
    const int lane = threadIdx.x & 31;
    enumerate_singles(C, R, sink);
    for (int s = 0; s < 2; ++s) {
        const u8* occ = s ? R.occb : R.occa;
        const u8* vir = s ? R.virb : R.vira;
        const int no = s ? R.nb : R.na, nv = s ? R.nvb : R.nva;
        if (no < 2 || nv < 2) continue;
        const int npv = nv * (nv - 1) / 2;
        for (int x1 = 0; x1 < no; ++x1)
            for (int x2 = x1 + 1; x2 < no; ++x2) {
                const int h1 = occ[x1], h2 = occ[x2];
                for (int t0 = 0; t0 < npv; t0 += 32) {
                    Cand c;
                    const int t = t0 + lane;
                    c.valid = t < npv;
                    c.single = false;
                    c.a = R.a;
                    c.b = R.b;
                    c.h = 0.0;
                    if (c.valid) {
                        int y1 = 0, rem = t;          // t-th pair y1 < y2, lexicographic
                        while (rem >= nv - 1 - y1) { rem -= nv - 1 - y1; ++y1; }
                        const int p1 = vir[y1], p2 = vir[y1 + 1 + rem];
                        const u64 m = (1ull << h1) | (1ull << h2) | (1ull << p1) | (1ull << p2);
                        if (s) c.b ^= m; else c.a ^= m;
                        const int i = 2 * h2 + s, j = 2 * h1 + s, A = 2 * p2 + s, B = 2 * p1 + s;
                        c.h = double_elem(R.a, R.b, i, j, A, B, anti_so_of(C.eri, i, j, A, B));
                    }
                    sink.step(c);
                }
            }
    }
    if (!R.na || !R.nva || !R.nb || !R.nvb) return;
    const int nsb = R.nb * R.nvb;
    for (int xa = 0; xa < R.na; ++xa)
        for (int ya = 0; ya < R.nva; ++ya) {
            const int ha = R.occa[xa], pa = R.vira[ya];
            const u64 ka = R.a ^ (1ull << ha) ^ (1ull << pa);
            for (int t0 = 0; t0 < nsb; t0 += 32) {
                Cand c;
                const int t = t0 + lane;
                c.valid = t < nsb;
                c.single = false;
                c.a = ka;
                c.b = R.b;
                c.h = 0.0;
                if (c.valid) {
                    const int hb = R.occb[t / R.nvb], pb = R.virb[t % R.nvb];
                    c.b = R.b ^ (1ull << hb) ^ (1ull << pb);
                    const int sa = 2 * ha, sb = 2 * hb + 1, ta = 2 * pa, tb = 2 * pb + 1;
                    const int i = max(sa, sb), j = min(sa, sb), A = max(ta, tb), B = min(ta, tb);
                    c.h = double_elem(R.a, R.b, i, j, A, B, anti_so_of(C.eri, i, j, A, B));
                }
                sink.step(c);
            }
        }
}

}  // namespace dnq
