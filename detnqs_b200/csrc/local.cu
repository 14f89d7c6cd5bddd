// local.cu -- matrix-free contraction sigma_i = sum_j H_ij c_j over a fixed
// basis and the variational energy E = sum_i c_i sigma_i
// (compute_variational_energy, local_conn.cpp:148-229).
//
// Large bases are matched by string groups (contract_strings, vvstr.cu); the
// others, and those the groups do not take (64 orbitals, duplicates, mixed
// electron counts), by the walk here.
//
// Same warp-per-row walk as the builder; hits in the basis are accumulated
// per lane with Dot2 (TwoProduct + TwoSum) and merged across the warp, and
// the row energies are summed with Dot2 again, so the result carries about
// twice FP64 precision before the final rounding.

#include "gen.cuh"

namespace dnq {

void check_orbitals(const u64* d, i64 n, int n_orb, cudaStream_t s);
void launch_diag(const dnq_ctx_s* c, const u64* d, i64 n, double* out, cudaStream_t s);
bool contract_strings(dnq_ctx_s* ctx, const u64* V, i64 n, const double* cd, int n_orb,
                      double single_thr, double cut, double* sigma, cudaStream_t s, double* e);

namespace {

constexpr int kWarps = 8;

__device__ __forceinline__ void tsum(double a, double b, double& s, double& e) {
    s = __dadd_rn(a, b);
    const double z = __dsub_rn(s, a);
    e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, z)), __dsub_rn(b, z));
}

struct DD {
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add_prod(double a, double b) {
        const double p = __dmul_rn(a, b);
        const double pe = fma(a, b, -p);
        double s2, e;
        tsum(s, p, s2, e);
        s = s2;
        c = __dadd_rn(c, __dadd_rn(e, pe));
    }
    __device__ __forceinline__ void merge(double os, double oc) {
        double s2, e;
        tsum(s, os, s2, e);
        s = s2;
        c = __dadd_rn(__dadd_rn(c, oc), e);
    }
};

struct ContractParams {
    CtxView C;
    DetMapView map;
    const u64* V;
    i64 n;
    const double* coeff;
    const double* diag;
    int n_orb;
    double single_thr;
    double cut;
    const i64* plen;
    int* next_row;
    double* part;     // per block (s, c)
    double* sigma;    // optional per-row sigma_i
};

struct ContractSink {
    const ContractParams& P;
    DD acc;
    __device__ explicit ContractSink(const ContractParams& p) : P(p) {}
    __device__ __forceinline__ void step(const Cand& c) {
        if (!c.valid) return;
        const double ah = fabs(c.h);
        if (!(ah > (c.single ? P.single_thr : kElemThresh))) return;
        const long long j = P.map.find(c.a, c.b);
        if (j >= 0) acc.add_prod(c.h, __ldg(&P.coeff[j]));
    }
};

__global__ void __launch_bounds__(kWarps * 32) k_contract(ContractParams P) {
    __shared__ WarpRow rows[kWarps];
    __shared__ double bs[kWarps], bc[kWarps];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpRow& R = rows[w];
    DD etot;   // meaningful in lane 0
    for (;;) {
        int r = 0;
        if (lane == 0) r = atomicAdd(P.next_row, 1);
        r = __shfl_sync(0xffffffffu, r, 0);
        if (r >= P.n) break;
        const double ci = P.coeff[r];
        if (ci * ci < 1e-12) {                  // local_conn.cpp:188
            if (P.sigma && lane == 0) P.sigma[r] = 0.0;
            continue;
        }
        load_row(R, P.V[2 * (i64)r], P.V[2 * (i64)r + 1], P.n_orb);
        ContractSink sink(P);
        enumerate_row(P.C, R, P.plen, P.cut, sink);
        DD sg = sink.acc;
        for (int o = 16; o; o >>= 1) {
            const double os = __shfl_xor_sync(0xffffffffu, sg.s, o);
            const double oc = __shfl_xor_sync(0xffffffffu, sg.c, o);
            sg.merge(os, oc);
        }
        if (lane == 0) {
            const double hd = P.diag[r];
            if (fabs(hd) > kElemThresh) sg.add_prod(hd, ci);
            const double sigma = sg.s + sg.c;
            if (P.sigma) P.sigma[r] = sigma;
            etot.add_prod(ci, sg.s);
            etot.add_prod(ci, sg.c);
        }
        __syncwarp();
    }
    if (lane == 0) { bs[w] = etot.s; bc[w] = etot.c; }
    __syncthreads();
    if (threadIdx.x == 0) {
        DD b;
        for (int k = 0; k < kWarps; ++k) b.merge(bs[k], bc[k]);
        P.part[2 * blockIdx.x] = b.s;
        P.part[2 * blockIdx.x + 1] = b.c;
    }
}

__global__ void k_final(const double* part, int nb, double* out) {
    if (threadIdx.x || blockIdx.x) return;
    DD a;
    for (int k = 0; k < nb; ++k) a.merge(part[2 * k], part[2 * k + 1]);
    *out = a.s + a.c;
}

// Prefix length of every table row for one cut; *kept sums them.
__global__ void k_prefix(PairTableView T, i64 nrows, double cut, i64* plen,
                         unsigned long long* kept) {
    unsigned long long sum = 0;
    for (i64 r = blockIdx.x * (i64)blockDim.x + threadIdx.x; r < nrows;
         r += (i64)gridDim.x * blockDim.x) {
        const i64 lo = T.off[r], len = T.off[r + 1] - lo;
        i64 L = 0, R = cut <= 0.0 ? 0 : len;
        while (L < R) {
            const i64 mid = L + (R - L) / 2;
            if (fabs(T.v[lo + mid]) >= cut) L = mid + 1; else R = mid;
        }
        if (cut <= 0.0) L = len;
        plen[r] = L;
        sum += L;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(kept, sum);
}

}  // namespace

// Whether the string groups contract faster than the candidate walk.  The
// walk takes about 0.1 us per candidate of a row (a warp steps through 32 at
// a time, a hash probe each) for every 2,500 rows, the groups 500 us more
// than the walk's own fixed cost, most of it sorting and indexing the
// basis.  Measured (walk / groups, us): 703 / 792 at 9.7e6 candidates (3,000
// rows of 14 orbitals), 1,726 / 876 at 3.2e7, 51,633 / 1,714 at 1.35e9 (20,011
// rows of 30 orbitals); 352 / 903 when a cut of 0.1 leaves few of 2.7e7.
// kept = share of the doubles the cut keeps.
bool contract_by_strings(i64 n, int n_orb, int na, int nb, double kept) {
    const double va = n_orb - na, vb = n_orb - nb;
    const double singles = na * va + nb * vb;
    const double doubles = 0.25 * na * (na - 1.0) * va * (va - 1.0) +
                           0.25 * nb * (nb - 1.0) * vb * (vb - 1.0) + na * va * nb * vb;
    return (singles + kept * doubles) * std::max(1.0, (double)n / 2500.0) > 5000.0;
}

// sigma (optional) and E for a fixed basis; returns E on the host.
double contract_energy(dnq_ctx_s* ctx, const u64* Vd, i64 n, const double* cd, int n_orb,
                       bool use_hb, double eps1, double* sigma, cudaStream_t s) {
    const double single_thr = use_hb ? std::max(eps1, kElemThresh) : kElemThresh;   // :176-178
    const double cut = use_hb ? hb_cutoff(ctx, eps1) : full_cutoff();
    const PairTableView tab = ctx->view().tab;
    DBuf<i64> plen(ctx->tab.n_rows, s);
    DBuf<unsigned long long> kept(1, s);
    DNQ_CUDA(cudaMemsetAsync(kept.p, 0, 8, s));
    k_prefix<<<64, 256, 0, s>>>(tab, ctx->tab.n_rows, cut, plen.p, kept.p);
    DNQ_CHECK_LAUNCH();
    if (n_orb < 64 && !default_options().force_walk) {
        u64 d0[2];
        unsigned long long hk = 0;
        DNQ_CUDA(cudaMemcpyAsync(d0, Vd, sizeof(d0), cudaMemcpyDeviceToHost, s));
        DNQ_CUDA(cudaMemcpyAsync(&hk, kept.p, 8, cudaMemcpyDeviceToHost, s));
        DNQ_CUDA(cudaStreamSynchronize(s));
        if (contract_by_strings(n, n_orb, __builtin_popcountll(d0[0]),
                                __builtin_popcountll(d0[1]),
                                (double)hk / std::max<double>(1.0, (double)ctx->tab.n_entries))) {
            try {
                double e = 0.0;
                if (contract_strings(ctx, Vd, n, cd, n_orb, single_thr, cut, sigma, s, &e))
                    return e;
            } catch (const Error& x) {   // the indices did not fit: the walk needs a map only
                if (x.code != DNQ_ERR_OUT_OF_MEMORY) throw;
            }
        }
    }
    DetMap map;
    build_detmap(map, Vd, n, false, s);
    DBuf<double> diag(n, s);
    launch_diag(ctx, Vd, n, diag.p, s);
    ContractParams P{};
    P.C = ctx->view();
    P.map = map.view();
    P.V = Vd;
    P.n = n;
    P.coeff = cd;
    P.diag = diag.p;
    P.n_orb = n_orb;
    P.single_thr = single_thr;
    P.cut = cut;
    P.plen = plen.p;
    DBuf<int> next(1, s);
    DNQ_CUDA(cudaMemsetAsync(next.p, 0, 4, s));
    P.next_row = next.p;
    int per_sm = 0;
    DNQ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_contract, kWarps * 32, 0));
    const int grid = std::max(1, per_sm) * sm_count(ctx->device);
    DBuf<double> part(2 * grid, s), out(1, s);
    P.part = part.p;
    P.sigma = sigma;
    k_contract<<<grid, kWarps * 32, 0, s>>>(P);
    DNQ_CHECK_LAUNCH();
    k_final<<<1, 32, 0, s>>>(part.p, grid, out.p);
    DNQ_CHECK_LAUNCH();
    double e = 0.0;
    DNQ_CUDA(cudaMemcpyAsync(&e, out.p, 8, cudaMemcpyDeviceToHost, s));
    DNQ_CUDA(cudaStreamSynchronize(s));
    return e;
}

}  // namespace dnq

using namespace dnq;

extern "C" {

int dnq_variational_energy(dnq_ctx_t ctx, const uint64_t* dets, int64_t n,
                           const double* coeffs, int n_orb, int use_heatbath, double eps1,
                           double* out, void* stream) {
    DNQ_API_BEGIN
    require_narrow(ctx);
    require(ctx && out, DNQ_ERR_INVALID, "null argument");
    require(n >= 0, DNQ_ERR_INVALID, "negative size");
    if (n == 0) { *out = 0.0; return DNQ_OK; }
    require(dets && coeffs, DNQ_ERR_INVALID, "null argument");
    require(n_orb >= 1 && n_orb <= ctx->n, DNQ_ERR_INVALID,
            "n_orb must be in [1, number of orbitals of the integral context]");
    if (use_heatbath)
        require(ctx->has_hb, DNQ_ERR_NO_HEATBATH,
                "compute_variational_energy: Heat-Bath mode requires non-null hb_table");
    DeviceGuard g(ctx->device);
    cudaStream_t s = (cudaStream_t)stream;
    DIn<u64> d(dets, 2 * n, s);
    DIn<double> c(coeffs, n, s);
    check_orbitals(d.p, n, n_orb, s);
    *out = contract_energy(ctx, d.p, n, c.p, n_orb, use_heatbath != 0, eps1, nullptr, s);
    DNQ_API_END
}

}  // extern "C"
