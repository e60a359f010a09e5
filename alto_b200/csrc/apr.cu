// apr.cu -- CP-APR (multiplicative update) on the device.
//
// Replaces cp_apr_alto (IntelLabs/ALTO include/apr.hpp:984-1376) and
// tt_logLikelihood<LIT> (:851-982).  Order of operations follows the
// reference: KruskalModelNormalize, then per outer iteration and mode n the
// kappa fix (iter > 0), RedistributeLambda, up to max_inner rounds of
// {Phi, KKT violation, B *= Phi} with the early exit when the violation is
// below epsilon (skipped in bench mode), and KruskalModelNormalizeMode.  The
// KKT violation and the log-likelihood accumulate in FP64.
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "dense.cuh"
#include "mttkrp_kernels.cuh"
#include "mttkrp_plan.h"

namespace altob {

// |min(B, 1 - Phi)| max-reduced (apr.hpp:1210-1216); with `mult`, also
// B *= Phi (apr.hpp:1226-1231) in the same pass.  stop (if given): nothing is
// done once it is set.
template <typename FT, int VEC>
__global__ void __launch_bounds__(256) k_kkt(FT* __restrict__ B, const FT* __restrict__ Phi, u64 n,
                                             double* __restrict__ kkt, int mult, const int* __restrict__ stop)
{
    typedef typename VecT<FT, VEC>::T V;
    if (stop && *stop) return;
    __shared__ double red[8];
    double m = 0.0;
    for (u64 e = (u64)blockIdx.x * blockDim.x + threadIdx.x; e < n / VEC; e += (u64)gridDim.x * blockDim.x) {
        V bv = reinterpret_cast<const V*>(B)[e];
        const V pv = reinterpret_cast<const V*>(Phi)[e];
        FT* b = reinterpret_cast<FT*>(&bv);
        const FT* p = reinterpret_cast<const FT*>(&pv);
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
            m = fmax(m, fabs(fmin((double)b[k], 1.0 - (double)p[k])));
            if (mult) b[k] = (FT)((double)b[k] * (double)p[k]);
        }
        if (mult) reinterpret_cast<V*>(B)[e] = bv;
    }
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) m = fmax(m, red[w]);
        atomicMax(reinterpret_cast<unsigned long long*>(kkt), (unsigned long long)__double_as_longlong(m));
    }
}

template <typename FT>
__global__ void k_mult(FT* __restrict__ B, const FT* __restrict__ Phi, u64 n)
{
    for (u64 e = (u64)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (u64)gridDim.x * blockDim.x)
        B[e] = (FT)((double)B[e] * (double)Phi[e]);
}

// What a mode's queued inner rounds leave on the device: the violation of the
// round in flight (two slots, so the next one is zero before its round
// starts), that of the last round, how many rounds ran, and the flag that ends
// them.  A fixed size: the limit on the rounds may be any int.
struct Rounds {
    double kkt[2];
    double last;
    int count, stop;
};

// The end of inner round r without the host: records it, and stops the mode's
// rounds when the violation is below eps (every block reads the same value;
// one of them sets the flag that later launches read), else B *= Phi, and Phi
// is zeroed for the next round.
template <typename FT, int VEC>
__global__ void __launch_bounds__(256) k_round_end(FT* __restrict__ B, FT* __restrict__ Phi, u64 n,
                                                   Rounds* rd, int r, double eps, int zero)
{
    typedef typename VecT<FT, VEC>::T V;
    if (*(volatile int*)&rd->stop) return;
    const double kkt = rd->kkt[r & 1];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        rd->kkt[(r + 1) & 1] = 0.0;
        rd->last = kkt;
        rd->count = r + 1;
    }
    if (kkt < eps) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *(volatile int*)&rd->stop = 1;
        return;
    }
    for (u64 e = (u64)blockIdx.x * blockDim.x + threadIdx.x; e < n / VEC; e += (u64)gridDim.x * blockDim.x) {
        V bv = reinterpret_cast<const V*>(B)[e];
        const V pv = reinterpret_cast<const V*>(Phi)[e];
        FT* b = reinterpret_cast<FT*>(&bv);
        const FT* p = reinterpret_cast<const FT*>(&pv);
#pragma unroll
        for (int k = 0; k < VEC; ++k) b[k] = (FT)((double)b[k] * (double)p[k]);
        reinterpret_cast<V*>(B)[e] = bv;
        if (zero) vstore_zero<FT, VEC>(Phi + e * VEC);
    }
}

// The two above, in 16-byte pieces where B allows it (Phi is aligned).
template <typename FT>
static altob_status launch_kkt(FT* B, const FT* Phi, u64 n, double* kkt, int mult, const int* stop, cudaStream_t st)
{
    constexpr int V = 16 / sizeof(FT);
    const bool vec = ptr_aligned16(B) && n % V == 0;
    const u64 pieces = vec ? n / V : n;
    const int g = (int)std::max<u64>(1, std::min<u64>((pieces + 511) / 512, (u64)num_sms() * 8));
    if (vec) k_kkt<FT, V><<<g, 256, 0, st>>>(B, Phi, n, kkt, mult, stop);
    else k_kkt<FT, 1><<<g, 256, 0, st>>>(B, Phi, n, kkt, mult, stop);
    ALTOB_LAUNCH_CHECK();
    return ALTOB_OK;
}

template <typename FT>
static altob_status launch_round_end(FT* B, FT* Phi, u64 n, Rounds* rd, int r, double eps, int zero, cudaStream_t st)
{
    constexpr int V = 16 / sizeof(FT);
    const bool vec = ptr_aligned16(B) && n % V == 0;
    const u64 pieces = vec ? n / V : n;
    const int g = (int)std::max<u64>(1, std::min<u64>((pieces + 511) / 512, (u64)num_sms() * 8));
    if (vec) k_round_end<FT, V><<<g, 256, 0, st>>>(B, Phi, n, rd, r, eps, zero);
    else k_round_end<FT, 1><<<g, 256, 0, st>>>(B, Phi, n, rd, r, eps, zero);
    ALTOB_LAUNCH_CHECK();
    return ALTOB_OK;
}

// Kappa fix (apr.hpp:1176-1189).
template <typename FT>
__global__ void k_kappa(FT* __restrict__ B, const FT* __restrict__ Phi, u64 n, double kappa_tol, double kappa)
{
    for (u64 e = (u64)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (u64)gridDim.x * blockDim.x)
        if ((double)B[e] < kappa_tol && (double)Phi[e] > 1.0) B[e] = (FT)((double)B[e] + kappa);
}

template <typename FT>
struct LLArgs {
    KeySrc key;
    const void* vals;
    altob_dtype vdt;
    u64 nnz;
    int nmode, R;
    double eps;
    const FT* U[ALTOB_MAX_MODES];
    Fields fld;
};

// sum_nnz v * log(max(sum_r prod_n U_n[i_n, r], eps)) (apr.hpp:913-943).
//
// A warp takes 32 consecutive nonzeros: a lane decodes its own key, then the
// lane groups of LPN lanes walk their own LPN nonzeros one after the other
// with the row indices shuffled from the owning lane, so a row is read by
// neighbouring lanes in VEC-wide pieces (coalesced; all LPN x NM gathers of a
// step are independent).  Each lane keeps LPN partial dot products; a
// transposing butterfly (LPN - 1 exchanges instead of LPN log2 LPN) leaves
// the total of nonzero k of the group on its lane k, the lane that owns its
// value, and one log serves 32 nonzeros.  Products and sums in FP64.
// Bound: the L1 gathers (NM rows of R elements per nonzero).  One thread per
// nonzero, which this replaces, read 8 bytes per 32-byte sector request: the
// whole call took 1267 us for 4.7M nonzeros, order 4, rank 16, FP64; now 265.
template <typename FT, int NM, int LPN, int VEC>
__global__ void __launch_bounds__(256) k_loglik(LLArgs<FT> a, double* __restrict__ acc)
{
    constexpr int MM = NM ? NM : ALTOB_MAX_MODES;
    const int nmode = NM ? NM : a.nmode;
    const int R = a.R, lane = threadIdx.x & 31, sub = lane % LPN, base = lane - sub;
    __shared__ double red[8];
    double s = 0.0;
    const u64 step = (u64)gridDim.x * blockDim.x;
    for (u64 i0 = (u64)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < a.nnz; i0 += step) {
        const u64 i = i0 + lane;
        const bool ok = i < a.nnz;
        u32 c[MM];
        double v = 0.0;
#pragma unroll
        for (int m = 0; m < MM; ++m) c[m] = 0;  // past the end: row 0 of every factor, value 0
        if (ok) {
            const u64 lo = a.key.klo[i], hi = key_hi(a.key, i);
#pragma unroll
            for (int m = 0; m < MM; ++m)
                if (NM != 0 || m < nmode) c[m] = field(lo, hi, a.fld.pos[m], a.fld.mask[m]);
            v = a.vdt == ALTOB_U32   ? (double)reinterpret_cast<const u32*>(a.vals)[i]
                : a.vdt == ALTOB_F64 ? reinterpret_cast<const double*>(a.vals)[i]
                                     : (double)reinterpret_cast<const float*>(a.vals)[i];
        }
        double part[LPN];
#pragma unroll
        for (int k = 0; k < LPN; ++k) part[k] = 0.0;
        for (int r0 = 0; r0 < R; r0 += LPN * VEC) {
            // lanes past the rank read the row's last elements and drop them
            const int col = min(r0 + sub * VEC, R - VEC);
            const bool in = r0 + sub * VEC < R;
#pragma unroll
            for (int k = 0; k < LPN; ++k) {
                FT x[MM][VEC];
#pragma unroll
                for (int m = 0; m < MM; ++m) {
                    if (NM == 0 && m >= nmode) break;
                    const u32 row = __shfl_sync(0xffffffffu, c[m], base + k);
                    vload<FT, VEC>(a.U[m] + (size_t)row * R + col, x[m]);
                }
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    double p = (double)x[0][e];
#pragma unroll
                    for (int m = 1; m < MM; ++m) {
                        if (NM == 0 && m >= nmode) break;
                        p *= (double)x[m][e];
                    }
                    if (in) part[k] += p;
                }
            }
        }
#pragma unroll
        for (int o = LPN / 2; o > 0; o >>= 1) {
            // lanes with bit o keep the upper half of the nonzeros, the others the lower half
            const bool up = sub & o;
#pragma unroll
            for (int k = 0; k < o; ++k) {
                const double give = up ? part[k] : part[k + o];
                const double keep = up ? part[k + o] : part[k];
                part[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        double t = part[0];
        if (t < a.eps) t = a.eps;
        if (ok) s += v * log(t);
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)blockDim.x / 32; ++w) t += red[w];
        atomicAdd(acc, t);
    }
}

static int ew_grid(u64 n)
{
    u64 b = (n + 256 * 8 - 1) / (256 * 8);
    return (int)std::max<u64>(1, std::min<u64>(b, (u64)num_sms() * 8));
}

template <typename FT, int NM>
static void launch_loglik(const LLArgs<FT>& a, bool vec, int grid, double* acc, cudaStream_t st)
{
    constexpr int V = 16 / sizeof(FT);
    // four lanes where they hold a whole row, else eight walking it in pieces
    if (vec && a.R <= 4 * V) k_loglik<FT, NM, 4, V><<<grid, 256, 0, st>>>(a, acc);
    else if (vec) k_loglik<FT, NM, 8, V><<<grid, 256, 0, st>>>(a, acc);
    else k_loglik<FT, NM, 8, 1><<<grid, 256, 0, st>>>(a, acc);
}

// Adds the log-likelihood sum to *acc (zeroed by the caller).
template <typename FT>
static altob_status loglik_sum(const altob_tensor* t, FT** U, int R, double eps, double* acc, cudaStream_t st)
{
    if (t->nnz == 0) return ALTOB_OK;
    LLArgs<FT> a;
    memset(&a, 0, sizeof(a));
    a.key = key_src(t);
    a.vals = t->d_vals;
    a.vdt = t->vdt;
    a.nnz = t->nnz;
    a.nmode = t->nmode;
    a.R = R;
    a.eps = eps;
    bool vec = R % (16 / sizeof(FT)) == 0;
    for (int m = 0; m < t->nmode; ++m) {
        a.U[m] = U[m];
        vec = vec && ptr_aligned16(U[m]);
    }
    a.fld = t->fld;
    const int g = (int)std::max<u64>(1, std::min<u64>((t->nnz + 255) / 256, (u64)num_sms() * 8));
    switch (t->nmode) {
    case 3: launch_loglik<FT, 3>(a, vec, g, acc, st); break;
    case 4: launch_loglik<FT, 4>(a, vec, g, acc, st); break;
    case 5: launch_loglik<FT, 5>(a, vec, g, acc, st); break;
    default: launch_loglik<FT, 0>(a, vec, g, acc, st); break;
    }
    ALTOB_LAUNCH_CHECK();
    return ALTOB_OK;
}

struct AprScratch {
    double *lam, *colacc, *llacc, *kkt, *G, *inner, *fit, *normAT;
    Rounds* rounds;  // one per mode
    int* info;
};

// tt_logLikelihood (apr.hpp:851-982): lambda into mode 0, log-likelihood
// minus sum(U_0), then mode 0 renormalised by its column 1-norms.
// The caller provides every scratch word: lam (R) and acc (R column sums, the
// log-likelihood, the sum of U_0; one contiguous block, zeroed here in one
// call and read back in one copy).  This function and the helpers it calls
// must not allocate device memory, since altob_loglik_noalloc passes its
// fixed array here.
template <typename FT>
static altob_status loglik_impl(altob_tensor* t, FT** U, double* lam, double* acc, int R, double eps, double* out,
                                cudaStream_t st)
{
    ALTOB_CUDA(cudaMemsetAsync(acc, 0, (size_t)(R + 2) * sizeof(double), st));
    ALTOB_TRY(mul_cols<FT>(U[0], t->dims[0], R, lam, st));
    ALTOB_TRY(loglik_sum<FT>(t, U, R, eps, acc + R, st));
    ALTOB_TRY(colsum_abs_sum<FT>(U[0], t->dims[0], R, acc, acc + R + 1, st));
    ALTOB_TRY(div_cols<FT>(U[0], t->dims[0], R, acc, lam, true, st));
    double h[2];
    ALTOB_CUDA(cudaMemcpyAsync(h, acc + R, sizeof(h), cudaMemcpyDeviceToHost, st));
    ALTOB_CUDA(cudaStreamSynchronize(st));
    *out = h[0] - h[1];
    return ALTOB_OK;
}

// How Phi is formed: precomputed Khatri-Rao rows (the reference's PRE build)
// when a mode runs more than one inner iteration, in the row-ordered stream
// (PHI_ROWS: rows, values and stream positions kept per mode) when that fits
// in a quarter of free memory, else in ALTO order (PHI_PRE, the tiled
// kernel), else on the fly (PHI_OTF).  ALTOB_APR_PHI=rows|pre|otf forces one.
enum AprPhi { PHI_OTF = 0, PHI_PRE = 1, PHI_ROWS = 2 };

static AprPhi apr_phi_kind(const altob_tensor* t, int R, size_t fsz, int max_inner)
{
    const char* v = getenv("ALTOB_APR_PHI");
    if (v && !strcmp(v, "otf")) return PHI_OTF;
    if (v && !strcmp(v, "pre")) return PHI_PRE;
    if (v && !strcmp(v, "rows")) return PHI_ROWS;
    if (max_inner < 2) return PHI_OTF;
    const double nnz = (double)t->nnz, rows = nnz * ((double)R * fsz + t->nmode * (8.0 + fsz) + 24.0);
    // what an earlier solve left in the pool needs no question about free
    // memory (cudaMemGetInfo can take milliseconds)
    const size_t kept = pool_unused();
    if (rows <= (double)kept) return PHI_ROWS;
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) return PHI_OTF;
    fr += kept;
    if (rows <= 0.25 * (double)fr) return PHI_ROWS;
    return nnz * R * fsz <= 0.25 * (double)fr ? PHI_PRE : PHI_OTF;
}

// Rounds queued between two reads of the stop flag.
constexpr int APR_GROUP = 2;

// Two pinned words and events for reading a device flag behind the queue.
struct PollFlag {
    volatile int* h = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    bool init()
    {
        struct Words {  // kept while the host thread lives
            int* p = nullptr;
            ~Words()
            {
                if (p) cudaFreeHost(p);
            }
        };
        static thread_local Words words;
        cudaError_t e = cudaSuccess;
        if (!words.p) e = cudaHostAlloc((void**)&words.p, 2 * sizeof(int), cudaHostAllocPortable);
        if (e != cudaSuccess) words.p = nullptr;
        h = words.p;
        for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess;
    }
    ~PollFlag()
    {
        for (int k = 0; k < 2; ++k)
            if (ev[k]) cudaEventDestroy(ev[k]);
    }
};

template <typename FT>
static altob_status cp_apr_impl(altob_tensor* t, FT** U, FT* lam_io, int R, int max_iters, int max_inner,
                                double eps, double eps_div_zero, double kappa_tol, double kappa, int dobench,
                                double* summary, cudaStream_t st)
{
    const int N = t->nmode;
    const altob_dtype ft = sizeof(FT) == 8 ? ALTOB_F64 : ALTOB_F32;
    size_t phi_elems = 0;
    std::vector<size_t> phi_off(N);
    for (int n = 0; n < N; ++n) {
        phi_off[n] = phi_elems;
        phi_elems += (t->dims[n] * R + 63) & ~(size_t)63;
    }
    constexpr size_t RD = sizeof(Rounds) / sizeof(double);
    size_t nd = 5 * (size_t)R + (size_t)N * R * R + (size_t)N * RD + 16;
    size_t bytes = nd * sizeof(double) + 256 + phi_elems * sizeof(FT) + 256;
    void* base = nullptr;
    ALTOB_TRY(tensor_scratch(t, bytes, &base));
    double* d = (double*)base;
    AprScratch s;
    s.lam = d;
    d += R;
    s.colacc = d;
    d += R;
    s.inner = d;
    d += R;
    s.G = d;
    d += (size_t)N * R * R;
    s.kkt = d;
    d += 8;  // one per mode
    s.fit = d++;
    s.normAT = d++;
    s.llacc = d;
    d += R + 2;
    s.rounds = (Rounds*)d;
    d += (size_t)N * RD;
    s.info = (int*)d;
    d += 2;
    FT* phi_base = (FT*)(((uintptr_t)d + 255) & ~(uintptr_t)255);
    std::vector<FT*> Phi(N);
    for (int n = 0; n < N; ++n) Phi[n] = phi_base + phi_off[n];

    // KruskalModelNormalize (src/kruskal_model.cpp:128-176)
    ALTOB_TRY(vec_from<FT>(s.lam, lam_io, R, st));
    for (int n = 0; n < N; ++n) {
        ALTOB_TRY(colsum_abs<FT>(U[n], t->dims[n], R, s.colacc, st));
        ALTOB_TRY(div_cols<FT>(U[n], t->dims[n], R, s.colacc, s.lam, false, st));
    }
    std::vector<double> kkt_iter(max_iters + 1, 0.0), kmode(N, 0.0);
    std::vector<int> ninner(max_iters + 1, 0);
    void* pi = nullptr;  // nnz x R precomputed rows
    u32 *rows = nullptr, *inv = nullptr;  // row-ordered stream: N x nnz each
    FT* svals = nullptr;
    struct PiFree {
        void *p, *r, *i, *v;
        ~PiFree()
        {
            dfree(p);
            dfree(r);
            dfree(i);
            dfree(v);
        }
    } pi_free{nullptr, nullptr, nullptr, nullptr};
    const u64 nnz = t->nnz;
    // per-mode stride of the row-ordered stream: a multiple of 4 elements, so
    // every mode's arrays start 16-byte aligned and may be read to a multiple
    // of 4 past their end (bulk copies of whole 16-byte units)
    const u64 nnzp = (nnz + 3) & ~3ull;
    AprPhi kind = nnz ? apr_phi_kind(t, R, sizeof(FT), max_inner) : PHI_OTF;
    // Memory can go to other streams between the choice and the allocations
    // (concurrent requests of a server): an allocation that fails falls back
    // to the next path, which gives the same Phi.
    auto drop_stream = [&]() {
        dfree(rows);
        dfree(inv);
        dfree(svals);
        rows = inv = nullptr;
        svals = nullptr;
        pi_free.r = pi_free.i = pi_free.v = nullptr;
    };
    if (kind == PHI_ROWS) {
        altob_status a = dmalloc_t(&rows, (size_t)N * nnzp);
        pi_free.r = rows;
        if (a == ALTOB_OK) a = dmalloc_t(&inv, (size_t)N * nnzp);
        pi_free.i = inv;
        if (a == ALTOB_OK) a = dmalloc_t(&svals, (size_t)N * nnzp);
        pi_free.v = svals;
        for (int n = 0; n < N && a == ALTOB_OK; ++n)
            a = mode_order_device(t, n, ft, rows + (size_t)n * nnzp, svals + (size_t)n * nnzp,
                                  inv + (size_t)n * nnzp, st);
        if (a == ALTOB_ERR_NOMEM) {
            drop_stream();
            kind = PHI_PRE;
        } else if (a != ALTOB_OK) {
            return a;
        }
    }
    if (kind != PHI_OTF) {
        const altob_status a = dmalloc(&pi, nnz * (size_t)R * sizeof(FT));
        if (a == ALTOB_ERR_NOMEM) {
            drop_stream();
            pi = nullptr;
            kind = PHI_OTF;
        } else if (a != ALTOB_OK) {
            return a;
        }
        pi_free.p = pi;
    }
    // rounds without the host in between: the row-ordered stream through the
    // register-staged kernel (the opt-in bulk-copy kernel takes no stop flag),
    // while the host can have its poll words; else the host drives every round
    PollFlag poll;
    const bool queued = rows && !env_int("ALTOB_PHI_TMA", 0) && poll.init();
    std::vector<Rounds> hrounds(N);
    int iter;
    for (iter = 0; iter < max_iters; ++iter) {
        bool converged = false;
        if (dobench) ALTOB_CUDA(cudaMemsetAsync(s.kkt, 0, N * sizeof(double), st));
        for (int n = 0; n < N; ++n) {
            const u64 sz = t->dims[n] * (u64)R;
            FT* B = U[n];
            if (iter > 0 && sz) {
                k_kappa<FT><<<ew_grid(sz), 256, 0, st>>>(B, Phi[n], sz, kappa_tol, kappa);
                ALTOB_LAUNCH_CHECK();
            }
            // RedistributeLambda (lambda is 1 from here to the normalisation that sets it again)
            ALTOB_TRY(mul_cols<FT>(B, t->dims[n], R, s.lam, st));
            const u32* inv_n = rows ? inv + (size_t)n * nnzp : nullptr;
            if (pi) ALTOB_TRY(pi_device(t, n, ft, (void* const*)U, (u64)R, pi, st, inv_n));
            if (queued) {
                // every round of the mode is queued without waiting for its
                // violation: the rounds after the one that meets eps return at
                // once.  The stop flag is polled one group of rounds behind,
                // so the device never waits for the host and few empty rounds
                // are queued.
                Rounds* rd = s.rounds + n;
                int* stop = &rd->stop;
                const double stop_eps = dobench ? -1.0 : eps;  // bench mode: all rounds
                ALTOB_CUDA(cudaMemsetAsync(rd, 0, sizeof(Rounds), st));
                ALTOB_CUDA(cudaMemsetAsync(Phi[n], 0, sz * sizeof(FT), st));
                int group = 0;
                for (int r = 0; r < max_inner; ++r) {
                    ALTOB_TRY(phi_rows_device(t, n, ft, pi, rows + (size_t)n * nnzp, svals + (size_t)n * nnzp, B, (u64)R,
                                              eps_div_zero, Phi[n], st, true, stop));
                    ALTOB_TRY(launch_kkt<FT>(B, Phi[n], sz, rd->kkt + (r & 1), 0, stop, st));
                    ALTOB_TRY(launch_round_end<FT>(B, Phi[n], sz, rd, r, stop_eps, r + 1 < max_inner, st));
                    if (dobench || r + 1 == max_inner || (r + 1) % APR_GROUP) continue;
                    ALTOB_CUDA(cudaMemcpyAsync((int*)poll.h + group % 2, stop, sizeof(int), cudaMemcpyDeviceToHost, st));
                    ALTOB_CUDA(cudaEventRecord(poll.ev[group % 2], st));
                    if (group > 0) {
                        ALTOB_CUDA(cudaEventSynchronize(poll.ev[(group - 1) % 2]));
                        if (poll.h[(group - 1) % 2]) break;
                    }
                    ++group;
                }
            } else {
            for (int inner = 0; inner < max_inner; ++inner) {
                ninner[iter]++;
                if (rows)
                    ALTOB_TRY(phi_rows_device(t, n, ft, pi, rows + (size_t)n * nnzp, svals + (size_t)n * nnzp, B,
                                              (u64)R, eps_div_zero, Phi[n], st, true));
                else if (pi) ALTOB_TRY(phi_pre_device(t, n, ft, pi, B, (u64)R, eps_div_zero, Phi[n], st));
                else ALTOB_TRY(phi_device(t, n, ft, (void* const*)U, (u64)R, eps_div_zero, Phi[n], st));
                if (dobench) {
                    // no early exit: the violation of the last round is what the reference reports
                    ALTOB_CUDA(cudaMemsetAsync(s.kkt + n, 0, sizeof(double), st));
                    ALTOB_TRY(launch_kkt<FT>(B, Phi[n], sz, s.kkt + n, 1, nullptr, st));
                } else {
                    ALTOB_CUDA(cudaMemsetAsync(s.kkt + n, 0, sizeof(double), st));
                    ALTOB_TRY(launch_kkt<FT>(B, Phi[n], sz, s.kkt + n, 0, nullptr, st));
                    double kv = 0.0;
                    ALTOB_CUDA(cudaMemcpyAsync(&kv, s.kkt + n, sizeof(double), cudaMemcpyDeviceToHost, st));
                    ALTOB_CUDA(cudaStreamSynchronize(st));
                    kmode[n] = kv;
                    if (kv < eps) break;
                    if (sz) k_mult<FT><<<ew_grid(sz), 256, 0, st>>>(B, Phi[n], sz);
                    ALTOB_LAUNCH_CHECK();
                }
            }
            }
            // KruskalModelNormalizeMode (src/kruskal_model.cpp:178-222)
            ALTOB_TRY(colsum_abs<FT>(B, t->dims[n], R, s.colacc, st));
            ALTOB_TRY(div_cols<FT>(B, t->dims[n], R, s.colacc, s.lam, true, st));
        }
        if (queued) {
            ALTOB_CUDA(cudaMemcpyAsync(hrounds.data(), s.rounds, N * sizeof(Rounds), cudaMemcpyDeviceToHost, st));
            ALTOB_CUDA(cudaStreamSynchronize(st));
            for (int n = 0; n < N; ++n) {
                ninner[iter] += hrounds[n].count;
                kmode[n] = hrounds[n].last;
            }
        } else if (dobench) {
            ALTOB_CUDA(cudaMemcpyAsync(kmode.data(), s.kkt, N * sizeof(double), cudaMemcpyDeviceToHost, st));
            ALTOB_CUDA(cudaStreamSynchronize(st));
        }
        kkt_iter[iter] = kmode[0];
        for (int n = 1; n < N; ++n) kkt_iter[iter] = std::fmax(kkt_iter[iter], kmode[n]);
        // apr.hpp:1261; the first iteration has no predecessor to compare with
        if (iter > 0 && std::fabs(kkt_iter[iter] - kkt_iter[iter - 1]) <= eps * eps && !dobench) converged = true;
        if (converged) break;
    }
    int tot_inner = 0;
    for (int i = 0; i < iter; ++i) tot_inner += ninner[i];
    double ll = 0.0;
    ALTOB_TRY(loglik_impl<FT>(t, U, s.lam, s.llacc, R, eps_div_zero, &ll, st));

    // least-squares fit of the final model (apr.hpp:1301-1330)
    for (int n = 0; n < N - 1; ++n)
        ALTOB_TRY(gram<FT>(U[n], t->dims[n], R, s.G + (size_t)n * R * R, nullptr, nullptr, nullptr, nullptr, st));
    FT* mt = Phi[N - 1];
    {
        std::vector<void*> tmpU(N);
        for (int n = 0; n < N; ++n) tmpU[n] = U[n];
        tmpU[N - 1] = mt;
        // summed run by run, as this fit always was: per-CTA copies of a short
        // last mode would move the reported FP32 fit by about 1.5e-6 of its
        // value (4.7M counts, fit 4.6e-7: 1.7e-6 from the FP64 solve's fit so,
        // under 1e-7 with copies), away from what earlier runs reported
        ALTOB_TRY(mttkrp_device(t, N - 1, ft, tmpU.data(), (u64)R, 0, ALTOB_ALGO_AUTO, st, MT_RUN_SUMS));
    }
    ALTOB_TRY(gram<FT>(U[N - 1], t->dims[N - 1], R, s.G + (size_t)(N - 1) * R * R, nullptr, nullptr, mt, s.inner,
                       st));
    ALTOB_TRY(value_sumsq(t, s.normAT, st));
    double normAT = 0.0;
    ALTOB_CUDA(cudaMemcpyAsync(&normAT, s.normAT, sizeof(double), cudaMemcpyDeviceToHost, st));
    ALTOB_CUDA(cudaStreamSynchronize(st));
    ALTOB_TRY(fit_from(s.G, N, R, s.lam, s.inner, normAT, s.fit, st));
    double fit = 0.0;
    ALTOB_CUDA(cudaMemcpyAsync(&fit, s.fit, sizeof(double), cudaMemcpyDeviceToHost, st));
    ALTOB_TRY(vec_to<FT>(lam_io, s.lam, R, st));
    ALTOB_CUDA(cudaStreamSynchronize(st));
    if (t->h_tma_err && *t->h_tma_err)
        return fail(ALTOB_ERR_CUDA, "a bulk-copy-staged Phi pass ran out of a wait limit");
    if (summary) {
        summary[0] = ll;
        summary[1] = fit;
        summary[2] = iter > 0 ? kkt_iter[iter - 1] : kkt_iter[0];
        summary[3] = iter;
        summary[4] = tot_inner;
    }
    return ALTOB_OK;
}

}  // namespace altob

using namespace altob;

extern "C" {

altob_status altob_cp_apr(altob_tensor* t, altob_dtype ftype, void* const* d_factors, void* d_lambda, uint64_t rank,
                          int max_iters, int max_inner, double epsilon, double eps_div_zero, double kappa_tol,
                          double kappa, int dobench, double* summary, void* stream)
{
    ALTOB_TRY(check_model(t, ftype, d_factors, rank));
    if (!d_lambda) return fail(ALTOB_ERR_ARG, "lambda is NULL");
    if (max_iters < 1 || max_inner < 1) return fail(ALTOB_ERR_ARG, "iteration counts must be >= 1");
    if (t->nnz == 0) return fail(ALTOB_ERR_ARG, "CP-APR on an empty tensor");
    cudaStream_t st = (cudaStream_t)stream;
    StreamScope scope(st);
    if (ftype == ALTOB_F64)
        return cp_apr_impl<double>(t, (double**)d_factors, (double*)d_lambda, (int)rank, max_iters, max_inner,
                                   epsilon, eps_div_zero, kappa_tol, kappa, dobench, summary, st);
    return cp_apr_impl<float>(t, (float**)d_factors, (float*)d_lambda, (int)rank, max_iters, max_inner, epsilon,
                              eps_div_zero, kappa_tol, kappa, dobench, summary, st);
}

altob_status altob_loglik(altob_tensor* t, altob_dtype ftype, void* const* d_factors, void* d_lambda, uint64_t rank,
                          double eps_div_zero, double* loglik, void* stream)
{
    ALTOB_TRY(check_model(t, ftype, d_factors, rank));
    if (!d_lambda || !loglik) return fail(ALTOB_ERR_ARG, "NULL argument");
    cudaStream_t st = (cudaStream_t)stream;
    StreamScope scope(st);
    const int R = (int)rank;
    void* base = nullptr;
    ALTOB_TRY(tensor_scratch(t, (4 * (size_t)R + 8) * sizeof(double), &base));
    double* d = (double*)base;
    double *lam = d, *acc = d + R;
    if (ftype == ALTOB_F64) {
        ALTOB_TRY(vec_from<double>(lam, (const double*)d_lambda, R, st));
        ALTOB_TRY(loglik_impl<double>(t, (double**)d_factors, lam, acc, R, eps_div_zero, loglik, st));
        ALTOB_TRY(vec_to<double>((double*)d_lambda, lam, R, st));
    } else {
        ALTOB_TRY(vec_from<float>(lam, (const float*)d_lambda, R, st));
        ALTOB_TRY(loglik_impl<float>(t, (float**)d_factors, lam, acc, R, eps_div_zero, loglik, st));
        ALTOB_TRY(vec_to<float>((float*)d_lambda, lam, R, st));
    }
    ALTOB_CUDA(cudaStreamSynchronize(st));
    return ALTOB_OK;
}

}  // extern "C"


// ---------------------------------------------------------------------------
// altob_loglik_noalloc: the log-likelihood for callers that cannot allocate
// device memory.  Some callers own every byte of device memory through their
// own pool or arena, run where the CUDA allocator must not be entered, or
// need a call whose memory footprint is fixed before it runs; altob_loglik
// takes its scratch from the tensor handle's cache, which may call
// cudaMalloc.  This variant keeps its scratch in the file-scope array below
// instead.  The caller still passes the tensor, factors and lambda.

namespace altob {

// Largest rank the fixed scratch holds (the library's model rank limit):
// lambda and column sums (2R doubles) plus the two accumulators;
// 2 * 112 + 8 doubles = 1856 bytes per device.
constexpr int LOGLIK_NOALLOC_MAX_RANK = 112;
static __device__ __align__(256) double g_loglik_scratch[2 * LOGLIK_NOALLOC_MAX_RANK + 8];

// Device address of g_loglik_scratch on the current device.  Host code may
// not use the array's name as a device pointer, so the address is looked up
// once per device (on the first call there) and cached.
static altob_status loglik_scratch_address(double** out)
{
    static std::mutex mu;
    static std::vector<double*> addr;
    int dev = 0;
    ALTOB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if ((size_t)dev >= addr.size()) addr.resize((size_t)dev + 1, nullptr);
    if (!addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_loglik_scratch);
        if (e != cudaSuccess || !p)
            return fail(ALTOB_ERR_CUDA, std::string("cudaGetSymbolAddress(g_loglik_scratch): ") + cudaGetErrorString(e));
        addr[dev] = (double*)p;
    }
    *out = addr[dev];
    return ALTOB_OK;
}

}  // namespace altob

extern "C" altob_status altob_loglik_noalloc(altob_tensor* t, altob_dtype ftype, void* const* d_factors,
                                             void* d_lambda, uint64_t rank, double eps_div_zero, double* loglik,
                                             void* stream)
{
    if (rank > (uint64_t)LOGLIK_NOALLOC_MAX_RANK)
        return fail(ALTOB_ERR_ARG, "altob_loglik_noalloc: rank " + std::to_string(rank) +
                                       " exceeds the fixed scratch (maximum rank " +
                                       std::to_string(LOGLIK_NOALLOC_MAX_RANK) + ")");
    ALTOB_TRY(check_model(t, ftype, d_factors, rank));
    if (!d_lambda || !loglik) return fail(ALTOB_ERR_ARG, "NULL argument");
    double* d = nullptr;
    ALTOB_TRY(loglik_scratch_address(&d));
    cudaStream_t st = (cudaStream_t)stream;
    const int R = (int)rank;
    // every scratch word is written before it is read in this call:
    // lambda is loaded from d_lambda, the others are zeroed by their kernels
    double *lam = d, *acc = d + R;
    if (ftype == ALTOB_F64) {
        ALTOB_TRY(vec_from<double>(lam, (const double*)d_lambda, R, st));
        ALTOB_TRY(loglik_impl<double>(t, (double**)d_factors, lam, acc, R, eps_div_zero, loglik, st));
        ALTOB_TRY(vec_to<double>((double*)d_lambda, lam, R, st));
    } else {
        ALTOB_TRY(vec_from<float>(lam, (const float*)d_lambda, R, st));
        ALTOB_TRY(loglik_impl<float>(t, (float**)d_factors, lam, acc, R, eps_div_zero, loglik, st));
        ALTOB_TRY(vec_to<float>((float*)d_lambda, lam, R, st));
    }
    ALTOB_CUDA(cudaStreamSynchronize(st));
    return ALTOB_OK;
}
