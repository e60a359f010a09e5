// build.cu -- ALTO tensor build on the device.
//
// Replaces create_alto (IntelLabs/ALTO include/alto.hpp:108-294):
//   setup_packed_alto  (alto.hpp:669-770)  -> host, make_masks()
//   pdep linearization (alto.hpp:184-202)  -> k_linearize (field layout), digits gathered in the sort
//   sort_alto          (alto.hpp:772-803)  -> alto_sort (radix.cu)
//   oidx               (alto.hpp:246-285)  -> radix sort of mode indices
//   prtn_alto          (alto.hpp:805-899)  -> k_intervals
//   CR bits            (alto.hpp:930-1027) -> k_cr_shared + k_cr_set
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "internal.cuh"

namespace altob {

// ------------------------------------------------------------- errors

static thread_local std::string g_last_error;

void set_error(const std::string& msg) { g_last_error = msg; }

altob_status fail(altob_status s, const std::string& msg)
{
    set_error(msg);
    return s;
}

static thread_local cudaStream_t g_alloc_stream = 0;

StreamScope::StreamScope(cudaStream_t s) : prev(g_alloc_stream) { g_alloc_stream = s; }
StreamScope::~StreamScope() { g_alloc_stream = prev; }

// The library's own stream-ordered pool of the current device.  The default
// pool hands unused memory back to the system at every synchronisation, which
// made a build spend 8 ms in its 22 allocations; this one keeps up to 1/32 of
// the device's memory (5.7 GB of 180) between calls.  Kept memory is returned
// by altob_trim_memory, and by the driver when another allocation of the
// process needs it (with 3.2 GB kept, 174.4 free, a cudaMalloc of 176.0 GB was
// given).  nullptr: pools cannot be made here, use the default one.
static cudaMemPool_t device_pool()
{
    static std::mutex mu;
    static std::vector<std::pair<bool, cudaMemPool_t>> pools;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= (int)pools.size()) pools.resize(dev + 1, {false, nullptr});
    if (!pools[dev].first) {
        cudaMemPoolProps pr;
        memset(&pr, 0, sizeof(pr));
        pr.allocType = cudaMemAllocationTypePinned;
        pr.location.type = cudaMemLocationTypeDevice;
        pr.location.id = dev;
        size_t fr = 0, tot = 0;
        cudaMemPool_t p = nullptr;
        if (cudaMemGetInfo(&fr, &tot) == cudaSuccess && cudaMemPoolCreate(&p, &pr) == cudaSuccess) {
            u64 keep = tot / 32;
            cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        } else {
            cudaGetLastError();
            p = nullptr;
        }
        pools[dev] = {true, p};
    }
    return pools[dev].second;
}

size_t pool_unused()
{
    cudaMemPool_t p = device_pool();
    u64 reserved = 0, used = 0;
    if (!p || cudaMemPoolGetAttribute(p, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(p, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return reserved > used ? (size_t)(reserved - used) : 0;
}

altob_status dmalloc(void** p, size_t bytes)
{
    *p = nullptr;
    cudaMemPool_t pool = device_pool();
    cudaError_t e = pool ? cudaMallocFromPoolAsync(p, bytes ? bytes : 1, pool, g_alloc_stream)
                         : cudaMallocAsync(p, bytes ? bytes : 1, g_alloc_stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return fail(e == cudaErrorMemoryAllocation ? ALTOB_ERR_NOMEM : ALTOB_ERR_CUDA,
                    std::string("cudaMalloc(") + std::to_string(bytes) + "): " + cudaGetErrorString(e));
    }
    return ALTOB_OK;
}

void dfree(void* p)
{
    if (p) cudaFreeAsync(p, g_alloc_stream);
}

altob_status tensor_scratch(altob_tensor* t, size_t bytes, void** out)
{
    if (bytes > t->scratch_bytes) {
        if (t->scratch) {
            dfree(t->scratch);  // stream-ordered: after this stream's earlier uses
            t->scratch = nullptr;
            t->scratch_bytes = 0;
        }
        size_t want = std::max(bytes, (size_t)1 << 20);
        ALTOB_TRY(dmalloc(&t->scratch, want));
        t->scratch_bytes = want;
    }
    *out = t->scratch;
    return ALTOB_OK;
}

bool stream_capturing(cudaStream_t st)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return cs != cudaStreamCaptureStatusNone;
}

// Buffers that outlive the call are never grown while st is being captured:
// the allocation would belong to the graph.  A buffer that a captured call
// has used stays allocated until the handle is destroyed, since the graph
// keeps its address: it is set aside when a later call needs a larger one.
static altob_status grow_buf(altob_tensor* t, HandleBuf* b, size_t bytes, void** out, cudaStream_t st)
{
    const bool cap = stream_capturing(st);
    if (bytes > b->bytes) {
        if (cap) return fail(ALTOB_ERR_NOMEM, "a handle's buffer cannot grow during stream capture");
        if (b->in_graph) t->set_aside.push_back({b->p, b->bytes});
        else dfree(b->p);
        *b = HandleBuf();
        ALTOB_TRY(dmalloc(&b->p, bytes));
        b->bytes = bytes;
    }
    b->in_graph = b->in_graph || cap;
    *out = b->p;
    return ALTOB_OK;
}

altob_status tensor_hotbuf(altob_tensor* t, size_t bytes, void** out, cudaStream_t st)
{
    return grow_buf(t, &t->hotbuf, bytes, out, st);
}

altob_status tensor_padbuf(altob_tensor* t, size_t bytes, void** out, cudaStream_t st)
{
    return grow_buf(t, &t->padbuf, bytes, out, st);
}

altob_status tensor_enter(altob_tensor* t, cudaStream_t st)
{
    if (!t->use_ev || t->use_stream == st || stream_capturing(st)) return ALTOB_OK;
    ALTOB_CUDA(cudaStreamWaitEvent(st, t->use_ev, 0));
    return ALTOB_OK;
}

altob_status tensor_leave(altob_tensor* t, cudaStream_t st)
{
    if (stream_capturing(st)) return ALTOB_OK;
    if (!t->use_ev) ALTOB_CUDA(cudaEventCreateWithFlags(&t->use_ev, cudaEventDisableTiming));
    ALTOB_CUDA(cudaEventRecord(t->use_ev, st));
    t->use_stream = st;
    return ALTOB_OK;
}

// SM count of the current device, cached per device ordinal.
int num_sms()
{
    static std::mutex mu;
    static std::vector<int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= (int)cache.size()) cache.resize(dev + 1, 0);
    if (cache[dev] <= 0) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cache[dev] = sms > 0 ? sms : 148;
    }
    return cache[dev];
}

// ------------------------------------------------------------ masks

static int mode_bits(u64 d) { return d <= 1 ? 0 : 64 - __builtin_clzll(d - 1); }

// setup_packed_alto(LSB_FIRST, SHORT_FIRST), alto.hpp:669-770: modes in
// ascending bit count (ties in mode order), one bit per mode per level,
// starting at the least significant bit.
static int make_masks(int nmode, const u64* dims, u128* masks, int* order)
{
    int bits[ALTOB_MAX_MODES], total = 0;
    for (int n = 0; n < nmode; ++n) {
        bits[n] = mode_bits(dims[n]);
        order[n] = n;
        total += bits[n];
        masks[n] = 0;
    }
    std::stable_sort(order, order + nmode, [&](int a, int b) { return bits[a] < bits[b]; });
    int shift = 0;
    for (int level = 0;; ++level) {
        bool done = true;
        for (int k = 0; k < nmode; ++k) {
            int n = order[k];
            if (level < bits[n]) {
                masks[n] |= (u128)1 << shift;
                ++shift;
                done = false;
            }
        }
        if (done) break;
    }
    return total;
}

Decoder make_decoder(int nmode, const u128* masks, int alto_bits)
{
    Decoder d;
    memset(&d, 0, sizeof(d));
    d.nmode = nmode;
    d.nwords = std::max(1, (alto_bits + 31) / 32);
    for (int n = 0; n < nmode; ++n) {
        u32 off = 0;
        for (int w = 0; w < 4; ++w) {
            u32 m = (u32)(masks[n] >> (32 * w));
            WordDec& wd = d.md[n].w[w];
            wd.m = m;
            wd.off = m ? off : 0;
            compress_moves(m, wd.mv);
            off += __builtin_popcount(m);
        }
    }
    return d;
}

// ------------------------------------------------------ build kernels

// Linearization (alto.hpp:184-202) straight into the device's field layout:
// every mode index at its bit field, bits past 64 in `hi` (HI wide, or none).
// The ALTO order of these keys is read off them digit by digit when they are
// sorted.  Also validates every coordinate against its dimension.
struct DimMax {
    u64 d[ALTOB_MAX_MODES];
};

template <typename HI>
__global__ void __launch_bounds__(256) k_linearize(const u64* __restrict__ cidx, u64 nnz, Fields f, DimMax dm,
                                                   u64* __restrict__ klo, HI* __restrict__ khi, int* __restrict__ bad)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (u64)gridDim.x * blockDim.x) {
        u64 lo = 0, hi = 0;
#pragma unroll
        for (int m = 0; m < ALTOB_MAX_MODES; ++m) {
            if (m >= f.nmode) break;
            u64 c = cidx[(u64)m * nnz + i];
            if (c >= dm.d[m]) {
                atomicExch(bad, 1);
                c = 0;
            }
            const u32 p = f.pos[m];
            if (p < 64) {
                lo |= c << p;
                if (p > 32) hi |= c >> (64 - p);
            } else {
                hi |= c << (p - 64);
            }
        }
        klo[i] = lo;
        if (khi) khi[i] = (HI)hi;
    }
}

// The high words of a sort as explicit 64-bit words.
template <typename HI>
__global__ void k_widen_hi(const HI* __restrict__ in, u64 n, u64* __restrict__ out)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        out[i] = in ? (u64)in[i] : 0;
}

template <typename VI, typename VO>
__global__ void k_gather_vals(const VI* __restrict__ in, const u32* __restrict__ perm, u64 n, VO* __restrict__ out)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        out[i] = (VO)in[perm[i]];
}

// Field layout -> interleaved ALTO key (for altob_dump); bits at and above
// alto_bits (the CR bits) are copied unchanged.
__global__ void k_interleave(const u64* __restrict__ klo, KeySrc ks, int alto_bits, u64 n, Decoder dec, Fields f,
                             u64* __restrict__ olo, u64* __restrict__ ohi)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 lo = klo[i], hi = key_hi(ks, i);
        u32 w[4] = {0, 0, 0, 0};
        for (int m = 0; m < dec.nmode; ++m) {
            const u32 c = field(lo, hi, f.pos[m], f.mask[m]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const WordDec& wd = dec.md[m].w[q];
                if (q < dec.nwords && wd.m) w[q] |= expand32(c >> wd.off, wd);
            }
        }
        u64 ilo = (u64)w[0] | ((u64)w[1] << 32), ihi = (u64)w[2] | ((u64)w[3] << 32);
        if (alto_bits < 64) ilo |= lo & (~0ull << alto_bits);
        if (alto_bits <= 64) ihi |= hi;  // every high bit is a CR bit
        else ihi |= hi & (~0ull << (alto_bits - 64));
        olo[i] = ilo;
        ohi[i] = ihi;
    }
}

// Mode indices of the sorted keys (for the oidx sort).
template <typename HI>
__global__ void k_mode_keys(const u64* __restrict__ klo, const HI* __restrict__ khi, u64 n, Fields f, int mode,
                            u32* __restrict__ out)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        out[i] = field(klo[i], khi ? (u64)khi[i] : 0ull, f.pos[mode], f.mask[mode]);
}

__global__ void k_init_intervals(u64* iv, int nprtn, int nmode, u64 d0, u64 d1, u64 d2, u64 d3, u64 d4)
{
    const u64 dm[5] = {d0, d1, d2, d3, d4};
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nprtn * nmode) {
        iv[2 * k] = dm[k % nmode];
        iv[2 * k + 1] = 0;
    }
}

// Per-partition min / max of every mode index (prtn_alto, alto.hpp:874-899).
// A warp walks IV_CHUNK consecutive keys, keeps the extremes of the current
// partition in registers and adds them to the table once per partition it
// meets (one atomic pair per 32 keys took 452 us on 20.2M keys).
constexpr u64 IV_CHUNK = 1024;

template <typename HI>
__global__ void __launch_bounds__(256) k_intervals(const u64* __restrict__ klo, const HI* __restrict__ khi, u64 n,
                                                   Fields f, u64 per, u64* __restrict__ iv)
{
    const int lane = threadIdx.x & 31;
    const u64 nw = ((u64)gridDim.x * blockDim.x) >> 5;
    for (u64 c = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * IV_CHUNK < n; c += nw) {
        u64 i0 = c * IV_CHUNK;
        const u64 stop = min(n, i0 + IV_CHUNK);
        u64 p = i0 / per;
        while (i0 < stop) {
            const u64 seg = min(stop, (p + 1) * per);
            u32 mn[ALTOB_MAX_MODES], mx[ALTOB_MAX_MODES];
#pragma unroll
            for (int m = 0; m < ALTOB_MAX_MODES; ++m) {
                mn[m] = 0xffffffffu;
                mx[m] = 0;
            }
#pragma unroll 4
            for (u64 i = i0 + lane; i < seg; i += 32) {
                const u64 lo = klo[i], hi = khi ? (u64)khi[i] : 0;
#pragma unroll
                for (int m = 0; m < ALTOB_MAX_MODES; ++m) {
                    if (m >= f.nmode) break;
                    const u32 x = field(lo, hi, f.pos[m], f.mask[m]);
                    mn[m] = min(mn[m], x);
                    mx[m] = max(mx[m], x);
                }
            }
#pragma unroll
            for (int m = 0; m < ALTOB_MAX_MODES; ++m) {
                if (m >= f.nmode) break;
                const u32 a = __reduce_min_sync(0xffffffffu, mn[m]), b = __reduce_max_sync(0xffffffffu, mx[m]);
                if (lane == 0) {
                    u64* e = iv + (p * f.nmode + m) * 2;
                    atomicMin((unsigned long long*)e, (unsigned long long)a);
                    atomicMax((unsigned long long*)(e + 1), (unsigned long long)b);
                }
            }
            i0 = seg;
            ++p;
        }
    }
}

struct CrArgs {
    int* owner[ALTOB_MAX_MODES];
    int bitpos[ALTOB_MAX_MODES];  // -1 = no CR bit for this mode
};

// Fibers that several partitions share (alto.hpp:970-996), from the mode's
// sorted order: a fiber's nonzeros stand together with ascending positions,
// so it is shared iff two neighbours lie in different partitions.  (Claiming
// owners with one compare-and-swap per nonzero took 3558 us on 20.2M
// nonzeros, serialised on the head rows.)
__global__ void k_cr_shared(const u32* __restrict__ key, const u32* __restrict__ pos, u64 n, u32 per,
                            int* __restrict__ owner)
{
    for (u64 k = (u64)blockIdx.x * blockDim.x + threadIdx.x; k + 1 < n; k += (u64)gridDim.x * blockDim.x) {
        const u32 c = key[k];
        if (c == key[k + 1] && pos[k] / per != pos[k + 1] / per) owner[c] = -1;
    }
}

// Sets the CR bits of nonzeros whose fiber is shared (alto.hpp:998-1019) in
// klo and the explicit high words khi (if any); src holds the high words the
// mode indices are read from.
template <typename HI>
__global__ void k_cr_set(u64* __restrict__ klo, u64* __restrict__ khi, u64 n, Fields f, CrArgs a,
                         const HI* __restrict__ src)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 lo = klo[i], hi = src ? (u64)src[i] : 0;
        u64 add_lo = 0, add_hi = 0;
        for (int m = 0; m < f.nmode; ++m) {
            int b = a.bitpos[m];
            if (b < 0) continue;
            u32 c = field(lo, hi, f.pos[m], f.mask[m]);
            if (a.owner[m][c] == -1) {
                if (b < 64) add_lo |= 1ull << b;
                else add_hi |= 1ull << (b - 64);
            }
        }
        if (add_lo) klo[i] = lo | add_lo;
        if (add_hi && khi) khi[i] = hi | add_hi;
    }
}

// Positions where the high key word changes (for the run table) and a
// check that it never decreases; either outcome that rules the table out ends
// the search.
template <typename HI>
__global__ void k_hi_runs(const HI* __restrict__ khi, u64 n, u64* __restrict__ starts, u32 cap,
                          u32* __restrict__ count, u32* __restrict__ decreasing)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        if (i == 0 || khi[i] != khi[i - 1]) {
            if (*(volatile u32*)decreasing || *(volatile u32*)count > cap) return;
            if (i > 0 && khi[i] < khi[i - 1]) atomicExch(decreasing, 1u);
            u32 k = atomicAdd(count, 1u);
            if (k < cap) starts[k] = i;
        }
    }
}

template <typename HI>
__global__ void k_gather_hi(const HI* __restrict__ src, const u64* __restrict__ idx, u32 n, u64* __restrict__ out)
{
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = (u64)src[idx[i]];
}

// Explicit high key word of every nonzero of a tensor that keeps them as a
// run table.
__global__ void k_expand_hi(KeySrc key, u64 n, u64* __restrict__ hi)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        hi[i] = key_hi(key, i);
}

static int intervals_grid(u64 n)
{
    const u64 warps = (n + IV_CHUNK - 1) / IV_CHUNK;
    return (int)std::max<u64>(1, std::min<u64>((warps + 7) / 8, (u64)num_sms() * 8));
}

static int grid_for(u64 n, int threads)
{
    u64 blocks = (n + threads - 1) / threads;
    u64 cap = (u64)num_sms() * 16;
    return (int)std::max<u64>(1, std::min(blocks, cap));
}

// ------------------------------------------------------------ create

// HI: the type the key bits past 64 have while they are sorted (hi_bytes
// wide; 0: the keys fit 64 bits).
template <typename HI>
static altob_status build(altob_tensor* t, const u64* d_cidx, const void* d_vals_in, altob_dtype vin, int hi_bytes,
                          cudaStream_t st)
{
    const u64 nnz = t->nnz;
    u64 *klo = nullptr, *klo2 = nullptr, *khi64 = nullptr, *starts = nullptr, *d_iv = nullptr;
    HI *khi = nullptr, *khi2 = nullptr;
    u32 *perm = nullptr, *perm2 = nullptr;
    u32* flags = nullptr;  // a coordinate out of range | high-word runs | a high word decreases
    CrArgs ca;
    memset(&ca, 0, sizeof(ca));
    altob_status s = ALTOB_OK;
    auto cleanup = [&] {
        dfree(klo2);
        dfree(khi);
        dfree(khi2);
        dfree(perm);
        dfree(perm2);
        dfree(flags);
        dfree(starts);
        dfree(d_iv);
        for (int n = 0; n < ALTOB_MAX_MODES; ++n) dfree(ca.owner[n]);
        if (s != ALTOB_OK) {
            dfree(klo);
            dfree(khi64);
            cudaStreamSynchronize(st);  // the caller's arrays are not read after the return
        }
    };
#define BTRY(x)             \
    do {                    \
        s = (x);            \
        if (s != ALTOB_OK) { \
            cleanup();      \
            return s;       \
        }                   \
    } while (0)
#define BLAUNCH(what)                                                                             \
    do {                                                                                          \
        const cudaError_t e_ = cudaGetLastError();                                                \
        if (e_ != cudaSuccess)                                                                    \
            BTRY(fail(ALTOB_ERR_CUDA, std::string(what " launch: ") + cudaGetErrorString(e_)));   \
    } while (0)
    const int grid = grid_for(nnz, 256);
    BTRY(dmalloc_t(&klo, nnz));
    BTRY(dmalloc_t(&klo2, nnz));
    if (hi_bytes) {
        BTRY(dmalloc_t(&khi, nnz));
        BTRY(dmalloc_t(&khi2, nnz));
    }
    BTRY(dmalloc_t(&perm, nnz));
    BTRY(dmalloc_t(&perm2, nnz));
    BTRY(dmalloc_t(&flags, 3));
    cudaMemsetAsync(flags, 0, 3 * sizeof(u32), st);
    DimMax dm;
    for (int n = 0; n < ALTOB_MAX_MODES; ++n) dm.d[n] = n < t->nmode ? t->dims[n] : 1;
    if (nnz) {
        k_linearize<HI><<<grid, 256, 0, st>>>(d_cidx, nnz, t->fld, dm, klo, khi, (int*)flags);
        BLAUNCH("k_linearize");
    }
    bool in_alt = false;
    BTRY(alto_sort(klo, khi, perm, klo2, khi2, perm2, nnz, hi_bytes, t->masks, t->fld, t->alto_bits, st, &in_alt));
    if (in_alt) {
        std::swap(klo, klo2);
        std::swap(khi, khi2);
        std::swap(perm, perm2);
    }
    // values in sorted order, converted to the stored dtype
    size_t vsz = val_size(t->vdt);
    BTRY(dmalloc(&t->d_vals, nnz * vsz + 16));
    if (nnz) {
#define GATHER(VI, VO) \
    k_gather_vals<VI, VO><<<grid, 256, 0, st>>>((const VI*)d_vals_in, perm, nnz, (VO*)t->d_vals)
        if (vin == ALTOB_F64 && t->vdt == ALTOB_F64) GATHER(double, double);
        else if (vin == ALTOB_F64 && t->vdt == ALTOB_F32) GATHER(double, float);
        else if (vin == ALTOB_F32 && t->vdt == ALTOB_F32) GATHER(float, float);
        else if (vin == ALTOB_F32 && t->vdt == ALTOB_F64) GATHER(float, double);
        else if (vin == ALTOB_U32 && t->vdt == ALTOB_U32) GATHER(u32, u32);
        else if (vin == ALTOB_F64 && t->vdt == ALTOB_U32) GATHER(double, u32);
        else BTRY(fail(ALTOB_ERR_UNSUPPORTED, "value dtype conversion not supported"));
#undef GATHER
        BLAUNCH("k_gather_vals");
    }

    const int np = t->nprtn, nm = t->nmode;
    const u64 per = (nnz + (u64)np - 1) / (u64)np;
    // which modes get CR bits (alto.hpp:932-968): all of them have an oidx
    int free_bits = t->lit_bits - t->alto_bits;
    bool any_cr = false, cr_hi = false;
    t->alto_cr_mask = 0;
    for (int n = 0; n < nm; ++n) {
        ca.bitpos[n] = -1;
        t->cr_masks[n] = 0;
        if (fib_reuse(t, n) <= 4 && free_bits) {
            int b = t->lit_bits - free_bits;
            ca.bitpos[n] = b;
            t->cr_masks[n] = (u128)1 << b;
            t->alto_cr_mask |= t->cr_masks[n];
            --free_bits;
            any_cr = true;
            cr_hi = cr_hi || b >= 64;
        }
    }
    // oidx for low-reuse modes (alto.hpp:246-285)
    t->is_oidx = 0;
    for (int n = 0; n < t->nmode; ++n)
        if (fib_reuse(t, n) <= 4) t->is_oidx = 1;
    if (t->is_oidx && nnz) {
        for (int n = 0; n < t->nmode; ++n) {
            if (fib_reuse(t, n) > 4) continue;
            // klo2 / perm2 are free at this point: two 32-bit key arrays, one payload
            u32 *mk = (u32*)klo2, *ox2 = nullptr;
            BTRY(dmalloc_t(&ox2, nnz));
            k_mode_keys<HI><<<grid, 256, 0, st>>>(klo, khi, nnz, t->fld, n, mk);
            bool alt2 = false;
            s = radix_argsort_u32(mk, perm2, mk + nnz, ox2, nnz, mode_bits(t->dims[n]), st, &alt2);
            if (s == ALTOB_OK && ca.bitpos[n] >= 0) s = dmalloc_t(&ca.owner[n], t->dims[n]);
            if (s != ALTOB_OK) {
                dfree(ox2);
                cleanup();
                return s;
            }
            if (ca.bitpos[n] >= 0) {
                cudaMemsetAsync(ca.owner[n], 0, t->dims[n] * sizeof(int), st);
                k_cr_shared<<<grid, 256, 0, st>>>(alt2 ? mk + nnz : mk, alt2 ? ox2 : perm2, nnz, (u32)per, ca.owner[n]);
                BLAUNCH("k_cr_shared");
            }
            if (alt2) {
                t->d_oidx[n] = ox2;
            } else {
                t->d_oidx[n] = perm2;
                perm2 = ox2;
            }
        }
    }

    // partitions (alto.hpp:822-836) and intervals (:874-899)
    t->prtn_ptr.assign(np + 1, 0);
    for (int p = 0; p < np; ++p) t->prtn_ptr[p + 1] = std::min<u64>((u64)(p + 1) * per, nnz);
    BTRY(dmalloc_t(&d_iv, (u64)np * nm * 2));
    k_init_intervals<<<(np * nm + 255) / 256, 256, 0, st>>>(d_iv, np, nm, dm.d[0], dm.d[1], dm.d[2], dm.d[3], dm.d[4]);
    if (nnz) k_intervals<HI><<<intervals_grid(nnz), 256, 0, st>>>(klo, khi, nnz, t->fld, per, d_iv);
    BLAUNCH("k_intervals");
    t->intervals.assign((size_t)np * nm * 2, 0);

    if (any_cr && nnz) {
        if (cr_hi) {  // CR bits past 64: explicit high words
            BTRY(dmalloc_t(&khi64, nnz));
            k_widen_hi<HI><<<grid, 256, 0, st>>>(khi, nnz, khi64);
        }
        k_cr_set<<<grid, 256, 0, st>>>(klo, khi64, nnz, t->fld, ca, khi);
        BLAUNCH("CR bits");
    }
    // high key words: a run table when they never decrease along the stream
    // (the usual case: they are the top ALTO bits), else one word per nonzero
    const u32 cap = 1u << 16;
    const bool has_hi = t->kw == 2 && nnz;
    if (has_hi) {
        BTRY(dmalloc_t(&starts, cap));
        if (khi64) k_hi_runs<u64><<<grid, 256, 0, st>>>(khi64, nnz, starts, cap, flags + 1, flags + 2);
        else k_hi_runs<HI><<<grid, 256, 0, st>>>(khi, nnz, starts, cap, flags + 1, flags + 2);
        BLAUNCH("k_hi_runs");
    }
    // one wait for the whole build
    u32 hf[3] = {0, 0, 0};
    cudaMemcpyAsync(hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(t->intervals.data(), d_iv, t->intervals.size() * sizeof(u64), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) BTRY(fail(ALTOB_ERR_CUDA, std::string("tensor build: ") + cudaGetErrorString(e)));
    if (hf[0]) BTRY(fail(ALTOB_ERR_ARG, "a coordinate is not below its dimension"));
    if (has_hi && hf[2] == 0 && hf[1] <= cap) {
        std::vector<u64> hs(hf[1]);
        cudaMemcpyAsync(hs.data(), starts, hf[1] * sizeof(u64), cudaMemcpyDeviceToHost, st);
        cudaStreamSynchronize(st);
        std::sort(hs.begin(), hs.end());
        u64 *rs = nullptr, *rv = nullptr;
        s = dmalloc_t(&rs, hf[1]);
        if (s == ALTOB_OK) s = dmalloc_t(&rv, hf[1]);
        if (s == ALTOB_OK) {
            cudaMemcpyAsync(rs, hs.data(), hf[1] * sizeof(u64), cudaMemcpyHostToDevice, st);
            const unsigned g = std::max(1u, (hf[1] + 255) / 256);
            if (khi64) k_gather_hi<u64><<<g, 256, 0, st>>>(khi64, rs, hf[1], rv);
            else k_gather_hi<HI><<<g, 256, 0, st>>>(khi, rs, hf[1], rv);
            e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) s = fail(ALTOB_ERR_CUDA, std::string("high-word runs: ") + cudaGetErrorString(e));
        }
        if (s != ALTOB_OK) {
            dfree(rs);
            dfree(rv);
            cleanup();
            return s;
        }
        t->d_run_start = rs;
        t->d_run_val = rv;
        t->nrun = (int)hf[1];
        dfree(khi64);
        khi64 = nullptr;
    } else if (has_hi && !khi64) {
        BTRY(dmalloc_t(&khi64, nnz));
        k_widen_hi<HI><<<grid, 256, 0, st>>>(khi, nnz, khi64);
        e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) BTRY(fail(ALTOB_ERR_CUDA, std::string("high words: ") + cudaGetErrorString(e)));
    }
    t->d_klo = klo;
    t->d_khi = khi64;
    cleanup();
#undef BTRY
#undef BLAUNCH
    t->device_bytes = nnz * (8 * (t->d_khi ? 2 : 1) + vsz) + (u64)t->nrun * 16;
    for (int n = 0; n < nm; ++n)
        if (t->d_oidx[n]) t->device_bytes += nnz * 4;
    return ALTOB_OK;
}

static altob_status create_common(int nmode, const u64* dims, u64 nnz, const u64* d_cidx, const void* d_vals,
                                  altob_dtype vdt, int nprtn, int lit_bits, cudaStream_t st, altob_tensor** out)
{
    if (!out) return fail(ALTOB_ERR_ARG, "out is NULL");
    *out = nullptr;
    if (nmode < 1 || nmode > ALTOB_MAX_MODES) return fail(ALTOB_ERR_ARG, "nmode must be 1..5");
    if (nprtn < 1) return fail(ALTOB_ERR_ARG, "nprtn must be >= 1");
    if (lit_bits != 0 && lit_bits != 64 && lit_bits != 128) return fail(ALTOB_ERR_ARG, "lit_bits must be 0, 64 or 128");
    if (nnz >= (1ull << 32)) return fail(ALTOB_ERR_UNSUPPORTED, "nnz must be below 2^32");
    if (vdt != ALTOB_F64 && vdt != ALTOB_F32 && vdt != ALTOB_U32) return fail(ALTOB_ERR_ARG, "bad value dtype");
    for (int n = 0; n < nmode; ++n) {
        if (dims[n] == 0) return fail(ALTOB_ERR_ARG, "a dimension is 0");
        if (dims[n] >= (1ull << 32)) return fail(ALTOB_ERR_UNSUPPORTED, "dimensions of 2^32 or more are not supported");
    }
    if (nnz && (!d_cidx || !d_vals)) return fail(ALTOB_ERR_ARG, "cidx / vals is NULL");
    altob_tensor* t = new altob_tensor();
    cudaGetDevice(&t->device);
    t->nmode = nmode;
    t->nprtn = nprtn;
    t->nnz = nnz;
    t->vdt = vdt;
    for (int n = 0; n < nmode; ++n) t->dims[n] = dims[n];
    int total = make_masks(nmode, dims, t->masks, t->order);
    if (lit_bits == 0) lit_bits = total <= 64 ? 64 : 128;
    if (total > lit_bits) {
        delete t;
        return fail(ALTOB_ERR_BITS, "ALTO bits (" + std::to_string(total) + ") exceed the " +
                                        std::to_string(lit_bits) + "-bit index");
    }
    t->lit_bits = lit_bits;
    t->alto_bits = total;
    t->alto_mask = 0;
    for (int n = 0; n < nmode; ++n) t->alto_mask |= t->masks[n];
    int ncr = 0, fb = lit_bits - total;
    for (int n = 0; n < nmode; ++n)
        if (fib_reuse(t, n) <= 4 && fb) {
            ++ncr;
            --fb;
        }
    t->kw = (total + ncr > 64) ? 2 : 1;
    t->dec = make_decoder(nmode, t->masks, total);
    t->fld.nmode = nmode;
    {
        u32 p = 0;
        for (int k = 0; k < nmode; ++k) {
            const int n = t->order[k];
            const int b = mode_bits(dims[n]);
            t->fld.pos[n] = p;
            t->fld.mask[n] = b >= 32 ? 0xffffffffu : ((1u << b) - 1u);
            p += b;
        }
    }
    const int hi_bits = total - 64;
    altob_status s = hi_bits <= 0    ? build<unsigned char>(t, d_cidx, d_vals, vdt, 0, st)
                     : hi_bits <= 8  ? build<unsigned char>(t, d_cidx, d_vals, vdt, 1, st)
                     : hi_bits <= 32 ? build<u32>(t, d_cidx, d_vals, vdt, 4, st)
                                     : build<u64>(t, d_cidx, d_vals, vdt, 8, st);
    if (s != ALTOB_OK) {
        altob_destroy(t);
        return s;
    }
    *out = t;
    return ALTOB_OK;
}

// The reference's interleaved keys (default encoding, CR bits included) of
// every nonzero, into device arrays.
altob_status interleaved_keys(const altob_tensor* t, u64* olo, u64* ohi, cudaStream_t st)
{
    if (!t->nnz) return ALTOB_OK;
    k_interleave<<<grid_for(t->nnz, 256), 256, 0, st>>>(t->d_klo, key_src(t), t->alto_bits, t->nnz, t->dec, t->fld,
                                                        olo, ohi);
    ALTOB_LAUNCH_CHECK();
    return ALTOB_OK;
}

// A contiguous range [begin, end) of a tensor's ALTO stream as a tensor of
// its own (one GPU's share of a sharded MTTKRP or CP-ALS; the split follows
// the reference's equal-nnz partition rule, alto.hpp:822-836).  Keys, values
// and high words are copied; oidx (for the slice's own low-reuse modes, as
// alto.hpp:246-285 decides them from its nonzero count), partitions and
// intervals (alto.hpp:822-899) are computed for the slice.  The slice has no
// CR masks: its keys keep the parent's CR bits, which no mode field reads.
static altob_status slice_impl(const altob_tensor* t, u64 begin, u64 end, int nprtn, cudaStream_t st,
                               altob_tensor* s)
{
    const u64 n = end - begin;
    s->device = t->device;
    s->nmode = t->nmode;
    s->nprtn = nprtn;
    s->lit_bits = t->lit_bits;
    s->alto_bits = t->alto_bits;
    s->kw = t->kw;
    s->vdt = t->vdt;
    s->nnz = n;
    for (int m = 0; m < ALTOB_MAX_MODES; ++m) {
        s->dims[m] = t->dims[m];
        s->masks[m] = t->masks[m];
        s->order[m] = t->order[m];
    }
    s->alto_mask = t->alto_mask;
    s->dec = t->dec;
    s->fld = t->fld;
    const size_t vsz = val_size(t->vdt);
    ALTOB_TRY(dmalloc_t(&s->d_klo, n));
    ALTOB_TRY(dmalloc(&s->d_vals, n * vsz + 16));
    if (n) {
        ALTOB_CUDA(cudaMemcpyAsync(s->d_klo, t->d_klo + begin, n * 8, cudaMemcpyDeviceToDevice, st));
        ALTOB_CUDA(cudaMemcpyAsync(s->d_vals, (const char*)t->d_vals + begin * vsz, n * vsz, cudaMemcpyDeviceToDevice,
                                   st));
    }
    if (t->d_khi) {
        ALTOB_TRY(dmalloc_t(&s->d_khi, n));
        if (n) ALTOB_CUDA(cudaMemcpyAsync(s->d_khi, t->d_khi + begin, n * 8, cudaMemcpyDeviceToDevice, st));
    } else if (t->nrun) {  // the runs that overlap the range, starts relative to it
        std::vector<u64> rs(t->nrun), rv(t->nrun), ns, nv;
        ALTOB_CUDA(cudaMemcpyAsync(rs.data(), t->d_run_start, rs.size() * 8, cudaMemcpyDeviceToHost, st));
        ALTOB_CUDA(cudaMemcpyAsync(rv.data(), t->d_run_val, rv.size() * 8, cudaMemcpyDeviceToHost, st));
        ALTOB_CUDA(cudaStreamSynchronize(st));
        for (int r = 0; r < t->nrun; ++r) {
            const u64 stop = r + 1 < t->nrun ? rs[r + 1] : t->nnz;
            if (stop <= begin || rs[r] >= end) continue;
            ns.push_back(std::max(rs[r], begin) - begin);
            nv.push_back(rv[r]);
        }
        if (ns.empty()) {  // empty slice
            ns.push_back(0);
            nv.push_back(0);
        }
        ALTOB_TRY(dmalloc_t(&s->d_run_start, ns.size()));
        ALTOB_TRY(dmalloc_t(&s->d_run_val, nv.size()));
        ALTOB_CUDA(cudaMemcpyAsync(s->d_run_start, ns.data(), ns.size() * 8, cudaMemcpyHostToDevice, st));
        ALTOB_CUDA(cudaMemcpyAsync(s->d_run_val, nv.data(), nv.size() * 8, cudaMemcpyHostToDevice, st));
        s->nrun = (int)ns.size();
    }
    // explicit high words for the oidx and interval kernels (a run table is
    // expanded into a temporary array)
    const u64* hi = s->d_khi;
    u64* hi_tmp = nullptr;
    struct HiFree {
        u64** p;
        ~HiFree() { dfree(*p); }
    } hi_free{&hi_tmp};
    if (!hi && s->nrun && n) {
        ALTOB_TRY(dmalloc_t(&hi_tmp, n));
        k_expand_hi<<<grid_for(n, 256), 256, 0, st>>>(key_src(s), n, hi_tmp);
        if (cudaGetLastError() != cudaSuccess) return fail(ALTOB_ERR_CUDA, "k_expand_hi launch failed");
        hi = hi_tmp;
    }
    // oidx of the slice's low-reuse modes
    s->is_oidx = 0;
    for (int m = 0; m < s->nmode; ++m)
        if (fib_reuse(s, m) <= 4) s->is_oidx = 1;
    if (s->is_oidx && n) {
        for (int m = 0; m < s->nmode; ++m) {
            if (fib_reuse(s, m) > 4) continue;
            u32 *mk = nullptr, *mk2 = nullptr;
            u32 *io = nullptr, *io2 = nullptr;
            altob_status a = dmalloc_t(&mk, n);
            if (a == ALTOB_OK) a = dmalloc_t(&mk2, n);
            if (a == ALTOB_OK) a = dmalloc_t(&io, n);
            if (a == ALTOB_OK) a = dmalloc_t(&io2, n);
            bool alt = false;
            if (a == ALTOB_OK) {
                k_mode_keys<u64><<<grid_for(n, 256), 256, 0, st>>>(s->d_klo, hi, n, s->fld, m, mk);
                if (cudaGetLastError() != cudaSuccess) a = fail(ALTOB_ERR_CUDA, "k_mode_keys launch failed");
            }
            if (a == ALTOB_OK) a = radix_argsort_u32(mk, io, mk2, io2, n, mode_bits(s->dims[m]), st, &alt);
            dfree(mk);
            dfree(mk2);
            if (a == ALTOB_OK) {
                s->d_oidx[m] = alt ? io2 : io;
                dfree(alt ? io : io2);
            } else {
                dfree(io);
                dfree(io2);
                return a;
            }
        }
    }
    // partitions and intervals of the slice
    const int np = nprtn, nm = s->nmode;
    const u64 per = (n + (u64)np - 1) / (u64)np;
    s->prtn_ptr.assign(np + 1, 0);
    for (int p = 0; p < np; ++p) s->prtn_ptr[p + 1] = std::min<u64>((u64)(p + 1) * per, n);
    u64 dm[5] = {1, 1, 1, 1, 1};
    for (int m = 0; m < nm; ++m) dm[m] = s->dims[m];
    u64* d_iv = nullptr;
    ALTOB_TRY(dmalloc_t(&d_iv, (u64)np * nm * 2));
    k_init_intervals<<<(np * nm + 255) / 256, 256, 0, st>>>(d_iv, np, nm, dm[0], dm[1], dm[2], dm[3], dm[4]);
    if (n) k_intervals<u64><<<intervals_grid(n), 256, 0, st>>>(s->d_klo, hi, n, s->fld, per, d_iv);
    s->intervals.assign((size_t)np * nm * 2, 0);
    cudaMemcpyAsync(s->intervals.data(), d_iv, s->intervals.size() * sizeof(u64), cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    dfree(d_iv);
    if (e != cudaSuccess) return fail(ALTOB_ERR_CUDA, std::string("slice: ") + cudaGetErrorString(e));
    s->device_bytes = n * (8 * (s->d_khi ? 2 : 1) + vsz) + (u64)s->nrun * 16;
    for (int m = 0; m < nm; ++m)
        if (s->d_oidx[m]) s->device_bytes += n * 4;
    return ALTOB_OK;
}

}  // namespace altob

using namespace altob;

extern "C" {

const char* altob_status_string(altob_status s)
{
    switch (s) {
    case ALTOB_OK: return "ok";
    case ALTOB_ERR_ARG: return "invalid argument";
    case ALTOB_ERR_BITS: return "ALTO bits exceed the index width";
    case ALTOB_ERR_CUDA: return "CUDA error";
    case ALTOB_ERR_NOMEM: return "out of memory";
    case ALTOB_ERR_IO: return "I/O error";
    case ALTOB_ERR_UNSUPPORTED: return "unsupported";
    case ALTOB_ERR_NOT_FOUND: return "no CUDA device";
    }
    return "unknown status";
}

const char* altob_last_error(void) { return g_last_error.c_str(); }

const char* altob_version(void) { return "alto_b200 0.1.0 (sm_100a)"; }

altob_status altob_trim_memory(void)
{
    cudaMemPool_t p = device_pool();
    if (p) ALTOB_CUDA(cudaMemPoolTrimTo(p, 0));
    return ALTOB_OK;
}

altob_status altob_create(int nmode, const uint64_t* dims, uint64_t nnz, const uint64_t* cidx, const void* vals,
                          altob_dtype val_dtype, int nprtn, int lit_bits, void* stream, altob_tensor** out)
{
    if (!dims) return fail(ALTOB_ERR_ARG, "dims is NULL");
    if (nmode < 1 || nmode > ALTOB_MAX_MODES) return fail(ALTOB_ERR_ARG, "nmode must be 1..5");
    cudaStream_t st = (cudaStream_t)stream;
    StreamScope scope(st);
    u64* d_cidx = nullptr;
    void* d_vals = nullptr;
    size_t vsz = val_size(val_dtype);
    if (nnz) {
        if (!cidx || !vals) return fail(ALTOB_ERR_ARG, "cidx / vals is NULL");
        ALTOB_TRY(dmalloc_t(&d_cidx, (u64)nmode * nnz));
        altob_status s = dmalloc(&d_vals, nnz * vsz);
        if (s != ALTOB_OK) {
            dfree(d_cidx);
            return s;
        }
        cudaMemcpyAsync(d_cidx, cidx, (u64)nmode * nnz * sizeof(u64), cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(d_vals, vals, nnz * vsz, cudaMemcpyHostToDevice, st);
    }
    altob_status s = create_common(nmode, dims, nnz, d_cidx, d_vals, val_dtype, nprtn, lit_bits, st, out);
    cudaStreamSynchronize(st);
    dfree(d_cidx);
    dfree(d_vals);
    return s;
}

altob_status altob_create_device(int nmode, const uint64_t* dims, uint64_t nnz, const uint64_t* d_cidx,
                                 const void* d_vals, altob_dtype val_dtype, int nprtn, int lit_bits, void* stream,
                                 altob_tensor** out)
{
    if (!dims) return fail(ALTOB_ERR_ARG, "dims is NULL");
    StreamScope scope((cudaStream_t)stream);
    return create_common(nmode, dims, nnz, d_cidx, d_vals, val_dtype, nprtn, lit_bits, (cudaStream_t)stream, out);
}

altob_status altob_slice(const altob_tensor* t, uint64_t begin, uint64_t end, int nprtn, void* stream,
                         altob_tensor** out)
{
    if (!t || !out) return fail(ALTOB_ERR_ARG, "NULL argument");
    *out = nullptr;
    if (begin > end || end > t->nnz) return fail(ALTOB_ERR_ARG, "slice range outside the tensor");
    if (nprtn < 1) return fail(ALTOB_ERR_ARG, "nprtn must be >= 1");
    cudaStream_t st = (cudaStream_t)stream;
    StreamScope scope(st);
    ALTOB_TRY(tensor_enter(const_cast<altob_tensor*>(t), st));
    altob_tensor* s = new altob_tensor();
    const altob_status r = slice_impl(t, begin, end, nprtn, st, s);
    tensor_leave(const_cast<altob_tensor*>(t), st);
    if (r != ALTOB_OK) {
        altob_destroy(s);
        return r;
    }
    *out = s;
    return ALTOB_OK;
}

altob_status altob_destroy(altob_tensor* t)
{
    if (!t) return ALTOB_OK;
    // frees are ordered on the legacy default stream, i.e. after the work
    // already issued on blocking streams; work on non-blocking streams that
    // uses the tensor must be finished by the caller first
    StreamScope scope(0);
    if (t->use_ev) {  // after the last call that used the handle, on any stream
        cudaStreamWaitEvent(0, t->use_ev, 0);
        cudaEventDestroy(t->use_ev);
    }
    dfree(t->d_klo);
    dfree(t->d_khi);
    dfree(t->d_run_start);
    dfree(t->d_run_val);
    dfree(t->d_vals);
    for (int n = 0; n < ALTOB_MAX_MODES; ++n) dfree(t->d_oidx[n]);
    for (int n = 0; n < ALTOB_MAX_MODES; ++n) dfree(t->d_plan[n]);
    dfree(t->scratch);
    dfree(t->hotbuf.p);
    dfree(t->padbuf.p);
    for (const altob::HandleBuf& b : t->set_aside) dfree(b.p);
    dfree(t->d_tma_err);
    if (t->h_tma_err) {
        cudaStreamSynchronize(0);  // the flag's last copy was ordered before the frees above
        cudaFreeHost(t->h_tma_err);
    }
    delete t;
    return ALTOB_OK;
}

altob_status altob_get_info(const altob_tensor* t, altob_info* o)
{
    if (!t || !o) return fail(ALTOB_ERR_ARG, "NULL argument");
    memset(o, 0, sizeof(*o));
    o->nmode = t->nmode;
    o->nprtn = t->nprtn;
    o->lit_bits = t->lit_bits;
    o->alto_bits = t->alto_bits;
    o->is_oidx = t->is_oidx;
    o->val_dtype = t->vdt;
    o->nnz = t->nnz;
    for (int n = 0; n < t->nmode; ++n) {
        o->dims[n] = t->dims[n];
        o->mode_masks[n][0] = (u64)t->masks[n];
        o->mode_masks[n][1] = (u64)(t->masks[n] >> 64);
        o->cr_masks[n][0] = (u64)t->cr_masks[n];
        o->cr_masks[n][1] = (u64)(t->cr_masks[n] >> 64);
    }
    o->alto_mask[0] = (u64)t->alto_mask;
    o->alto_mask[1] = (u64)(t->alto_mask >> 64);
    o->alto_cr_mask[0] = (u64)t->alto_cr_mask;
    o->alto_cr_mask[1] = (u64)(t->alto_cr_mask >> 64);
    o->device_bytes = t->device_bytes + t->scratch_bytes + t->hotbuf.bytes + t->padbuf.bytes;
    for (const altob::HandleBuf& b : t->set_aside) o->device_bytes += b.bytes;
    o->key_bytes = t->d_khi ? 16 : 8;
    o->nruns = t->nrun;
    o->tma_err = t->h_tma_err ? (int)*t->h_tma_err : 0;
    for (int n = 0; n < t->nmode; ++n)
        if (t->d_plan[n]) {
            o->plan_modes |= 1 << n;
            o->plan_bytes += t->nnz * sizeof(uint16_t);
        }
    return ALTOB_OK;
}

altob_status altob_dump(const altob_tensor* t, uint64_t* idx, void* vals, uint64_t* prtn_ptr, uint64_t* intervals,
                        uint64_t* oidx, void* stream)
{
    if (!t) return fail(ALTOB_ERR_ARG, "NULL tensor");
    cudaStream_t st = (cudaStream_t)stream;
    StreamScope scope(st);
    const u64 nnz = t->nnz;
    if (idx && nnz) {
        u64 *olo = nullptr, *ohi = nullptr;
        ALTOB_TRY(dmalloc_t(&olo, nnz));
        altob_status s = dmalloc_t(&ohi, nnz);
        if (s != ALTOB_OK) {
            dfree(olo);
            return s;
        }
        k_interleave<<<grid_for(nnz, 256), 256, 0, st>>>(t->d_klo, key_src(t), t->alto_bits, nnz, t->dec, t->fld,
                                                         olo, ohi);
        std::vector<u64> lo(nnz), hi(nnz);
        cudaMemcpyAsync(lo.data(), olo, nnz * 8, cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(hi.data(), ohi, nnz * 8, cudaMemcpyDeviceToHost, st);
        cudaError_t e = cudaStreamSynchronize(st);
        dfree(olo);
        dfree(ohi);
        if (e != cudaSuccess) return fail(ALTOB_ERR_CUDA, std::string("dump: ") + cudaGetErrorString(e));
        for (u64 i = 0; i < nnz; ++i) {
            idx[2 * i] = lo[i];
            idx[2 * i + 1] = hi[i];
        }
    }
    if (vals && nnz) ALTOB_CUDA(cudaMemcpyAsync(vals, t->d_vals, nnz * val_size(t->vdt), cudaMemcpyDeviceToHost, st));
    if (prtn_ptr) memcpy(prtn_ptr, t->prtn_ptr.data(), t->prtn_ptr.size() * sizeof(u64));
    if (intervals) memcpy(intervals, t->intervals.data(), t->intervals.size() * sizeof(u64));
    if (oidx && nnz) {
        std::vector<u32> tmp(nnz);
        for (int n = 0; n < t->nmode; ++n) {
            if (!t->d_oidx[n]) continue;
            ALTOB_CUDA(cudaMemcpyAsync(tmp.data(), t->d_oidx[n], nnz * 4, cudaMemcpyDeviceToHost, st));
            ALTOB_CUDA(cudaStreamSynchronize(st));
            for (u64 i = 0; i < nnz; ++i) oidx[(u64)n * nnz + i] = tmp[i];
        }
    }
    ALTOB_CUDA(cudaStreamSynchronize(st));
    return ALTOB_OK;
}

}  // extern "C"
