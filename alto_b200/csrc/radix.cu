// radix.cu -- stable LSD radix sort of (key, payload) pairs, 8-bit digits.
//
// The ALTO build sorts the linearized keys (sort_alto, IntelLabs/ALTO
// include/alto.hpp:772-803), the oidx and the CP-APR row order sort mode
// indices (alto.hpp:246-285).  Per pass: digit histogram of every tile, one
// exclusive scan of the digit-major table, and a scatter that first sorts its
// tile in shared memory and then writes runs of equal digits.
//
// Bound: memory traffic of the scatter (a key and payload read and written
// per pass).  Each warp ranks its own 256 keys with match_any against
// counters of its own (no block barrier per round), one block scan turns the
// counters into positions, and the staged tile leaves in digit order, so the
// writes are runs of ~16 elements instead of single elements.  On 20.2M keys
// of 65 bits a pass took 470 us (histogram, scan, scatter with four barriers
// per 256 keys and 8-byte writes at random); now 274 us, 236 of them the
// scatter.
//
// Keys may be stored in a layout that is not their sort order (the device key
// holds every mode index as a bit field): a digit is then gathered from up to
// five bit fields and put together by small tables (KeyDigit), which is what
// makes the interleaved keys, and the pass that re-encodes them after the
// sort, unnecessary.
#include <algorithm>
#include <type_traits>

#include "internal.cuh"

namespace altob {

// ----------------------------------------------------------- scans
// Exclusive prefix sum of u32 values in place (sum < 2^32).

static constexpr int SC_THREADS = 1024;
static constexpr int SC_IPT = 4;
static constexpr int SC_CHUNK = SC_THREADS * SC_IPT;

__device__ __forceinline__ u32 block_excl_scan(u32 v, u32* total, u32* warp_sums)
{
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    u32 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        u32 y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        u32 s = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            u32 y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) warp_sums[lane] = s;
    }
    __syncthreads();
    u32 base = warp ? warp_sums[warp - 1] : 0;
    *total = warp_sums[nw - 1];
    __syncthreads();
    return base + x - v;
}

__global__ void k_scan_reduce(const u32* in, u64 n, u32* bsum)
{
    __shared__ u32 ws[32];
    u64 base = (u64)blockIdx.x * SC_CHUNK + (u64)threadIdx.x * SC_IPT;
    u32 s = 0;
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k)
        if (base + k < n) s += in[base + k];
    u32 tot;
    block_excl_scan(s, &tot, ws);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void k_scan_top(u32* bsum, u32 nb)
{
    __shared__ u32 ws[32];
    u32 carry = 0;
    for (u32 b0 = 0; b0 < nb; b0 += blockDim.x) {
        u32 i = b0 + threadIdx.x;
        u32 v = i < nb ? bsum[i] : 0;
        u32 tot;
        u32 ex = block_excl_scan(v, &tot, ws);
        if (i < nb) bsum[i] = carry + ex;
        carry += tot;
    }
}

// bsum: exclusive offsets of the blocks, or nullptr when one block scans all.
__global__ void k_scan_down(u32* data, u64 n, const u32* bsum)
{
    __shared__ u32 ws[32];
    u32 carry = bsum ? bsum[blockIdx.x] : 0;
    const u64 stop = bsum ? min(n, ((u64)blockIdx.x + 1) * SC_CHUNK) : n;
    for (u64 b0 = (u64)blockIdx.x * SC_CHUNK; b0 < stop; b0 += SC_CHUNK) {
        const u64 base = b0 + (u64)threadIdx.x * SC_IPT;
        u32 v[SC_IPT];
        u32 s = 0;
#pragma unroll
        for (int k = 0; k < SC_IPT; ++k) {
            v[k] = base + k < n ? data[base + k] : 0;
            s += v[k];
        }
        u32 tot;
        u32 ex = block_excl_scan(s, &tot, ws) + carry;
#pragma unroll
        for (int k = 0; k < SC_IPT; ++k) {
            if (base + k < n) data[base + k] = ex;
            ex += v[k];
        }
        carry += tot;
    }
}

static altob_status excl_scan_u32(u32* data, u64 n, u32* bsum, cudaStream_t st)
{
    u32 nb = (u32)((n + SC_CHUNK - 1) / SC_CHUNK);
    if (nb == 0) return ALTOB_OK;
    if (nb <= 8) {  // one launch: a block walks a few chunks in about the time two more launches take
        k_scan_down<<<1, SC_THREADS, 0, st>>>(data, n, nullptr);
        ALTOB_LAUNCH_CHECK();
        return ALTOB_OK;
    }
    k_scan_reduce<<<nb, SC_THREADS, 0, st>>>(data, n, bsum);
    ALTOB_LAUNCH_CHECK();
    k_scan_top<<<1, SC_THREADS, 0, st>>>(bsum, nb);
    ALTOB_LAUNCH_CHECK();
    k_scan_down<<<nb, SC_THREADS, 0, st>>>(data, n, bsum);
    ALTOB_LAUNCH_CHECK();
    return ALTOB_OK;
}

// ------------------------------------------------------------ passes

static constexpr int RS_TILE = 4096;
static constexpr int RH_THREADS = 256;  // histogram
static constexpr int RH_IPT = RS_TILE / RH_THREADS;
static constexpr int RS_THREADS = 512;  // scatter: 8 keys a thread keep it at 64 registers, two blocks a SM
static constexpr int RS_WARPS = RS_THREADS / 32;
static constexpr int RS_IPT = RS_TILE / RS_THREADS;

// High key words: none, or 8, 32 or 64 bits of them.
struct NoHi {
};
template <typename HI>
__device__ __forceinline__ u64 hi_get(const HI* p, u64 i) { return (u64)p[i]; }
template <>
__device__ __forceinline__ u64 hi_get<NoHi>(const NoHi*, u64) { return 0; }

// A pass's digit tables (KeyDigit::lut) into shared memory.
__device__ __forceinline__ void load_lut(const KeyDigit& d, u32* lut)
{
    for (int k = threadIdx.x; k < KEY_DIGIT_LUT / 4; k += blockDim.x) lut[k] = d.lut[k];
}

template <typename LO, bool PIECES>
__device__ __forceinline__ u32 key_digit(LO lo, u64 hi, const KeyDigit& d, const u32* lut32)
{
    const unsigned char* lut = reinterpret_cast<const unsigned char*>(lut32);
    if constexpr (!PIECES) {
        return (u32)((d.pos[0] >= 64 ? hi >> (d.pos[0] - 64) : (u64)lo >> d.pos[0])) & 0xffu;
    } else {
        u32 r = 0;
#pragma unroll
        for (int m = 0; m < ALTOB_MAX_MODES; ++m) {
            if (m >= d.pieces) break;
            r |= lut[d.off[m] + field((u64)lo, hi, d.pos[m], d.mask[m])];
        }
        return r;
    }
}

// Counts one digit per lane (256: none) in the warp's counters.  The first
// lane's digit is counted once for all lanes that share it: the high digits of
// skewed keys are mostly equal, and one atomic per key on one counter
// serialises.
__device__ __forceinline__ void count_digit(u32* h, u32 d)
{
    const u32 d0 = __shfl_sync(0xffffffffu, d, 0);
    const u32 eq = __ballot_sync(0xffffffffu, d == d0);
    if (d == d0) {
        if ((threadIdx.x & 31) == 0 && d < 256u) atomicAdd(&h[d], (u32)__popc(eq));
    } else if (d < 256u) {
        atomicAdd(&h[d], 1u);
    }
}

__device__ __forceinline__ void write_hist(const u32 (*h)[256], u32* hist, u32 ntiles)
{
    const u32 d = threadIdx.x;
    u32 s = 0;
#pragma unroll
    for (int w = 0; w < RH_THREADS / 32; ++w) s += h[w][d];
    hist[(u64)d * ntiles + blockIdx.x] = s;
}

// First pass: digits of the keys (kept in dig) and their histogram per tile.
template <typename LO, typename HI, bool PIECES>
__global__ void __launch_bounds__(RH_THREADS) k_rs_first(const LO* __restrict__ klo, const HI* __restrict__ khi, u64 n,
                                                         KeyDigit dg, unsigned char* __restrict__ dig,
                                                         u32* __restrict__ hist, u32 ntiles)
{
    __shared__ u32 h[RH_THREADS / 32][256];
    __shared__ u32 lut[KEY_DIGIT_LUT / 4];
    for (int j = threadIdx.x; j < RH_THREADS / 32 * 256; j += RH_THREADS) (&h[0][0])[j] = 0;
    if (PIECES) load_lut(dg, lut);
    __syncthreads();
    const u64 base = (u64)blockIdx.x * RS_TILE;
#pragma unroll 4
    for (int k = 0; k < RH_IPT; ++k) {
        const u64 i = base + (u64)k * RH_THREADS + threadIdx.x;
        u32 d = 256u;
        if (i < n) {
            d = key_digit<LO, PIECES>(klo[i], dg.need_hi ? hi_get<HI>(khi, i) : 0, dg, lut);
            dig[i] = (unsigned char)d;
        }
        count_digit(h[threadIdx.x >> 5], d);
    }
    __syncthreads();
    write_hist(h, hist, ntiles);
}

// Later passes: histogram of the digits that the previous scatter left in dig.
static __global__ void __launch_bounds__(RH_THREADS) k_rs_hist(const unsigned char* __restrict__ dig, u64 n,
                                                               u32* __restrict__ hist, u32 ntiles)
{
    __shared__ u32 h[RH_THREADS / 32][256];
    for (int j = threadIdx.x; j < RH_THREADS / 32 * 256; j += RH_THREADS) (&h[0][0])[j] = 0;
    __syncthreads();
    const u64 i0 = (u64)blockIdx.x * RS_TILE + (u64)threadIdx.x * 16;
    // (dig is readable to a multiple of 16 past n)
    const uint4 v = i0 < n ? *reinterpret_cast<const uint4*>(dig + i0) : make_uint4(0, 0, 0, 0);
    const u32 w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 16; ++k)
        count_digit(h[threadIdx.x >> 5], i0 + k < n ? w[k / 4] >> (8 * (k % 4)) & 0xffu : 256u);
    __syncthreads();
    write_hist(h, hist, ntiles);
}

// Shared memory of the scatter: the staged tile (low words, payloads, digits,
// next digits, high words) and the warps' counters.
template <typename LO, typename HI>
struct ScatterSmem {
    static constexpr bool HAS_HI = !std::is_same<HI, NoHi>::value;
    static constexpr int PAY = RS_TILE * (int)sizeof(LO), HIW = PAY + RS_TILE * 4,
                         DIG = HIW + (HAS_HI ? RS_TILE * (int)sizeof(HI) : 0), NEXT = DIG + RS_TILE,
                         CNT = NEXT + RS_TILE, BYTES = CNT + RS_WARPS * 256 * 2;
};

// One pass: every key of the tile to its place.  pay == nullptr: the payload
// of position i is i (the first pass).  odig (if given) receives the digits of
// the next pass, `next`.
template <typename LO, typename HI, bool PIECES>
__global__ void __launch_bounds__(RS_THREADS, 2) k_rs_scatter(const LO* __restrict__ klo, const HI* __restrict__ khi,
                                                              const u32* __restrict__ pay,
                                                              const unsigned char* __restrict__ dig,
                                                              LO* __restrict__ olo, HI* __restrict__ ohi,
                                                              u32* __restrict__ opay, unsigned char* __restrict__ odig,
                                                              u64 n, KeyDigit next, const u32* __restrict__ offs,
                                                              u32 ntiles)
{
    typedef ScatterSmem<LO, HI> Sm;
    constexpr bool HAS_HI = Sm::HAS_HI;
    extern __shared__ __align__(16) unsigned char rsm[];
    LO* slo = reinterpret_cast<LO*>(rsm);
    u32* spy = reinterpret_cast<u32*>(rsm + Sm::PAY);
    HI* shi = reinterpret_cast<HI*>(rsm + Sm::HIW);
    unsigned char* sdig = rsm + Sm::DIG;
    unsigned char* snext = rsm + Sm::NEXT;
    unsigned short(*wcnt)[256] = reinterpret_cast<unsigned short(*)[256]>(rsm + Sm::CNT);
    __shared__ u32 gofs[256];
    __shared__ u32 wsum[8];
    __shared__ u32 lut[KEY_DIGIT_LUT / 4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int j = tid; j < RS_WARPS * 128; j += RS_THREADS) reinterpret_cast<u32*>(&wcnt[0][0])[j] = 0;
    if (PIECES && odig) load_lut(next, lut);
    const u64 base = (u64)blockIdx.x * RS_TILE;
    const int nvalid = (int)min((u64)RS_TILE, n - base);
    // element k of a lane: position warp * 256 + k * 32 + lane of the tile
    LO lo[RS_IPT];
    HI hi[RS_IPT];
    u32 py[RS_IPT], dd[RS_IPT];
#pragma unroll
    for (int k = 0; k < RS_IPT; ++k) {
        const int p = warp * (32 * RS_IPT) + k * 32 + lane;
        lo[k] = LO(0);
        py[k] = 0;
        dd[k] = 256u;
        if constexpr (HAS_HI) hi[k] = HI(0);
        if (p < nvalid) {
            dd[k] = dig[base + p];
            lo[k] = klo[base + p];
            if constexpr (HAS_HI) hi[k] = khi[base + p];
            py[k] = pay ? pay[base + p] : (u32)(base + p);
        }
    }
    __syncthreads();
    // ranks inside the warp: equal digits of a round share one counter update
    u32 rk[RS_IPT];
#pragma unroll
    for (int k = 0; k < RS_IPT; ++k) {
        const u32 d = dd[k];
        const u32 peers = __match_any_sync(0xffffffffu, d);
        const u32 below = __popc(peers & ((1u << lane) - 1u));
        u32 c = 0;
        if (d < 256u) c = wcnt[warp][d];
        __syncwarp();
        if (d < 256u && below == 0) wcnt[warp][d] = (unsigned short)(c + __popc(peers));
        __syncwarp();
        rk[k] = c + below;
    }
    __syncthreads();
    // positions: digits in order, inside a digit the warps in order
    u32 t = 0, x = 0;
    if (tid < 256) {
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) t += wcnt[w][tid];
        x = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
    }
    __syncthreads();
    if (tid < 256) {
        u32 start = x - t;
#pragma unroll
        for (int w = 0; w < 8; ++w)
            if (w < warp) start += wsum[w];
        gofs[tid] = offs[(u64)tid * ntiles + blockIdx.x] - start;
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) {
            const u32 c = wcnt[w][tid];
            wcnt[w][tid] = (unsigned short)start;
            start += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RS_IPT; ++k) {
        const u32 d = dd[k];
        if (d >= 256u) continue;
        const u32 p = wcnt[warp][d] + rk[k];
        sdig[p] = (unsigned char)d;
        slo[p] = lo[k];
        spy[p] = py[k];
        u64 h = 0;
        if constexpr (HAS_HI) {
            shi[p] = hi[k];
            h = (u64)hi[k];
        }
        if (odig) snext[p] = (unsigned char)key_digit<LO, PIECES>(lo[k], h, next, lut);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RS_IPT; ++k) {
        const int p = k * RS_THREADS + tid;
        if (p >= nvalid) break;
        const u32 dst = gofs[sdig[p]] + (u32)p;
        olo[dst] = slo[p];
        opay[dst] = spy[p];
        if constexpr (HAS_HI) ohi[dst] = shi[p];
        if (odig) odig[dst] = snext[p];
    }
}

// Runs the passes `dg[0 .. npass)`; the result is in the alt arrays when
// *result_in_alt.  iota: the payload of position i starts as i (pay's initial
// contents are not read).
template <typename LO, typename HI, bool PIECES>
static altob_status sort_passes(LO* klo, HI* khi, u32* pay, LO* klo_alt, HI* khi_alt, u32* pay_alt, u64 n,
                                const KeyDigit* dg, int npass, bool iota, cudaStream_t st, bool* result_in_alt)
{
    *result_in_alt = false;
    constexpr int smem = ScatterSmem<LO, HI>::BYTES;
    ALTOB_CUDA(cudaFuncSetAttribute(k_rs_scatter<LO, HI, PIECES>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const u32 ntiles = (u32)((n + RS_TILE - 1) / RS_TILE);
    const u64 hn = (u64)ntiles * 256, dn = (n + 255) & ~255ull;
    u32* hist = nullptr;
    ALTOB_TRY(dmalloc((void**)&hist, (hn + hn / SC_CHUNK + 64) * 4 + 2 * dn));
    u32* bsum = hist + hn;
    // the digits of the current and the next pass
    unsigned char* dcur = (unsigned char*)(((uintptr_t)(bsum + hn / SC_CHUNK + 2) + 15) & ~(uintptr_t)15);
    unsigned char* dnext = dcur + dn;
    altob_status s = ALTOB_OK;
    bool alt = false;
    for (int p = 0; p < npass && s == ALTOB_OK; ++p) {
        LO *slo = alt ? klo_alt : klo, *dlo = alt ? klo : klo_alt;
        HI *shi = alt ? khi_alt : khi, *dhi = alt ? khi : khi_alt;
        u32 *sp = alt ? pay_alt : pay, *dp = alt ? pay : pay_alt;
        if (p == 0 && iota) sp = nullptr;
        if (p == 0) k_rs_first<LO, HI, PIECES><<<ntiles, RH_THREADS, 0, st>>>(slo, shi, n, dg[0], dcur, hist, ntiles);
        else k_rs_hist<<<ntiles, RH_THREADS, 0, st>>>(dcur, n, hist, ntiles);
        s = excl_scan_u32(hist, hn, bsum, st);
        if (s != ALTOB_OK) break;
        const bool last = p + 1 == npass;
        k_rs_scatter<LO, HI, PIECES><<<ntiles, RS_THREADS, smem, st>>>(slo, shi, sp, dcur, dlo, dhi, dp,
                                                                      last ? nullptr : dnext, n, dg[last ? p : p + 1],
                                                                      hist, ntiles);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) s = fail(ALTOB_ERR_CUDA, std::string("radix scatter: ") + cudaGetErrorString(e));
        alt = !alt;
        std::swap(dcur, dnext);
    }
    dfree(hist);
    *result_in_alt = alt;
    return s;
}

static int plain_digits(int nbits, KeyDigit* dg)
{
    int np = 0;
    for (int shift = 0; shift < nbits; shift += 8) {
        dg[np] = KeyDigit();
        dg[np].pos[0] = (u32)shift;
        dg[np].need_hi = shift >= 64;
        ++np;
    }
    return np;
}

altob_status radix_sort_pairs(u64* klo, u64* khi, u32* pay, u64* klo_alt, u64* khi_alt, u32* pay_alt, u64 n,
                              int kw, int nbits, cudaStream_t st, bool* result_in_alt)
{
    *result_in_alt = false;
    if (n <= 1 || nbits <= 0) return ALTOB_OK;
    KeyDigit dg[16];
    const int np = plain_digits(nbits, dg);
    if (kw == 2)
        return sort_passes<u64, u64, false>(klo, khi, pay, klo_alt, khi_alt, pay_alt, n, dg, np, false, st,
                                            result_in_alt);
    return sort_passes<u64, NoHi, false>(klo, nullptr, pay, klo_alt, nullptr, pay_alt, n, dg, np, false, st,
                                         result_in_alt);
}

// Payload i of an unsorted or empty-key sort (no pass ran).
__global__ void k_iota(u32* p, u64 n)
{
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) p[i] = (u32)i;
}

static altob_status fill_iota(u32* p, u64 n, cudaStream_t st)
{
    if (!n) return ALTOB_OK;
    k_iota<<<(unsigned)std::min<u64>((n + 255) / 256, (u64)num_sms() * 8), 256, 0, st>>>(p, n);
    ALTOB_LAUNCH_CHECK();
    return ALTOB_OK;
}

altob_status radix_argsort_u32(u32* key, u32* perm, u32* key_alt, u32* perm_alt, u64 n, int nbits, cudaStream_t st,
                               bool* result_in_alt)
{
    *result_in_alt = false;
    if (n <= 1 || nbits <= 0) return fill_iota(perm, n, st);
    KeyDigit dg[16];
    const int np = plain_digits(std::min(nbits, 32), dg);
    return sort_passes<u32, NoHi, false>(key, nullptr, perm, key_alt, nullptr, perm_alt, n, dg, np, true, st,
                                         result_in_alt);
}

// Digit p of the ALTO order (bits [8p, 8p + 8)) gathered from field keys: the
// bits of mode m there are consecutive bits of its index.
static int alto_digits(const u128* masks, const Fields& f, int alto_bits, KeyDigit* dg)
{
    int np = 0;
    for (int shift = 0; shift < alto_bits; shift += 8, ++np) {
        KeyDigit& d = dg[np];
        d = KeyDigit();
        for (int m = 0; m < f.nmode; ++m) {
            const u32 here = (u32)(masks[m] >> shift) & 0xffu;
            if (!here) continue;
            u128 below = masks[m] & (((u128)1 << shift) - 1);
            const int first = __builtin_popcountll((u64)below) + __builtin_popcountll((u64)(below >> 64));
            const int n = __builtin_popcount(here), k = d.pieces;
            d.pos[k] = f.pos[m] + (u32)first;
            d.mask[k] = (1u << n) - 1u;
            d.off[k] = k ? d.off[k - 1] + d.mask[k - 1] + 1u : 0u;
            for (u32 v = 0; v <= d.mask[k]; ++v) {  // v's bits where the digit has this mode's
                u32 r = 0, b = 0;
                for (int p = 0; p < 8; ++p)
                    if (here >> p & 1u) r |= (v >> b++ & 1u) << p;
                const u32 e = d.off[k] + v;
                d.lut[e / 4] |= r << (8 * (e % 4));
            }
            if (d.pos[k] + n > 64) d.need_hi = 1;
            ++d.pieces;
        }
    }
    return np;
}

altob_status alto_sort(u64* klo, void* khi, u32* perm, u64* klo_alt, void* khi_alt, u32* perm_alt, u64 n, int hi_bytes,
                       const u128* masks, const Fields& f, int alto_bits, cudaStream_t st, bool* result_in_alt)
{
    *result_in_alt = false;
    if (n <= 1 || alto_bits <= 0) return fill_iota(perm, n, st);
    KeyDigit dg[16];
    const int np = alto_digits(masks, f, alto_bits, dg);
    switch (hi_bytes) {
    case 0:
        return sort_passes<u64, NoHi, true>(klo, nullptr, perm, klo_alt, nullptr, perm_alt, n, dg, np, true, st,
                                            result_in_alt);
    case 1:
        return sort_passes<u64, unsigned char, true>(klo, (unsigned char*)khi, perm, klo_alt, (unsigned char*)khi_alt,
                                                     perm_alt, n, dg, np, true, st, result_in_alt);
    case 4:
        return sort_passes<u64, u32, true>(klo, (u32*)khi, perm, klo_alt, (u32*)khi_alt, perm_alt, n, dg, np, true, st,
                                           result_in_alt);
    }
    return sort_passes<u64, u64, true>(klo, (u64*)khi, perm, klo_alt, (u64*)khi_alt, perm_alt, n, dg, np, true, st,
                                       result_in_alt);
}

}  // namespace altob
