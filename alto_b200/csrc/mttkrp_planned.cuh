// mttkrp_planned.cuh -- MTTKRP on the ALTO stream with a per-mode tile plan.
//
// Replaces mttkrp_alto_da_mem_pull (IntelLabs/ALTO include/alto.hpp:
// 1227-1318) for modes with fiber reuse above 4.  The grouped kernel
// (mttkrp_kernels.cuh) sorts every tile of the stream by output row on each
// launch: slot claims, a scan and a counting-sort scatter, about 40% of its
// instructions.  That order depends only on the tensor and the mode, so it is
// computed once (k_tile_plan) and kept beside the stream as a 16-bit position
// per nonzero and mode ("tile plan": where the nonzero goes in its tile's
// records sorted by the mode's index, ties in stream order).  A launch then
// reads key, value and plan entry (14 B per nonzero instead of 12), decodes
// the mode indices and writes each record straight to its sorted slot in
// shared memory; the run phase is the grouped kernel's (lean_runs: running
// row sums in registers, one vector atomic per run, per-CTA hot-row
// accumulators for long runs).
//
// The same body serves two more paths that used to sort every tile on every
// launch in the grouped kernel:
//   * modes read through oidx (alto.hpp:1320-1415): the permuted stream is
//     already in target order, so the record of position g goes to slot g and
//     no plan is needed;
//   * the CP-APR Phi (apr.hpp:383-848): the run loop keeps the target's
//     factor row beside the run sum and re-reads it only when the row changes.
//
// The plan is the tile-local analogue of the reference's oidx (alto.hpp:
// 246-285: a full permutation per low-reuse mode); it is built on the first
// MTTKRP of a mode and freed with the tensor.
#pragma once

#include "mttkrp_kernels.cuh"

namespace altob {

typedef uint16_t u16;

// Default tile of the planned kernels (nonzeros per tile; plan entries are
// below the tile size).
constexpr int PT_TILE = 1024;

// Decoded high key word of the nonzeros of one tile: one value for the whole
// tile unless it spans a run boundary of the high-word table (then two), or
// more than two runs (then a search per nonzero).
struct TileHi {
    u64 hcur = 0, hnext = 0, nstart = ~0ull;
    bool slow = false;
    __device__ __forceinline__ void init(const KeySrc& k, u64 g0, int tile)
    {
        if (k.khi || k.nrun == 0) return;
        const int r = run_of(k, g0);
        hcur = k.run_val[r];
        if (r + 1 < k.nrun) {
            nstart = k.run_start[r + 1];
            hnext = k.run_val[r + 1];
            if (r + 2 < k.nrun && k.run_start[r + 2] < g0 + (u64)tile) slow = true;
        }
    }
    __device__ __forceinline__ u64 get(const KeySrc& k, u64 g) const
    {
        if (k.khi) return k.khi[g];
        if (k.nrun == 0) return 0;
        if (slow) return key_hi(k, g);
        return g >= nstart ? hnext : hcur;
    }
};

// ------------------------------------------------------------ plan build
//
// One CTA per tile sorts (mode index, position in the tile) and writes, for
// nonzero g, its sorted rank inside its tile.  A thread holds IPT elements in
// registers (element e of the tile: thread e / IPT), so the bitonic network
// exchanges inside a thread for distances below IPT, by warp shuffles up to a
// warp's 32 * IPT elements and through shared memory only above (6 of the 55
// steps for 1024 elements).  The elements are 32-bit, (index - smallest index
// of the tile) * TILE + position, unless the indices of the tile span more
// than 32 bits hold (then 64-bit).  Bound by its own instructions: 1024-key
// networks entirely in shared memory with 64-bit keys, which this replaces,
// took 0.93 ms for 20M nonzeros and one mode.  Positions past the end of the
// stream sort last and are not written.
constexpr int TP_IPT = 4;

template <typename K>
__device__ __forceinline__ void cmp_swap(K& x, K& y, bool up)
{
    const K lo = x < y ? x : y, hi = x < y ? y : x;
    x = up ? lo : hi;
    y = up ? hi : lo;
}

template <int TILE, typename K>
__device__ __forceinline__ void tile_sort(K (&x)[TP_IPT], K* s)
{
    const int tid = threadIdx.x, e0 = tid * TP_IPT;
#pragma unroll
    for (int k = 2; k <= TILE; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32 * TP_IPT) {  // partner in another warp
                __syncthreads();
#pragma unroll
                for (int q = 0; q < TP_IPT; ++q) s[q * (TILE / TP_IPT) + tid] = x[q];
                __syncthreads();
                const bool up = (e0 & k) == 0, low = (e0 & j) == 0;
#pragma unroll
                for (int q = 0; q < TP_IPT; ++q) {
                    const K y = s[q * (TILE / TP_IPT) + (tid ^ (j / TP_IPT))];
                    const K mn = x[q] < y ? x[q] : y, mx = x[q] < y ? y : x[q];
                    x[q] = up == low ? mn : mx;
                }
            } else if (j >= TP_IPT) {  // partner in another lane
                const bool up = (e0 & k) == 0, low = (e0 & j) == 0;
#pragma unroll
                for (int q = 0; q < TP_IPT; ++q) {
                    const K y = __shfl_xor_sync(0xffffffffu, x[q], j / TP_IPT);
                    const K mn = x[q] < y ? x[q] : y, mx = x[q] < y ? y : x[q];
                    x[q] = up == low ? mn : mx;
                }
            } else {
#pragma unroll
                for (int q = 0; q < TP_IPT; ++q)
                    if ((q & j) == 0) cmp_swap(x[q], x[q | j], ((e0 + q) & k) == 0);
            }
        }
    }
}

template <int TILE>
__global__ void __launch_bounds__(TILE / TP_IPT) k_tile_plan(KeySrc key, Fields fld, u64 nnz, int mode, u16* plan)
{
    constexpr int NT = TILE / TP_IPT, NW = NT / 32;
    __shared__ unsigned long long s[TILE];
    __shared__ u32 wmin[NW], wmax[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u64 g0 = (u64)blockIdx.x * TILE;
    const int nvalid = (int)min((u64)TILE, nnz - g0);
    // loaded strided (coalesced); where an element starts out is free
    u32 row[TP_IPT];
    u32 mn = 0xffffffffu, mx = 0;
#pragma unroll
    for (int q = 0; q < TP_IPT; ++q) {
        const int i = q * NT + tid;
        row[q] = 0;
        if (i < nvalid) {
            const u64 g = g0 + i;
            const u64 lo = key.klo[g];
            const u64 hi = key.khi ? key.khi[g] : (key.nrun ? key_hi(key, g) : 0);
            row[q] = field(lo, hi, fld.pos[mode], fld.mask[mode]);
            mn = min(mn, row[q]);
            mx = max(mx, row[q]);
        }
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) {
        wmin[warp] = mn;
        wmax[warp] = mx;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        mn = min(mn, wmin[w]);
        mx = max(mx, wmax[w]);
    }
    if (mx - mn < 0xffffffffu / TILE) {  // uniform in the CTA; strictly below: ~0 marks positions past the end
        u32 x[TP_IPT];
#pragma unroll
        for (int q = 0; q < TP_IPT; ++q) {
            const int i = q * NT + tid;
            x[q] = i < nvalid ? (row[q] - mn) * TILE + (u32)i : 0xffffffffu;
        }
        tile_sort<TILE>(x, reinterpret_cast<u32*>(s));
#pragma unroll
        for (int q = 0; q < TP_IPT; ++q) {
            const int p = tid * TP_IPT + q;
            if (p < nvalid) plan[g0 + (x[q] & (TILE - 1))] = (u16)p;
        }
    } else {
        unsigned long long x[TP_IPT];
#pragma unroll
        for (int q = 0; q < TP_IPT; ++q) {
            const int i = q * NT + tid;
            x[q] = i < nvalid ? ((unsigned long long)row[q] << 32) | (u32)i : ~0ull;
        }
        tile_sort<TILE>(x, s);
#pragma unroll
        for (int q = 0; q < TP_IPT; ++q) {
            const int p = tid * TP_IPT + q;
            if (p < nvalid) plan[g0 + (u32)x[q]] = (u16)p;
        }
    }
}

// --------------------------------------------------------- planned MTTKRP

// Resident blocks per SM each instance is compiled for (a register cap; 0:
// the compiler's own choice).  The run loop waits on its row gathers, so more
// resident warps hide more of that latency until the loop spills.  FP32 order
// 3: 5 blocks of 8 warps (48 registers; 2.31 ms per mode at 4 blocks, 2.17 ms
// at 5 on the 100.85M-nonzero Zipf tensor; 3 blocks: 2.53 ms), 4 above rank
// 64 (32 lanes per nonzero spill at 48 registers).  FP32 orders 4-5 and Phi:
// 4 (on 18.9M nonzeros of order 4 at rank 16 Phi takes 490 us a mode at 3
// blocks, 467 at 4, 484 at 5; the order-4 MTTKRP 348, 350, 470).  FP64 orders 3
// and 4: 4 (order 4 at rank 16 takes 66 registers uncapped, three blocks: 579
// us a mode, 542 at four).
template <typename FT, int NM, int LPN, int CH, bool PHI>
constexpr int planned_min_blocks()
{
    if (CH != 1) return 0;
    if (sizeof(FT) != 4) return NM <= 4 ? 4 : 0;
    return NM == 3 && !PHI && LPN <= 16 ? 5 : 4;
}

// Record buffers of the planned kernel: two (the next tile's scatter
// overlaps this tile's runs, one barrier per tile) for FP32 order 3, one (two
// barriers, half the shared memory, more L1 for the gathers) where records
// are wider.
template <typename FT, int NM>
constexpr int planned_nbuf()
{
    return sizeof(FT) == 4 && NM == 3 ? 2 : 1;
}

// Nonzeros whose key, value and plan entry a thread loads together in the
// scatter phase: one.  Four in flight were the register peak of the kernel
// (order 4, rank 16, FP64, 18.9M nonzeros: 647 us a mode with four and two
// buffers, 560 with one and one).
constexpr int PLANNED_Q = 1;

// A planned record holds MM + FW words: [target index, the other modes'
// indices, the value].  Four words are one 16-byte record; wider ones keep
// words 1-4 in a 16-byte array and the rest (the target index and one or two
// more words) in a second, narrower array, so an order-4 FP32 or order-3 FP64
// record takes 20 bytes and two loads of 16 and 4 bytes instead of 32 bytes.
template <typename FT, int MM>
struct PlanRec {
    static constexpr int W = MM + (int)(sizeof(FT) / 4);
    static constexpr int BW = W <= 4 ? 0 : W == 5 ? 1 : W == 6 ? 2 : 4;  // words of the second array
    static_assert(W <= 8, "record words");

    static __device__ __forceinline__ void store(u32* A, u32* B, int slot, const u32* w)
    {
        if constexpr (BW == 0) {
            *reinterpret_cast<uint4*>(A + (size_t)slot * 4) = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
            *reinterpret_cast<uint4*>(A + (size_t)slot * 4) = make_uint4(w[1], w[2], w[3], w[4]);
            if constexpr (BW == 1) B[slot] = w[0];
            else if constexpr (BW == 2) *reinterpret_cast<uint2*>(B + (size_t)slot * 2) = make_uint2(w[0], w[5]);
            else *reinterpret_cast<uint4*>(B + (size_t)slot * 4) = make_uint4(w[0], w[5], w[6], W > 7 ? w[7] : 0u);
        }
    }
    static __device__ __forceinline__ void load(const u32* A, const u32* B, int slot, u32* w)
    {
        const uint4 t = *reinterpret_cast<const uint4*>(A + (size_t)slot * 4);
        if constexpr (BW == 0) {
            w[0] = t.x;
            w[1] = t.y;
            w[2] = t.z;
            w[3] = t.w;
        } else {
            w[1] = t.x;
            w[2] = t.y;
            w[3] = t.z;
            w[4] = t.w;
            if constexpr (BW == 1) {
                w[0] = B[slot];
            } else if constexpr (BW == 2) {
                const uint2 b = *reinterpret_cast<const uint2*>(B + (size_t)slot * 2);
                w[0] = b.x;
                w[5] = b.y;
            } else {
                const uint4 b = *reinterpret_cast<const uint4*>(B + (size_t)slot * 4);
                w[0] = b.x;
                w[5] = b.y;
                w[6] = b.z;
                if constexpr (W > 7) w[7] = b.w;
            }
        }
    }
};

// Records a lane group takes per tile (lpn lanes per nonzero).
constexpr int planned_ipg(int pt, int lpn) { return pt / (MT_WARPS * (32 / lpn)); }
constexpr int log2c(int x) { return x <= 1 ? 0 : 1 + log2c(x / 2); }

// Record words per slot of a run-time order, and the dynamic shared memory of
// the planned kernel: nbuf run-ordered record buffers (one padding record per
// lane-group stretch) and the hot-row tags.
inline int planned_rec_words(int nmode, size_t fsz)
{
    const int w = nmode + (int)(fsz / 4);
    return w <= 4 ? 4 : w <= 6 ? w : 8;
}
inline size_t planned_smem(int nmode, size_t fsz, int hot, int lpn, int pt, int nbuf)
{
    return (size_t)nbuf * (size_t)(pt + pt / planned_ipg(pt, lpn)) * planned_rec_words(nmode, fsz) * 4 + (size_t)hot * 4;
}

// Phase A of a planned tile: every thread loads key, value and plan entry
// of its nonzeros (QM in flight at a time), decodes the mode indices and
// writes the record [target, other modes..., value] to its run-ordered slot
// (one padding record per 2^PSH).  Reading through a permutation (oidx) the
// stream is in target order already and the slot is the position itself.
template <typename FT, typename VT, int MM, int PT, int PSH, int QM = 4, bool PERM = false>
__device__ __forceinline__ void planned_scatter(const TiledArgs<FT>& a, u64 g0, int nvalid, u32* srec, u32* srecb = nullptr)
{
    typedef PlanRec<FT, MM> Rec;
    constexpr int FW = (int)(sizeof(FT) / 4);
    constexpr int IPT = PT / MT_THREADS;
    constexpr int IPQ = IPT < QM ? IPT : QM;
    const int tid = threadIdx.x, target = a.target;
    const VT* vals = reinterpret_cast<const VT*>(a.vals);
    TileHi th;
    if constexpr (PERM) th.slow = true;
    else th.init(a.key, g0, PT);
#pragma unroll
    for (int k0 = 0; k0 < IPT; k0 += IPQ) {
        u64 lo[IPQ];
        VT vv[IPQ];
        u32 ps[IPQ];
#pragma unroll
        for (int k = 0; k < IPQ; ++k) {
            const int it = tid + (k0 + k) * MT_THREADS;
            if (it < nvalid) {
                const u64 g = g0 + it;
                if constexpr (PERM) {
                    ps[k] = a.perm[g];  // read position
                    lo[k] = a.key.klo[ps[k]];
                    vv[k] = vals[ps[k]];
                } else {
                    lo[k] = __ldcs(reinterpret_cast<const unsigned long long*>(a.key.klo) + g);
                    vv[k] = ldcs_val(vals + g);
                    ps[k] = __ldcs(reinterpret_cast<const unsigned short*>(a.plan) + g);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < IPQ; ++k) {
            const int it = tid + (k0 + k) * MT_THREADS;
            if (it < nvalid) {
                const u64 hi = th.get(a.key, PERM ? (u64)ps[k] : g0 + it);
                u32 c[MM];
#pragma unroll
                for (int m = 0; m < MM; ++m) c[m] = field(lo[k], hi, a.fld.pos[m], a.fld.mask[m]);
                u32 w[Rec::W];
                w[0] = c[0];
#pragma unroll
                for (int m = 1; m < MM; ++m)
                    if (m == target) w[0] = c[m];
#pragma unroll
                for (int s = 1; s < MM; ++s) w[s] = s - 1 < target ? c[s - 1] : c[s];
                const FT fv = (FT)vv[k];
                if constexpr (FW == 1) {
                    w[MM] = __float_as_uint((float)fv);
                } else {
                    const unsigned long long bits = (unsigned long long)__double_as_longlong((double)fv);
                    w[MM] = (u32)bits;
                    w[MM + 1] = (u32)(bits >> 32);
                }
                Rec::store(srec, srecb, rslot_t<PSH>(PERM ? it : (int)ps[k]), w);
            }
        }
    }
}

// Phase B: the lane group walks its stretch [p0, pe) of the run-ordered
// records two at a time (both records' gathers issued before either is
// added) and keeps the run sum of its current output row in registers.
// A run's sum goes to its row of `out` with one vector atomic, or, if the run
// has a.hot_minrun nonzeros, to the CTA's hot-row slot.
// MTTKRP adds v * row_1 * ... * row_{N-1} (the products in the order of
// nz_row); PHI adds (v / max(<B[row], pi>, eps)) pi with pi the same product
// without v and B[row] held in registers for the run.
template <typename FT, int MM, int LPN, int VEC, int CH, int PSH, bool PHI, bool HOT = true>
__device__ __forceinline__ void planned_runs(const TiledArgs<FT>& a, const GroupedSmem& gs, const u32* srec,
                                             const u32* srecb, const FT* const* Uo, FT* out, int p0, int pe, int R,
                                             int sub, unsigned gmask)
{
    typedef PlanRec<FT, MM> Rec;
    const u32 Ru = (u32)R;
    // Lanes past the rank (R below LPN * VEC * CH) load the row's last
    // elements, so every load stays inside its row; only r0 < R is written.
    int col[CH];
    bool in[CH];
#pragma unroll
    for (int ch = 0; ch < CH; ++ch) {
        col[ch] = min((ch * LPN + sub) * VEC, R - VEC);
        in[ch] = (ch * LPN + sub) * VEC < R;
    }
    const FT* Ub[MM - 1];
#pragma unroll
    for (int k = 0; k < MM - 1; ++k) Ub[k] = Uo[k] + (CH == 1 ? col[0] : 0);
    const FT* Bt = PHI ? a.U[a.target] + (CH == 1 ? col[0] : 0) : nullptr;
    auto vl = [&](const FT* base, u32 row, FT (*y)[VEC]) {
        const FT* r = base + (size_t)row * Ru;
#pragma unroll
        for (int ch = 0; ch < CH; ++ch) vload<FT, VEC>(CH == 1 ? r : r + col[ch], y[ch]);
    };
    u32 cur = 0xffffffffu;
    int len = 0;
    const int hmin = a.hot_minrun ? a.hot_minrun : GT_HOT_MINRUN;
    FT acc[CH][VEC];
    FT bc[PHI ? CH : 1][VEC];
#pragma unroll
    for (int ch = 0; ch < CH; ++ch)
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[ch][e] = FT(0);
    auto flush = [&]() {
        if (cur != 0xffffffffu)
            flush_run<FT, VEC, CH, LPN>(out, gs, HOT && len >= hmin ? a.hot : 0, a.hot_acc, gmask, cur, R, sub,
                                            acc);
    };
    // the Khatri-Rao product of a record into x (times its value for MTTKRP)
    auto product = [&](const u32* w, FT (*y)[CH][VEC], FT (*x)[VEC]) {
        if constexpr (PHI) {
#pragma unroll
            for (int ch = 0; ch < CH; ++ch)
#pragma unroll
                for (int e = 0; e < VEC; ++e) x[ch][e] = in[ch] ? y[0][ch][e] : FT(0);
        } else {
            const FT v = rec_val<FT, MM>(w);
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) {
#pragma unroll
                for (int e = 0; e < VEC; ++e) x[ch][e] = v;
                vmul<FT, VEC>(x[ch], y[0][ch]);
            }
        }
#pragma unroll
        for (int k = 1; k < MM - 1; ++k)
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) vmul<FT, VEC>(x[ch], y[k][ch]);
    };
    auto add = [&](const u32* w, FT (*x)[VEC]) {
        if (w[0] != cur) {
            flush();
            cur = w[0];
            len = 1;
#pragma unroll
            for (int ch = 0; ch < CH; ++ch)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[ch][e] = x[ch][e];
        } else {
            run_add<FT, VEC, CH>(acc, x);
            ++len;
        }
    };
    auto dot = [&](FT (*b)[VEC], FT (*x)[VEC]) {
        FT d = FT(0);
#pragma unroll
        for (int ch = 0; ch < CH; ++ch)
#pragma unroll
            for (int e = 0; e < VEC; ++e) d += b[ch][e] * x[ch][e];
        return d;
    };
    auto scale = [&](const u32* w, FT d, FT (*x)[VEC]) {
        const FT sc = rec_val<FT, MM>(w) / (d > a.eps ? d : a.eps);
#pragma unroll
        for (int ch = 0; ch < CH; ++ch)
#pragma unroll
            for (int e = 0; e < VEC; ++e) x[ch][e] *= sc;
    };
    int p = p0;
    for (; p + 1 < pe; p += 2) {
        u32 w0[Rec::W], w1[Rec::W];
        Rec::load(srec, srecb, rslot_t<PSH>(p), w0);
        Rec::load(srec, srecb, rslot_t<PSH>(p + 1), w1);
        FT y0[MM - 1][CH][VEC], y1[MM - 1][CH][VEC];
#pragma unroll
        for (int k = 0; k < MM - 1; ++k) {
            vl(Ub[k], w0[1 + k], y0[k]);
            vl(Ub[k], w1[1 + k], y1[k]);
        }
        FT x0[CH][VEC], x1[CH][VEC];
        if constexpr (PHI) {
            FT b0[CH][VEC];
            if (w0[0] != cur) vl(Bt, w0[0], bc);
#pragma unroll
            for (int ch = 0; ch < CH; ++ch)
#pragma unroll
                for (int e = 0; e < VEC; ++e) b0[ch][e] = bc[ch][e];
            if (w1[0] != w0[0]) vl(Bt, w1[0], bc);
            product(w0, y0, x0);
            product(w1, y1, x1);
            FT d0 = dot(b0, x0), d1 = dot(bc, x1);
#pragma unroll
            for (int o = LPN / 2; o > 0; o >>= 1) {
                d0 += __shfl_xor_sync(gmask, d0, o, LPN);
                d1 += __shfl_xor_sync(gmask, d1, o, LPN);
            }
            scale(w0, d0, x0);
            scale(w1, d1, x1);
            add(w0, x0);
            add(w1, x1);
        } else {
            product(w0, y0, x0);
            add(w0, x0);
            product(w1, y1, x1);
            add(w1, x1);
        }
    }
    if (p < pe) {
        u32 w0[Rec::W];
        Rec::load(srec, srecb, rslot_t<PSH>(p), w0);
        FT y0[MM - 1][CH][VEC], x0[CH][VEC];
#pragma unroll
        for (int k = 0; k < MM - 1; ++k) vl(Ub[k], w0[1 + k], y0[k]);
        product(w0, y0, x0);
        if constexpr (PHI) {
            if (w0[0] != cur) vl(Bt, w0[0], bc);
            FT d0 = dot(bc, x0);
#pragma unroll
            for (int o = LPN / 2; o > 0; o >>= 1) d0 += __shfl_xor_sync(gmask, d0, o, LPN);
            scale(w0, d0, x0);
        }
        add(w0, x0);
    }
    flush();
}

// One planned tile with one record buffer (the batched kernel): scatter,
// barrier, runs, barrier.
template <typename FT, typename VT, int NM, int LPN, int VEC>
__device__ __forceinline__ void planned_tile(const TiledArgs<FT>& a, u64 ti, const GroupedSmem& gs, u32* srecb)
{
    constexpr int NPW = 32 / LPN;
    constexpr int IPG = PT_TILE / (MT_WARPS * NPW);
    constexpr int PSH = log2c(IPG);
    static_assert(NM >= 3 && NM <= ALTOB_MAX_MODES, "static order 3..5");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane % LPN, q = lane / LPN;
    const unsigned gmask = (0xffffffffu >> (32 - LPN)) << (q * LPN);
    const u64 g0 = ti * (u64)PT_TILE;
    const int nvalid = (int)min((u64)PT_TILE, a.nnz - g0);
    if (a.perm) planned_scatter<FT, VT, NM, PT_TILE, PSH, PLANNED_Q, true>(a, g0, nvalid, gs.srec, srecb);
    else planned_scatter<FT, VT, NM, PT_TILE, PSH, PLANNED_Q>(a, g0, nvalid, gs.srec, srecb);
    __syncthreads();
    const int p0 = (warp * NPW + q) * IPG;
    const FT* Uo[NM - 1];
#pragma unroll
    for (int k = 0; k < NM - 1; ++k) Uo[k] = a.U[k < a.target ? k : k + 1];
    planned_runs<FT, NM, LPN, VEC, 1, PSH, false>(a, gs, gs.srec, srecb, Uo, a.out, p0, min(p0 + IPG, nvalid), a.R, sub,
                                                          gmask);
    __syncthreads();
}

// PT: nonzeros per tile (the plan's tile); NBUF: record buffers (2: the
// next tile's scatter overlaps this tile's runs, one barrier per tile; 1:
// two barriers per tile, half the shared memory, so more of the SM's
// 256 KB stays L1 cache for the row gathers).  2^split_shift CTAs share a
// tile: each scatters all of it and walks its share of every lane group's
// stretch.  With WHOLE the output is short enough that every CTA adds into
// a copy of its own, which reaches the output once per CTA: fewer FP32
// additions per row and no contention on the rows of a short mode.
template <typename FT, typename VT, int NM, int LPN, int VEC, int CH, bool PHI, bool PERM, bool WHOLE, int PT, int NBUF>
__device__ __forceinline__ void planned_body(const TiledArgs<FT>& a)
{
    constexpr int MM = NM;
    constexpr int NPW = 32 / LPN;
    constexpr int NGRP = MT_WARPS * NPW;
    constexpr int IPG = PT / NGRP;
    constexpr int PSH = log2c(IPG);
    constexpr int SREC = PT + PT / IPG;
    constexpr int BW = PlanRec<FT, MM>::BW;
    static_assert(IPG == planned_ipg(PT, LPN) && (1 << PSH) == IPG, "lane-group stretch");
    static_assert(NM >= 3 && NM <= ALTOB_MAX_MODES, "static order 3..5");
    static_assert(NBUF == 1 || NBUF == 2, "record buffers");
    static_assert(SREC % 4 == 0, "second record array on a 16-byte boundary");
    extern __shared__ __align__(16) unsigned char smem[];
    u32* const buf = reinterpret_cast<u32*>(smem);
    GroupedSmem gs = {};
    gs.htag = buf + (size_t)NBUF * SREC * (4 + BW);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int R = a.R, target = a.target;
    const int sub = lane % LPN, q = lane / LPN;
    const int grp = warp * NPW + q;
    const unsigned gmask = (0xffffffffu >> (32 - LPN)) << (q * LPN);
    const int slots = WHOLE ? a.whole : a.hot;
    if (slots) {
        FT* hacc = a.hot_acc + (size_t)blockIdx.x * slots * R;
        if (!WHOLE)
            for (int k = tid; k < slots; k += MT_THREADS) gs.htag[k] = 0;
        for (int k = tid * VEC; k < slots * R; k += MT_THREADS * VEC) vstore_zero<FT, VEC>(hacc + k);
        __syncthreads();  // the zeroed accumulators precede every run flush
    }

    const int ssh = a.split_shift;
    const u64 nitems = a.ntiles << ssh;
    int b = 0;
    for (u64 it = blockIdx.x; it < nitems; it += gridDim.x, b ^= NBUF - 1) {
        u32* srec = buf + (size_t)b * SREC * (4 + BW);
        u32* srecb = BW ? srec + (size_t)SREC * 4 : nullptr;
        const u64 g0 = (it >> ssh) * (u64)PT;
        const int nvalid = (int)min((u64)PT, a.nnz - g0);
        // ---- A: load key, value and plan entry; record into its sorted slot
        planned_scatter<FT, VT, MM, PT, PSH, PLANNED_Q, PERM>(a, g0, nvalid, srec, srecb);
        // with two buffers one barrier per tile: the buffer written next tile
        // was last read before this barrier
        __syncthreads();
        // up to here only keys, values and the plan were read (and the CTA's
        // own accumulators written); factors and output may still be in the
        // hands of the kernel before this one
        if (it == blockIdx.x) grid_wait();
        // ---- B: runs of equal output rows
        const int ipg = IPG >> ssh;
        const int p0 = grp * IPG + (int)(it & ((1u << ssh) - 1u)) * ipg;
        const int pend = min(p0 + ipg, nvalid);
        const FT* Uo[MM - 1];  // from the parameters each tile: fewer live registers
#pragma unroll
        for (int k = 0; k < MM - 1; ++k) Uo[k] = a.U[k < target ? k : k + 1];
        FT* out = WHOLE ? a.hot_acc + (size_t)blockIdx.x * a.whole * R : a.out;
        if constexpr (!PHI && !WHOLE && CH == 1 && BW == 0) {
            gs.srec = srec;
            lean_runs<FT, MM, LPN, VEC, PSH>(a, gs, Uo, p0, pend, R, sub, gmask);
        } else {
            planned_runs<FT, MM, LPN, VEC, CH, PSH, PHI, !WHOLE>(a, gs, srec, srecb, Uo, out, p0, pend, R, sub, gmask);
        }
        if constexpr (NBUF == 1) __syncthreads();  // the records are overwritten next tile
    }
    if (slots) {  // the CTA's sums, once each (read from L2, where the atomics landed)
        const FT* hacc = a.hot_acc + (size_t)blockIdx.x * slots * R;
        typedef typename VecT<FT, VEC>::T V;
        __syncthreads();
        for (int k = tid * VEC; k < slots * R; k += MT_THREADS * VEC) {
            const int sl = k / R;
            const u32 row = WHOLE ? (u32)sl : gs.htag[sl] - 1u;
            if (row == 0xffffffffu) continue;
            const V v = __ldcg(reinterpret_cast<const V*>(hacc + k));
            const FT* x = reinterpret_cast<const FT*>(&v);
            bool any = false;  // rows this CTA never met stay zero
#pragma unroll
            for (int e = 0; e < VEC; ++e) any = any || x[e] != FT(0);
            if (any) gred<FT, VEC>(a.out + (size_t)row * R + (k - sl * R), x);
        }
    }
}

// MINB 0: the compiler's own register choice.
template <typename FT, typename VT, int NM, int LPN, int VEC, int CH, bool PHI, bool PERM, bool WHOLE, int MINB, int PT, int NBUF>
__global__ void __launch_bounds__(MT_THREADS, MINB ? MINB : 1) k_planned(TiledArgs<FT> a)
{
    planned_body<FT, VT, NM, LPN, VEC, CH, PHI, PERM, WHOLE, PT, NBUF>(a);
}

// Batched form: the tiles of many tensors (one TiledArgs each, same shape
// class and slot count) in one persistent launch.  tile_prefix[b] is the
// first global tile of tensor b; tensors whose active flag is 0 are skipped.
template <typename FT>
struct BatchTiles {
    const TiledArgs<FT>* args;
    const u64* tile_prefix;  // ntensors + 1
    const int* bid;          // batch index of each entry (for `active`)
    const int* active;
    int ntensors;
    int hslots;
    u64 total_tiles;
};

// Tensor of a global tile.  The tile prefixes and active flags of up to
// BT_CACHE tensors are kept in shared memory: in global memory every tile
// waited for about seven dependent loads (32 tensors, 4 iterations, together
// with the rank classes side by side: 11.5 -> 10.3 ms).
constexpr int BT_CACHE = 512;
struct BatchLookup {
    u32 pre[BT_CACHE];
    unsigned char act[BT_CACHE];
};

template <typename FT>
__device__ __forceinline__ void batch_lookup_init(const BatchTiles<FT>& bt, BatchLookup& c)
{
    if (bt.ntensors <= BT_CACHE)
        for (int i = threadIdx.x; i < bt.ntensors; i += blockDim.x) {
            c.pre[i] = (u32)bt.tile_prefix[i];
            c.act[i] = bt.active[bt.bid[i]] != 0;
        }
    __syncthreads();
}

// The last tensor whose first tile is at or before gt; *active its flag.
template <typename FT>
__device__ __forceinline__ int batch_owner(const BatchTiles<FT>& bt, const BatchLookup& c, u64 gt, bool* active)
{
    const bool cached = bt.ntensors <= BT_CACHE;
    int lo = 0, hi = bt.ntensors - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((cached ? (u64)c.pre[mid] : bt.tile_prefix[mid]) <= gt) lo = mid;
        else hi = mid - 1;
    }
    *active = cached ? c.act[lo] != 0 : bt.active[bt.bid[lo]] != 0;
    return lo;
}

template <typename FT, typename VT, int NM, int LPN, int VEC, int CH, bool PHI>
__device__ __forceinline__ void grouped_batch_body(const BatchTiles<FT>& bt)
{
    constexpr int MM = grouped_mm<NM>();
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ u32 statics[2 + MT_WARPS];
    const GroupedSmem gs = grouped_smem_ptrs<FT, MM>(smem, bt.hslots, statics);
    __shared__ BatchLookup lookup;
    batch_lookup_init(bt, lookup);
    grouped_init(gs, bt.hslots);
    for (u64 gt = blockIdx.x; gt < bt.total_tiles; gt += gridDim.x) {
        bool active;
        const int lo = batch_owner(bt, lookup, gt, &active);
        if (!active) continue;
        grouped_tile<FT, VT, NM, LPN, VEC, CH, PHI>(bt.args[lo], gt - bt.tile_prefix[lo], gs);
    }
}

template <typename FT, typename VT, int NM, int LPN, int VEC, int CH, bool PHI>
__global__ void __launch_bounds__(MT_THREADS) k_grouped_batch(BatchTiles<FT> bt)
{
    grouped_batch_body<FT, VT, NM, LPN, VEC, CH, PHI>(bt);
}

template <typename FT, typename VT, int NM, int LPN, int VEC, int CH, bool PHI, int MINB>
__global__ void __launch_bounds__(MT_THREADS, MINB) k_grouped_batch_mb(BatchTiles<FT> bt)
{
    grouped_batch_body<FT, VT, NM, LPN, VEC, CH, PHI>(bt);
}

// Batched planned MTTKRP: the tiles of the tensors whose target mode has a
// tile plan (same shape class), one persistent launch; single record buffer.
template <typename FT, typename VT, int NM, int LPN, int VEC>
__device__ __forceinline__ void planned_batch_body(const BatchTiles<FT>& bt)
{
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int SREC = PT_TILE + PT_TILE / planned_ipg(PT_TILE, LPN);
    GroupedSmem gs = {};
    gs.srec = reinterpret_cast<u32*>(smem);
    u32* srecb = gs.srec + (size_t)SREC * 4;
    __shared__ BatchLookup lookup;
    batch_lookup_init(bt, lookup);
    for (u64 gt = blockIdx.x; gt < bt.total_tiles; gt += gridDim.x) {
        bool active;
        const int lo = batch_owner(bt, lookup, gt, &active);
        if (!active) continue;
        planned_tile<FT, VT, NM, LPN, VEC>(bt.args[lo], gt - bt.tile_prefix[lo], gs, srecb);
    }
}

template <typename FT, typename VT, int NM, int LPN, int VEC>
__global__ void __launch_bounds__(MT_THREADS) k_planned_batch(BatchTiles<FT> bt)
{
    planned_batch_body<FT, VT, NM, LPN, VEC>(bt);
}

template <typename FT, typename VT, int NM, int LPN, int VEC, int MINB>
__global__ void __launch_bounds__(MT_THREADS, MINB) k_planned_batch_mb(BatchTiles<FT> bt)
{
    planned_batch_body<FT, VT, NM, LPN, VEC>(bt);
}

// Shared memory of the batched planned kernel: one run-ordered record buffer.
inline size_t planned_batch_smem(int nmode, size_t fsz, int lpn) { return planned_smem(nmode, fsz, 0, lpn, PT_TILE, 1); }

}  // namespace altob
