// k_conv.cu -- 3x3x3 "same" convolutions on the 5th-generation tensor cores
// (tcgen05.mma kind::f16, BF16 operands, FP32 accumulators in tensor memory),
// used by the learned preconditioner.
//
// Forward (and data-gradient, with the flipped/transposed weight image) as an
// implicit GEMM.  A persistent CTA takes blocks of one 128-cell x-tile, four
// output lines in j and KC levels, and marches through the block's input levels:
// six x-lines of 130 cells (one halo cell per side) per level, bulk-copied with
// one 2080-byte copy per (line, channel group).  In that no-swizzle K-major
// layout a tap's A operand is the line's matrix descriptor with the start address
// moved by (di+1) rows of 16 bytes.  One MMA multiplies a line by the stacked
// weights of the taps dj = 1, 0, -1 (N = 3 cout): the accumulators of the four
// output lines of a level lie side by side in tensor memory, so the three
// products land in neighbouring columns.  Four accumulator levels rotate (three
// being summed, one in the epilogue).  A copy warp, an MMA thread and four
// epilogue warps run side by side, tied by mbarriers.
// What bounds it: an MMA with N <= 64 takes as long as reading its A operand (4
// KB), so the taps are merged in N (13.5 MMAs per 128-cell tile and 16 input
// channels instead of 27), and a line is fetched 1.5 times instead of 9.  B200,
// 32 -> 32 channels at 64x64x48: 91 -> 46 us.  Convolutions to 16 channels merge
// all nine taps of a line (conv3_fwd9_kernel).
//
// Weight gradient: dW_tap[CIN x COUT] = sum over cells of X(v + tap)^T dY(v):
// the reduction runs over cells (the MMA's K), both operands MN-major straight
// from the same line images (8 cells x 8 channels = one 128-byte core matrix).
// A tile is TJ lines of dY (N = TJ cout) and the 3 (TJ + 2) input lines around
// them: rows of one M=128 operand are 16 consecutive (level, line, channel group)
// blocks at the fixed 2080-byte line stride, so one descriptor covers many taps;
// the three x-shifts are separate accumulators.  Of the line pairs in a product
// those within one line of each other are kept.  Each persistent CTA accumulates
// all of its tiles in TMEM, sums its pairs in shared memory and adds them to the
// FP32 gradient with 16-byte atomics.
// What bounds it: reading the A operand (4 KB an MMA), so several dY lines share
// it (16 MMAs per 128-cell line of 16 channels instead of 48), and the atomics of
// 148 CTAs.  128x128x32 (and its halves), a launch: 16 -> 16 97 -> 53 us, 32 -> 32
// 107 -> 58 us, 16 -> 32 95 -> 56 us, 32 -> 16 91 -> 53 us.
#include <cuda_bf16.h>
#include <limits.h>
#include <stdio.h>

#include <algorithm>

#include "kernels.h"
#include "tc05.cuh"
#include "unet.h"

namespace hw {

constexpr int TILE = 128;
constexpr int LROWS = TILE + 2;
constexpr int LG = LROWS * 16; // bytes of one (line, channel group) image with halo
constexpr int YG = TILE * 16;  // bytes of one (line, channel group) image without halo
constexpr int SG = 17 * 128;   // pitch of the images in a forward stage, which start SGO past a multiple of 128 bytes,
constexpr int SGO = 112;       // so that the core matrices of the unshifted taps are whole 128-byte lines (the other
                               // shifts straddle two: an MMA's operand read takes twice as long)
constexpr int up128(int b) { return (b + 127) / 128 * 128; }

__device__ __forceinline__ bool conv_gated(const SolveState *g)
{
    return g && *(volatile const int *)&g->stop != 0 && !g->profile;
}

__device__ __forceinline__ void unpack8(const uint4 &u, float (&f)[8])
{
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        float2 t = __bfloat1622float2(h[q]);
        f[2 * q] = t.x;
        f[2 * q + 1] = t.y;
    }
}

__device__ __forceinline__ uint4 pack8(const float *f)
{
    uint4 u;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
    for (int q = 0; q < 4; q++) h[q] = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
    return u;
}

template <int CIN, int COUT>
struct FwdCfg {
    static constexpr int GI = CIN / 8, GO = COUT / 8;
    static constexpr int TJ = 4, NL = TJ + 2;       // output and input lines of a block in j
    static constexpr int SLOTS = 4;                 // accumulator levels: three in the making, one in the epilogue
    static constexpr int WB = 27 * GI * COUT * 16;  // weight image bytes
    static constexpr int STAGE = NL * GI * SG;      // one input level's line images
    static constexpr int NCOL = SLOTS * TJ * COUT;  // all of the tensor memory
    static constexpr int NS = 3;                    // input levels in flight
    static constexpr int SMEM = up128(WB) + NS * STAGE + 256;
    static constexpr int PER_SM = 1;
    static_assert(CIN % 16 == 0 && COUT == 32 && NCOL == 512 && 3 * COUT <= 256, "channel counts");
    static_assert(SMEM <= 232448, "shared memory");
};

// How a launch splits the grid: blocks of one x-tile, TJ output lines in j and
// KC output levels, nkb of them in k, njb in j (k fastest).
struct ConvSplit {
    int KC, nkb, njb, units;
};

struct ConvBlock {
    int tx, j0, k0, nj, nk; // first output line and level, how many of each
    int lo, hi;             // input levels read (the halo levels are zero and left out)
};

__device__ __forceinline__ ConvBlock conv_block(const ActDims &d, const ConvSplit &p, int TJ, int u)
{
    ConvBlock b;
    b.k0 = u % p.nkb * p.KC;
    b.j0 = u / p.nkb % p.njb * TJ;
    b.tx = u / (p.nkb * p.njb);
    b.nj = min(TJ, d.ny - b.j0);
    b.nk = min(p.KC, d.nz - b.k0);
    b.lo = max(b.k0 - 1, 0);
    b.hi = min(b.k0 + b.nk, d.nz - 1);
    return b;
}

constexpr int CONV_THREADS = 192; // warps 0-3 epilogue (TMEM lanes 32 w .. 32 w + 31), 4 copies, 5 MMAs

// One input level's MMAs of the taps dk into one output level's accumulators d0
// (NJ output lines, or nj where NJ is 0): line l feeds the output lines l - 2 .. l
// with the taps dj = 1, 0, -1; fresh: the accumulators get their first products.
template <int CIN, int COUT, int NJ>
__device__ __forceinline__ void issue_taps(int nj, uint64_t a0, uint64_t b0, uint32_t d0, int dk, bool fresh)
{
    using C = FwdCfg<CIN, COUT>;
    const int lines = NJ ? NJ : nj;
    const uint64_t bk = b0 + (uint64_t)((dk * 3 * C::GI * 3 * COUT * 16) >> 4);
#pragma unroll
    for (int dil = 0; dil < 3; dil++)
#pragma unroll
        for (int c = 0; c < C::GI / 2; c++) {
            const uint64_t bt = bk + (uint64_t)(((dil * C::GI + 2 * c) * 3 * COUT * 16) >> 4);
#pragma unroll
            for (int l = 0; l < C::NL; l++) {
                if (l >= lines + 2) break;
                const int o0 = l - 2 > 0 ? l - 2 : 0, o1 = l < lines - 1 ? l : lines - 1;
                const uint64_t ad = a0 + (uint64_t)(((l * C::GI + 2 * c) * SG + dil * 16) >> 4);
                const uint64_t bd = bt + (uint64_t)((o0 - (l - 2)) * COUT); // without the taps of lines outside the block
                const uint32_t all = tc::idesc_bf16(128, 0, 0, 0) | ((uint32_t)((o1 - o0 + 1) * COUT / 8) << 17);
                if (dil == 0 && c == 0 && fresh) {
                    const int old = l - 1 < o1 ? l - 1 : o1;
                    if (old >= o0)
                        tc::mma_bf16(d0 + o0 * COUT, ad, bd,
                                     tc::idesc_bf16(128, 0, 0, 0) | ((uint32_t)((old - o0 + 1) * COUT / 8) << 17), 1u);
                    if (o1 == l) // output line l gets its first product
                        tc::mma_bf16(d0 + l * COUT, ad, bt + (uint64_t)(2 * COUT), tc::idesc_bf16(128, COUT, 0, 0), 0u);
                } else tc::mma_bf16(d0 + o0 * COUT, ad, bd, all, 1u);
            }
        }
}

// Bias, skip, ReLU, mask and the stores of one cell of one output line: v its
// sums, ex its skip (or else mask) values fetched ahead, at its act unit.
template <int COUT>
__device__ __forceinline__ void conv_store(const ConvArgs &a, float (&v)[COUT], const float (&bias)[COUT],
                                           const uint4 (&ex)[COUT / 8], long long at, int i, int k, int j)
{
    constexpr int GO = COUT / 8;
    const ActDims &dd = a.dout;
#pragma unroll
    for (int c = 0; c < COUT; c++) v[c] += bias[c];
    if (a.skip) {
#pragma unroll
        for (int g = 0; g < GO; g++) {
            float f[8];
            unpack8(ex[g], f);
#pragma unroll
            for (int e = 0; e < 8; e++) v[g * 8 + e] += f[e];
        }
    }
    if (a.relu) {
#pragma unroll
        for (int c = 0; c < COUT; c++) v[c] = fmaxf(v[c], 0.0f);
    }
    if (a.mask) {
#pragma unroll
        for (int g = 0; g < GO; g++) {
            float f[8];
            unpack8(a.skip ? a.mask[at + g * dd.PX] : ex[g], f);
#pragma unroll
            for (int e = 0; e < 8; e++) v[g * 8 + e] = f[e] > 0.0f ? v[g * 8 + e] : 0.0f;
        }
    }
    if (a.out) {
#pragma unroll
        for (int g = 0; g < GO; g++) a.out[at + g * dd.PX] = pack8(v + g * 8);
    }
    if (a.out0) a.out0[((long long)j * dd.nz + k) * dd.nx + i] = v[0];
}

// The skip (or else mask) values of a thread's cell in the output lines of a block's level.
template <int COUT, int TJ>
__device__ __forceinline__ void conv_extra(const ConvArgs &a, uint4 (&ex)[TJ][COUT / 8], long long base, long long js, int nj,
                                           bool live)
{
    const uint4 *extra = a.skip ? a.skip : a.mask;
#pragma unroll
    for (int o = 0; o < TJ; o++)
#pragma unroll
        for (int g = 0; g < COUT / 8; g++)
            ex[o][g] = extra && live && o < nj ? extra[base + o * js + g * a.dout.PX] : make_uint4(0, 0, 0, 0);
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(CONV_THREADS) conv3_fwd_kernel(ConvArgs a, ConvSplit p)
{
    using C = FwdCfg<CIN, COUT>;
    constexpr int NS = C::NS, TJ = C::TJ, SLOTS = C::SLOTS;
    if (conv_gated(a.gate)) return;
    extern __shared__ __align__(128) uint8_t sm[];
    uint8_t *wsm = sm, *stg = sm + up128(C::WB) + SGO;
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + up128(C::WB) + NS * C::STAGE + 128), *empty = full + NS, *tfull = empty + NS,
             *tempty = tfull + SLOTS;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(tempty + SLOTS);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const ActDims di = a.din, dd = a.dout;
    if (tid == 0) {
        for (int q = 0; q < NS; q++) {
            tc::mbar_init(&full[q], 1);
            tc::mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < SLOTS; q++) {
            tc::mbar_init(&tfull[q], 1);
            tc::mbar_init(&tempty[q], 4);
        }
        tc::mbar_fence_init();
    }
    if (warp == 0) tc::tmem_alloc(tslot, C::NCOL);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;
    bool ok = true;
    auto wait = [&](uint64_t *bar, int use) { // the use-th completion (from 0); on time-out: no more waits
        if (ok && !tc::mbar_wait(bar, use & 1)) {
            if (lane == 0) atomicExch(a.err, 1);
            ok = false;
        }
    };

    if (warp == 4) { // ---- copies: one input level per stage, one bulk copy per (line, channel group) ----
        const char *inb = reinterpret_cast<const char *>(a.in);
        int it = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
            const ConvBlock b = conv_block(di, p, TJ, u);
            for (int kk = b.lo; kk <= b.hi; kk++, it++) {
                const int s = it % NS;
                if (it >= NS) wait(&empty[s], it / NS - 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const int n = (b.nj + 2) * C::GI;
                if (lane == 0) tc::mbar_expect_tx(&full[s], n * LG + (it == 0 ? C::WB : 0));
                __syncwarp();
                if (it == 0 && lane == 31) tc::bulk_g2s(wsm, a.w, C::WB, &full[s]);
                for (int q = lane; q < n; q += 32) {
                    const int l = q / C::GI, g = q % C::GI; // input line j0 - 1 + l, level kk
                    const long long L = (long long)(b.j0 + l) * (di.nz + 2) + (kk + 1);
                    tc::bulk_g2s(stg + s * C::STAGE + q * SG, inb + ((L * C::GI + g) * di.PX + (long long)b.tx * TILE) * 16,
                                 LG, &full[s]);
                }
            }
            if (!ok) break;
        }
        // nothing in flight at the end: the last stages landed and were read
        for (int q = it > NS ? it - NS : 0; q < it; q++) {
            if (!tc::mbar_wait(&full[q % NS], (q / NS) & 1) && lane == 0) atomicExch(a.err, 1);
            wait(&empty[q % NS], q / NS);
        }
    } else if (warp == 5) { // ---- MMAs, one thread ----
        if (lane == 0) {
            // descriptors of the stage / weight bases; operands are byte offsets from them (start field = address >> 4)
            const uint64_t b0 = tc::sdesc(tc::smem_u32(wsm), 3 * COUT * 16, 128);
            int it = 0, n0 = 0; // n0: output levels of the blocks before
            for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
                const ConvBlock b = conv_block(di, p, TJ, u);
                for (int kk = b.lo; kk <= b.hi; kk++, it++) {
                    const int s = it % NS;
                    wait(&full[s], it / NS);
                    // output levels first touched here: their slots must be read out
                    for (int k = kk == b.lo ? b.k0 : kk + 1; k <= kk + 1 && k < b.k0 + b.nk; k++) {
                        const int n = n0 + k - b.k0;
                        if (n >= SLOTS) wait(&tempty[n % SLOTS], n / SLOTS - 1);
                    }
                    if (!ok) continue;
                    tc::fence_after();
                    const uint64_t a0 = tc::sdesc(tc::smem_u32(stg + s * C::STAGE), SG, 128);
                    for (int dk = 2; dk >= 0; dk--) { // tap dk - 1: output level k = kk - (dk - 1)
                        const int k = kk + 1 - dk;
                        if (k < b.k0 || k >= b.k0 + b.nk) continue;
                        const bool fresh = kk == max(k - 1, b.lo);
                        const uint32_t d0 = tmem + (uint32_t)((n0 + k - b.k0) % SLOTS * TJ * COUT);
                        // whole blocks with the line count known at compile time: the issuing thread
                        // then only adds constants to its descriptors
                        if (b.nj == TJ) issue_taps<CIN, COUT, TJ>(TJ, a0, b0, d0, dk, fresh);
                        else issue_taps<CIN, COUT, 0>(b.nj, a0, b0, d0, dk, fresh);
                    }
                    tc::mma_commit(&empty[s]);
                    if (kk - 1 >= b.k0) tc::mma_commit(&tfull[(n0 + kk - 1 - b.k0) % SLOTS]);
                    if (kk == b.hi && kk < b.k0 + b.nk) tc::mma_commit(&tfull[(n0 + kk - b.k0) % SLOTS]);
                }
                n0 += b.nk;
            }
        }
        __syncwarp();
    } else { // ---- epilogue: thread = cell of the x-tile ----
        float bias[COUT];
#pragma unroll
        for (int c = 0; c < COUT; c++) bias[c] = a.bias ? __ldg(a.bias + c) : 0.0f;
        int n = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
            const ConvBlock b = conv_block(di, p, TJ, u);
            const int i = b.tx * TILE + tid;
            const bool live = i < di.nx;
            const long long js = (long long)(dd.nz + 2) * C::GO * dd.PX; // from one line to the next in j
            for (int k = b.k0; k < b.k0 + b.nk; k++, n++) {
                const int slot = n % SLOTS;
                const long long base = act_unit(dd, i, k, b.j0, 0);
                // what the epilogue reads, fetched while the accumulators are still being summed
                uint4 ex[TJ][C::GO];
                conv_extra<COUT, TJ>(a, ex, base, js, b.nj, live);
                wait(&tfull[slot], n / SLOTS);
                tc::fence_after();
#pragma unroll
                for (int o = 0; o < TJ; o++) {
                    if (o >= b.nj) break;
                    uint32_t r[COUT / 16][16];
#pragma unroll
                    for (int q = 0; q < COUT / 16; q++)
                        tc::tmem_ld16_async(tmem + ((uint32_t)(warp * 32) << 16) +
                                                (uint32_t)((slot * TJ + o) * COUT + q * 16),
                                            r[q]);
                    float v[COUT];
#pragma unroll
                    for (int q = 0; q < COUT / 16; q++) {
                        tc::tmem_ld_wait(r[q]);
#pragma unroll
                        for (int e = 0; e < 16; e++) v[q * 16 + e] = __uint_as_float(r[q][e]);
                    }
                    if (o == b.nj - 1) { // the slot is read out
                        tc::fence_before();
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(&tempty[slot]);
                    }
                    if (live) conv_store<COUT>(a, v, bias, ex[o], base + o * js, i, k, b.j0 + o);
                }
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, C::NCOL);
}

// ---------------------------------------------------------------------------
// The same for 16 output channels with all nine taps (dj, dk) merged in N: the
// accumulators of an output line's three levels in the making lie side by side
// (column (3 o + slot) 16, slots rotating with the level), so one MMA of a line
// and x-shift feeds up to three output lines times three levels (N = 144): three
// MMAs per line and level instead of nine, for an operand read that costs as much
// each.  The rotation of the slots is in the weights (three images).  Every
// product accumulates; a slot is read out and zeroed before the next level's
// products, which the CTA next to it on the SM covers.  Levels outside the block
// that a block's first and last input levels also feed are zeroed without being
// stored.
// 16 -> 16 at 512x512x48 (B200), against the three-tap form above: 0.342 -> 0.183 ms (0.68 of measured HBM, 0.57 of
// measured BF16); 32 -> 16 at 256x256x48: 0.093 ms.
// ---------------------------------------------------------------------------
template <int CIN>
struct Fwd9Cfg {
    static constexpr int COUT = 16, GI = CIN / 8, GO = 2, TJ = 4, NL = TJ + 2;
    static constexpr int ROWS = 9 * COUT;                  // weight rows of one (rotation, x-shift, channel group)
    static constexpr int WB = 9 * GI * ROWS * 16;          // three images
    static constexpr int STAGE = NL * GI * SG;
    static constexpr int NCOL = 256, NS = 2;
    static constexpr int SMEM = up128(WB) + NS * STAGE + 256;
    static constexpr int PER_SM = SMEM <= 113 * 1024 ? 2 : 1;
    static_assert(SMEM <= 232448, "shared memory");
};

template <int CIN>
__global__ void __launch_bounds__(CONV_THREADS) conv3_fwd9_kernel(ConvArgs a, ConvSplit p)
{
    using C = Fwd9Cfg<CIN>;
    constexpr int NS = C::NS, TJ = C::TJ, COUT = C::COUT;
    if (conv_gated(a.gate)) return;
    extern __shared__ __align__(128) uint8_t sm[];
    uint8_t *wsm = sm, *stg = sm + up128(C::WB) + SGO;
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + up128(C::WB) + NS * C::STAGE + 128), *empty = full + NS,
             *summed = empty + NS, *drained = summed + 1;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(drained + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const ActDims di = a.din, dd = a.dout;
    if (tid == 0) {
        for (int q = 0; q < NS; q++) {
            tc::mbar_init(&full[q], 1);
            tc::mbar_init(&empty[q], 1);
        }
        tc::mbar_init(summed, 1);
        tc::mbar_init(drained, 4);
        tc::mbar_fence_init();
    }
    if (warp == 0) tc::tmem_alloc(tslot, C::NCOL);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;
    bool ok = true;
    auto wait = [&](uint64_t *bar, int use) { // the use-th completion (from 0); on time-out: no more waits
        if (ok && !tc::mbar_wait(bar, use & 1)) {
            if (lane == 0) atomicExch(a.err, 1);
            ok = false;
        }
    };

    if (warp == 4) { // ---- copies (as conv3_fwd_kernel) ----
        const char *inb = reinterpret_cast<const char *>(a.in);
        int it = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
            const ConvBlock b = conv_block(di, p, TJ, u);
            for (int kk = b.lo; kk <= b.hi; kk++, it++) {
                const int s = it % NS;
                if (it >= NS) wait(&empty[s], it / NS - 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const int n = (b.nj + 2) * C::GI;
                if (lane == 0) tc::mbar_expect_tx(&full[s], n * LG + (it == 0 ? C::WB : 0));
                __syncwarp();
                if (it == 0 && lane == 31) tc::bulk_g2s(wsm, a.w, C::WB, &full[s]);
                for (int q = lane; q < n; q += 32) {
                    const int l = q / C::GI, g = q % C::GI; // input line j0 - 1 + l, level kk
                    const long long L = (long long)(b.j0 + l) * (di.nz + 2) + (kk + 1);
                    tc::bulk_g2s(stg + s * C::STAGE + q * SG, inb + ((L * C::GI + g) * di.PX + (long long)b.tx * TILE) * 16,
                                 LG, &full[s]);
                }
            }
            if (!ok) break;
        }
        // nothing in flight at the end: the last stages landed and were read
        for (int q = it > NS ? it - NS : 0; q < it; q++) {
            if (!tc::mbar_wait(&full[q % NS], (q / NS) & 1) && lane == 0) atomicExch(a.err, 1);
            wait(&empty[q % NS], q / NS);
        }
    } else if (warp == 5) { // ---- MMAs, one thread ----
        if (lane == 0) {
            const uint64_t b0 = tc::sdesc(tc::smem_u32(wsm), C::ROWS * 16, 128);
            int it = 0; // input level; its rotation (the slot of output level kk - 1) is it % 3
            for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
                const ConvBlock b = conv_block(di, p, TJ, u);
                for (int kk = b.lo; kk <= b.hi; kk++, it++) {
                    const int s = it % NS;
                    wait(&full[s], it / NS);
                    wait(drained, it); // completion 0: all columns zeroed at the start
                    if (!ok) continue;
                    tc::fence_after();
                    const uint64_t a0 = tc::sdesc(tc::smem_u32(stg + s * C::STAGE), SG, 128);
                    const uint64_t br = b0 + (uint64_t)((it % 3 * 3 * C::GI * C::ROWS * 16) >> 4);
#pragma unroll
                    for (int dil = 0; dil < 3; dil++)
#pragma unroll
                        for (int c = 0; c < C::GI / 2; c++) {
                            const uint64_t bt = br + (uint64_t)(((dil * C::GI + 2 * c) * C::ROWS * 16) >> 4);
#pragma unroll
                            for (int l = 0; l < C::NL; l++) {
                                if (l >= b.nj + 2) break;
                                const int o0 = l - 2 > 0 ? l - 2 : 0, o1 = min(l, b.nj - 1);
                                const uint64_t ad = a0 + (uint64_t)(((l * C::GI + 2 * c) * SG + dil * 16) >> 4);
                                tc::mma_bf16(tmem + o0 * 3 * COUT, ad, bt + (uint64_t)((o0 - (l - 2)) * 3 * COUT),
                                             tc::idesc_bf16(128, 0, 0, 0) | ((uint32_t)((o1 - o0 + 1) * 3 * COUT / 8) << 17), 1u);
                            }
                        }
                    tc::mma_commit(&empty[s]);
                    tc::mma_commit(summed);
                }
            }
        }
        __syncwarp();
    } else { // ---- epilogue: thread = cell of the x-tile ----
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int q = 0; q < 3 * TJ; q++) tc::tmem_zero16(lanes + q * COUT);
        tc::tmem_st_wait();
        auto hand_back = [&]() {
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(drained);
        };
        hand_back();
        float bias[COUT];
#pragma unroll
        for (int c = 0; c < COUT; c++) bias[c] = a.bias ? __ldg(a.bias + c) : 0.0f;
        const long long js = (long long)(dd.nz + 2) * C::GO * dd.PX; // from one line to the next in j
        int it = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
            const ConvBlock b = conv_block(di, p, TJ, u);
            const int i = b.tx * TILE + tid;
            const bool live = i < di.nx;
            for (int kk = b.lo; kk <= b.hi; kk++, it++) {
                // output level kk - 1 is complete after input level kk, and after the last one also kk, if it is the grid's last
                const int last = kk == b.hi ? 3 : 1;
                uint4 ex[TJ][C::GO];
                conv_extra<COUT, TJ>(a, ex, act_unit(dd, i, kk - 1, b.j0, 0), js, b.nj, live && kk > b.k0);
                wait(summed, it);
                tc::fence_after();
                for (int t = 0; t < last; t++) {
                    const int k = kk - 1 + t, slot = (it + t) % 3;
                    const bool store = k >= b.k0 && k < b.k0 + b.nk;
                    uint32_t r[TJ][16];
#pragma unroll
                    for (int o = 0; o < TJ; o++) tc::tmem_ld16_async(lanes + (uint32_t)((3 * o + slot) * COUT), r[o]);
#pragma unroll
                    for (int o = 0; o < TJ; o++) tc::tmem_ld_wait(r[o]);
#pragma unroll
                    for (int o = 0; o < TJ; o++) tc::tmem_zero16(lanes + (uint32_t)((3 * o + slot) * COUT));
                    tc::tmem_st_wait();
                    if (t == last - 1) hand_back();
                    if (!store || !live) continue;
                    const long long base = act_unit(dd, i, k, b.j0, 0);
                    if (t > 0) conv_extra<COUT, TJ>(a, ex, base, js, b.nj, live);
#pragma unroll
                    for (int o = 0; o < TJ; o++) {
                        if (o >= b.nj) break;
                        float v[COUT];
#pragma unroll
                        for (int e = 0; e < 16; e++) v[e] = __uint_as_float(r[o][e]);
                        conv_store<COUT>(a, v, bias, ex[o], base + o * js, i, k, b.j0 + o);
                    }
                }
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, C::NCOL);
}

template <int CIN, int COUT>
struct WgCfg {
    static constexpr int GI = CIN / 8, GO = COUT / 8;
    static constexpr int TJ = CIN == 16 ? (COUT == 16 ? 3 : 2) : COUT == 16 ? 2 : 1; // dY lines of a tile (tensor memory)
    static constexpr int NL = TJ + 2;            // input lines in j
    static constexpr int NB = 3 * NL * GI;       // (level, line, channel group) blocks of one x-shift
    static constexpr int NMC = (NB + 15) / 16;   // M = 128 row chunks
    static constexpr int N = TJ * COUT;
    static constexpr int XR = NMC * 16 * LG;     // input lines + slack read by the last chunk
    static constexpr int YR = TJ * GO * YG;
    static constexpr int STAGE = XR + YR;
    static constexpr int NEED = 3 * NMC * N;
    static constexpr int NCOL = NEED <= 32 ? 32 : NEED <= 64 ? 64 : NEED <= 128 ? 128 : NEED <= 256 ? 256 : 512;
    static constexpr int SMEM = 2 * STAGE + 64;
    static_assert(NEED <= 512, "tensor memory columns");
    static_assert(SMEM <= 232448, "shared memory");
    static_assert(27 * CIN * COUT * 4 <= 2 * STAGE, "the CTA's sums fit where the stages were");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(128) conv3_wgrad_kernel(WgradArgs a)
{
    using C = WgCfg<CIN, COUT>;
    constexpr int TJ = C::TJ, NL = C::NL;
    extern __shared__ __align__(128) uint8_t sm[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + 2 * C::STAGE); // copies of stage 0, 1; MMAs of stage 0, 1
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + 4);
    const int tid = threadIdx.x, warp = tid >> 5;
    const ActDims dx = a.dx, dy = a.ddy;
    const int ntx = (dx.nx + TILE - 1) / TILE, njb = (dx.ny + TJ - 1) / TJ;
    const int ntiles = ntx * dx.nz * njb;
    if (tid == 0) {
        for (int q = 0; q < 4; q++) tc::mbar_init(&bars[q], 1);
        tc::mbar_fence_init();
    }
    if (warp == 0) tc::tmem_alloc(tslot, C::NCOL);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;
    const char *xb = reinterpret_cast<const char *>(a.x);
    const char *yb = reinterpret_cast<const char *>(a.dy);

    // called by all lanes of warp 0; lines past the last block's end: the zero halo lines
    auto issue = [&](int tile, int s) {
        const int tx = tile % ntx, r = tile / ntx, k = r % dx.nz, j0 = r / dx.nz * TJ;
        const int lane = tid & 31;
        uint8_t *dst = sm + s * C::STAGE;
        if (lane == 0) tc::mbar_expect_tx(&bars[s], C::NB * LG + C::YR);
        __syncwarp();
        for (int q = lane; q < C::NB + TJ * C::GO; q += 32) {
            if (q < C::NB) {
                const int g = q % C::GI, l = q / C::GI % NL, kl = q / (C::GI * NL);
                const long long L = (long long)min(j0 + l, dx.ny + 1) * (dx.nz + 2) + (k + kl);
                tc::bulk_g2s(dst + q * LG, xb + ((L * C::GI + g) * dx.PX + (long long)tx * TILE) * 16, LG, &bars[s]);
            } else {
                const int p = q - C::NB, g = p % C::GO, o = p / C::GO;
                const long long L = (long long)(min(j0 + o, dy.ny) + 1) * (dy.nz + 2) + (k + 1);
                tc::bulk_g2s(dst + C::XR + p * YG, yb + ((L * C::GO + g) * dy.PX + (long long)tx * TILE + 1) * 16, YG,
                             &bars[s]);
            }
        }
    };

    // dY lines of a tile: those past a short last block's end take no part, since zero
    // times an infinite input of the last line is not zero
    const int whole = ntx * dx.nz * (njb - 1), rest = dx.ny - (njb - 1) * TJ; // tiles of whole blocks, the last block's lines
    auto lines = [&](int tile) { return tile < whole ? TJ : rest; };
    float db[COUT];
#pragma unroll
    for (int c = 0; c < COUT; c++) db[c] = 0.0f;
    bool ok = true;
    int it = 0, tile = blockIdx.x;
    if (warp == 0 && tile < ntiles) issue(tile, 0);
    for (; tile < ntiles; tile += gridDim.x, it++) {
        const int s = it & 1;
        const bool got = tc::mbar_wait(&bars[s], (it >> 1) & 1);
        if (!__syncthreads_and(got)) { ok = false; break; }
        const uint8_t *st = sm + s * C::STAGE;
        if (tid == 0) {
            tc::fence_after();
            const uint64_t a0 = tc::sdesc(tc::smem_u32(st), 128, LG);
            const uint64_t b0 = tc::sdesc(tc::smem_u32(st) + C::XR, 128, YG);
            const uint32_t idesc = tc::idesc_bf16(128, 0, 1, 1) | ((uint32_t)(lines(tile) * COUT / 8) << 17);
#pragma unroll
            for (int dil = 0; dil < 3; dil++)
#pragma unroll
                for (int mc = 0; mc < C::NMC; mc++) {
                    const uint32_t d = tmem + (uint32_t)((dil * C::NMC + mc) * C::N);
#pragma unroll
                    for (int kc = 0; kc < TILE / 16; kc++) {
                        const uint64_t ad = a0 + (uint64_t)((mc * 16 * LG + dil * 16 + kc * 256) >> 4);
                        const uint64_t bd = b0 + (uint64_t)((kc * 256) >> 4);
                        tc::mma_bf16(d, ad, bd, idesc, (it > 0 || kc > 0) ? 1u : 0u);
                    }
                }
            tc::mma_commit(&bars[2 + s]);
        }
        // bias gradient: this thread's cell of the dy lines
#pragma unroll
        for (int p = 0; p < TJ * C::GO; p++) {
            float f[8];
            unpack8(*reinterpret_cast<const uint4 *>(st + C::XR + p * YG + tid * 16), f);
#pragma unroll
            for (int e = 0; e < 8; e++) db[p % C::GO * 8 + e] += f[e];
        }
        // the other stage's MMAs (the tile before) end while these run: the next tile's copies into it
        if (it > 0) {
            const bool done = tc::mbar_wait(&bars[2 + (s ^ 1)], ((it - 1) >> 1) & 1);
            if (!__syncthreads_and(done)) { ok = false; break; }
        }
        if (warp == 0 && tile + (int)gridDim.x < ntiles) issue(tile + gridDim.x, s ^ 1);
    }
    if (ok && it > 0) {
        const bool done = tc::mbar_wait(&bars[2 + ((it - 1) & 1)], ((it - 1) >> 1) & 1);
        ok = __syncthreads_and(done) != 0;
    }
    if (ok && it > 0) {
        tc::fence_after();
        // the products (input line l) x (dy line o) with l - o = dj + 1 belong to the tap dj: summed over o in
        // shared memory, one o at a time (each sum is then touched by one thread), then added to the gradient;
        // the tiles run up in j, so the CTA's first one has touched all lines that any has
        float *sum = reinterpret_cast<float *>(sm);
        const int used = lines(blockIdx.x);
#pragma unroll
        for (int o = 0; o < TJ; o++) {
            if (o >= used) break;
            for (int dil = 0; dil < 3; dil++)
                for (int mc = 0; mc < C::NMC; mc++)
#pragma unroll
                    for (int q = 0; q < COUT / 16; q++) {
                        float v[16];
                        tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) +
                                          (uint32_t)((dil * C::NMC + mc) * C::N + o * COUT + q * 16),
                                      v);
                        const int b = mc * 16 + tid / 8, g = b % C::GI, l = b / C::GI % NL, kl = b / (C::GI * NL);
                        if (b < C::NB && l >= o && l <= o + 2) {
                            const int t = (l - o) * 9 + kl * 3 + dil;
                            float4 *dst = reinterpret_cast<float4 *>(sum + (t * CIN + g * 8 + (tid & 7)) * COUT + q * 16);
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                float4 x = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
                                if (o > 0) {
                                    const float4 y = dst[e];
                                    x = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
                                }
                                dst[e] = x;
                            }
                        }
                    }
            __syncthreads();
        }
        // CTAs start at different places, so that they do not queue for the same addresses
        constexpr int Q = 27 * CIN * COUT / 4;
        const int q0 = (int)((long long)Q * blockIdx.x / gridDim.x);
        const bool vec = ((uintptr_t)a.dw & 15) == 0;
        for (int p = tid; p < Q; p += 128) {
            const int q = q0 + p < Q ? q0 + p : q0 + p - Q;
            const float4 x = reinterpret_cast<const float4 *>(sum)[q];
            if (vec) atomicAdd(reinterpret_cast<float4 *>(a.dw) + q, x);
            else {
                atomicAdd(a.dw + 4 * q, x.x);
                atomicAdd(a.dw + 4 * q + 1, x.y);
                atomicAdd(a.dw + 4 * q + 2, x.z);
                atomicAdd(a.dw + 4 * q + 3, x.w);
            }
        }
#pragma unroll
        for (int c = 0; c < COUT; c++) {
            float x = db[c];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if ((tid & 31) == 0) atomicAdd(a.db + c, x);
        }
    }
    if (!ok && tid == 0) {
        atomicExch(a.err, 1);
        // bounded waits for the copies and MMAs this CTA may still have in flight
        for (int q = 0; q < 4; q++) tc::mbar_wait(&bars[q], (uint32_t)((q & 1) == (it & 1) ? it >> 1 : (it - 1) >> 1) & 1, 100000000ull);
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, C::NCOL);
}

// ---------------------------------------------------------------------------
// Weight image of a conv cin -> cout, BF16.  cout = 32: per (dk, di) and group of 8
// input channels a column of 3 cout rows of 16 bytes, the taps dj = 1, 0, -1 below
// one another (the order of the output lines that they feed).  cout = 16: per
// rotation, di and group a column of 9 cout rows, the taps dj = 1, 0, -1 and below
// each the three slots, slot s of rotation q holding the tap dk that feeds it.
static bool merged9(int cout) { return cout == 16; }

__device__ __forceinline__ void wimage_put(__nv_bfloat16 *img, int t, int ci, int co, int cin, int cout, int nine, float w)
{
    const __nv_bfloat16 v = __float2bfloat16_rn(w);
    const int tj = t / 9, tk = t / 3 % 3, ti = t % 3, g = ci / 8, e = ci & 7, G = cin / 8;
    if (!nine) {
        img[(((tk * 3 + ti) * G + g) * 3 * cout + (2 - tj) * cout + co) * 8 + e] = v;
        return;
    }
    for (int q = 0; q < 3; q++) { // rotation q: slot q holds output level kk - 1 (tap dk = 1), the next ones kk and kk + 1
        const int slot = (q + 2 - tk) % 3;
        img[(((q * 3 + ti) * G + g) * 9 * cout + ((2 - tj) * 3 + slot) * cout + co) * 8 + e] = v;
    }
}

__global__ void conv_pack_fwd_kernel(const float *__restrict__ W, int cin, int cout, int nine, __nv_bfloat16 *__restrict__ img)
{
    const int n = 27 * cin * cout;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int t = q / (cin * cout), r = q % (cin * cout), ci = r / cout, co = r % cout;
        wimage_put(img, t, ci, co, cin, cout, nine, W[q]);
    }
}

// image of the conv cout -> cin whose output is the data gradient:
// W'[t'][ci' = co][co' = ci] = W[26 - t'][ci][co]
__global__ void conv_pack_bwd_kernel(const float *__restrict__ W, int cin, int cout, int nine, __nv_bfloat16 *__restrict__ img)
{
    const int n = 27 * cin * cout;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int t = q / (cin * cout), r = q % (cin * cout), ci = r / cout, co = r % cout;
        wimage_put(img, 26 - t, co, ci, cout, cin, nine, W[q]);
    }
}

// room for the image of either direction
size_t conv_wimage_bytes(int cin, int cout) { return (size_t)27 * cin * cout * 2 * 3; }

void conv_pack_fwd(const float *W, int cin, int cout, uint4 *img, cudaStream_t s)
{
    conv_pack_fwd_kernel<<<(27 * cin * cout + 255) / 256, 256, 0, s>>>(W, cin, cout, merged9(cout), (__nv_bfloat16 *)img);
    count_launch(1);
}

void conv_pack_bwd(const float *W, int cin, int cout, uint4 *img, cudaStream_t s)
{
    conv_pack_bwd_kernel<<<(27 * cin * cout + 255) / 256, 256, 0, s>>>(W, cin, cout, merged9(cin), (__nv_bfloat16 *)img);
    count_launch(1);
}

static int sm_count()
{
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

// Levels per block: as few rounds of `resident` blocks, each of KC levels and
// about three more in halo levels, fill and drain, as any split of nz gives.
static ConvSplit conv_split(const ActDims &d, int TJ, int resident)
{
    ConvSplit best{};
    long long cost = -1;
    const long long cols = (long long)((d.nx + TILE - 1) / TILE) * ((d.ny + TJ - 1) / TJ);
    for (int n = 1; n <= d.nz; n++) {
        const int KC = (d.nz + n - 1) / n, nkb = (d.nz + KC - 1) / KC;
        const long long units = cols * nkb, c = (units + resident - 1) / resident * (KC + 3);
        if (units > INT_MAX) break;
        if (cost < 0 || c < cost) {
            cost = c;
            best = ConvSplit{KC, nkb, (d.ny + TJ - 1) / TJ, (int)units};
        }
    }
    return best;
}

static bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

template <typename C>
static int launch_fwd(void (*kernel)(ConvArgs, ConvSplit), int ci, int co, const ConvArgs &a, cudaStream_t s)
{
    static const bool attr = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) == cudaSuccess;
    if (!attr) return -1;
    const ConvSplit p = conv_split(a.din, C::TJ, sm_count() * C::PER_SM);
    const int grid = std::min(p.units, sm_count() * C::PER_SM);
    if (grid <= 0) return 0;
    char name[32];
    snprintf(name, sizeof(name), "conv3_fwd_%dx%d", ci, co);
    const double cells = (double)a.din.nx * a.din.ny * a.din.nz;
    ProfScope ps_(name, cells * 2.0 * (ci + co), s);
    kernel<<<grid, CONV_THREADS, C::SMEM, s>>>(a, p);
    count_launch(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <int CI, int CO>
static int launch_wgrad(const WgradArgs &a, cudaStream_t s)
{
    using C = WgCfg<CI, CO>;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(conv3_wgrad_kernel<CI, CO>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) !=
            cudaSuccess)
            return -1;
        attr = true;
    }
    const long long ntiles = (long long)((a.dx.nx + TILE - 1) / TILE) * a.dx.nz * ((a.dx.ny + C::TJ - 1) / C::TJ);
    if (ntiles > INT_MAX) return -2;
    const int grid = (int)(ntiles < sm_count() ? ntiles : sm_count()); // 1 CTA per SM (TMEM / smem)
    if (grid <= 0) return 0;
    char name[32];
    snprintf(name, sizeof(name), "conv3_wgrad_%dx%d", CI, CO);
    const double cells = (double)a.dx.nx * a.dx.ny * a.dx.nz;
    ProfScope ps_(name, cells * 2.0 * (CI + CO), s);
    conv3_wgrad_kernel<CI, CO><<<grid, 128, C::SMEM, s>>>(a);
    count_launch(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

static bool dims_ok(const ActDims &a, int C)
{
    return a.nx > 0 && a.ny > 0 && a.nz > 0 && a.G * 8 == C && a.PX == act_pitch(a.nx);
}

int conv3_fwd(int cin, int cout, const ConvArgs &a, cudaStream_t s)
{
    if (!dims_ok(a.din, cin) || !dims_ok(a.dout, cout) || a.din.nx != a.dout.nx || a.din.ny != a.dout.ny ||
        a.din.nz != a.dout.nz || !a.in || !a.w || !a.err)
        return -2;
    if (!aligned16(a.in) || !aligned16(a.w) || !aligned16(a.out) || !aligned16(a.skip) || !aligned16(a.mask)) return -2;
    if (cin == 16 && cout == 16) return launch_fwd<Fwd9Cfg<16>>(conv3_fwd9_kernel<16>, 16, 16, a, s);
    if (cin == 16 && cout == 32) return launch_fwd<FwdCfg<16, 32>>(conv3_fwd_kernel<16, 32>, 16, 32, a, s);
    if (cin == 32 && cout == 32) return launch_fwd<FwdCfg<32, 32>>(conv3_fwd_kernel<32, 32>, 32, 32, a, s);
    if (cin == 32 && cout == 16) return launch_fwd<Fwd9Cfg<32>>(conv3_fwd9_kernel<32>, 32, 16, a, s);
    return -2;
}

int conv3_wgrad(int cin, int cout, const WgradArgs &a, cudaStream_t s)
{
    if (!dims_ok(a.dx, cin) || !dims_ok(a.ddy, cout) || a.dx.nx != a.ddy.nx || a.dx.ny != a.ddy.ny ||
        a.dx.nz != a.ddy.nz || !a.x || !a.dy || !a.dw || !a.db || !a.err)
        return -2;
    if (!aligned16(a.x) || !aligned16(a.dy)) return -2;
    if (cin == 16 && cout == 16) return launch_wgrad<16, 16>(a, s);
    if (cin == 16 && cout == 32) return launch_wgrad<16, 32>(a, s);
    if (cin == 32 && cout == 32) return launch_wgrad<32, 32>(a, s);
    if (cin == 32 && cout == 16) return launch_wgrad<32, 16>(a, s);
    return -2;
}

}  // namespace hw
