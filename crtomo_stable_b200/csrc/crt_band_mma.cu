// crt_band_mma.cu -- band factorisation of a few systems with the window in
// registers and its update on the FP64 tensor pipe (the interior systems of
// the Schur forward, one per wavenumber; prepared rows, in-place factor and
// progress as k_band_factor_blk's).
//
// With one CTA per system and no more systems than SMs, the time is one
// CTA's chain of panels.  k_band_factor_blk keeps the window in shared memory
// and updates it by 4 x 4 multiply-add tiles: for a half-bandwidth of 128 a
// panel of 8 columns moved 0.9 MB through shared memory (16,600 cycles a
// panel, four times the FP64 pipe's share), and for narrow bands the phases'
// instructions, issued by few warps at one in four cycles, made 1,340 cycles a
// column.  Measured, the factor alone (16 wavenumbers of a half-bandwidth of
// 128, 14 of 101, 12 of 40, 10 of 21; 12 real ones of 36): 31.7 -> 25.6, 19.6 ->
// 13.1, 2.69 -> 2.08, 0.81 -> 0.57; 3.35 -> 1.92 ms.  A panel at 128 is now
// 13,400 cycles, 4,350 of them the FP64 pipe's.
//
// Here the window's 8 x 8 tiles (slot blocks X >= Y; row r in slot r mod Wn)
// are the accumulators of m8n8k4 products and stay in the registers of their
// warp; only the panel passes through shared memory.  Per panel of 8 columns:
//   1. the rows below solve their 8 entries against the block factor, a
//      thread each;
//   2. the update warps first update the next panel's tiles and hand them to
//      shared memory; then warp 0 factors the next diagonal block (a lane per
//      row, every lane forming the pivot's root, so a column costs one shuffle
//      and the root's latency) while the update warps do the rest;
//      the panel's own tiles take the next 8 prepared rows, which one bulk
//      copy brought into a staging buffer a panel ahead.
//
// Every entry takes its updates in ascending columns, as fused multiply-adds
// in fms_acc's order, so the factor's bits are those of k_band_factor_blk.
// There the two products of an imaginary part are taken with the operand of
// the larger slot first, in a window of roundup(mb + P, P) rows for a panel of
// P columns; `Wv` and `H4` restate that order: a pair of rows (r, c), r > c,
// has r's entry first unless a multiple of Wv lies between them, and for P = 4
// the second four columns of a panel take the first four's as such pairs.
#include "crt_band.h"

#include <type_traits>

namespace {

constexpr int FP = 8;   // panel columns = rows of a slot block

template <typename T> struct FPad { static constexpr int v = 32 / (int)sizeof(T); };

template <typename T> __device__ __forceinline__ T shfl_t(T v, int src);
template <> __device__ __forceinline__ double shfl_t<double>(double v, int src)
{
    return __shfl_sync(0xffffffffu, v, src);
}
template <> __device__ __forceinline__ cd shfl_t<cd>(cd v, int src)
{
    return cd{__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
}

// Products by a reciprocal pivot in the forms k_band_factor_blk compiles to,
// within its diagonal block (`row` false) and in its rows below it.
__device__ __forceinline__ cd mul_inv(cd a, cd inv, bool row)
{
    const double p = __dmul_rn(a.x, inv.y), q = __dmul_rn(a.y, inv.x);
    return cd{fma(a.x, inv.x, -__dmul_rn(a.y, inv.y)), row ? fma(a.y, inv.x, p) : fma(a.x, inv.y, q)};
}
__device__ __forceinline__ double mul_inv(double a, double inv, bool) { return a * inv; }

// fms_acc(acc, a, b), or fms_acc(acc, b, a) when rev: the imaginary part's two
// products in the other order
__device__ __forceinline__ void fms_ord(cd& acc, cd a, cd b, bool rev)
{
    acc.x = fma(-a.x, b.x, acc.x);
    acc.x = fma(a.y, b.y, acc.x);
    acc.y = fma(-(rev ? a.y : a.x), rev ? b.x : b.y, acc.y);
    acc.y = fma(-(rev ? a.x : a.y), rev ? b.y : b.x, acc.y);
}
__device__ __forceinline__ void fms_ord(double& acc, double a, double b, bool) { fms_acc(acc, a, b); }

// Warp 0 for the diagonal blocks and NU update warps of MT tiles each (at least
// NB (NB + 1) / 2 in all; at 512 threads a thread has 128 registers).  H4: the
// order of P = 4 columns (Wv may be an odd multiple of 4); else of 8.
template <typename T, int NU, int MT, bool H4>
__global__ void __launch_bounds__(32 * (NU + 1), 1) k_band_factor_mma(BandArgs<T> A, int NB, int Wv)
{
    constexpr bool CPLX = std::is_same<T, cd>::value;
    constexpr int NT = 32 * (NU + 1), ST = FP + FPad<T>::v;
    using Tile = MmaTile<T>;
    constexpr int KC = Tile::KC;
    extern __shared__ __align__(16) unsigned char fm_dyn[];
    const int n = A.n, mb = A.mb, W = A.W, Wn = FP * NB;
    T* stage = reinterpret_cast<T*>(fm_dyn);   // [2][FP * W] prepared rows
    T* pan = stage + 2 * FP * W;               // [Wn][ST] the panel's L of every slot
    T* raw = pan + (size_t)Wn * ST;            // [Wn][ST] the next panel's entries before its solve
    __shared__ T LD[FP][2 * FP];               // the diagonal block, LD[t][j] = L(p0 + j, p0 + t)
    __shared__ T LDi[FP];                      // its reciprocal pivots
    __shared__ int bseg[64][2];                // a slot block's halves: rows / Wv
    __shared__ unsigned short txy[NU * MT];    // tile q = (warp - 1) + NU i of update warp `warp`: X | Y << 8
    __shared__ int s_err;
    __shared__ __align__(8) unsigned long long bar[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, sys = A.sys0 + b;
    T* Lc = A.Lws + (size_t)b * A.lstride;
    auto publish = [&](int c) {
        if (A.progress && tid == NT - 1) {
            __threadfence();
            asm volatile("st.release.gpu.global.s32 [%0], %1;\n" ::"l"(A.progress + b), "r"(c) : "memory");
        }
    };
    if (A.started && tid == 0) atomicAdd(A.started, 1);
    if (A.status[sys] != 0) {   // zero diagonal found by the preparation pass
        publish(n);
        return;
    }
    if (tid == 0) {
        s_err = 0;
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
    }
    if (H4 && tid < 2 * NB) bseg[tid >> 1][tid & 1] = 4 * tid / Wv;
    for (int q = tid; q < NU * MT; q += NT) {
        int X = 0;
        while ((X + 1) * (X + 2) / 2 <= q) ++X;
        txy[q] = X < NB ? X | (q - X * (X + 1) / 2) << 8 : 0xffff;
    }
    __syncthreads();

    // prepared rows [r0, r0 + FP) into stage[buf], by the last thread
    auto fetch = [&](int r0, int buf) {
        if (tid == NT - 1 && r0 < n) {
            const int bytes = min(FP, n - r0) * W * (int)sizeof(T);
            mbar_expect_tx(&bar[buf], bytes);
            bulk_g2s(stage + (size_t)buf * FP * W, Lc + (size_t)r0 * W, bytes, &bar[buf]);
        }
    };
    Tile acc[MT];
    constexpr unsigned short NONE = 0xffff;
    const unsigned short* mine = txy + max(warp - 1, 0);   // this warp's tiles
    const int lr = lane >> 2, lc = 2 * (lane & 3);   // the lane's row and first column in a tile
    // initial window: rows 0 .. Wn - 1
#pragma unroll
    for (int i = 0; i < MT; ++i)
        if (warp > 0 && mine[NU * i] != NONE) {
            const int r = FP * (mine[NU * i] & 0xff) + lr;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int d = r - (FP * (mine[NU * i] >> 8) + lc + q);
                acc[i].set(q, r < n && d >= 0 && d <= mb ? Lc[(size_t)r * W + d] : Sc<T>::zero());
            }
        }
    // a tile of the panel in block P as raw[slot][panel column]
    auto put_raw = [&](const Tile& t, int X, int Y, int P) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (Y == P) raw[(FP * X + lr) * ST + lc + q] = t.get(q);
            else raw[(FP * Y + lc + q) * ST + lr] = t.get(q);
        }
    };
#pragma unroll
    for (int i = 0; i < MT; ++i)
        if (warp > 0 && mine[NU * i] >> 8 == 0) put_raw(acc[i], mine[NU * i] & 0xff, 0, 0);
    fetch(Wn, 0);
    __syncthreads();

    // Diagonal block of the panel at p0 (slot block P): lane 4 j + g holds row j's
    // entries of columns g and g + 4 (a warp on its own issues an instruction
    // every four cycles or so: few instructions per lane).  Every lane forms
    // the pivot's root and reciprocal.
    auto diag_block = [&](int p0, int P) {
        const int npp = min(FP, n - p0), j = lane >> 2, g = lane & 3;
        const T* row = raw + (FP * P + j) * ST;
        T a0 = row[g], a1 = row[g + 4];   // entries above the diagonal are not used
        T piv = shfl_t(a0, 0);
#pragma unroll
        for (int t = 0; t < FP; ++t) {
            if (t >= npp) break;
            if (Sc<T>::bad_pivot(piv)) s_err = CRT_ERR_PIVOT;
            T root, inv;
            root_fx(piv, root, inv);
            const T l = j == t ? root : mul_inv(t < 4 ? a0 : a1, inv, H4 && (j >> 2) != (t >> 2));
            if (t + 1 < FP) {
                const T lr_ = shfl_t(l, (lane & ~3) | (t & 3));              // L(j, t)
                if (t < 3) fms_acc(a0, lr_, shfl_t(l, 4 * g + (t & 3)));
                fms_acc(a1, lr_, shfl_t(l, 4 * (g + 4) + (t & 3)));
                piv = shfl_t(t + 1 < 4 ? a0 : a1, 4 * (t + 1) + ((t + 1) & 3));
            }
            if (g == (t & 3) && j >= t && j < npp) {
                LD[t][j] = l;
                if (j - t <= mb) Lc[(size_t)(p0 + t) * W + (j - t)] = l;
            }
            if (lane == 0) LDi[t] = inv;
        }
    };
    if (warp == 0) diag_block(0, 0);
    __syncthreads();

    // tile (X, Y) minus the panel's product, P0 = the panel's block
    auto update = [&](Tile& t, int X, int Y, int P0) {
        const T* ap = pan + (FP * X + lr) * ST + Tile::kk();
        const T* bp = pan + (FP * Y + lr) * ST + Tile::kk();
        if constexpr (!CPLX) {
#pragma unroll
            for (int k = 0; k < FP; k += KC) t.mma(Tile::lda_neg(ap + k), Tile::ldb(bp + k));
        } else {
            const int part = lane & 1;
            const double *a = reinterpret_cast<const double*>(ap) + part, *b = reinterpret_cast<const double*>(bp) + part;
            const double *ya = a, *yb = b + 1 - 2 * part;   // the imaginary part's factors, X's entry first
            if (H4) {
                // whether rows of X come after rows of Y, and which halves of the
                // two blocks have a multiple of Wv between them
                const bool xlater = X == Y || (X >= P0) == (Y >= P0) ? X >= Y : X < P0;
                const int sx0 = bseg[X][0], sx1 = bseg[X][1], sy0 = bseg[Y][0], sy1 = bseg[Y][1];
                if (sx0 != sx1 || sy0 != sy1) {
                    // a multiple of Wv inside a block: its halves one by one (or, in
                    // both blocks, the four pairs), the other rows and columns zeroed
                    const bool hx = sx0 != sx1, hy = sy0 != sy1;
#pragma unroll 1
                    for (int h = 0; h < 4; ++h) {
                        if ((!hx && (h & 2)) || (!hy && (h & 1))) continue;
                        const bool first = xlater == ((h & 2 ? sx1 : sx0) == (h & 1 ? sy1 : sy0));
                        const double *ha = first ? a : a + 1 - 2 * part, *hb = first ? yb : b;
                        const bool inx = !hx || lane >> 4 == h >> 1, iny = !hy || lane >> 4 == (h & 1);
#pragma unroll
                        for (int k = 0; k < 2 * FP; k += 2 * KC) dmma(t.y0, t.y1, inx ? -ha[k] : 0.0, iny ? hb[k] : 0.0);
                    }
#pragma unroll
                    for (int k = 0; k < 2 * FP; k += 2 * KC) dmma(t.x0, t.x1, part ? a[k] : -a[k], b[k]);
                    return;
                }
                if (xlater != (sx0 == sy0)) {
                    ya = a + 1 - 2 * part;
                    yb = b;
                }
            }
#pragma unroll
            for (int k = 0; k < 2 * FP; k += 2 * KC) {
                const double v = a[k];
                dmma(t.x0, t.x1, part ? v : -v, b[k]);
                dmma(t.y0, t.y1, -(H4 ? ya[k] : v), yb[k]);
            }
        }
    };

    if (warp == 0) {
        // the diagonal blocks: each once its panel's entries are in raw
        for (int i0 = FP, P = 1; i0 < n && !s_err; i0 += FP, P = P + 1 == NB ? 0 : P + 1) {
            asm volatile("bar.sync 1, %0;\n" ::"n"(NT) : "memory");
            diag_block(i0, P);
            __syncthreads();
        }
    } else {
        int P = 0, p = 0;   // the panel's slot block, the panels taken
        for (int i0 = 0; !s_err; i0 += FP, ++p) {
            const int Q = P + 1 == NB ? 0 : P + 1, inext = i0 + FP;
            fetch(inext + Wn, (p + 1) & 1);
            // ---- 1. rows below the panel, four columns at a time
            for (int x = tid - 32; x < Wn; x += NT - 32) {
                const int xb = x >> 3;
                if (xb == P) continue;
                const int r = i0 + FP * (xb - P + (xb < P ? NB : 0)) + (x & 7);
                T* px = pan + x * ST;
                if (r < n && r - i0 < mb + FP) {
                    const T* rx = raw + x * ST;
                    // P = 4 columns of the order: the second half's rows against r
                    const bool rev = CPLX && H4 && bseg[xb][(x >> 2) & 1] != bseg[P][1];
#pragma unroll
                    for (int h = 0; h < FP; h += 4) {
                        T s[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t) s[t] = rx[h + t];
#pragma unroll
                        for (int u = 0; u < h; ++u) {
                            const T lu = px[u];
#pragma unroll
                            for (int t = 0; t < 4; ++t) fms_ord(s[t], lu, LD[u][4 + t], rev);
                        }
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            s[t] = mul_inv(s[t], LDi[h + t], true);
#pragma unroll
                            for (int t2 = t + 1; t2 < 4; ++t2) fms_acc(s[t2], s[t], LD[h + t][h + t2]);
                            px[h + t] = s[t];
                            const int d = r - (i0 + h + t);
                            if (d <= mb) Lc[(size_t)(i0 + h + t) * W + d] = s[t];
                        }
                    }
                } else {
#pragma unroll
                    for (int t = 0; t < FP; ++t) px[t] = Sc<T>::zero();
                }
            }
            asm volatile("bar.sync 2, %0;\n" ::"n"(NT - 32) : "memory");
            // columns [0, i0 + FP) are final (the diagonal blocks were written a panel ago)
            if ((p & 7) == 7) publish(min(n, inext));
            if (inext >= n) break;
            // ---- 2. the next panel's tiles, then the rest of the window
            const T* sg = stage + (size_t)(p & 1) * FP * W;
            const int rn = i0 + Wn;   // the first of the rows that take the panel's slots
            // (this panel's updates read the other blocks' entries of bseg only)
            if (H4 && tid - 32 < 2) bseg[P][tid - 32] = (rn + 4 * (tid - 32)) / Wv;
            if (rn < n && !mbar_wait(&bar[p & 1], (p >> 1) & 1)) s_err = CRT_ERR_CUDA;
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    const int X = mine[NU * i] & 0xff, Y = mine[NU * i] >> 8;
                    if (X == 0xff || (X == Q || Y == Q) != (pass == 0)) continue;
                    if (X != P && Y != P) {
                        update(acc[i], X, Y, P);
                    } else {
                        // new rows a = lr (X == P) or lc + q against the other block's rows
                        const int o = X == P ? Y : X, off = o == P ? 0 : Wn - FP * (o - P + (o < P ? NB : 0));
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int a = X == P ? lr : lc + q, d = off + (X == P ? lr - lc - q : lc + q - lr);
                            acc[i].set(q, d >= 0 && d <= mb && rn + a < n ? sg[a * W + d] : Sc<T>::zero());
                        }
                        // the staging buffer's next writer is the async (bulk copy) proxy
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    }
                    if (pass == 0) put_raw(acc[i], X, Y, Q);
                }
                if (pass == 0) asm volatile("bar.arrive 1, %0;\n" ::"n"(NT) : "memory");
            }
            P = Q;
            __syncthreads();
        }
        // Copy c (rows Wn + 8 c on) is awaited by panel c, a panel after its
        // start: when a pivot ends the loop with p panels taken, copy p is in
        // flight (and p - 1, if its wait gave up).  The CTA's shared memory
        // must not be left to it.
        if (tid == NT - 1 && s_err)
            for (int c = max(0, p - 1); c <= p; ++c)
                if (Wn + FP * c < n) mbar_wait(&bar[c & 1], (c >> 1) & 1);
    }
    __syncthreads();
    if (tid == 0 && s_err) A.status[sys] = s_err;
    publish(n);
}

int mma_blocks(int mb) { return (mb + FP + FP - 1) / FP; }

template <typename T>
size_t mma_smem(int mb, int W)
{
    return ((size_t)2 * FP * W + 2 * (size_t)FP * mma_blocks(mb) * (FP + FPad<T>::v)) * sizeof(T);
}

}  // namespace

template <typename T>
bool band_mma_fits(int mb) { return mb >= 1 && mma_blocks(mb) <= 17; }

template <typename T>
void launch_band_factor_mma(const BandArgs<T>& a, cudaStream_t st)
{
    const int NB = mma_blocks(a.mb);
    // the order of products of k_band_factor_blk with the panel its tuner picks
    // for few complex systems of this band (4: up to 14 % faster there up to 76
    // and, 512 threads against 512, from 89 to 100)
    const int pv = std::is_same<T, cd>::value && (a.mb <= 76 || (a.mb >= 89 && a.mb <= 100)) ? 4 : 8;
    const int Wv = (a.mb + 2 * pv - 1) / pv * pv;
    const size_t smem = mma_smem<T>(a.mb, a.W);
    auto go = [&](auto kern, int nu) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<a.nsys, 32 * (nu + 1), smem, st>>>(a, NB, Wv);
    };
    constexpr bool H4 = std::is_same<T, cd>::value;
    // a tile per update warp while the tiles fit, then as few as 15 warps allow
    // (half-bandwidth 21: 0.57 ms with a tile per warp, 0.66 with four on three)
    if (NB <= 4) go(k_band_factor_mma<T, 10, 1, H4>, 10);
    else if (NB <= 5) go(k_band_factor_mma<T, 15, 1, H4>, 15);
    else if (NB <= 7) go(k_band_factor_mma<T, 15, 2, H4>, 15);
    else if (NB <= 9) go(k_band_factor_mma<T, 15, 3, H4>, 15);
    else if (NB <= 10) go(k_band_factor_mma<T, 15, 4, H4>, 15);
    else if (pv == 8 && NB <= 12) go(k_band_factor_mma<T, 15, 6, false>, 15);
    else if (pv == 8 && NB <= 14) go(k_band_factor_mma<T, 15, 7, false>, 15);
    else if (pv == 8) go(k_band_factor_mma<T, 15, 11, false>, 15);
    else go(k_band_factor_mma<T, 15, 7, true>, 15);
}

template bool band_mma_fits<cd>(int);
template bool band_mma_fits<double>(int);
template void launch_band_factor_mma<cd>(const BandArgs<cd>&, cudaStream_t);
template void launch_band_factor_mma<double>(const BandArgs<double>&, cudaStream_t);
