// crt_schur.cu -- forward model by elimination of the mixed-boundary nodes
// (see crt_schur.h for the algebra).  Kernels, in the order they run:
//
//   k_schur_rhs_src / k_schur_rhs_cpl  the columns F r_I (one per source
//       electrode) and F A_IG (one per boundary node) of the interior
//       solves, and the coupling values a(g, i) kept for later steps;
//   k_schur_transpose  the interior factor reversed and row-packed, so the
//       back substitution runs as a forward sweep;
//   k_schur_sweep   banded triangular sweep of 16 columns per CTA (forward for
//       all columns, each block from its first non-zero row; back for the
//       source columns), the triangle of a block beside the update by the
//       block before on the FP64 tensor pipe;
//   k_schur_gram    C = V^T [u^ | V^] per wavenumber (tiled GEMM on the FP64
//       tensor pipe that skips the rows where a column is still zero);
//   k_schur_ll      per (k, l): S_l = A_GG(l) - V^T V^, left-looking blocked
//       Cholesky (unconjugated, complex symmetric as src/chol.f90:44-78), the
//       forward solve fused into the factorisation, the back solve by panels
//       (k_schur_chol, right-looking, for the larger boundaries: ll_staged);
//   k_schur_zrebuild  z^ = u^ - V^ p_G (tiled GEMM);
//   k_schur_out_gam p_G into kpot at the boundary nodes.
#include "crt_schur.h"

#include <cstdlib>
#include <cstring>

#include <algorithm>
#include <cstdio>
#include <numeric>
#include <type_traits>
#include <utility>

// ---------------------------------------------------------------------------
// Host plan.
int schur_plan_host(const AssemblyLists& full, int n, const std::vector<int>& gamma_nodes,
                    const std::vector<int>& enr0, int lsink, int nsink0, SchurHost& o)
{
    o = SchurHost{};
    o.n = n;
    o.L = (int)enr0.size();
    std::vector<int> posI(n, -1), posG(n, -1);
    std::vector<char> isg(n, 0);
    for (int v : gamma_nodes)
        if (v >= 0 && v < n) isg[v] = 1;
    for (int v = 0; v < n; ++v) {
        if (isg[v]) {
            posG[v] = (int)o.gam.size();
            o.gam.push_back(v);
        } else {
            posI[v] = (int)o.permI.size();
            o.permI.push_back(v);
        }
    }
    o.nI = (int)o.permI.size();
    o.m = (int)o.gam.size();
    if (o.nI == 0 || o.m == 0 || o.m > SCHUR_MMAX) return CRT_ERR_ARG;
    AssemblyLists& li = o.lists_I;
    li.row_ptr.assign(1, 0);
    li.ent_ptr.assign(1, 0);
    std::vector<std::vector<std::pair<int, int>>> cpl(o.m);   // per g: (interior position, gather entry)
    for (int r = 0; r < n; ++r) {
        const int pr = posI[r];
        for (int e = full.row_ptr[r]; e < full.row_ptr[r + 1]; ++e) {
            const int c = r - full.ent_d[e];
            if (pr >= 0 && posI[c] >= 0) {
                li.ent_d.push_back(pr - posI[c]);
                for (int q = full.ent_ptr[e]; q < full.ent_ptr[e + 1]; ++q) {
                    // a mixed-boundary segment couples boundary nodes only
                    if (full.con_code[q] < 0) return CRT_ERR_ARG;
                    li.con_code.push_back(full.con_code[q]);
                    li.con_sig.push_back(full.con_sig[q]);
                }
                li.ent_ptr.push_back((int)li.con_code.size());
                o.mbI = std::max(o.mbI, pr - posI[c]);
            } else if (pr >= 0) {
                cpl[posG[c]].push_back({pr, e});
            } else if (posI[c] >= 0) {
                cpl[posG[r]].push_back({posI[c], e});
            } else {
                o.gg_g.push_back(posG[r]);   // r >= c, so g >= h
                o.gg_h.push_back(posG[c]);
                o.gg_ent.push_back(e);
            }
        }
        if (pr >= 0) {
            li.row_ptr.push_back((int)li.ent_d.size());
            li.max_row_entries = std::max(li.max_row_entries, li.row_ptr.back() - li.row_ptr[li.row_ptr.size() - 2]);
        }
    }
    // rows of D_l: the G-G entries with a mixed-boundary contribution, both
    // triangles, by row
    {
        std::vector<std::vector<std::pair<int, int>>> bd(o.m);
        for (size_t q = 0; q < o.gg_ent.size(); ++q) {
            const int e = o.gg_ent[q];
            bool mixed = false;
            for (int c = full.ent_ptr[e]; c < full.ent_ptr[e + 1]; ++c) mixed |= full.con_code[c] < 0;
            if (!mixed) continue;
            bd[o.gg_g[q]].push_back({o.gg_h[q], e});
            if (o.gg_g[q] != o.gg_h[q]) bd[o.gg_h[q]].push_back({o.gg_g[q], e});
        }
        o.bd_ptr.assign(1, 0);
        for (int g = 0; g < o.m; ++g) {
            std::sort(bd[g].begin(), bd[g].end());
            for (auto& he : bd[g]) {
                o.bd_col.push_back(he.first);
                o.bd_ent.push_back(he.second);
            }
            o.bd_ptr.push_back((int)o.bd_col.size());
        }
    }
    o.gi_ptr.assign(1, 0);
    std::vector<int> first(o.L + o.m, o.nI);
    for (int g = 0; g < o.m; ++g) {
        std::sort(cpl[g].begin(), cpl[g].end());
        for (auto& pe : cpl[g]) {
            o.gi_pos.push_back(pe.first);
            o.gi_ent.push_back(pe.second);
            o.gi_g.push_back(g);
            first[o.L + g] = std::min(first[o.L + g], pe.first);
        }
        o.gi_ptr.push_back((int)o.gi_pos.size());
    }
    o.posI_src.resize(o.L);
    o.posG_src.resize(o.L);
    o.posI_sink = lsink ? posI[nsink0] : -1;
    o.posG_sink = lsink ? posG[nsink0] : -1;
    for (int l = 0; l < o.L; ++l) {
        o.posI_src[l] = posI[enr0[l]];
        o.posG_src[l] = posG[enr0[l]];
        if (o.posI_src[l] >= 0) first[l] = std::min(first[l], o.posI_src[l]);
        if (o.posI_sink >= 0) first[l] = std::min(first[l], o.posI_sink);
    }
    o.first = first;
    o.gsort.resize(o.m);
    std::iota(o.gsort.begin(), o.gsort.end(), 0);
    std::stable_sort(o.gsort.begin(), o.gsort.end(), [&](int a, int b) { return first[o.L + a] < first[o.L + b]; });
    o.gfirst.resize(o.m);
    for (int q = 0; q < o.m; ++q) o.gfirst[q] = first[o.L + o.gsort[q]];
    // columns by their first non-zero row, so that a block's forward pass
    // starts where its earliest column does
    const int ncol = o.L + o.m;
    o.col_order.resize(ncol);
    std::iota(o.col_order.begin(), o.col_order.end(), 0);
    std::stable_sort(o.col_order.begin(), o.col_order.end(), [&](int a, int b) { return first[a] < first[b]; });
    for (int b0 = 0; b0 < ncol; b0 += SCHUR_MS_R) {
        const int f = first[o.col_order[b0]];
        o.blk_start.push_back(f >= o.nI ? o.nI : f / SCHUR_MS_BB * SCHUR_MS_BB);
    }
    return CRT_OK;
}

namespace {

template <typename T> __device__ __forceinline__ T shfl_w(T v, int src, int width);
template <> __device__ __forceinline__ double shfl_w<double>(double v, int src, int width)
{
    return __shfl_sync(0xffffffffu, v, src, width);
}
template <> __device__ __forceinline__ cd shfl_w<cd>(cd v, int src, int width)
{
    return cd{__shfl_sync(0xffffffffu, v.x, src, width), __shfl_sync(0xffffffffu, v.y, src, width)};
}
// acc += a b (complex: four fused multiply-adds)
__device__ __forceinline__ void fma_acc(cd& acc, cd a, cd b)
{
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(a.y, b.x, acc.y);
}
__device__ __forceinline__ void fma_acc(double& acc, double a, double b) { acc = fma(a, b, acc); }

template <typename T> __device__ __forceinline__ T shfl_xor_t(T v, int mask);
template <> __device__ __forceinline__ double shfl_xor_t<double>(double v, int mask)
{
    return __shfl_xor_sync(0xffffffffu, v, mask);
}
template <> __device__ __forceinline__ cd shfl_xor_t<cd>(cd v, int mask)
{
    return cd{__shfl_xor_sync(0xffffffffu, v.x, mask), __shfl_xor_sync(0xffffffffu, v.y, mask)};
}

// one element global -> shared, asynchronously (cp.async; both addresses
// aligned to the element)
template <typename T> __device__ __forceinline__ void cp_async_elem(T* dst, const T* src);
template <> __device__ __forceinline__ void cp_async_elem<cd>(cd* dst, const cd* src) { cp_async16(dst, src); }
template <> __device__ __forceinline__ void cp_async_elem<double>(double* dst, const double* src)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src) : "memory");
}

// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_schur_rhs_src(SchurArgs s, const double* __restrict__ fakws, T* X)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= s.K * s.L) return;
    const int k = idx / s.L, l = idx % s.L;
    T* col = X + ((size_t)k * s.ncol + l) * s.nI;
    const double* fk = fakws + (size_t)k * s.nI;
    // r = e_src - e_sink (A pot = r; the reference's b = -r, src/kompab.f90),
    // scaled by fak
    if (s.posI_src[l] >= 0) col[s.posI_src[l]] = scale(Sc<T>::one(), fk[s.posI_src[l]]);
    if (s.lsink && s.posI_sink >= 0) col[s.posI_sink] -= scale(Sc<T>::one(), fk[s.posI_sink]);
}

template <typename T>
__global__ void k_schur_rhs_cpl(SchurArgs s, BandArgs<T> A, const double* __restrict__ fakws, T* X, T* cval)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)s.K * s.ncpl) return;
    const int k = (int)(idx / s.ncpl), q = (int)(idx % s.ncpl);
    // an interior-boundary entry has area contributions only (l unused)
    const T a = band_assemble_entry<T>(A, s.gi_ent[q], k, 0);
    cval[idx] = a;
    const int i = s.gi_pos[q];
    X[((size_t)k * s.ncol + s.L + s.gi_g[q]) * s.nI + i] = scale(a, fakws[(size_t)k * s.nI + i]);
}

// Lrev[k][c'][d] = L(r, r - d), r = n - 1 - c' (0 where r - d < 0).
template <typename T>
__global__ void k_schur_transpose(SchurArgs s, const T* __restrict__ Lws, T* Lrev)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int n = s.nI, W = s.WI;
    const long long per = (long long)n * W;
    if (idx >= (long long)s.nk * per) return;
    const int k = s.k0 + (int)(idx / per), cp = (int)((idx % per) / W), d = (int)(idx % W);
    const int r = n - 1 - cp, c = r - d;
    const T* Lk = Lws + (size_t)k * per;
    Lrev[(size_t)k * per + idx % per] = (c >= 0 && d <= s.mbI) ? Lk[(size_t)c * W + d] : Sc<T>::zero();
}

// ---------------------------------------------------------------------------
// Banded lower-triangular sweep L z = b for SW_R columns per CTA: grid (K,
// column blocks).  The factor's columns stream through shared memory SW_BB at
// a time (one bulk copy each, NB buffers, bounded mbarrier wait), the
// right-hand sides live in a window Z of WZ rows (row r at slot r mod WZ, WZ
// >= mb + 3 SW_BB), their rows arriving by cp.async: block b starts the copies
// of rows c0 + 16 + mb .. c0 + 31 + mb.  Phase A of block b + 1 touches rows
// below c0 + 16 + mb only where mb >= 16, so there they may still be in flight
// when it begins; in narrower bands its triangle (rows c0 + 16 .. c0 + 31)
// reaches them, and block b waits for its own copies (schur_sweep_in_flight).
// Per block b (rows c0 .. c0 + 15), between barriers:
//   A. warps 0 and 1 solve the block's triangle for eight columns each (a lane
//      per column, 8 x 8 triangles in registers, the product between them on
//      the tensor pipe) while the other warps take block b - 1's columns into
//      the rows past block b;
//   B. four warps take block b's columns into block b + 1's rows, a tile each,
//      another starts the next factor copy, the rest write block b's rows out.
// The updates are m8n8k4 FP64 tensor products.  Every row takes its columns
// in ascending order by fused multiply-adds in fms_acc's order.  Bound by the
// block's chain: 4,900 cycles at a half-bandwidth of 128 (phase A 3,800, its
// products alone 2,050 on the FP64 pipe; B 700), 2,900 at 21.  As 4 x 2
// multiply-add tiles per thread and a half-warp per triangle column it was
// 11,800 (back sweep of 128 sources, 492 electrodes: 11.2 -> 4.7 ms; 101 at
// a half-bandwidth of 21: 0.38 -> 0.13).
//   back == 0: forward sweep of X's columns (col_order, from each block's
//     first non-zero row), in place;
//   back == 1: the back sweep L^T x^ = z^ of the source columns: Lws holds
//     the reversed row-packed factor and the rows are read reversed; the
//     solution goes out as kpot = fak x^ at the interior rows' nodes.
constexpr int SW_R = SCHUR_MS_R, SW_BB = SCHUR_MS_BB;

// Rows of the window are padded so that the eight rows of a tile differ in banks.
template <typename T> struct SweepRow { static constexpr int v = SW_R + (sizeof(T) == 16 ? 1 : 4); };

// Operands of the sweep's products: the factor's entry negated once for both
// chains of a complex product, the sign between them with the solution's.
template <typename T> struct SweepTile;
template <> struct SweepTile<cd> : MmaTile<cd> {
    __device__ __forceinline__ static double lda_neg(const cd* a)
    {
        return -reinterpret_cast<const double*>(a)[threadIdx.x & 1];
    }
    __device__ __forceinline__ static B ldb(const cd* b)
    {
        const double* p = reinterpret_cast<const double*>(b);
        const double v = p[threadIdx.x & 1];
        return B{(threadIdx.x & 1) ? -v : v, p[(threadIdx.x & 1) ^ 1]};
    }
    __device__ __forceinline__ void mma(double a, const B& b)
    {
        dmma(x0, x1, a, b.n);
        dmma(y0, y1, a, b.s);
    }
};
template <> struct SweepTile<double> : MmaTile<double> {};

template <typename T, int NT, int NB, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_schur_sweep(SchurArgs s, const T* __restrict__ Lws, const double* __restrict__ fakws, T* X, cd* kpot, int n_kpot,
                  int WZ, int in_flight, int back)
{
    constexpr int R = SW_R, BB = SW_BB, RS = SweepRow<T>::v;
    constexpr int NU = NT / 32 - 2;                              // update warps
    constexpr int FW = 4, OT = NT - 32 * (FW + 1), NE = (BB * R + OT - 1) / OT;   // phase B: the fetching warp; threads and entries of the rows out
    static_assert(NU >= 4 && OT >= 32, "warps of phase B: four tiles, one to fetch, the others the rows out");
    using Tile = SweepTile<T>;
    constexpr int KC = Tile::KC;
    extern __shared__ __align__(16) unsigned char sw_dyn[];
    const int W = s.WI, n = s.nI, mb = s.mbI;
    T* Lb = reinterpret_cast<T*>(sw_dyn);   // [NB][BB * W]
    T* Z = Lb + NB * BB * W;                // [WZ][RS]
    __shared__ T dinv[2][BB];
    __shared__ int colid[R];
    __shared__ __align__(8) unsigned long long bar[NB];
    __shared__ int s_err;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // wavenumbers along x: the CTAs start in the order of their blocks'
    // first rows, longest passes first over all wavenumbers
    const int blk = blockIdx.y, k = s.k0 + blockIdx.x;
    const int start = back ? 0 : s.blk_start[blk];
    if (start >= n) return;   // every column of the block is zero, and so is its solution
    const T* Lk = Lws + (size_t)k * n * W;
    if (tid < R) {
        const int c = blk * R + tid;
        colid[tid] = back ? (c < s.L ? c : -1) : (c < s.ncol ? s.col_order[c] : -1);
    }
    if (tid == 0) {
        s_err = 0;
        for (int q = 0; q < NB; ++q) mbar_init(&bar[q], 1);
    }
    __syncthreads();
    auto fetch = [&](int c0, int buf) {   // by one thread
        if (s.progress && !s_err) {
            // the factor's columns [c0, c0 + BB) are final once its
            // progress passes them.  The wait gives up after about 4 s,
            // or at once when another CTA of this wavenumber gave up
            // (status set); the result is then flagged as failed, and an
            // error that the factor recorded stays.
            const int want = min(n, c0 + BB);
            long polls = 0;
            int got;
            while (true) {
                asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(got) : "l"(s.progress + k) : "memory");
                if (got >= want) break;
                if (*(volatile const int*)(s.status + k) != 0 || ++polls > (1L << 22)) {
                    s_err = 1;
                    atomicCAS(&s.status[k], 0, (int)CRT_ERR_CUDA);
                    break;
                }
                __nanosleep(256);
            }
            // the copy below reads them through the async proxy
            asm volatile("fence.proxy.async.global;\n" ::: "memory");
        }
        const int bytes = min(BB, n - c0) * W * (int)sizeof(T);
        mbar_expect_tx(&bar[buf], bytes);
        bulk_g2s(Lb + (size_t)buf * BB * W, Lk + (size_t)c0 * W, bytes, &bar[buf]);
    };
    // the reciprocals of a block's diagonal, by one warp once its copy has landed
    auto pivots = [&](int buf, int phase, T* di) {
        if (!mbar_wait(&bar[buf], phase)) s_err = 1;
        if (lane < BB) di[lane] = recip_fx(Lb[(size_t)(buf * BB + lane) * W]);
    };
    auto colp = [&](int j) { return X + ((size_t)k * s.ncol + colid[j]) * n; };   // the column's rows in X
    auto copy_row = [&](int j, int r, T* dst) {
        if (colid[j] >= 0) cp_async_elem<T>(dst, colp(j) + (back ? n - 1 - r : r));
        else *dst = Sc<T>::zero();
    };
    const int lr = lane >> 2, lg = lane & 3;
    // NR tiles of 8 rows (slots sr and, `step` slots on, sr2) x NC tiles of 8
    // columns from column j0 minus a factor block Lq whose solution rows begin
    // at slot sb; the tiles' rows are d0, d0 + step below the block's first
    // row, and those from dhi on are left as they are
    auto update = [&](auto nr_, auto nc_, const T* Lq, int sb, const int* sr, int d0, int step, int dhi, int j0) {
        constexpr int NR = decltype(nr_)::value, NC = decltype(nc_)::value;
        Tile acc[NR][NC];
        T* zp[NR];
        const T* ap[NR];
        const int kk = Tile::kk();
#pragma unroll
        for (int a = 0; a < NR; ++a) {
            zp[a] = Z + (size_t)(sr[a] + lr) * RS + j0 + 2 * lg;
            ap[a] = Lq + kk * (W - 1) + d0 + a * step + lr;   // column u is u (W - 1) on
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int q = 0; q < 2; ++q) acc[a][c].set(q, zp[a][8 * c + q]);
        }
        const T* bp = Z + (size_t)(sb + kk) * RS + j0 + lr;
        static_assert(BB % KC == 0, "whole products");
        auto products = [&](auto edge_) {
            constexpr bool edge = decltype(edge_)::value;   // some entries lie outside the band
#pragma unroll
            for (int u = 0; u < BB; u += KC) {
                typename Tile::B b[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) b[c] = Tile::ldb(bp + u * RS + 8 * c);
#pragma unroll
                for (int a = 0; a < NR; ++a) {
                    double av;
                    if (edge) {
                        const int over = max(0, d0 + a * step + lr - kk - u - mb);   // rows past the band: read its last entry
                        av = Tile::lda_neg(ap[a] + u * (W - 1) - over);
                        if (over) av = 0.0;
                    } else {
                        av = Tile::lda_neg(ap[a] + u * (W - 1));
                    }
#pragma unroll
                    for (int c = 0; c < NC; ++c) acc[a][c].mma(av, b[c]);
                }
            }
        };
        if (d0 + (NR - 1) * step + 7 <= mb) products(std::false_type{});
        else products(std::true_type{});
#pragma unroll
        for (int a = 0; a < NR; ++a)
            if (d0 + a * step + lr < dhi)
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int q = 0; q < 2; ++q) zp[a][8 * c + q] = acc[a][c].get(q);
    };
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    // eight rows (slots from zh) of a block's triangle whose first column is
    // Lh, for eight columns of the window: a lane per column, the other
    // lanes repeat them
    auto triangle = [&](auto wide_, const T* Lh, const T* dh, T* zh) {
        constexpr bool wide = decltype(wide_)::value;   // mb >= 7: every entry is stored
        auto l = [&](int t, int u) { return wide || t - u <= mb ? Lh[u * W + (t - u)] : Sc<T>::zero(); };
        T* zc = zh + (lane & 7);
        T z[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) z[t] = zc[(size_t)t * RS];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            z[u] = mul_fx(dh[u], z[u]);
#pragma unroll
            for (int t = u + 1; t < 8; ++t) fms_acc(z[t], l(t, u), z[u]);
        }
        if (lane < 8)
#pragma unroll
            for (int t = 0; t < 8; ++t) zc[(size_t)t * RS] = z[t];
        __syncwarp();
    };
    for (int r = start + tid / R; r < min(n, start + BB + mb); r += NT / R) copy_row(tid % R, r, Z + (size_t)(r % WZ) * RS + tid % R);
    cp_async_commit();
    if (warp == FW) {
        if (lane == 0) {
            fetch(start, 0);
            if (NB == 3 && start + BB < n) fetch(start + BB, 1);
        }
        __syncwarp();
        pivots(0, 0, dinv[0]);
    }
    cp_async_wait_group<0>();
    __syncthreads();
    int bi = 0, phs = 0, sc = start % WZ;   // sc: slot of the block's first row (WZ is a multiple of BB)
    auto slot = [&](int d) { return sc + d < WZ ? sc + d : sc + d - WZ; };   // slot of row c0 + d, 0 <= d < WZ
    for (int c0 = start; c0 < n; c0 += BB, ++bi) {
        const int cur = bi % NB, prv = (bi + NB - 1) % NB, nxt = (bi + 1) % NB, sp = sc ? sc - BB : WZ - BB;
        if (!mbar_wait(&bar[cur], phs >> cur & 1)) s_err = 1;
        phs ^= 1 << cur;
        const T* Lc = Lb + (size_t)cur * BB * W;
        const T* Lp = Lb + (size_t)prv * BB * W;
        T* zb = Z + (size_t)sc * RS;
        int node[NE];
        double fk[NE];
        if (warp < 2) {
            // A. the triangle: rows 0-7, their products into rows 8-15, rows 8-15
            T* zh = zb + 8 * warp;
            auto tri = [&](const T* Lh, const T* dh, T* z) {
                if (mb >= 7) triangle(std::true_type{}, Lh, dh, z);
                else triangle(std::false_type{}, Lh, dh, z);
            };
            const T* di = dinv[bi & 1];
            tri(Lc, di, zh);
            {
                Tile acc;
                T* z8 = zh + (8 + lr) * RS + 2 * lg;
                acc.set(0, z8[0]);
                acc.set(1, z8[1]);
                const int d0 = 8 + lr - Tile::kk();
                const T* bp = zh + Tile::kk() * RS + lr;
                const T* ap = Lc + Tile::kk() * W + d0;
#pragma unroll
                for (int u = 0; u < 8; u += KC)
                    {
                    const int over = max(0, d0 - u - mb);
                    const double av = Tile::lda_neg(ap + u * (W - 1) - over);
                    acc.mma(over ? 0.0 : av, Tile::ldb(bp + u * RS));
                }
                z8[0] = acc.get(0);
                z8[1] = acc.get(1);
            }
            __syncwarp();
            tri(Lc + 8 * W, di + 8, zh + 8 * RS);
        } else {
            // A. the rows that block b + 1 needs start; block b - 1 into the
            // rows [c0 + BB, c0 + mb); the next block's pivots
#pragma unroll
            for (int e = tid - 64; e < BB * R; e += 32 * NU) {
                const int t = e % BB, r = c0 + BB + mb + t;
                if (r < n) copy_row(e / BB, r, Z + (size_t)slot(BB + mb + t) * RS + e / BB);
            }
            cp_async_commit();
            if (back && warp > FW)   // for phase B
#pragma unroll
                for (int q = 0; q < NE; ++q) {
                    const int i = n - 1 - (c0 + (tid - 32 * (FW + 1) + q * OT) % BB);
                    if (i >= 0) {
                        node[q] = s.permI[i];
                        fk[q] = fakws[(size_t)k * n + i];
                    }
                }
            if (c0 > start) {
                const int dhi = min(n - c0, mb);   // rows below c0
                int d = BB + 8 * (warp - 2);
                for (; d + 8 * NU < dhi; d += 16 * NU) {
                    const int sr[2] = {slot(d), slot(d + 8 * NU)};
                    update(I2{}, I2{}, Lp, sp, sr, d + BB, 8 * NU, dhi + BB, 0);
                }
                if (d < dhi) {
                    const int sr[1] = {slot(d)};
                    update(I1{}, I2{}, Lp, sp, sr, d + BB, 0, dhi + BB, 0);
                }
            }
            if (NB == 3 && warp == NT / 32 - 1 && c0 + BB < n) pivots(nxt, phs >> nxt & 1, dinv[bi + 1 & 1]);
            if (in_flight) cp_async_wait_group<1>();
            else cp_async_wait_group<0>();
        }
        // block b-1's buffer is the destination of a copy below
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (warp < 4) {
            // B. block b into block b+1's rows
            const int d = BB + 8 * (warp >> 1), sr[1] = {slot(d)};
            if (c0 + d < n) update(I1{}, I1{}, Lc, sc, sr, d, 0, min(n - c0, BB + mb), 8 * (warp & 1));
        } else if (warp == FW) {
            if (lane == 0 && c0 + (NB - 1) * BB < n) fetch(c0 + (NB - 1) * BB, prv);
            __syncwarp();
            if (NB == 2 && c0 + BB < n) pivots(nxt, phs >> nxt & 1, dinv[bi + 1 & 1]);
        } else {
            // B. block b's rows out
#pragma unroll
            for (int q = 0; q < NE; ++q) {
                const int e = tid - 32 * (FW + 1) + q * OT, t = e % BB, j = e / BB;
                if (j < R && c0 + t < n && colid[j] >= 0) {
                    const T v = zb[(size_t)t * RS + j];
                    if (!back) colp(j)[c0 + t] = v;
                    else kpot[((size_t)k * s.L + colid[j]) * n_kpot + node[q]] = Sc<T>::to_cd(scale(v, fk[q]));
                }
            }
        }
        __syncthreads();
        sc = sc + BB < WZ ? sc + BB : 0;
    }
    cp_async_wait_group<0>();
    if (tid == 0 && s_err) atomicCAS(&s.status[k], 0, (int)CRT_ERR_CUDA);
}

// ---------------------------------------------------------------------------
// C[k][c][g] = sum_i V^[i][g] X[i][c] over the rows where both columns can
// be non-zero, on the FP64 tensor pipe: tiles TG (g) x TC (c), warps of
// (8 WG) x (8 WC), the rows staged GRAM_TI at a time, NS - 1 stages ahead.
// Bound by the pipe and by the operands from L2 (1 KB per 4,096 multiply-adds
// of a 32 x 32 tile); with the multiply-adds on the FP64 cores, 4 x 4 per
// thread, their shared-memory operands bound it (60k triangles 14.3 -> 9.2 ms,
// 20k cells 7.2 -> 4.0 ms, 12,960 cells real 0.72 -> 0.35 ms).
// Every entry is summed over ascending rows.  The tiles of the V^T V^ block
// above its diagonal are skipped (the Cholesky reads the lower triangle).
// A row run of a column is padded by 32 bytes, so the four rows x 32 bytes
// that a half-warp reads at once lie in different banks.
constexpr int GRAM_TI = 16;
template <typename T> struct RunPad { static constexpr int v = 32 / (int)sizeof(T); };

template <typename T, int TG, int TC, int WG, int WC, int NS>
__global__ void __launch_bounds__(TG / (8 * WG) * (TC / (8 * WC)) * 32)
    k_schur_gram(SchurArgs s, const T* __restrict__ X, T* C)
{
    constexpr int TI = GRAM_TI, ST = TI + RunPad<T>::v, NW = TC / (8 * WC), NT = TG / (8 * WG) * NW * 32;
    using Tile = MmaTile<T>;
    constexpr int KC = Tile::KC;
    extern __shared__ __align__(16) unsigned char gram_dyn[];   // NS stages of both operands
    T* buf0 = reinterpret_cast<T*>(gram_dyn);                   // [NS][TG + TC][ST]
    __shared__ int s_i0;
    // wavenumbers along x, so the long tiles (early first rows) of every
    // wavenumber start first
    const int tid = threadIdx.x, k = s.k0 + blockIdx.x;
    const int g0 = blockIdx.y * TG, c0 = blockIdx.z * TC;
    const int m = s.m, L = s.L, nI = s.nI, ncol = s.ncol;
    if (c0 >= L && c0 - L > g0 + TG - 1) return;
    if (tid < 32) {
        int fg = nI, fc = nI;
        for (int q = tid; q < TG && g0 + q < m; q += 32) fg = min(fg, s.first[L + g0 + q]);
        for (int q = tid; q < TC && c0 + q < ncol; q += 32) fc = min(fc, s.first[c0 + q]);
        const int f = max(__reduce_min_sync(0xffffffffu, fg), __reduce_min_sync(0xffffffffu, fc));
        if (tid == 0) s_i0 = f / TI * TI;
    }
    __syncthreads();
    const int i0 = s_i0, nt = (nI - i0 + TI - 1) / TI;
    const int lane = tid & 31, warp = tid >> 5, wg = warp / NW * 8 * WG, wc = warp % NW * 8 * WC;
    Tile acc[WG][WC];
    const T* Xk = X + (size_t)k * ncol * nI;
    // rows [i0 + t TI, + TI) of the tile's columns into stage t % NS
    auto stage = [&](int t) {
        T* dst = buf0 + (size_t)(t % NS) * (TG + TC) * ST;
        const int r0 = i0 + t * TI;
        for (int idx = tid; idx < TI * (TG + TC); idx += NT) {
            const int q = idx / TI, ii = idx % TI;
            const int c = q < TG ? (g0 + q < m ? L + g0 + q : -1) : (c0 + q - TG < ncol ? c0 + q - TG : -1);
            T* d = dst + q * ST + ii;
            if (c >= 0 && r0 + ii < nI) cp_async_elem<T>(d, Xk + (size_t)c * nI + r0 + ii);
            else *d = Sc<T>::zero();
        }
    };
    for (int t = 0; t < NS - 1; ++t) {
        if (t < nt) stage(t);
        cp_async_commit();
    }
    for (int t = 0; t < nt; ++t) {
        cp_async_wait_group<NS - 2>();
        __syncthreads();   // stage t has landed; the last readers of stage t - 1 are through
        if (t + NS - 1 < nt) stage(t + NS - 1);
        cp_async_commit();
        const T* As = buf0 + (size_t)(t % NS) * (TG + TC) * ST;
        const T* ap = As + (wg + (lane >> 2)) * ST + Tile::kk();
        const T* bp = As + (TG + wc + (lane >> 2)) * ST + Tile::kk();
#pragma unroll
        for (int ii = 0; ii < TI; ii += KC) {
            typename Tile::A a[WG];
            typename Tile::B b[WC];
#pragma unroll
            for (int x = 0; x < WG; ++x) a[x] = Tile::lda(ap + x * 8 * ST + ii);
#pragma unroll
            for (int y = 0; y < WC; ++y) b[y] = Tile::ldb(bp + y * 8 * ST + ii);
#pragma unroll
            for (int x = 0; x < WG; ++x)
#pragma unroll
                for (int y = 0; y < WC; ++y) acc[x][y].mma(a[x], b[y]);
        }
    }
    cp_async_wait_group<0>();
#pragma unroll
    for (int y = 0; y < WC; ++y)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int cc = c0 + wc + 8 * y + 2 * (lane & 3) + q;
            if (cc >= ncol) continue;
#pragma unroll
            for (int x = 0; x < WG; ++x) {
                const int g = g0 + wg + 8 * x + (lane >> 2);
                if (g < m) C[((size_t)k * ncol + cc) * m + g] = acc[x][y].get(q);
            }
        }
}

// ---------------------------------------------------------------------------
// Dense Cholesky of the Schur complements, one CTA per (k, l) system:
// S = A_GG(l) - C_VV (lower triangle, column-major, in the workspace),
// right-looking with an NB-column panel in shared memory; the forward solve
// L y = r_G - C[l] rides along each column, the back solve L^T x = y goes
// panel by panel from the last (dot products of the panel columns, then the
// panel's triangle on one warp).
//
// PF: the next super-tile's entries are loaded into registers while the
// current one is updated (one CTA per SM); without, two CTAs share an SM and
// hide each other's latency.
// REF: the reference factors of the iterative form instead, one per
// (wavenumber, electrode group) b: S0 + the group's mean mixed-boundary part
// (S0 from C), factored in place without a right-hand side; a non-positive
// pivot is counted in *nonconv.
template <typename T, int NT, int NB, bool PF, bool REF = false>
__global__ void __launch_bounds__(NT, PF ? 1 : 2) k_schur_chol(SchurArgs s, BandArgs<T> A, const T* __restrict__ C,
                                                               T* Sws, T* xg, int sys0, int* nonconv = nullptr)
{
    static_assert(NT == 256 && NB <= 16, "chol layout");
    extern __shared__ __align__(16) unsigned char ch_dyn[];
    const int m = s.m;
    T* P = reinterpret_cast<T*>(ch_dyn);   // panel [NB][m]: P[t m + r] = L(r, p0 + t)
    T* y = P + (size_t)NB * m;             // [m]
    __shared__ int s_err;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, sys = sys0 + b;
    const int k = REF ? b / s.ngrp : sys / s.L, l = REF ? (b % s.ngrp) * s.grp : sys % s.L;
    T* S = Sws + (size_t)b * m * m;
    const T* Ck = C + (size_t)k * s.ncol * m;
    if (tid == 0) s_err = 0;
    if constexpr (REF) {
        const T* S0k = C;   // REF: C is S0 ([k][m][m], both triangles)
        for (int c = 0; c < m; ++c)
            for (int r = c + tid; r < m; r += NT) S[(size_t)c * m + r] = S0k[((size_t)k * m + c) * m + r];
        for (int g = tid; g < m; g += NT) y[g] = Sc<T>::zero();
        __syncthreads();
        const int nl = min(s.grp, s.L - l);
        for (int g = tid; g < m; g += NT)
            for (int q = s.bd_ptr[g]; q < s.bd_ptr[g + 1]; ++q) {
                const int h = s.bd_col[q];
                if (h <= g) S[(size_t)h * m + g] += band_assemble_part<T>(A, s.bd_ent[q], k, l, nl, 1);
            }
    } else {
        for (int c = 0; c < m; ++c) {
            const T* src = Ck + (size_t)(s.L + c) * m;
            for (int r = c + tid; r < m; r += NT) S[(size_t)c * m + r] = -src[r];
        }
        for (int g = tid; g < m; g += NT) {
            T v = -Ck[(size_t)l * m + g];
            if (g == s.posG_src[l]) v += Sc<T>::one();
            if (s.lsink && g == s.posG_sink) v -= Sc<T>::one();
            y[g] = v;
        }
        __syncthreads();
        for (int q = tid; q < s.ngg; q += NT) {
            const T a = band_assemble_entry<T>(A, s.gg_ent[q], k, l);
            S[(size_t)s.gg_h[q] * m + s.gg_g[q]] += a;
        }
    }
    __syncthreads();
    for (int p0 = 0; p0 < m; p0 += NB) {
        const int nb = min(NB, m - p0);
        for (int t = 0; t < nb; ++t)
            for (int r = p0 + tid; r < m; r += NT) P[t * m + r] = S[(size_t)(p0 + t) * m + r];
        __syncthreads();
        for (int t = 0; t < nb; ++t) {
            const int c = p0 + t;
            const T piv = P[t * m + c];
            if (Sc<T>::bad_pivot(piv)) s_err = CRT_ERR_PIVOT;
            T root, inv;
            Sc<T>::sqrt_recip(piv, root, inv);
            const T yc = Sc<T>::mul(y[c], inv);
            __syncthreads();   // every thread has read the pivot and y[c]
            for (int r = c + 1 + tid; r < m; r += NT) {
                const T lv = Sc<T>::mul(P[t * m + r], inv);
                P[t * m + r] = lv;
                fms_acc(y[r], lv, yc);
            }
            if (tid == 0) {
                P[t * m + c] = root;
                y[c] = yc;
            }
            __syncthreads();
            const int rows = m - c - 1;
            for (int idx = tid; idx < (nb - t - 1) * rows; idx += NT) {
                const int tt = t + 1 + idx / rows, r = c + 1 + idx % rows;
                if (r >= p0 + tt) fms_acc(P[tt * m + r], P[t * m + r], P[t * m + p0 + tt]);
            }
            __syncthreads();
        }
        if (s_err) break;
        for (int t = 0; t < nb; ++t)
            for (int r = p0 + t + tid; r < m; r += NT) S[(size_t)(p0 + t) * m + r] = P[t * m + r];
        // trailing update of the lower triangle below the panel by 64 x 64
        // super-tiles (their lower triangle on the diagonal): thread (ti, tj)
        // owns rows ti + 16 a and columns tj + 16 c of each, so a warp's
        // loads of S are two 256-byte runs and its panel reads consecutive
        // words; the next super-tile's entries load while the current one
        // is updated
        const int q0 = p0 + nb, mt = m - q0;
        if (mt > 0) {
            const int NS = (mt + 63) / 64, nst = NS * (NS + 1) / 2;
            const int ti = tid & 15, tj = tid >> 4;
            auto st_origin = [&](int st, int& R0, int& C0) {
                int SX = (int)((sqrtf(8.0f * st + 1.0f) - 1.0f) * 0.5f);
                while ((SX + 1) * (SX + 2) / 2 <= st) ++SX;
                while (SX * (SX + 1) / 2 > st) --SX;
                R0 = q0 + 64 * SX;
                C0 = q0 + 64 * (st - SX * (SX + 1) / 2);
            };
            auto st_load = [&](int st, T (&v)[4][4]) {
                int R0, C0;
                st_origin(st, R0, C0);
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int r = R0 + ti + 16 * a, cc = C0 + tj + 16 * c;
                        v[a][c] = (r < m && cc < m && r >= cc) ? S[(size_t)cc * m + r] : Sc<T>::zero();
                    }
            };
            T cur[4][4], nxt[4][4];
            st_load(0, cur);
            for (int st = 0; st < nst; ++st) {
                if (PF && st + 1 < nst) st_load(st + 1, nxt);
                int R0, C0;
                st_origin(st, R0, C0);
                for (int t = 0; t < nb; ++t) {
                    T pr[4], pc[4];
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        const int r = R0 + ti + 16 * a, cc = C0 + tj + 16 * a;
                        pr[a] = r < m ? P[t * m + r] : Sc<T>::zero();
                        pc[a] = cc < m ? P[t * m + cc] : Sc<T>::zero();
                    }
#pragma unroll
                    for (int a = 0; a < 4; ++a)
#pragma unroll
                        for (int c = 0; c < 4; ++c) fms_acc(cur[a][c], pr[a], pc[c]);
                }
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int r = R0 + ti + 16 * a, cc = C0 + tj + 16 * c;
                        if (r < m && cc < m && r >= cc) S[(size_t)cc * m + r] = cur[a][c];
                        if (PF) cur[a][c] = nxt[a][c];
                    }
                if (!PF && st + 1 < nst) st_load(st + 1, cur);
            }
        }
        __syncthreads();
    }
    if constexpr (REF) {
        if (s_err && tid == 0) atomicAdd(nonconv, 1);
        return;
    }
    if (s_err) {
        if (tid == 0) atomicMax(&s.status[sys], s_err);
        return;
    }
    // L^T x = y, panel by panel from the last
    for (int p0 = (m - 1) / NB * NB; p0 >= 0; p0 -= NB) {
        const int nb = min(NB, m - p0);
        for (int t = 0; t < nb; ++t)
            for (int r = p0 + tid; r < m; r += NT) P[t * m + r] = S[(size_t)(p0 + t) * m + r];
        __syncthreads();
        {   // y[p0 + t] -= sum over solved rows r >= p0 + nb of L(r, p0 + t) x_r
            const int t = tid >> 4, sl = tid & 15;
            T part = Sc<T>::zero();
            if (t < nb)
                for (int r = p0 + nb + sl; r < m; r += 16) fma_acc(part, P[t * m + r], y[r]);
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) part += shfl_xor_t(part, off);
            if (sl == 0 && t < nb) y[p0 + t] -= part;
        }
        __syncthreads();
        if (warp == 0) {   // the panel's triangle of L^T, lane t = row p0 + t
            T v = lane < nb ? y[p0 + lane] : Sc<T>::zero();
            for (int u = nb - 1; u >= 0; --u) {
                if (lane == u) v = Sc<T>::mul(v, Sc<T>::recip(P[u * m + p0 + u]));
                const T x = shfl_w(v, u, 32);
                if (lane < u) fms_acc(v, P[lane * m + p0 + u], x);
            }
            if (lane < nb) y[p0 + lane] = v;
        }
        __syncthreads();
    }
    for (int g = tid; g < m; g += NT) xg[(size_t)sys * m + g] = y[g];
}

// ---------------------------------------------------------------------------
// The same factorisation left-looking, on the FP64 tensor pipe, a CTA per
// system: per block column of 8, every 8 x 8 tile below the diagonal is
// summed over the finished columns in registers (a warp per row block, m8n8k4
// products in ascending columns), the diagonal block is factored by one warp
// and the rows below are solved by a thread each; nothing is written twice.
// The right-looking form's three barriers and shared-memory passes per column
// and its trailing update through L2 took 4,900 cycles a column (m = 101,
// complex).  Measured, all systems: 400 of m = 101 complex 0.50 -> 0.33 ms, 576
// of 181 complex 1.43 -> 1.02, 1,152 of 253 real 3.23 -> 1.88; the reference
// factors of 128 groups of 492: 3.4 -> 3.0.  The factor lies in shared memory where two CTAs share an SM
// (SM), packed by block columns, else column-major in the workspace, its
// finished block columns staged one ahead by cp.async.  Entries take their
// updates in the same order and form as there, and the back solve keeps its
// panels of NBP columns and their partial sums: the same bits.
constexpr int LL_NT = 256;
// entries of the packed factor: block columns of 8 padded runs (a product's k
// columns x four rows in different banks)
__host__ __device__ inline size_t ll_packed(int m)
{
    const size_t nbk = (m + 7) / 8;
    return 8 * (nbk * (8 * nbk + 4) - 4 * nbk * (nbk - 1));
}
template <typename T> size_t ll_smem(int m, bool sm)
{
    const size_t m8 = (m + 7) / 8 * 8;
    return (m8 * (8 + RunPad<T>::v) + m8 + (sm ? ll_packed(m) : 2 * 8 * (m8 + 4))) * sizeof(T);
}

template <typename T, bool SM, bool REF, int NT, int U>
__global__ void __launch_bounds__(NT, 512 / NT) k_schur_ll(SchurArgs s, BandArgs<T> A, const T* __restrict__ C, T* Sws,
                                                           T* xg, int sys0, int NBP, int* nonconv)
{
    constexpr int ST = 8 + RunPad<T>::v, NW = NT / 32;
    using Tile = MmaTile<T>;
    constexpr int KC = Tile::KC;
    extern __shared__ __align__(16) unsigned char ll_dyn[];
    const int m = s.m, nbk = (m + 7) / 8, m8 = 8 * nbk;
    T* pan = reinterpret_cast<T*>(ll_dyn);   // [m8][ST] the block column before its solve
    T* y = pan + (size_t)m8 * ST;            // [m8]
    T* pack = y + m8;                        // the packed factor, or the two stages [8][m8 + 4]
    __shared__ T LD[8][8], LDi[8], zb[8];    // LD[t][j] = L(c0 + j, c0 + t)
    __shared__ int s_err;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, sys = sys0 + b;
    const int k = REF ? b / s.ngrp : sys / s.L, l = REF ? (b % s.ngrp) * s.grp : sys % s.L;
    T* S = Sws + (size_t)b * m * m;
    const T* Ck = C + (size_t)k * s.ncol * m;
    // block column J: entry (r, 8 J + t) at blk(J)[t ld(J) + r] (r >= 8 J)
    auto ld = [&](int J) { return SM ? m8 - 8 * J + 4 : m; };
    auto blk = [&](int J) -> T* {
        // packed: block columns 0 .. J-1 take the sum of 8 (m8 - 8 j + 4)
        return SM ? pack + 8 * (J * (m8 + 4) - 4 * J * (J - 1)) - 8 * J : S + (size_t)8 * J * m;
    };
    auto at = [&](int r, int c) -> T& { return blk(c >> 3)[(c & 7) * ld(c >> 3) + r]; };
    if (tid == 0) s_err = 0;
    // eight columns of loads in flight per thread
    for (int J = 0; J < nbk; ++J) {
        T* cp = blk(J);
        const int lj = ld(J), nc = min(8, m - 8 * J);
        const T* src = REF ? C + ((size_t)k * m + 8 * J) * m : Ck + (size_t)(s.L + 8 * J) * m;
        for (int r = 8 * J + tid; r < m; r += NT) {
            T v[8];
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (t < nc && r >= 8 * J + t) v[t] = src[(size_t)t * m + r];
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (t < nc && r >= 8 * J + t) cp[t * lj + r] = REF ? v[t] : -v[t];   // REF: C is S0
        }
    }
    for (int g = tid; g < m8; g += NT) {
        T v = Sc<T>::zero();
        if (!REF && g < m) {
            v = -Ck[(size_t)l * m + g];
            if (g == s.posG_src[l]) v += Sc<T>::one();
            if (s.lsink && g == s.posG_sink) v -= Sc<T>::one();
        }
        y[g] = v;
    }
    __syncthreads();
    if constexpr (REF) {
        const int nl = min(s.grp, s.L - l);
        for (int g = tid; g < m; g += NT)
            for (int q = s.bd_ptr[g]; q < s.bd_ptr[g + 1]; ++q) {
                const int h = s.bd_col[q];
                if (h <= g) at(g, h) += band_assemble_part<T>(A, s.bd_ent[q], k, l, nl, 1);
            }
    } else {
        for (int q = tid; q < s.ngg; q += NT) at(s.gg_g[q], s.gg_h[q]) += band_assemble_entry<T>(A, s.gg_ent[q], k, l);
    }
    __syncthreads();
    const int lr = lane >> 2, lc = 2 * (lane & 3);
    for (int J = 0; J < nbk; ++J) {
        const int c0 = 8 * J, npp = min(8, m - c0), lj = ld(J);
        T* cb = blk(J);
        // block column K's rows from c0 on into stage K % 2
        const int sl = m8 - c0 + 4;
        auto stage = [&](int K) {
            if (SM || K >= J) return;
            const T* src = S + (size_t)8 * K * m;
            T* dst = pack + (K & 1) * 8 * (m8 + 4) - c0;
            for (int t = warp; t < 8; t += NW)
                for (int r = c0 + lane; r < m; r += 32) cp_async_elem<T>(dst + t * sl + r, src + (size_t)t * m + r);
        };
        // tiles (I, J) minus the finished columns, U row blocks of a warp at a time
        for (int I0 = J; I0 < nbk; I0 += U * NW) {
            Tile acc[U];
            int row[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int r = 8 * (I0 + warp + u * NW) + lr;
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    acc[u].set(q, r < m && c0 + lc + q <= r ? cb[(lc + q) * lj + r] : Sc<T>::zero());
                row[u] = min(r, m - 1);   // rows past the end repeat the last one
            }
            const int rj = min(c0 + lr, m - 1), nu = min(U, (nbk - I0 - warp + NW - 1) / NW);
            stage(0);
            cp_async_commit();
            for (int K = 0; K < J; ++K) {
                const T* kc = SM ? blk(K) : pack + (K & 1) * 8 * (m8 + 4) - c0;
                const int kl = SM ? ld(K) : sl;
                if (!SM) {
                    cp_async_wait_group<0>();
                    __syncthreads();   // stage K has landed, stage K - 1's readers are through
                    stage(K + 1);
                    cp_async_commit();
                }
                kc += Tile::kk() * kl;
#pragma unroll
                for (int t = 0; t < 8; t += KC) {
                    const typename Tile::B bf = Tile::ldb(kc + t * kl + rj);
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (u < nu) acc[u].mma(Tile::lda_neg(kc + t * kl + row[u]), bf);
                }
            }
            if (!SM) __syncthreads();   // the stages may be filled again
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (u < nu)
#pragma unroll
                    for (int q = 0; q < 2; ++q) pan[(8 * (I0 + warp + u * NW) + lr) * ST + lc + q] = acc[u].get(q);
        }
        __syncthreads();
        if (warp == 0) {
            // the diagonal block: lane 4 j + g holds row j's entries of columns
            // g and g + 4, and y of its row
            const int j = lane >> 2, g = lane & 3;
            T a0 = pan[(c0 + j) * ST + g], a1 = pan[(c0 + j) * ST + g + 4], yj = y[c0 + j];
            T piv = shfl_w(a0, 0, 32);
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                if (t >= npp) break;
                if (Sc<T>::bad_pivot(piv)) s_err = CRT_ERR_PIVOT;
                T root, inv;
                root_fx(piv, root, inv);
                const T lt = j == t ? root : mul_fx(t < 4 ? a0 : a1, inv);
                const T yc = mul_fx(yj, inv);
                const T z = shfl_w(yc, 4 * t, 32);
                const T lrow = shfl_w(lt, (lane & ~3) | (t & 3), 32);   // L(j, t)
                if (j > t) fms_acc(yj, lrow, z);
                if (t + 1 < 8) {
                    if (t < 3) fms_acc(a0, lrow, shfl_w(lt, 4 * g + (t & 3), 32));
                    fms_acc(a1, lrow, shfl_w(lt, 4 * (g + 4) + (t & 3), 32));
                    piv = shfl_w(t + 1 < 4 ? a0 : a1, 4 * (t + 1) + ((t + 1) & 3), 32);
                }
                if (g == (t & 3) && j >= t && j < npp) {
                    LD[t][j] = lt;
                    cb[t * lj + c0 + j] = lt;
                }
                if (lane == 0) {
                    LDi[t] = inv;
                    zb[t] = z;
                    y[c0 + t] = z;
                }
            }
        }
        __syncthreads();
        if (s_err) break;
        // the rows below (a full block: there are rows only then)
        for (int r = c0 + 8 + tid; r < m; r += NT) {
            const T* px = pan + r * ST;
            T v[8], yr = REF ? Sc<T>::zero() : y[r];
#pragma unroll
            for (int t = 0; t < 8; ++t) v[t] = px[t];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                v[t] = mul_fx(v[t], LDi[t]);
#pragma unroll
                for (int t2 = t + 1; t2 < 8; ++t2) fms_acc(v[t2], v[t], LD[t][t2]);
                if (!REF) fms_acc(yr, v[t], zb[t]);
                cb[t * lj + r] = v[t];
            }
            if (!REF) y[r] = yr;
        }
        __syncthreads();
    }
    if constexpr (REF) {
        if (s_err && tid == 0) atomicAdd(nonconv, 1);
        return;
    }
    if (s_err) {
        if (tid == 0) atomicMax(&s.status[sys], s_err);
        return;
    }
    // L^T x = y, panel by panel from the last
    for (int p0 = (m - 1) / NBP * NBP; p0 >= 0; p0 -= NBP) {
        const int nb = min(NBP, m - p0);
        {   // y[p0 + t] -= sum over solved rows r >= p0 + nb of L(r, p0 + t) x_r
            const int t = tid >> 4, sl = tid & 15;   // NT = 256 here
            T part = Sc<T>::zero();
            if (t < nb) {
                const T* cp = &at(0, p0 + t);
#pragma unroll 4
                for (int r = p0 + nb + sl; r < m; r += 16) fma_acc(part, cp[r], y[r]);
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) part += shfl_xor_t(part, off);
            if (sl == 0 && t < nb) y[p0 + t] -= part;
        }
        __syncthreads();
        if (warp == 0) {   // the panel's triangle of L^T, lane t = row p0 + t
            const T* cl = &at(0, p0 + min(lane, nb - 1));
            T v = lane < nb ? y[p0 + lane] : Sc<T>::zero();
            const T rc = recip_fx(cl[p0 + min(lane, nb - 1)]);
            for (int u = nb - 1; u >= 0; --u) {
                const T lu = lane < u ? cl[p0 + u] : Sc<T>::zero();
                if (lane == u) v = mul_fx(v, rc);
                const T x = shfl_w(v, u, 32);
                if (lane < u) fms_acc(v, lu, x);
            }
            if (lane < nb) y[p0 + lane] = v;
        }
        __syncthreads();
    }
    for (int g = tid; g < m; g += NT) xg[(size_t)sys * m + g] = y[g];
}

// |Re| + |Im| (the convergence test's magnitude)
__device__ __forceinline__ double mag1(double a) { return fabs(a); }
__device__ __forceinline__ double mag1(cd a) { return fabs(a.x) + fabs(a.y); }

// ---------------------------------------------------------------------------
// Iterative form.  S0[k] = A_GG^area - V^T V^, both triangles, column-major:
// first -C_VV (C's lower triangle, mirrored), then the area part of every G-G
// entry (each pair g >= h occurs once in the gg list).
template <typename T>
__global__ void k_schur_s0_vv(SchurArgs s, const T* __restrict__ C, T* S0)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int m = s.m;
    if (idx >= (long long)s.K * m * m) return;
    const int k = (int)(idx / ((long long)m * m)), c = (int)((idx / m) % m), r = (int)(idx % m);
    const int hi = max(r, c), lo = min(r, c);
    S0[idx] = -C[((size_t)k * s.ncol + s.L + lo) * m + hi];
}

template <typename T>
__global__ void k_schur_s0_area(SchurArgs s, BandArgs<T> A, T* S0)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)s.K * s.ngg) return;
    const int k = (int)(idx / s.ngg), q = (int)(idx % s.ngg), m = s.m;
    const T a = band_assemble_part<T>(A, s.gg_ent[q], k, 0, 1, 0);
    const int g = s.gg_g[q], h = s.gg_h[q];
    T* Sk = S0 + (size_t)k * m * m;
    Sk[(size_t)h * m + g] += a;
    if (g != h) Sk[(size_t)g * m + h] += a;
}

// The preconditioned iteration for NS systems of one electrode group (one
// CTA): x_0 = 0, r = b - S_l x, z = S_ref^-1 r, x += z, until
// max |z| <= tol max |x| for every system.  X and R/Z live in shared memory,
// a system's column contiguous ([NS][m], so that threads over rows touch
// consecutive words); S0 and the reference factor stream from L2.  The
// products S0 X read S0 by columns (coalesced over the rows); D_l X uses the
// boundary rows (bd_*); the triangular solves go by 16-column panels (one
// warp per system solves a panel's triangle, all threads update the rows
// below, or, backwards, reduce the solved rows into the panel).
// Bound by the panels' chains: the pivots' reciprocals are staged with the
// diagonal block, and the factor's entries (and the next block) are loaded
// ahead of the triangle that they wait for.  1,414 systems of 401 boundary
// nodes: 5.2 -> 4.2 ms; 2,048 of 492: 10.1 -> 8.3.
constexpr int SCHUR_IT_NS = 8;
constexpr int SCHUR_IT_NT = 256;
constexpr int SCHUR_IT_PB = 16;

template <typename T>
__global__ void k_schur_dvals(SchurArgs s, BandArgs<T> A, T* Dv)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)s.K * s.L * s.nbd) return;
    const int q = (int)(idx % s.nbd);
    const long long kl = idx / s.nbd;
    const int k = (int)(kl / s.L), l = (int)(kl % s.L);
    Dv[idx] = band_assemble_part<T>(A, s.bd_ent[q], k, l, 1, 1);
}

// NS systems per CTA (8, or 4 at two CTAs per SM: MINB); each system's
// arithmetic does not depend on NS.
template <typename T, int NS = SCHUR_IT_NS, int MINB = 1>
__global__ void __launch_bounds__(SCHUR_IT_NT, MINB) k_schur_iter(SchurArgs s, BandArgs<T> A, const T* __restrict__ C,
                                                                 const T* __restrict__ S0, const T* __restrict__ Lref,
                                                                 const T* __restrict__ Dv, T* xg, int maxit,
                                                                 double tol, int* nonconv)
{
    constexpr int NT = SCHUR_IT_NT, PB = SCHUR_IT_PB;
    extern __shared__ __align__(16) unsigned char it_dyn[];
    const int m = s.m, L = s.L;
    T* X = reinterpret_cast<T*>(it_dyn);   // [NS][m]: system j's column at j m
    T* Z = X + (size_t)m * NS;              // [NS][m]
    __shared__ double s_dx[NS], s_x[NS], s_dprev[NS];
    __shared__ int s_go;
    __shared__ T Ld[PB][PB + 1];   // the panel's diagonal block, Ld[c][r] = L(p0 + r, p0 + c)
    __shared__ T Ldi[PB];          // its reciprocal pivots
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cpg = (s.grp + NS - 1) / NS;             // CTAs per group
    const int b = blockIdx.x, half = b % cpg, kg = b / cpg, g = kg % s.ngrp, k = kg / s.ngrp;
    const int l0 = g * s.grp + half * NS;
    const int l1 = min(min(L, (g + 1) * s.grp), l0 + NS);
    const int ns = l1 - l0;
    if (ns <= 0) return;
    const T* Ck = C + (size_t)k * s.ncol * m;
    const T* Sk = S0 + (size_t)k * m * m;
    const T* Lg = Lref + (size_t)kg * m * m;
    auto bval = [&](int r, int j) {
        const int l = l0 + j;
        T v = -Ck[(size_t)l * m + r];
        if (r == s.posG_src[l]) v += Sc<T>::one();
        if (s.lsink && r == s.posG_sink) v -= Sc<T>::one();
        return v;
    };
    for (int i = tid; i < m * NS; i += NT) {
        const int j = i / m, r = i % m;
        X[i] = Sc<T>::zero();
        Z[i] = j < ns ? bval(r, j) : Sc<T>::zero();
    }
    __syncthreads();
    int it = 0;
    for (;; ++it) {
        if (it > 0) {
            // Z = b - S0 X - D_l X (rows r = tid, tid + NT, ...)
            for (int r = tid; r < m; r += NT) {
                T acc[NS];
#pragma unroll
                for (int j = 0; j < NS; ++j) acc[j] = j < ns ? bval(r, j) : Sc<T>::zero();
#pragma unroll 8
                for (int c = 0; c < m; ++c) {
                    const T a = Sk[(size_t)c * m + r];
#pragma unroll
                    for (int j = 0; j < NS; ++j) fms_acc(acc[j], a, X[j * m + c]);
                }
                const T* Dk = Dv + ((size_t)k * L + l0) * s.nbd;
                for (int q = s.bd_ptr[r]; q < s.bd_ptr[r + 1]; ++q) {
                    const int c = s.bd_col[q];
#pragma unroll
                    for (int j = 0; j < NS; ++j)
                        if (j < ns) fms_acc(acc[j], Dk[(size_t)j * s.nbd + q], X[j * m + c]);
                }
#pragma unroll
                for (int j = 0; j < NS; ++j) Z[j * m + r] = acc[j];
            }
            __syncthreads();
        }
        // thread's entry of the diagonal block at p0, and its store (with the
        // pivot's reciprocal) once the block before is done with
        static_assert(NT == PB * PB, "a thread per entry");
        const int dc = tid / PB, dr = tid % PB;
        auto load_diag = [&](int p0) {
            return p0 < m && dr >= dc && p0 + dr < m ? Lg[(size_t)(p0 + dc) * m + p0 + dr] : Sc<T>::zero();
        };
        auto store_diag = [&](T d) {
            Ld[dc][dr] = d;
            if (dc == dr) Ldi[dc] = recip_fx(d);
        };
        // forward: L y = z, by panels
        store_diag(load_diag(0));
        for (int p0 = 0; p0 < m; p0 += PB) {
            const int nb = min(PB, m - p0);
            // the factor's entries below the panel, and the next diagonal
            // block, are on their way while the panel's triangle is solved
            T a[PB];
            const int r0 = p0 + nb + tid;
#pragma unroll
            for (int u = 0; u < PB; ++u) a[u] = u < nb && r0 < m ? Lg[(size_t)(p0 + u) * m + r0] : Sc<T>::zero();
            const T dn = load_diag(p0 + PB);
            __syncthreads();
            if (warp < NS) {   // warp j: system j, lane t: row p0 + t
                const int j = warp;
                T v = lane < nb ? Z[j * m + p0 + lane] : Sc<T>::zero();
#pragma unroll
                for (int u = 0; u < PB; ++u) {
                    if (u < nb) {
                        if (lane == u) v = mul_fx(v, Ldi[u]);
                        const T xu = shfl_w(v, u, 32);
                        if (lane > u && lane < nb) fms_acc(v, Ld[u][lane], xu);
                    }
                }
                if (lane < nb) Z[j * m + p0 + lane] = v;
            }
            __syncthreads();
            store_diag(dn);
            for (int r = r0; r < m; r += NT) {
                T acc[NS];
#pragma unroll
                for (int j = 0; j < NS; ++j) acc[j] = Z[j * m + r];
                if (r > r0)
#pragma unroll
                    for (int u = 0; u < PB; ++u) a[u] = u < nb ? Lg[(size_t)(p0 + u) * m + r] : Sc<T>::zero();
#pragma unroll
                for (int u = 0; u < PB; ++u)
#pragma unroll
                    for (int j = 0; j < NS; ++j) fms_acc(acc[j], a[u], Z[j * m + p0 + u]);
#pragma unroll
                for (int j = 0; j < NS; ++j) Z[j * m + r] = acc[j];
            }
        }
        __syncthreads();
        // backward: L^T x = y, by panels from the last
        for (int p0 = (m - 1) / PB * PB; p0 >= 0; p0 -= PB) {
            const int nb = min(PB, m - p0);
            {   // y[p0 + t] -= sum over solved rows r >= p0 + nb of L(r, p0 + t) x_r: 16 threads per column t
                const int t = tid >> 4, sl = tid & 15;
                const T d = load_diag(p0);
                T part[NS];
#pragma unroll
                for (int j = 0; j < NS; ++j) part[j] = Sc<T>::zero();
                if (t < nb) {
                    const T* col = Lg + (size_t)(p0 + t) * m;
                    constexpr int RU = 8;   // rows in flight
                    for (int r = p0 + nb + sl; r < m; r += 16 * RU) {
                        T a[RU];
#pragma unroll
                        for (int u = 0; u < RU; ++u) a[u] = r + 16 * u < m ? col[r + 16 * u] : Sc<T>::zero();
#pragma unroll
                        for (int u = 0; u < RU; ++u)
                            if (r + 16 * u < m)
#pragma unroll
                                for (int j = 0; j < NS; ++j) fma_acc(part[j], a[u], Z[j * m + r + 16 * u]);
                    }
                }
#pragma unroll
                for (int j = 0; j < NS; ++j) {
#pragma unroll
                    for (int off = 8; off > 0; off >>= 1) part[j] += shfl_xor_t(part[j], off);
                }
                __syncthreads();
                if (sl == 0 && t < nb)
#pragma unroll
                    for (int j = 0; j < NS; ++j) Z[j * m + p0 + t] -= part[j];
                store_diag(d);
            }
            __syncthreads();
            if (warp < NS) {   // the panel's triangle of L^T, lane t = row p0 + t
                const int j = warp;
                T v = lane < nb ? Z[j * m + p0 + lane] : Sc<T>::zero();
#pragma unroll
                for (int u = PB - 1; u >= 0; --u) {
                    if (u < nb) {
                        if (lane == u) v = mul_fx(v, Ldi[u]);
                        const T xu = shfl_w(v, u, 32);
                        if (lane < u) fms_acc(v, Ld[lane][u], xu);
                    }
                }
                if (lane < nb) Z[j * m + p0 + lane] = v;
            }
            __syncthreads();
        }
        // x += z; convergence: max |z| <= tol max |x| per system
        if (tid < NS) {
            s_dx[tid] = 0.0;
            s_x[tid] = 0.0;
        }
        __syncthreads();
        {
            // the NT / NS threads of system j (NT / NS a multiple of 32):
            // rows r = i, i + NT / NS, ..., then their warps
            constexpr int TPS = NT / NS;
            static_assert(TPS % 32 == 0, "whole warps per system");
            const int j = tid / TPS, i = tid % TPS;
            double dmax = 0.0, xmax = 0.0;
            for (int r = i; r < m; r += TPS) {
                const T z = Z[j * m + r];
                const T x = X[j * m + r] + z;
                X[j * m + r] = x;
                dmax = fmax(dmax, mag1(z));
                xmax = fmax(xmax, mag1(x));
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, off));
                xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, off));
            }
            if (lane == 0) {
                atomicMax(reinterpret_cast<unsigned long long*>(&s_dx[j]), __double_as_longlong(dmax));
                atomicMax(reinterpret_cast<unsigned long long*>(&s_x[j]), __double_as_longlong(xmax));
            }
        }
        __syncthreads();
        if (tid == 0) {
            // converged: the correction at tol of the solution, or no longer
            // contracting at the rounding level of the residual (a small
            // correction that did not halve)
            int go = 0;
            for (int j = 0; j < ns; ++j) {
                const bool done = s_dx[j] <= tol * s_x[j] ||
                                  (it >= 2 && s_dx[j] > 0.5 * s_dprev[j] && s_dx[j] <= 1e-9 * s_x[j]);
                go |= !done;
                s_dprev[j] = s_dx[j];
            }
            s_go = go;
        }
        __syncthreads();
        if (!s_go) break;
        if (it + 1 >= maxit) {
            if (tid == 0) atomicAdd(nonconv, ns);
            return;
        }
    }
    if (tid == 0) atomicAdd(nonconv + 1, ns * (it + 1));   // system-iterations, for the work count
    for (int i = tid; i < m * ns; i += NT) {
        const int j = i / m, r = i % m;
        xg[((size_t)k * L + l0 + j) * m + r] = X[j * m + r];
    }
}

// ---------------------------------------------------------------------------
// z^_l = u^_l - V^ p_G on the FP64 tensor pipe (60k triangles 5.6 -> 5.0 ms
// against 4 x 4 multiply-adds per thread): tiles of 64 interior rows x 32
// electrodes (8 warps of 16 x 16); the boundary columns in the order of their
// first row, so a tile stops at the first column that is zero on all its rows.
template <typename T>
__global__ void __launch_bounds__(256) k_schur_zrebuild(SchurArgs s, T* X, const T* __restrict__ xg)
{
    constexpr int TI = 64, TL = 32, TG = 16, NS = 3, NT = 256;
    // [boundary column][row] and [electrode][boundary column] runs, padded so
    // that what a half-warp reads at once (the columns of one product x four
    // rows, four electrodes x the columns) lies in different banks
    constexpr int SA = TI + 4, SB = TG + RunPad<T>::v;
    using Tile = MmaTile<T>;
    constexpr int KC = Tile::KC;
    extern __shared__ __align__(16) unsigned char zr_dyn[];
    T* buf0 = reinterpret_cast<T*>(zr_dyn);   // [NS][TG * SA + TL * SB]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // wavenumbers along x and the row blocks from the last: a late row block
    // meets the most boundary columns, so the longest tiles start first
    const int k = s.k0 + blockIdx.x, i0 = (gridDim.y - 1 - blockIdx.y) * TI, l0 = blockIdx.z * TL;
    const int m = s.m, nI = s.nI, L = s.L;
    T* Xk = X + (size_t)k * s.ncol * nI;
    // boundary columns [TG t, TG t + TG) of both operands into stage t % NS
    auto stage = [&](int t) {
        T* As = buf0 + (size_t)(t % NS) * (TG * SA + TL * SB);
        T* Bs = As + TG * SA;
        for (int idx = tid; idx < TG * TI; idx += NT) {
            const int gg = idx / TI, ii = idx % TI;
            const int g = TG * t + gg < m ? s.gsort[TG * t + gg] : -1;
            if (g >= 0 && i0 + ii < nI) cp_async_elem<T>(As + gg * SA + ii, Xk + (size_t)(L + g) * nI + i0 + ii);
            else As[gg * SA + ii] = Sc<T>::zero();
        }
        for (int idx = tid; idx < TG * TL; idx += NT) {
            const int ll = idx / TG, gg = idx % TG;
            const int g = TG * t + gg < m ? s.gsort[TG * t + gg] : -1;
            if (g >= 0 && l0 + ll < L) cp_async_elem<T>(Bs + ll * SB + gg, xg + ((size_t)k * L + l0 + ll) * m + g);
            else Bs[ll * SB + gg] = Sc<T>::zero();
        }
    };
    // the boundary columns in the order of their first rows: a block whose
    // first column starts below this tile ends the loop
    auto live = [&](int t) { return TG * t < m && s.gfirst[TG * t] < i0 + TI; };
    int nt = 0;
    {   // the live blocks lead
        int lo = 0, hi = (m + TG - 1) / TG;
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (live(mid)) lo = mid + 1;
            else hi = mid;
        }
        nt = lo;
    }
    Tile acc[2][2];
    const int wi = warp / 2 * 16, wl = warp % 2 * 16;
    for (int t = 0; t < NS - 1; ++t) {
        if (t < nt) stage(t);
        cp_async_commit();
    }
    for (int t = 0; t < nt; ++t) {
        cp_async_wait_group<NS - 2>();
        __syncthreads();   // stage t has landed; the last readers of stage t - 1 are through
        if (t + NS - 1 < nt) stage(t + NS - 1);
        cp_async_commit();
        const T* As = buf0 + (size_t)(t % NS) * (TG * SA + TL * SB);
        const T* ap = As + Tile::kk() * SA + wi + (lane >> 2);
        const T* bp = As + TG * SA + (wl + (lane >> 2)) * SB + Tile::kk();
#pragma unroll
        for (int gg = 0; gg < TG; gg += KC) {
            typename Tile::A a[2];
            typename Tile::B b[2];
#pragma unroll
            for (int x = 0; x < 2; ++x) a[x] = Tile::lda(ap + gg * SA + 8 * x);
#pragma unroll
            for (int y = 0; y < 2; ++y) b[y] = Tile::ldb(bp + 8 * y * SB + gg);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < 2; ++y) acc[x][y].mma(a[x], b[y]);
        }
    }
    cp_async_wait_group<0>();
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int l = l0 + wl + 8 * y + 2 * (lane & 3) + q;
            if (l >= L) continue;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int i = i0 + wi + 8 * x + (lane >> 2);
                if (i < nI) Xk[(size_t)l * nI + i] -= acc[x][y].get(q);
            }
        }
}

template <typename T>
__global__ void k_schur_out_gam(SchurArgs s, const T* __restrict__ xg, int n, cd* kpot)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)s.nk * s.L * s.m) return;
    const int g = (int)(idx % s.m);
    const long long kl = (long long)s.k0 * s.L + idx / s.m;   // k L + l
    kpot[kl * n + s.gam[g]] = Sc<T>::to_cd(xg[kl * s.m + g]);
}

int sm_count()
{
    int nsm = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

// window rows: mb + 3 BB (the rows of a block, the band below it, and two
// blocks arriving ahead), a multiple of BB
int sweep_wz(int mbI) { return (mbI + 4 * SW_BB - 1) / SW_BB * SW_BB; }

}  // namespace

// dynamic shared memory of a sweep with nb factor buffers
template <typename T> static size_t sweep_smem(int mbI, int WI, int nb)
{
    return ((size_t)nb * SW_BB * WI + (size_t)sweep_wz(mbI) * SweepRow<T>::v) * sizeof(T);
}

template <typename T> size_t schur_sweep_smem(int mbI, int WI) { return sweep_smem<T>(mbI, WI, 3); }

int schur_sweep_in_flight(int mbI) { return mbI >= SW_BB ? 1 : 0; }

namespace {

// One launch of the sweep.  Launches of more CTAs than SMs pair two on an SM,
// each with two factor buffers, while both fit (complex half-bandwidths to
// 128): one's chain runs beside the other's updates.  Smaller ones give a CTA
// its SM and three buffers, a block's pivots ahead of it.  Measured, paired
// against alone: 128 sources and 492 boundary nodes at a half-bandwidth of
// 128, the forward sweep's part after the factor (624 CTAs) 4.4 ms against
// 6.5, the back sweep (128 CTAs) 6.3 against 4.7; 96 and 253 at 36, real, 0.02
// against 0.23 (264 CTAs) and 0.75 against 0.50 (72).
template <typename T>
void sweep(const SchurArgs& s, int nblk, const T* Lws, const double* fakws, T* X, cd* kpot, int n_kpot, int back,
           cudaStream_t st)
{
    constexpr int NT = 320;
    const size_t two = sweep_smem<T>(s.mbI, s.WI, 2);
    const bool pair = (long long)s.nk * nblk > sm_count() && 2 * (two + 2048) <= 228 * 1024;
    const size_t smem = pair ? two : schur_sweep_smem<T>(s.mbI, s.WI);
    auto kern = pair ? k_schur_sweep<T, NT, 2, 2> : k_schur_sweep<T, NT, 3, 1>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<dim3(s.nk, nblk), NT, smem, st>>>(s, Lws, fakws, X, kpot, n_kpot, sweep_wz(s.mbI),
                                            schur_sweep_in_flight(s.mbI), back);
}

}  // namespace

// ---------------------------------------------------------------------------
template <typename T>
void launch_schur_rhs(const SchurArgs& s, const BandArgs<T>& full, const double* fakws, T* X, T* cval, cudaStream_t st)
{
    const int ns = s.K * s.L;
    k_schur_rhs_src<T><<<(ns + 127) / 128, 128, 0, st>>>(s, fakws, X);
    const long long nc = (long long)s.K * s.ncpl;
    if (nc > 0) k_schur_rhs_cpl<T><<<(unsigned)((nc + 255) / 256), 256, 0, st>>>(s, full, fakws, X, cval);
}

template <typename T>
void launch_schur_transpose(const SchurArgs& s, const T* Lws, T* Lrev, cudaStream_t st)
{
    const long long tot = (long long)s.nk * s.nI * s.WI;
    k_schur_transpose<T><<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(s, Lws, Lrev);
}

template <typename T>
void launch_schur_forward(const SchurArgs& s, const T* Lws, T* X, cudaStream_t st)
{
    sweep<T>(s, s.nblk, Lws, nullptr, X, nullptr, 0, 0, st);
}

// One thread: returns once `want` CTAs of the concurrent factor have begun
// (bounded: about 2 s), so that the sweep's CTAs, which wait on that
// factor's progress, never take SMs the factor still needs.
__global__ void k_wait_started(const int* started, int want, int* status)
{
    long polls = 0;
    while (*(volatile const int*)started < want) {
        if (++polls > (1L << 21)) {
            atomicMax(status, (int)CRT_ERR_CUDA);
            return;
        }
        __nanosleep(1000);
    }
}

void launch_wait_started(const int* started, int want, int* status, cudaStream_t st)
{
    k_wait_started<<<1, 1, 0, st>>>(started, want, status);
}

template <typename T>
void launch_schur_gram(const SchurArgs& s, const T* X, T* C, cudaStream_t st)
{
    auto go = [&](auto kern, int TG, int TC, int nt, int ns) {
        const int smem = ns * (TG + TC) * (GRAM_TI + RunPad<T>::v) * (int)sizeof(T);
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        kern<<<dim3(s.nk, (s.m + TG - 1) / TG, (s.ncol + TC - 1) / TC), nt, smem, st>>>(s, X, C);
    };
    // 32 x 32 tiles, or 32 x 16 where there would be fewer than five per SM
    // (8,000 triangles and 48 electrodes, 12 wavenumbers: 0.34 against 0.45
    // ms; 60k triangles: 9.7 against 9.2 ms, the other way).  64-wide tiles
    // lose on every size (60k triangles: 12.5 ms at 64 x 64, 10.8 at 64 x 32):
    // a tile runs from the earliest row of its columns, and its serial sum
    // over the rows is the longest CTA's time.
    if ((long long)s.nk * ((s.m + 31) / 32) * ((s.ncol + 31) / 32) >= 5 * sm_count())
        go(k_schur_gram<T, 32, 32, 2, 2, 4>, 32, 32, 128, 4);
    else
        go(k_schur_gram<T, 32, 16, 2, 1, 4>, 32, 16, 128, 4);
}

// columns per panel of the back solve (its partial sums' order): 12, or 16
// above 553 complex boundary nodes
template <typename T>
static int ll_back_panel(int m) { return 2 * ((size_t)13 * m * sizeof(T) + 1024) <= 227 * 1024 ? 12 : 16; }

// Whether nsys systems of m boundary nodes go left-looking with their stages
// in shared memory: always while two such CTAs share an SM (complex to 256
// nodes, real to 488), and above only where every system has an SM of its
// own, up to a size at which the right-looking form's two CTAs win even there.
// Left and right in ms, complex: 1,152 systems of 241 nodes 3.95 and 4.57, of
// 261 6.48 and 5.26, of 401 18.9 and 13.4; 140 of 361 1.84 and 1.96, of 401
// 2.42 and 2.45, of 481 3.88 and 3.72.  Real: 1,152 of 481 10.3 and 12.0, of
// 521 16.1 and 14.5, of 767 61 and 41; 140 of 601 3.53 and 3.78, of 701 5.57
// and 5.42.  The two give the same bits.
template <typename T>
static bool ll_staged(int m, int nsys)
{
    const size_t smem = ll_smem<T>(m, false), cta = 2560;   // a CTA's static shared memory and the driver's share
    if (2 * (smem + cta) <= 228 * 1024) return true;
    return nsys <= sm_count() && m <= (std::is_same<T, cd>::value ? 400 : 640);
}

template <typename T>
void launch_schur_chol(const SchurArgs& s, const BandArgs<T>& full, const T* C, T* Sws, T* xg, int sys0, int nsys,
                       cudaStream_t st)
{
    constexpr size_t lim = 227 * 1024;
    auto go = [&](auto kern, size_t smem) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<nsys, LL_NT, smem, st>>>(s, full, C, Sws, xg, sys0, ll_back_panel<T>(s.m), nullptr);
    };
    // the factor in shared memory where two CTAs fit an SM (complex m = 101,
    // 400 systems: 0.33 against 0.34 ms staged; real m = 181 with one CTA per
    // SM 0.50 against 0.54)
    if (2 * (ll_smem<T>(s.m, true) + 2048) <= lim) {
        go(k_schur_ll<T, true, false, LL_NT, 4>, ll_smem<T>(s.m, true));
        return;
    }
    if (ll_staged<T>(s.m, nsys)) {
        go(k_schur_ll<T, false, false, LL_NT, 4>, ll_smem<T>(s.m, false));
        return;
    }
    // right-looking: two CTAs per SM with 12-column panels up to 553 complex
    // boundary nodes, else one with 16
    constexpr int NT = 256;
    const size_t smem16 = ((size_t)16 * s.m + s.m) * sizeof(T), smem12 = ((size_t)12 * s.m + s.m) * sizeof(T);
    if (ll_back_panel<T>(s.m) == 12) {
        auto kern = k_schur_chol<T, NT, 12, false>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem12);
        kern<<<nsys, NT, smem12, st>>>(s, full, C, Sws, xg, sys0, nullptr);
    } else if constexpr (std::is_same<T, cd>::value) {   // real: SCHUR_MMAX nodes take 12
        auto kern = k_schur_chol<T, NT, 16, true>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem16);
        kern<<<nsys, NT, smem16, st>>>(s, full, C, Sws, xg, sys0, nullptr);
    }
}

template <typename T>
void launch_schur_s0(const SchurArgs& s, const BandArgs<T>& full, const T* C, T* S0, cudaStream_t st)
{
    const long long tot = (long long)s.K * s.m * s.m;
    k_schur_s0_vv<T><<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(s, C, S0);
    const long long ng = (long long)s.K * s.ngg;
    if (ng > 0) k_schur_s0_area<T><<<(unsigned)((ng + 255) / 256), 256, 0, st>>>(s, full, S0);
}

template <typename T>
void launch_schur_ref(const SchurArgs& s, const BandArgs<T>& full, const T* S0, T* Lref, int* nonconv, cudaStream_t st)
{
    const int nref = s.K * s.ngrp;
    const size_t smem = ll_smem<T>(s.m, false);
    // left-looking with 512 threads on an SM while its stages fit (complex to
    // 528 boundary nodes) and every factor has an SM (complex, 128 of 492: 3.0
    // ms against 3.4 right-looking, but 300 of 441 0.5 longer); real up to 640
    // nodes at any number (300 of 521 1.1 shorter, 450 of 761 2.2 longer)
    const bool real = std::is_same<T, double>::value;
    if (smem <= 227 * 1024 && (nref <= sm_count() || (real && s.m <= 640))) {
        auto kern = k_schur_ll<T, false, true, 512, 4>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<nref, 512, smem, st>>>(s, full, S0, Lref, nullptr, 0, 0, nonconv);
        return;
    }
    constexpr int NT = 256;
    const size_t smem12 = ((size_t)12 * s.m + s.m) * sizeof(T), smem16 = ((size_t)16 * s.m + s.m) * sizeof(T);
    if (ll_back_panel<T>(s.m) == 12) {
        auto kern = k_schur_chol<T, NT, 12, false, true>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem12);
        kern<<<nref, NT, smem12, st>>>(s, full, S0, Lref, nullptr, 0, nonconv);
    } else if constexpr (std::is_same<T, cd>::value) {   // real: SCHUR_MMAX nodes take 12
        auto kern = k_schur_chol<T, NT, 16, true, true>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem16);
        kern<<<nref, NT, smem16, st>>>(s, full, S0, Lref, nullptr, 0, nonconv);
    }
}

template <typename T>
size_t schur_iter_smem(int m) { return 2 * (size_t)m * SCHUR_IT_NS * sizeof(T); }

template <typename T>
void launch_schur_dvals(const SchurArgs& s, const BandArgs<T>& full, T* Dv, cudaStream_t st)
{
    const long long tot = (long long)s.K * s.L * s.nbd;
    if (tot > 0) k_schur_dvals<T><<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(s, full, Dv);
}

template <typename T>
void launch_schur_iter(const SchurArgs& s, const BandArgs<T>& full, const T* C, const T* S0, const T* Lref,
                       const T* Dv, T* xg, int maxit, double tol, int* nonconv, cudaStream_t st)
{
    // four systems per CTA at two CTAs per SM (electrode solves 13.6 against
    // 15.9 ms with eight at one on the 60k-triangle mesh: the panel solves
    // are chains of dependent steps, and two CTAs hide each other's
    // latency; two systems at three CTAs per SM measured 14.8 ms);
    // CRT_B200_SCHUR_IT_NS=8 keeps eight
    const char* nv = std::getenv("CRT_B200_SCHUR_IT_NS");
    if (!(nv && std::strcmp(nv, "8") == 0) && 2 * (2 * (size_t)s.m * 4 * sizeof(T)) <= 227 * 1024) {
        const size_t smem = 2 * (size_t)s.m * 4 * sizeof(T);
        const int cpg = (s.grp + 3) / 4;
        auto kern = k_schur_iter<T, 4, 2>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<s.K * s.ngrp * cpg, SCHUR_IT_NT, smem, st>>>(s, full, C, S0, Lref, Dv, xg, maxit, tol, nonconv);
        return;
    }
    const size_t smem = schur_iter_smem<T>(s.m);
    const int cpg = (s.grp + SCHUR_IT_NS - 1) / SCHUR_IT_NS;
    auto kern = k_schur_iter<T>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<s.K * s.ngrp * cpg, SCHUR_IT_NT, smem, st>>>(s, full, C, S0, Lref, Dv, xg, maxit, tol, nonconv);
}

template <typename T>
void launch_schur_zrebuild(const SchurArgs& s, T* X, const T* xg, cudaStream_t st)
{
    dim3 grid(s.nk, (s.nI + 63) / 64, (s.L + 31) / 32);
    constexpr int smem = 3 * (16 * (64 + 4) + 32 * (16 + RunPad<T>::v)) *
                         (int)sizeof(T);   // three stages of both operands
    cudaFuncSetAttribute(k_schur_zrebuild<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k_schur_zrebuild<T><<<grid, 256, smem, st>>>(s, X, xg);
}

template <typename T>
void launch_schur_back(const SchurArgs& s, const T* Lrev, const double* fakws, const T* X, const T* xg, int n,
                       cd* kpot, cudaStream_t st)
{
    sweep<T>(s, (s.L + SW_R - 1) / SW_R, Lrev, fakws, const_cast<T*>(X), kpot, n, 1, st);
    const long long tot = (long long)s.nk * s.L * s.m;
    k_schur_out_gam<T><<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(s, xg, n, kpot);
}

template size_t schur_sweep_smem<cd>(int, int);
template size_t schur_sweep_smem<double>(int, int);
template void launch_schur_rhs<cd>(const SchurArgs&, const BandArgs<cd>&, const double*, cd*, cd*, cudaStream_t);
template void launch_schur_rhs<double>(const SchurArgs&, const BandArgs<double>&, const double*, double*, double*,
                                       cudaStream_t);
template void launch_schur_transpose<cd>(const SchurArgs&, const cd*, cd*, cudaStream_t);
template void launch_schur_transpose<double>(const SchurArgs&, const double*, double*, cudaStream_t);
template void launch_schur_forward<cd>(const SchurArgs&, const cd*, cd*, cudaStream_t);
template void launch_schur_forward<double>(const SchurArgs&, const double*, double*, cudaStream_t);
template void launch_schur_gram<cd>(const SchurArgs&, const cd*, cd*, cudaStream_t);
template void launch_schur_gram<double>(const SchurArgs&, const double*, double*, cudaStream_t);
template void launch_schur_chol<cd>(const SchurArgs&, const BandArgs<cd>&, const cd*, cd*, cd*, int, int, cudaStream_t);
template void launch_schur_chol<double>(const SchurArgs&, const BandArgs<double>&, const double*, double*, double*,
                                        int, int, cudaStream_t);
template void launch_schur_zrebuild<cd>(const SchurArgs&, cd*, const cd*, cudaStream_t);
template void launch_schur_zrebuild<double>(const SchurArgs&, double*, const double*, cudaStream_t);
template void launch_schur_back<cd>(const SchurArgs&, const cd*, const double*, const cd*, const cd*, int, cd*,
                                    cudaStream_t);
template void launch_schur_back<double>(const SchurArgs&, const double*, const double*, const double*, const double*,
                                        int, cd*, cudaStream_t);
template void launch_schur_s0<cd>(const SchurArgs&, const BandArgs<cd>&, const cd*, cd*, cudaStream_t);
template void launch_schur_s0<double>(const SchurArgs&, const BandArgs<double>&, const double*, double*, cudaStream_t);
template void launch_schur_ref<cd>(const SchurArgs&, const BandArgs<cd>&, const cd*, cd*, int*, cudaStream_t);
template void launch_schur_ref<double>(const SchurArgs&, const BandArgs<double>&, const double*, double*, int*,
                                       cudaStream_t);
template void launch_schur_dvals<cd>(const SchurArgs&, const BandArgs<cd>&, cd*, cudaStream_t);
template void launch_schur_dvals<double>(const SchurArgs&, const BandArgs<double>&, double*, cudaStream_t);
template void launch_schur_iter<cd>(const SchurArgs&, const BandArgs<cd>&, const cd*, const cd*, const cd*,
                                    const cd*, cd*, int, double, int*, cudaStream_t);
template void launch_schur_iter<double>(const SchurArgs&, const BandArgs<double>&, const double*, const double*,
                                        const double*, const double*, double*, int, double, int*, cudaStream_t);
template size_t schur_iter_smem<cd>(int);
template size_t schur_iter_smem<double>(int);
