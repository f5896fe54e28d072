// Supernodal triangular solve kernels (sm_100a).
//
// The right-hand sides live on the device in the permuted numbering, column
// major with leading dimension ldy.  A solve with a block-lower panel P (the L
// panel, or the U^T panel of an LU factor) is, level by level:
//   forward   y_k <- P_kk^{-1} y_k;  y[rows(k)] -= P_off(k) y_k       (diag kernels, k_fwd_update)
//   backward  x_k <- P_kk^{-T} (x_k - P_off(k)^T x[rows(k)])            (k_bwd_update, diag kernels)
// which restates solve_cblk_ztrsmsp_forward / _backward
// (kernels/solve_ztrsmsp.c:302, :468) and solve_blok_ztrsm / _zgemm (:76, :160)
// with the step table of pastix_subtask_solve_adv (sopalin/pastix_task_solve.c:543-649):
//   POTRF  L (non-unit) then L^T;  SYTRF  L (unit), D, L^T (unit);
//   GETRF  L (unit) then U through the stored U^T panel (non-unit).
// Independent cblks of one level run in one launch.  The off-diagonal
// products use 64 x 64 tiles of the panel (rows x columns) so that a level's
// wide cblks spread over many CTAs; partial sums go to the right-hand sides by
// atomics.  Diagonal blocks of wide cblks are applied with the inverted 32 x 32
// sub-blocks kept by the factorization (a blocked triangular solve whose
// diagonal steps are small matrix-vector products); narrow cblks use
// substitution by one warp per right-hand side.
#include "device.cuh"

#include <cooperative_groups.h>

namespace pgpu {

constexpr int ST_R = 64, ST_C = 64;  // solve update tile: panel rows x panel columns

// ---------------------------------------------------------------------------
// Narrow cblks: substitution, blocks of 32 rows on the lanes of a warp, one
// warp per right-hand side.
// ---------------------------------------------------------------------------
template <typename T, int RC>
__global__ void __launch_bounds__(256) k_fwd_diag(DevStruct s, const int *__restrict__ list, const T *P, int unit,
                                                   T *Y, int ldy, int nrhs) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *y = reinterpret_cast<T *>(smem_raw);  // nc x RC
    const int k = list[blockIdx.x];
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const int j0 = blockIdx.y * RC;
    const int nr = min(RC, nrhs - j0);
    const T *D = P + s.cb_coef[k];
    const int tid = threadIdx.x, nt = blockDim.x;
    pdl_trigger();
    pdl_wait();
    for (int e = tid; e < nc * nr; e += nt) {
        int i = e % nc, j = e / nc;
        y[i + j * nc] = Y[(fc + i) + (size_t)(j0 + j) * ldy];
    }
    __syncthreads();
    for (int jb = 0; jb < nc; jb += 32) {
        const int nb = min(32, nc - jb);
        {
            const int lane = tid & 31, warp = tid >> 5;
            const T rd = (!unit && lane < nb) ? T(1) / D[(jb + lane) + (size_t)(jb + lane) * st] : T(1);
            T drow[32];  // row jb + lane of the block, loaded before the dependent sweep
#pragma unroll
            for (int c = 0; c < 32; c++)
                drow[c] = (c < lane && lane < nb) ? D[(jb + lane) + (size_t)(jb + c) * st] : T(0);
            for (int j = warp; j < nr; j += nt / 32) {
                T v = (lane < nb) ? y[jb + lane + j * nc] : T(0);
#pragma unroll
                for (int c = 0; c < 32; c++) {
                    if (c < nb) {
                        if (lane == c) v *= rd;
                        const T vc = __shfl_sync(0xffffffffu, v, c);
                        v -= drow[c] * vc;
                    }
                }
                if (lane < nb) y[jb + lane + j * nc] = v;
            }
        }
        __syncthreads();
        for (int e = tid; e < (nc - jb - nb) * nr; e += nt) {
            int i = jb + nb + e % (nc - jb - nb), j = e / (nc - jb - nb);
            T acc = T(0);
            for (int c = 0; c < nb; c++) acc += D[i + (size_t)(jb + c) * st] * y[jb + c + j * nc];
            y[i + j * nc] -= acc;
        }
        __syncthreads();
    }
    for (int e = tid; e < nc * nr; e += nt) {
        int i = e % nc, j = e / nc;
        Y[(fc + i) + (size_t)(j0 + j) * ldy] = y[i + j * nc];
    }
}

template <typename T, int RC>
__global__ void __launch_bounds__(256) k_bwd_diag(DevStruct s, const int *__restrict__ list, const T *P, int unit,
                                                   T *Y, int ldy, int nrhs) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *y = reinterpret_cast<T *>(smem_raw);
    const int k = list[blockIdx.x];
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const int j0 = blockIdx.y * RC;
    const int nr = min(RC, nrhs - j0);
    const T *D = P + s.cb_coef[k];
    const int tid = threadIdx.x, nt = blockDim.x;
    pdl_trigger();
    pdl_wait();
    for (int e = tid; e < nc * nr; e += nt) {
        int i = e % nc, j = e / nc;
        y[i + j * nc] = Y[(fc + i) + (size_t)(j0 + j) * ldy];
    }
    __syncthreads();
    for (int je = nc; je > 0; je -= 32) {
        const int jb = max(0, je - 32);
        const int nb = je - jb;
        {
            const int lane = tid & 31, warp = tid >> 5;
            const T rd = (!unit && lane < nb) ? T(1) / D[(jb + lane) + (size_t)(jb + lane) * st] : T(1);
            T dcol[32];  // column jb + lane of the block, loaded before the dependent sweep
#pragma unroll
            for (int c = 0; c < 32; c++)
                dcol[c] = (lane < c && c < nb) ? D[(jb + c) + (size_t)(jb + lane) * st] : T(0);
            for (int j = warp; j < nr; j += nt / 32) {
                T v = (lane < nb) ? y[jb + lane + j * nc] : T(0);
#pragma unroll
                for (int c = 31; c >= 0; c--) {
                    if (c < nb) {
                        if (lane == c) v *= rd;
                        const T vc = __shfl_sync(0xffffffffu, v, c);
                        v -= dcol[c] * vc;
                    }
                }
                if (lane < nb) y[jb + lane + j * nc] = v;
            }
        }
        __syncthreads();
        for (int e = tid; e < jb * nr; e += nt) {
            int i = e % jb, j = e / jb;
            T acc = T(0);
            for (int c = 0; c < nb; c++) acc += D[(jb + c) + (size_t)i * st] * y[jb + c + j * nc];
            y[i + j * nc] -= acc;
        }
        __syncthreads();
    }
    for (int e = tid; e < nc * nr; e += nt) {
        int i = e % nc, j = e / nc;
        Y[(fc + i) + (size_t)(j0 + j) * ldy] = y[i + j * nc];
    }
}

// One right-hand side: one warp per narrow cblk (width <= 64, since
// stride * width <= 4096), eight cblks per CTA -- the leaves of the tree are
// tens of thousands of such cblks, and a CTA each left seven of its warps
// idle.  In levels of many narrow cblks (solve_fuse_rows) the warp also applies
// the rows below its diagonal block: as 64 x 64 update tiles a leaf of ten
// columns kept a sixth of a CTA's threads busy, and the backward sums went
// through atomics.  Lower four levels of the 100^3 Laplacian, FP32 factors,
// forward: 324 -> 100 us (B200).  y_k lives in two registers per lane (columns lane, 32 + lane); the
// substitution steps are those of k_fwd_diag / k_bwd_diag.
//
// The 32 x 32 block that the sweep starts with is loaded ahead of pdl_wait: it
// belongs to the factor, not to the kernel ahead.
template <typename T>
__device__ __forceinline__ void warp_fwd_load(const T *D, int st, int jb, int nb, int unit, int lane, T (&d)[32], T &rd) {
    rd = (!unit && lane < nb) ? T(1) / D[(jb + lane) + (size_t)(jb + lane) * st] : T(1);
#pragma unroll
    for (int c = 0; c < 32; c++) d[c] = (c < lane && lane < nb) ? D[(jb + lane) + (size_t)(jb + c) * st] : T(0);
}
template <typename T>
__device__ __forceinline__ T warp_fwd_block(const T (&d)[32], T rd, int nb, int lane, T v) {
#pragma unroll
    for (int c = 0; c < 32; c++) {
        if (c < nb) {
            if (lane == c) v *= rd;
            const T vc = __shfl_sync(0xffffffffu, v, c);
            v -= d[c] * vc;
        }
    }
    return v;
}
template <typename T>
__device__ __forceinline__ void warp_bwd_load(const T *D, int st, int jb, int nb, int unit, int lane, T (&d)[32], T &rd) {
    rd = (!unit && lane < nb) ? T(1) / D[(jb + lane) + (size_t)(jb + lane) * st] : T(1);
#pragma unroll
    for (int c = 0; c < 32; c++) d[c] = (lane < c && c < nb) ? D[(jb + c) + (size_t)(jb + lane) * st] : T(0);
}
template <typename T>
__device__ __forceinline__ T warp_bwd_block(const T (&d)[32], T rd, int nb, int lane, T v) {
#pragma unroll
    for (int c = 31; c >= 0; c--) {
        if (c < nb) {
            if (lane == c) v *= rd;
            const T vc = __shfl_sync(0xffffffffu, v, c);
            v -= d[c] * vc;
        }
    }
    return v;
}

// Sum over the 32 lanes of v[u] for every u at once (butterfly transpose
// reduction, 31 shuffles): on return lane l holds in v[0] the sum of v[l].
template <typename T>
__device__ __forceinline__ void lane_sums32(T (&v)[32], int lane) {
#pragma unroll
    for (int sft = 16; sft >= 1; sft >>= 1) {
        const bool upper = (lane & sft) != 0;
#pragma unroll
        for (int u = 0; u < sft; u++) {
            const T send = upper ? v[u] : v[u + sft];
            const T keep = upper ? v[u + sft] : v[u];
            v[u] = keep + __shfl_xor_sync(0xffffffffu, send, sft);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_fwd_diag_w(DevStruct s, const int *__restrict__ list, int count, const T *P,
                                                     int unit, T *Y, int rows) {
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (w >= count) return;  // whole warps; the others of the CTA wait
    const int k = list[w];
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const T *D = P + s.cb_coef[k];
    T d[32], rd;
    warp_fwd_load<T>(D, st, 0, min(32, nc), unit, lane, d, rd);
    pdl_wait();
    T y0 = lane < nc ? Y[fc + lane] : T(0);
    T y1 = 32 + lane < nc ? Y[fc + 32 + lane] : T(0);
    y0 = warp_fwd_block<T>(d, rd, min(32, nc), lane, y0);
    if (nc > 32) {  // rows 32 .. nc - 1 of the diagonal block: y1 -= D[32 + lane, 0..31] y0
        const int r = 32 + lane;
        T acc = T(0);
#pragma unroll
        for (int c = 0; c < 32; c++) {
            const T yc = __shfl_sync(0xffffffffu, y0, c);
            if (r < nc) acc += D[r + (size_t)c * st] * yc;
        }
        warp_fwd_load<T>(D, st, 32, nc - 32, unit, lane, d, rd);
        y1 = warp_fwd_block<T>(d, rd, nc - 32, lane, y1 - acc);
    }
    if (lane < nc) Y[fc + lane] = y0;
    if (32 + lane < nc) Y[fc + 32 + lane] = y1;
    if (!rows) return;
    // y[row(r)] -= P[r, :] y_k, two rows per lane, eight columns' loads in flight
    const int *ridx = s.rowidx + s.cb_rowidx[k];
    for (int r0 = nc; r0 < st; r0 += 64) {
        const int ra = r0 + lane, rb = ra + 32;
        T acc0 = T(0), acc1 = T(0);
        for (int c0 = 0; c0 < nc; c0 += 8) {
            T p0[8], p1[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                p0[u] = (ra < st && c0 + u < nc) ? D[ra + (size_t)(c0 + u) * st] : T(0);
                p1[u] = (rb < st && c0 + u < nc) ? D[rb + (size_t)(c0 + u) * st] : T(0);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const T yc = __shfl_sync(0xffffffffu, c0 < 32 ? y0 : y1, (c0 + u) & 31);
                acc0 += p0[u] * yc;
                acc1 += p1[u] * yc;
            }
        }
        if (ra < st) atomicAdd(&Y[ridx[ra]], -acc0);
        if (rb < st) atomicAdd(&Y[ridx[rb]], -acc1);
    }
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_bwd_diag_w(DevStruct s, const int *__restrict__ list, int count, const T *P,
                                                     int unit, T *Y, int rows) {
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (w >= count) return;
    const int k = list[w];
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const T *D = P + s.cb_coef[k];
    T d[32], rd;
    const int jl = nc > 32 ? 32 : 0;  // the last block goes first
    const int *ridx = s.rowidx + s.cb_rowidx[k];
    if (!rows) warp_bwd_load<T>(D, st, jl, nc - jl, unit, lane, d, rd);
    pdl_wait();
    T y0 = lane < nc ? Y[fc + lane] : T(0);
    T y1 = 32 + lane < nc ? Y[fc + 32 + lane] : T(0);
    // x_k -= P_off^T x[rows]: lanes over the rows, the 32 column sums by one butterfly
    for (int cb = jl; rows && cb >= 0; cb -= 32) {
        T v[32];
#pragma unroll
        for (int u = 0; u < 32; u++) v[u] = T(0);
        for (int r = nc + lane; r < st; r += 32) {
            const T xr = Y[ridx[r]];
#pragma unroll
            for (int u = 0; u < 32; u++)
                if (cb + u < nc) v[u] += D[r + (size_t)(cb + u) * st] * xr;
        }
        lane_sums32(v, lane);
        if (cb) y1 -= v[0];
        else y0 -= v[0];
    }
    if (rows) warp_bwd_load<T>(D, st, jl, nc - jl, unit, lane, d, rd);
    if (nc > 32) {  // the last block first, then its contribution to rows 0..31: y0 -= D[32 + c, lane] y1[c]
        y1 = warp_bwd_block<T>(d, rd, nc - 32, lane, y1);
        T acc = T(0);
#pragma unroll
        for (int c = 0; c < 32; c++) {
            const T yc = __shfl_sync(0xffffffffu, y1, c);
            if (32 + c < nc) acc += D[(32 + c) + (size_t)lane * st] * yc;
        }
        y0 -= acc;
        warp_bwd_load<T>(D, st, 0, 32, unit, lane, d, rd);
    }
    y0 = warp_bwd_block<T>(d, rd, min(32, nc), lane, y0);
    if (lane < nc) Y[fc + lane] = y0;
    if (32 + lane < nc) Y[fc + 32 + lane] = y1;
}

// ---------------------------------------------------------------------------
// Wide cblks: blocked diagonal solves with the inverted 32 x 32 sub-blocks Z
// (Z = T^{-1}, T the upper factor of the sub-block, see factor.cu):
//   forward   y_j <- S Z^T y_j,  then  y[below] -= P[below, j] y_j
//   backward  x_j -= P[below, j]^T x[below],  then  x_j <- Z S x_j
// with S = D (LDL^T, scaled) or I.  zside picks the Z set (GETRF: 0 = U, 1 = L^T).
// ---------------------------------------------------------------------------
// Diagonal steps with the full inverse of the block's triangular factor, kept
// (transposed, FP32) by the FP32 factorization for its TRSM: Pt = T^{-T},
// column major nc x nc, lower triangular.  Forward: y <- S Pt y; backward:
// x <- Pt^T S x (S = D for LDL^T, else I) -- the blocked steps of
// solve_cblk_ztrsmsp_forward / _backward as one dense product, for RC
// right-hand sides.  A cluster of TC CTAs shares one cblk: every CTA copies
// y_k to its shared memory, and the lower triangle of Pt is cut into 32 x 32
// tiles spread over the cluster's 8 * TC warps (at most two each, 32
// independent coalesced loads per lane), so that no warp walks a long row or
// column alone.  Partial sums go by distributed-shared-memory atomics to the
// CTA that owns the 32 outputs (block b -> CTA b % TC); a second cluster
// barrier orders every partial before the owners overwrite y_k in place.
constexpr int TC = 8;

// Tile t of the lower triangle of an nch x nch block grid, row by row:
// (i, jc) with jc <= i and t = i (i + 1) / 2 + jc.
__device__ __forceinline__ void tri_tile(int t, int &i, int &jc) {
    i = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
    while ((i + 1) * (i + 2) / 2 <= t) i++;
    while (i * (i + 1) / 2 > t) i--;
    jc = t - i * (i + 1) / 2;
}

template <typename T, int RC>
__global__ void __cluster_dims__(TC, 1, 1) __launch_bounds__(256)
    k_fwd_diag_tinv(DevStruct s, const int *__restrict__ list, int zside, int scaled, const T *Ldiag, T *Y, int ldy,
                    int nrhs, const float *__restrict__ tinv, const int64_t *__restrict__ ti_off) {
    __shared__ float ys[RC][384];
    __shared__ float acc[RC][384];
    pdl_trigger();
    const int k = list[blockIdx.x / TC];
    const int64_t off = ti_off[k];
    if (off < 0) return;  // the whole cluster leaves: k_fwd_diag_inv takes this cblk
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const int j0 = blockIdx.y * RC, nr = min(RC, nrhs - j0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int npad = 32 * ((nc + 31) / 32);  // whole 32-blocks: the tiles read ys up to npad
    const float *Pt = tinv + off + (size_t)zside * nc * nc;
    const int nch = (nc + 31) / 32, ntile = nch * (nch + 1) / 2;
    int t = rank * 8 + warp, i = 0, jc = 0;
    float p[32];
    auto load = [&]() {  // tile t: row block i, column block jc
        tri_tile(t, i, jc);
        const int r = 32 * i + lane, c0 = 32 * jc;
#pragma unroll
        for (int u = 0; u < 32; u++) p[u] = (r < nc && c0 + u < nc) ? Pt[r + (size_t)(c0 + u) * nc] : 0.f;
    };
    if (t < ntile) load();  // the inverse does not depend on the kernel ahead
    pdl_wait();
    for (int e = tid; e < npad * RC; e += blockDim.x) {
        const int i = e % npad, j = e / npad;
        ys[j][i] = (j < nr && i < nc) ? (float)Y[fc + i + (size_t)(j0 + j) * ldy] : 0.f;
        acc[j][i] = 0.f;
    }
    cluster.sync();  // every copy of y_k made, every accumulator cleared
    while (t < ntile) {
        const int r = 32 * i + lane, c0 = 32 * jc;
        float a[RC];
#pragma unroll
        for (int j = 0; j < RC; j++) a[j] = 0.f;
        if (r < nc) {
#pragma unroll
            for (int u = 0; u < 32; u++)
#pragma unroll
                for (int j = 0; j < RC; j++) a[j] += p[u] * ys[j][c0 + u];
            float *dst = cluster.map_shared_rank(&acc[0][0], i % TC);
#pragma unroll
            for (int j = 0; j < RC; j++)
                if (j < nr) atomicAdd(dst + j * 384 + r, a[j]);
        }
        t += TC * 8;
        if (t < ntile) load();
    }
    cluster.sync();  // every partial sum in place
    for (int cb = rank * 32; cb < nc; cb += TC * 32)
        for (int e = tid; e < 32 * RC; e += blockDim.x) {
            const int l = e & 31, j = e >> 5, c = cb + l;
            if (c < nc && j < nr) {
                float v = acc[j][c];
                if (scaled) v *= (float)Ldiag[s.cb_coef[k] + c + (size_t)c * st];
                Y[fc + c + (size_t)(j0 + j) * ldy] = (T)v;
            }
        }
}

// Groups of 8 right-hand sides: 8 products per loaded element make the work
// compute-heavy enough that 32-row (forward) or 32-column (backward) blocks
// round robin over the cluster's CTAs, with no cross-CTA partial sums, beat the
// tiled kernels (whose remote atomics grow with the number of right-hand
// sides); a single right-hand side uses the tiled kernels.
template <typename T, int RC>
__global__ void __cluster_dims__(TC, 1, 1) __launch_bounds__(256)
    k_fwd_diag_tinv_rr(DevStruct s, const int *__restrict__ list, int zside, int scaled, const T *Ldiag, T *Y, int ldy,
                    int nrhs, const float *__restrict__ tinv, const int64_t *__restrict__ ti_off) {
    __shared__ float ys[RC][384];
    __shared__ float part[8][RC][33];
    pdl_trigger();
    const int k = list[blockIdx.x / TC];
    const int64_t off = ti_off[k];
    if (off < 0) return;  // the whole cluster leaves: k_fwd_diag_inv takes this cblk
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const int j0 = blockIdx.y * RC, nr = min(RC, nrhs - j0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_wait();
    for (int e = tid; e < nc * RC; e += blockDim.x) {
        const int i = e % nc, j = e / nc;
        ys[j][i] = j < nr ? (float)Y[fc + i + (size_t)(j0 + j) * ldy] : 0.f;
    }
    cluster.sync();
    const float *Pt = tinv + off + (size_t)zside * nc * nc;
    for (int cb = rank * 32; cb < nc; cb += TC * 32) {
        const int c = cb + lane;
        const int kend = min(nc, cb + 32);  // Pt is lower triangular: columns past the block are zero
        float acc[RC];
#pragma unroll
        for (int j = 0; j < RC; j++) acc[j] = 0.f;
        if (c < nc) {
#pragma unroll 8
            for (int kk = warp; kk < kend; kk += 8) {
                const float pv = Pt[c + (size_t)kk * nc];
#pragma unroll
                for (int j = 0; j < RC; j++) acc[j] += pv * ys[j][kk];
            }
        }
#pragma unroll
        for (int j = 0; j < RC; j++) part[warp][j][lane] = acc[j];
        __syncthreads();
        for (int o = tid; o < 32 * RC; o += blockDim.x) {
            const int l = o & 31, j = o >> 5, cc = cb + l;
            if (cc < nc && j < nr) {
                float v = 0.f;
#pragma unroll
                for (int w = 0; w < 8; w++) v += part[w][j][l];
                if (scaled) v *= (float)Ldiag[s.cb_coef[k] + cc + (size_t)cc * st];
                Y[fc + cc + (size_t)(j0 + j) * ldy] = (T)v;
            }
        }
        __syncthreads();
    }
}

template <typename T, int RC>
__global__ void __cluster_dims__(TC, 1, 1) __launch_bounds__(256)
    k_bwd_diag_tinv_rr(DevStruct s, const int *__restrict__ list, int zside, int scaled, const T *Ldiag, T *Y, int ldy,
                    int nrhs, const float *__restrict__ tinv, const int64_t *__restrict__ ti_off) {
    __shared__ float xs[RC][384];
    pdl_trigger();
    const int k = list[blockIdx.x / TC];
    const int64_t off = ti_off[k];
    if (off < 0) return;  // the whole cluster leaves: k_bwd_diag_inv takes this cblk
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const int j0 = blockIdx.y * RC, nr = min(RC, nrhs - j0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_wait();
    for (int e = tid; e < nc * RC; e += blockDim.x) {
        const int i = e % nc, j = e / nc;
        float v = j < nr ? (float)Y[fc + i + (size_t)(j0 + j) * ldy] : 0.f;
        if (scaled) v *= (float)Ldiag[s.cb_coef[k] + i + (size_t)i * st];
        xs[j][i] = v;
    }
    cluster.sync();
    const float *Pt = tinv + off + (size_t)zside * nc * nc;
    // x_c = sum_{r >= c} Pt[r, c] xs[r]: four columns per warp, lanes over the rows (coalesced)
    for (int cb = rank * 32; cb < nc; cb += TC * 32) {
        const int c0 = cb + 4 * warp;
        float acc[4][RC];
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int j = 0; j < RC; j++) acc[u][j] = 0.f;
        for (int r = c0 + lane; r < nc; r += 32) {
            float pv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) pv[u] = (c0 + u < nc && r >= c0 + u) ? Pt[r + (size_t)(c0 + u) * nc] : 0.f;
#pragma unroll
            for (int j = 0; j < RC; j++) {
                const float xr = xs[j][r];
#pragma unroll
                for (int u = 0; u < 4; u++) acc[u][j] += pv[u] * xr;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int j = 0; j < RC; j++) {
                float v = acc[u][j];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0 && c0 + u < nc && j < nr) Y[fc + c0 + u + (size_t)(j0 + j) * ldy] = (T)v;
            }
    }
}

template <typename T, int RC>
__global__ void __cluster_dims__(TC, 1, 1) __launch_bounds__(256)
    k_bwd_diag_tinv(DevStruct s, const int *__restrict__ list, int zside, int scaled, const T *Ldiag, T *Y, int ldy,
                    int nrhs, const float *__restrict__ tinv, const int64_t *__restrict__ ti_off) {
    __shared__ float xs[RC][384];
    __shared__ float acc[RC][384];
    pdl_trigger();
    const int k = list[blockIdx.x / TC];
    const int64_t off = ti_off[k];
    if (off < 0) return;  // the whole cluster leaves: k_bwd_diag_inv takes this cblk
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const int j0 = blockIdx.y * RC, nr = min(RC, nrhs - j0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int npad = 32 * ((nc + 31) / 32);
    const float *Pt = tinv + off + (size_t)zside * nc * nc;
    // x_c = sum_{r >= c} Pt[r, c] xs[r]: tile (row block i, column block jc <= i), lanes over the rows
    const int nch = (nc + 31) / 32, ntile = nch * (nch + 1) / 2;
    int t = rank * 8 + warp, i = 0, jc = 0;
    float p[32];
    auto load = [&]() {
        tri_tile(t, i, jc);
        const int r = 32 * i + lane, c0 = 32 * jc;
#pragma unroll
        for (int u = 0; u < 32; u++)
            p[u] = (r < nc && c0 + u < nc && r >= c0 + u) ? Pt[r + (size_t)(c0 + u) * nc] : 0.f;
    };
    if (t < ntile) load();  // the inverse does not depend on the kernel ahead
    pdl_wait();
    for (int e = tid; e < npad * RC; e += blockDim.x) {
        const int i = e % npad, j = e / npad;
        float v = (j < nr && i < nc) ? (float)Y[fc + i + (size_t)(j0 + j) * ldy] : 0.f;
        if (scaled && i < nc) v *= (float)Ldiag[s.cb_coef[k] + i + (size_t)i * st];
        xs[j][i] = v;
        acc[j][i] = 0.f;
    }
    cluster.sync();
    while (t < ntile) {
        const int r = 32 * i + lane, c0 = 32 * jc;
        float *dst = cluster.map_shared_rank(&acc[0][0], jc % TC);
#pragma unroll
        for (int j = 0; j < RC; j++) {
            if (j >= nr) break;
            const float xr = r < nc ? xs[j][r] : 0.f;
            float v[32];
#pragma unroll
            for (int u = 0; u < 32; u++) v[u] = p[u] * xr;
            lane_sums32(v, lane);
            if (c0 + lane < nc) atomicAdd(dst + j * 384 + c0 + lane, v[0]);
        }
        t += TC * 8;
        if (t < ntile) load();
    }
    cluster.sync();  // every partial sum in place
    for (int cb = rank * 32; cb < nc; cb += TC * 32)
        for (int e = tid; e < 32 * RC; e += blockDim.x) {
            const int l = e & 31, j = e >> 5, c = cb + l;
            if (c < nc && j < nr) Y[fc + c + (size_t)(j0 + j) * ldy] = (T)acc[j][c];
        }
}

// Wide cblks without a kept full inverse (FP64 factors): the blocked solve with
// the inverted 32 x 32 sub-blocks, one CTA per cblk and right-hand-side group.
// Bound by latency: nc / 32 dependent steps, each a 32 x 32 product with Z and
// an update with a 32-column (forward) or 32-row (backward) strip of the block.
// Z and the strip of the next step are copied by cp.async into the second of
// two shared-memory stages while the current one is used, and the first two
// steps' copies are issued ahead of pdl_wait, so that no step waits for memory
// one element at a time.  Against a kernel whose steps loaded their own data:
// FP64 100^3 Laplacian, one RHS, all levels, forward 7.9 -> 2.7 ms and backward
// 3.9 -> 3.0 ms; 80^3, 16 RHS, 6.9 -> 3.0 and 11.2 -> 2.7 ms (events around
// every launch, B200); the whole 16-RHS solve with the update kernels below
// 24.6 -> 8.5 ms.
// One RHS: each warp forms the whole 32-vector yb (no barrier between the
// product with Z and the update).  Groups of 8: warp j forms column j; FP64
// applies the strip by DMMA (8 rows x 8 right-hand sides per fragment).
constexpr int SD_LDZ = 33;  // row stride of Z: lane-per-row and lane-per-column reads without bank conflicts
// Leading dimension of a forward strip of m rows: 4 mod 16, so that the DMMA
// fragment loads (4 columns x 4 rows per half warp) hit 16 different banks.
__host__ __device__ inline int sd_ldm(int m) { return ((m + 15) & ~15) + 4; }
// Backward strips hold 32 rows per column; rows are permuted by the column so
// that both a lane per column and the DMMA fragments are conflict-free.
__device__ __forceinline__ int sd_swz(int c, int r) { return 32 * c + (r ^ (4 * (c & 3) + ((c >> 2) & 3))); }
// Rows (columns) of a strip kept in shared memory: all of them up to widths of
// 384 columns; a wider cblk reads the rest of its strips from global memory.
__host__ __device__ inline long long sd_fixed_elems(int nc, int rc, bool scaled) {
    const int npad = (nc + 31) & ~31;
    return 2 * 32 * SD_LDZ + (long long)rc * npad + 8 * 32 + (rc > 1 ? 32 * rc : 0) + (scaled ? npad : 0);
}
constexpr long long SD_SMEM = 227 * 1024;
inline int sd_cap(int nc, int rc, bool scaled, int tsize) {
    const long long room = (SD_SMEM / tsize - sd_fixed_elems(nc, rc, scaled)) / 64 - 4;
    const int m = nc > 32 ? (nc - 1) & ~31 : 0;  // columns ahead of the last block: the longest backward strip
    return (int)(room < 16 ? 0 : (room < m ? room & ~15LL : m));
}
inline long long sd_smem_elems(int nc, int rc, bool scaled, int cap) {
    return sd_fixed_elems(nc, rc, scaled) + 2 * 32LL * sd_ldm(cap);
}
template <typename T>
__device__ __forceinline__ void cp_async_elem(T *smem, const T *gmem) {
    if (sizeof(T) == 8) cp_async8(smem, gmem, true);
    else cp_async4(smem, gmem, true);
}

template <typename T, int RC, bool FWD>
__global__ void __launch_bounds__(256) k_diag_inv(DevStruct s, const int *__restrict__ list, const T *P,
                                                  const T *__restrict__ dinv, int zside, int scaled, const T *Ldiag,
                                                  T *Y, int ldy, int nrhs, const float *__restrict__ tinv,
                                                  const int64_t *__restrict__ ti_off, int cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_trigger();
    const int k = list[blockIdx.x];
    if (tinv != nullptr && ti_off[k] >= 0) return;  // the kept full inverse is applied by k_*_diag_tinv
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const int j0 = blockIdx.y * RC, nr = min(RC, nrhs - j0);
    const T *D = P + s.cb_coef[k];
    const int nzb = (nc + 31) / 32, npad = 32 * nzb;
    const T *gZ = dinv + s.cb_dinv[k] + (size_t)(zside ? nzb : 0) * 1024;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ldm = sd_ldm(cap);
    const size_t stage_elems = 32 * SD_LDZ + 32 * (size_t)ldm;
    T *stage0 = reinterpret_cast<T *>(smem_raw);
    T *y = stage0 + 2 * stage_elems;  // npad x RC, a row's right-hand sides together
    T *yw = y + (size_t)RC * npad;    // RC == 1: one 32-vector per warp
    T *yb = yw + 8 * 32;              // RC > 1: 32 x RC
    T *ds = yb + (RC > 1 ? 32 * RC : 0);  // diagonal of D (scaled)
    // copies of step q (forward: block q; backward: block nzb - 1 - q) into stage q & 1
    auto prefetch = [&](int q) {
        if (q < nzb) {
            const int b = FWD ? q : nzb - 1 - q, jb = 32 * b;
            T *Zs = stage0 + (q & 1) * stage_elems, *Ds = Zs + 32 * SD_LDZ;
            for (int e = tid; e < 1024; e += 256) cp_async_elem(Zs + (e >> 5) * SD_LDZ + (e & 31), gZ + (size_t)b * 1024 + e);
            if (FWD) {  // rows below the block, one column of the block per warp
                const int m = min(cap, nc - jb - 32);
                for (int c = warp; c < 32; c += 8)
                    for (int r = lane; r < m; r += 32)
                        cp_async_elem(Ds + c * ldm + r, D + jb + 32 + r + (size_t)(jb + c) * st);
            } else {  // the block's rows in the columns ahead of it
                const int nb = min(32, nc - jb);
                for (int c = warp; c < min(cap, jb); c += 8)
                    if (lane < nb) cp_async_elem(Ds + sd_swz(c, lane), D + jb + lane + (size_t)c * st);
            }
        }
        cp_async_commit();
    };
    prefetch(0);
    prefetch(1);
    if (scaled)
        for (int i = tid; i < npad; i += 256) ds[i] = i < nc ? Ldiag[s.cb_coef[k] + i + (size_t)i * st] : T(0);
    pdl_wait();
    for (int j = 0; j < RC; j++)
        for (int i = tid; i < npad; i += 256)
            y[i * RC + j] = (i < nc && j < nr) ? Y[(fc + i) + (size_t)(j0 + j) * ldy] : T(0);
    for (int q = 0; q < nzb; q++) {
        const int b = FWD ? q : nzb - 1 - q, jb = 32 * b, nb = min(32, nc - jb);
        const T *Zs = stage0 + (q & 1) * stage_elems, *Ds = Zs + 32 * SD_LDZ;
        cp_async_wait<1>();
        __syncthreads();
        // the block's solution, column j by warp j (one RHS: by every warp): forward
        // S Z^T y, backward Z S x; Z is upper triangular
        const int jw = RC == 1 ? 0 : warp;
        T v0 = T(0), v1 = T(0), v2 = T(0), v3 = T(0);
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
            T yv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                yv[u] = y[(jb + c + u) * RC + jw];
                if (!FWD && scaled) yv[u] *= ds[jb + c + u];
            }
            const bool low = FWD;
            if (low ? (c + 0 <= lane) : (c + 0 >= lane && c + 0 < nb)) v0 += (FWD ? Zs[(c + 0) * SD_LDZ + lane] : Zs[lane * SD_LDZ + c + 0]) * yv[0];
            if (low ? (c + 1 <= lane) : (c + 1 >= lane && c + 1 < nb)) v1 += (FWD ? Zs[(c + 1) * SD_LDZ + lane] : Zs[lane * SD_LDZ + c + 1]) * yv[1];
            if (low ? (c + 2 <= lane) : (c + 2 >= lane && c + 2 < nb)) v2 += (FWD ? Zs[(c + 2) * SD_LDZ + lane] : Zs[lane * SD_LDZ + c + 2]) * yv[2];
            if (low ? (c + 3 <= lane) : (c + 3 >= lane && c + 3 < nb)) v3 += (FWD ? Zs[(c + 3) * SD_LDZ + lane] : Zs[lane * SD_LDZ + c + 3]) * yv[3];
        }
        T xv = (v0 + v1) + (v2 + v3);
        if (FWD && scaled) xv *= ds[jb + lane];
        if (lane >= nb) xv = T(0);
        const T *xb;
        if (RC == 1) {
            yw[32 * warp + lane] = xv;
            __syncwarp();
            xb = yw + 32 * warp;
            if (warp == 0 && lane < nb) Y[fc + jb + lane + (size_t)j0 * ldy] = xv;
        } else {
            yb[lane * RC + warp] = xv;
            if (warp < nr && lane < nb) Y[fc + jb + lane + (size_t)(j0 + warp) * ldy] = xv;
            __syncthreads();
            xb = yb;
        }
        // the strip's product with the block's solution, removed from the other rows
        const int m = FWD ? nc - jb - 32 : jb, r0 = FWD ? jb + 32 : 0;
        auto at = [&](int r, int c) -> T {
            if (!FWD && c >= nb) return T(0);  // rows past the end of a partial last block
            if (r < cap) return FWD ? Ds[c * ldm + r] : Ds[sd_swz(r, c)];
            return FWD ? D[r0 + r + (size_t)(jb + c) * st] : D[jb + c + (size_t)r * st];
        };
        if constexpr (RC > 1 && sizeof(T) == 8) {
            const int g = lane >> 2, t4 = lane & 3;
            double bf[8];
#pragma unroll
            for (int ks = 0; ks < 8; ks++) bf[ks] = (double)xb[(4 * ks + t4) * RC + g];
            for (int f = warp; 8 * f < m; f += 8) {
                const int r = 8 * f + g;
                double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
#pragma unroll
                for (int ks = 0; ks < 8; ks += 2) {
                    dmma884(a0[0], a0[1], r < m ? at(r, 4 * ks + t4) : 0.0, bf[ks]);
                    dmma884(a1[0], a1[1], r < m ? at(r, 4 * ks + 4 + t4) : 0.0, bf[ks + 1]);
                }
                if (r < m) {
                    y[(r0 + r) * RC + 2 * t4] -= (T)(a0[0] + a1[0]);
                    y[(r0 + r) * RC + 2 * t4 + 1] -= (T)(a0[1] + a1[1]);
                }
            }
        } else {
            for (int r = tid; r < m; r += 256) {
                T acc[RC], acd[RC];
#pragma unroll
                for (int j = 0; j < RC; j++) acc[j] = acd[j] = T(0);
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    const T p0 = at(r, c), p1 = at(r, c + 1);
#pragma unroll
                    for (int j = 0; j < RC; j++) {
                        acc[j] += p0 * xb[c * RC + j];
                        acd[j] += p1 * xb[(c + 1) * RC + j];
                    }
                }
#pragma unroll
                for (int j = 0; j < RC; j++) y[(r0 + r) * RC + j] -= acc[j] + acd[j];
            }
        }
        __syncthreads();  // the stage may be refilled, y is up to date
        prefetch(q + 2);
    }
}

// ---------------------------------------------------------------------------
// Off-diagonal products on 64 x 64 panel tiles (RowTile.r0 = first row, the
// tile's column block is blockIdx.z).  Forward: y[row(r)] -= P[r, cols] y_k[cols];
// backward: x_k[c] -= sum_r P[r, c] x[row(r)].  The panel tile and its row
// indices do not depend on the right-hand sides: they are loaded into registers
// ahead of pdl_wait, so that a level's panels stream in while the kernel ahead
// finishes.  A CTA applies its tile to `ng` groups of right-hand sides
// (blockIdx.y the first), so that a panel is read once for several groups.
// FP64 groups of 8 run on DMMA, the panel fragments in registers and 16 shared
// loads per thread (per-thread dot products needed 128): 80^3 Laplacian, 16 RHS,
// forward 3.4 -> 2.1 ms, backward 4.3 -> 2.2 ms per solve.
// ---------------------------------------------------------------------------
constexpr int ST_LDX = 12;  // right-hand sides per staged row: 12 keeps the DMMA B fragments conflict-free
template <typename T, int RC>
__global__ void __launch_bounds__(256) k_fwd_update(DevStruct s, const RowTile *__restrict__ tiles, const T *P,
                                                     T *Y, int ldy, int nrhs, int ng) {
    constexpr bool DM = RC > 1 && sizeof(T) == 8;
    constexpr int LDX = DM ? ST_LDX : RC;
    __shared__ __align__(16) T yk[ST_C * LDX];
    __shared__ __align__(16) T part[DM ? 1 : 4][DM ? 1 : ST_R * RC];
    pdl_trigger();
    const RowTile tl = tiles[blockIdx.x];
    const int k = tl.cblk;
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int c0 = blockIdx.z * ST_C;
    if (c0 >= nc) return;
    const int ncol = min(ST_C, nc - c0);
    const int st = s.cb_stride[k];
    const int rows = min(ST_R, st - tl.r0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const T *Pk = P + s.cb_coef[k] + tl.r0 + (size_t)c0 * st;
    const int *ridx = s.rowidx + s.cb_rowidx[k] + tl.r0;
    // FP64 groups of 8: DMMA fragments, warp w rows 8 w .. 8 w + 7; otherwise one row and 16 columns per thread
    const int g = lane >> 2, t4 = lane & 3;
    const int r = DM ? 8 * warp + g : tid % ST_R, q = tid / ST_R, cb = 16 * q;
    T p[16];
#pragma unroll
    for (int u = 0; u < 16; u++) {
        const int c = DM ? 4 * u + t4 : cb + u;
        p[u] = (r < rows && c < ncol) ? Pk[r + (size_t)c * st] : T(0);
    }
    const int gr = r < rows ? ridx[r] : 0;
    pdl_wait();
    for (int j0 = blockIdx.y * ng * RC; j0 < min(nrhs, (int)(blockIdx.y + 1) * ng * RC); j0 += RC) {
        const int nr = min(RC, nrhs - j0);
        for (int e = tid; e < ST_C * RC; e += 256) {
            const int c = e % ST_C, j = e / ST_C;
            yk[c * LDX + j] = (c < ncol && j < nr) ? Y[(fc + c0 + c) + (size_t)(j0 + j) * ldy] : T(0);
        }
        __syncthreads();
        if constexpr (DM) {
            double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
#pragma unroll
            for (int u = 0; u < 16; u += 2) {
                dmma884(a0[0], a0[1], p[u], yk[(4 * u + t4) * LDX + g]);
                dmma884(a1[0], a1[1], p[u + 1], yk[(4 * u + 4 + t4) * LDX + g]);
            }
            if (r < rows) {
                if (2 * t4 < nr) atomicAdd(&Y[gr + (size_t)(j0 + 2 * t4) * ldy], -(a0[0] + a1[0]));
                if (2 * t4 + 1 < nr) atomicAdd(&Y[gr + (size_t)(j0 + 2 * t4 + 1) * ldy], -(a0[1] + a1[1]));
            }
            __syncthreads();
        } else {
            T acc[RC];
#pragma unroll
            for (int j = 0; j < RC; j++) acc[j] = T(0);
#pragma unroll
            for (int u = 0; u < 16; u++)
#pragma unroll
                for (int j = 0; j < RC; j++) acc[j] += p[u] * yk[(cb + u) * LDX + j];
#pragma unroll
            for (int j = 0; j < RC; j++) part[q][r + j * ST_R] = acc[j];
            __syncthreads();
            for (int e = tid; e < ST_R * RC; e += 256) {  // e % ST_R = r for every e of this thread
                const int j = e / ST_R;
                if (r < rows && j < nr)
                    atomicAdd(&Y[gr + (size_t)(j0 + j) * ldy], -((part[0][e] + part[1][e]) + (part[2][e] + part[3][e])));
            }
        }
    }
}

template <typename T, int RC>
__global__ void __launch_bounds__(256) k_bwd_update(DevStruct s, const RowTile *__restrict__ tiles, const T *P,
                                                     T *Y, int ldy, int nrhs, int ng) {
    constexpr bool DM = RC > 1 && sizeof(T) == 8;
    constexpr int LDX = DM ? ST_LDX : RC;
    __shared__ __align__(16) T xr[ST_R * LDX];
    __shared__ T pt[DM ? 1 : ST_C * (ST_R + 1)];  // products (one RHS) or the transposed tile, row stride 65
    __shared__ T part[(!DM && RC > 1) ? 4 : 1][(!DM && RC > 1) ? ST_C * RC : 1];
    pdl_trigger();
    const RowTile tl = tiles[blockIdx.x];
    const int k = tl.cblk;
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int c0 = blockIdx.z * ST_C;
    if (c0 >= nc) return;
    const int ncol = min(ST_C, nc - c0);
    const int st = s.cb_stride[k];
    const int rows = min(ST_R, st - tl.r0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int *ridx = s.rowidx + s.cb_rowidx[k] + tl.r0;
    const T *Pk = P + s.cb_coef[k] + tl.r0 + (size_t)c0 * st;
    // FP64 groups of 8: DMMA fragments of the transposed tile, warp w columns 8 w .. 8 w + 7
    const int g = lane >> 2, t4 = lane & 3;
    const int r = tid % ST_R, q = tid / ST_R, cb = 16 * q;
    T p[16];
#pragma unroll
    for (int u = 0; u < 16; u++) {
        const int rr = DM ? 4 * u + t4 : r, c = DM ? 8 * warp + g : cb + u;
        p[u] = (rr < rows && c < ncol) ? Pk[rr + (size_t)c * st] : T(0);
    }
    const int gr = r < rows ? ridx[r] : 0;  // staging: rows e % ST_R = r for every e of this thread
    if constexpr (!DM && RC > 1) {
#pragma unroll
        for (int u = 0; u < 16; u++) pt[(cb + u) * (ST_R + 1) + r] = p[u];
    }
    pdl_wait();
    for (int j0 = blockIdx.y * ng * RC; j0 < min(nrhs, (int)(blockIdx.y + 1) * ng * RC); j0 += RC) {
        const int nr = min(RC, nrhs - j0);
        for (int e = tid; e < ST_R * RC; e += 256) {
            const int j = e / ST_R;
            xr[r * LDX + j] = (r < rows && j < nr) ? Y[gr + (size_t)(j0 + j) * ldy] : T(0);
        }
        __syncthreads();
        if constexpr (DM) {
            double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
#pragma unroll
            for (int u = 0; u < 16; u += 2) {
                dmma884(a0[0], a0[1], p[u], xr[(4 * u + t4) * LDX + g]);
                dmma884(a1[0], a1[1], p[u + 1], xr[(4 * u + 4 + t4) * LDX + g]);
            }
            const int c = 8 * warp + g;
            if (c < ncol) {
                T *yc = &Y[(fc + c0 + c) + (size_t)(j0 + 2 * t4) * ldy];
                if (2 * t4 < nr) atomicAdd(yc, -(a0[0] + a1[0]));
                if (2 * t4 + 1 < nr) atomicAdd(yc + ldy, -(a0[1] + a1[1]));
            }
            __syncthreads();
        } else if constexpr (RC == 1) {
            const T xv = xr[r];
#pragma unroll
            for (int u = 0; u < 16; u++) pt[(cb + u) * (ST_R + 1) + r] = p[u] * xv;
            __syncthreads();
            if (tid < ncol) {
                T v = T(0);
#pragma unroll 16
                for (int i = 0; i < ST_R; i++) v += pt[tid * (ST_R + 1) + i];
                atomicAdd(&Y[(fc + c0 + tid) + (size_t)j0 * ldy], -v);
            }
        } else {
            // out[c, j] = sum_r P[r, c] x[r, j]: column c = tid % 64, a quarter of the rows per thread
            T acc[RC];
#pragma unroll
            for (int j = 0; j < RC; j++) acc[j] = T(0);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const T pv = pt[r * (ST_R + 1) + 16 * q + i];
#pragma unroll
                for (int j = 0; j < RC; j++) acc[j] += pv * xr[(16 * q + i) * LDX + j];
            }
#pragma unroll
            for (int j = 0; j < RC; j++) part[q][r + j * ST_C] = acc[j];
            __syncthreads();
            for (int e = tid; e < ST_C * RC; e += 256) {
                const int j = e / ST_C;
                if (r < ncol && j < nr)
                    atomicAdd(&Y[(fc + c0 + r) + (size_t)(j0 + j) * ldy],
                              -((part[0][e] + part[1][e]) + (part[2][e] + part[3][e])));
            }
        }
    }
}

// Diagonal step of LDL^T: x_i /= D_i (solve_cblk_zdiag, kernels/solve_ztrsmsp.c:664).
template <typename T>
__global__ void k_diag_scale(DevStruct s, const T *L, T *Y, int ldy, int nrhs) {
    pdl_trigger();
    pdl_wait();
    const int k = blockIdx.x;
    const int fc = s.cb_fcol[k];
    const int nc = s.cb_lcol[k] - fc + 1;
    const int st = s.cb_stride[k];
    const T *D = L + s.cb_coef[k];
    for (int e = threadIdx.x; e < nc * nrhs; e += blockDim.x) {
        int i = e % nc, j = e / nc;
        Y[(fc + i) + (size_t)j * ldy] /= D[i + (size_t)i * st];
    }
}

// ------------------------------ launchers ---------------------------------
// Whether the diagonal kernels of a level's `count` narrow cblks apply their rows
// too: one right-hand side, and enough cblks that a warp each fills the SMs.
// The warp against the diagonal kernel and the update launch, FP64, us, forward and
// backward: 512^2 grid 512 cblks 10.7 | 13.2 and 11.0 | 12.1, 1024 8.1 | 13.2 and
// 10.8 | 13.3, 2048 6.4 | 15.9 and 9.4 | 18.8, 16385 35 | 85 and 53 | 123; 80^3
// Laplacian 2030 larger ones 19 | 38 and 30 | 46; 64 of the 512^2 grid's, larger
// still, 26 | 10 and 28 | 10.  The line lies at the smallest count that is clearly
// ahead both ways.
bool solve_fuse_rows(int count, int nrhs) { return nrhs == 1 && count >= 1024; }
// One right-hand side or groups of 8 (a group's missing columns are masked).
template <typename T>
void launch_fwd_diag(const DevStruct &s, const int *list, int count, int maxnc, const T *P, int unit, T *Y, int ldy,
                     int nrhs, cudaStream_t st) {
    if (count <= 0) return;
    if (nrhs == 1)  // narrow cblks (width <= 64): one warp each
        launch_k(k_fwd_diag_w<T>, dim3((count + 7) / 8), dim3(256), 0, st, s, list, count, P, unit, Y,
                 (int)solve_fuse_rows(count, nrhs));
    else
        launch_k(k_fwd_diag<T, 8>, dim3(count, (nrhs + 7) / 8), dim3(256), 8 * (size_t)maxnc * sizeof(T), st, s, list, P,
                 unit, Y, ldy, nrhs);
}
template <typename T>
void launch_bwd_diag(const DevStruct &s, const int *list, int count, int maxnc, const T *P, int unit, T *Y, int ldy,
                     int nrhs, cudaStream_t st) {
    if (count <= 0) return;
    if (nrhs == 1)
        launch_k(k_bwd_diag_w<T>, dim3((count + 7) / 8), dim3(256), 0, st, s, list, count, P, unit, Y,
                 (int)solve_fuse_rows(count, nrhs));
    else
        launch_k(k_bwd_diag<T, 8>, dim3(count, (nrhs + 7) / 8), dim3(256), 8 * (size_t)maxnc * sizeof(T), st, s, list, P,
                 unit, Y, ldy, nrhs);
}
// ntinv: how many cblks of the list have a kept full inverse (FP32 factors);
// those go to the 8-CTA cluster kernels, the rest to the blocked kernels, and
// a kernel with no cblk of its own is not launched.
template <typename T, bool FWD>
static void launch_diag_inv(const DevStruct &s, const int *list, int count, int maxnc, const T *P, const T *dinv,
                            int zside, int scaled, const T *Ld, T *Y, int ldy, int nrhs, const float *tinv,
                            const int64_t *ti_off, int ntinv, cudaStream_t st) {
    if (count <= 0) return;
    if (tinv == nullptr) ntinv = 0;
    const int ng = (nrhs + 7) / 8;
    if (ntinv > 0) {
        if (nrhs == 1)
            launch_k(FWD ? k_fwd_diag_tinv<T, 1> : k_bwd_diag_tinv<T, 1>, dim3(count * TC), dim3(256), 0, st, s, list,
                     zside, scaled, Ld, Y, ldy, nrhs, tinv, ti_off);
        else
            launch_k(FWD ? k_fwd_diag_tinv_rr<T, 8> : k_bwd_diag_tinv_rr<T, 8>, dim3(count * TC, ng), dim3(256), 0, st,
                     s, list, zside, scaled, Ld, Y, ldy, nrhs, tinv, ti_off);
    }
    if (ntinv < count) {
        const int rc = nrhs == 1 ? 1 : 8, cap = sd_cap(maxnc, rc, scaled != 0, (int)sizeof(T));
        const size_t smem = (size_t)sd_smem_elems(maxnc, rc, scaled != 0, cap) * sizeof(T);
        if (nrhs == 1)
            launch_k(k_diag_inv<T, 1, FWD>, dim3(count), dim3(256), smem, st, s, list, P, dinv, zside, scaled, Ld, Y, ldy,
                     nrhs, tinv, ti_off, cap);
        else
            launch_k(k_diag_inv<T, 8, FWD>, dim3(count, ng), dim3(256), smem, st, s, list, P, dinv, zside, scaled, Ld, Y,
                     ldy, nrhs, tinv, ti_off, cap);
    }
}
template <typename T>
void launch_fwd_diag_inv(const DevStruct &s, const int *list, int count, int maxnc, const T *P, const T *dinv,
                         int zside, int scaled, const T *Ld, T *Y, int ldy, int nrhs, const float *tinv,
                         const int64_t *ti_off, int ntinv, cudaStream_t st) {
    launch_diag_inv<T, true>(s, list, count, maxnc, P, dinv, zside, scaled, Ld, Y, ldy, nrhs, tinv, ti_off, ntinv, st);
}
template <typename T>
void launch_bwd_diag_inv(const DevStruct &s, const int *list, int count, int maxnc, const T *P, const T *dinv,
                         int zside, int scaled, const T *Ld, T *Y, int ldy, int nrhs, const float *tinv,
                         const int64_t *ti_off, int ntinv, cudaStream_t st) {
    launch_diag_inv<T, false>(s, list, count, maxnc, P, dinv, zside, scaled, Ld, Y, ldy, nrhs, tinv, ti_off, ntinv, st);
}
// Right-hand-side groups per CTA of the update kernels: all of them once the
// tiles alone give every SM its eight resident CTAs (a panel is then read once
// for all right-hand sides), one otherwise (the groups fill the SMs instead).
static int update_groups(long long ctas, int nrhs) {
    const int groups = (nrhs + 7) / 8;
    return ctas >= 8LL * 148 ? groups : 1;
}
template <typename T>
void launch_fwd_update(const DevStruct &s, const RowTile *tiles, int count, int maxnc, const T *P, T *Y, int ldy,
                       int nrhs, cudaStream_t st) {
    if (count <= 0) return;
    const int nz = (maxnc + ST_C - 1) / ST_C;
    const int ng = update_groups((long long)count * nz, nrhs), gy = ((nrhs + 7) / 8 + ng - 1) / ng;
    if (nrhs == 1) launch_k(k_fwd_update<T, 1>, dim3(count, 1, nz), dim3(256), 0, st, s, tiles, P, Y, ldy, nrhs, 1);
    else launch_k(k_fwd_update<T, 8>, dim3(count, gy, nz), dim3(256), 0, st, s, tiles, P, Y, ldy, nrhs, ng);
}
template <typename T>
void launch_bwd_update(const DevStruct &s, const RowTile *tiles, int count, int maxnc, const T *P, T *Y, int ldy,
                       int nrhs, cudaStream_t st) {
    if (count <= 0) return;
    const int nz = (maxnc + ST_C - 1) / ST_C;
    const int ng = update_groups((long long)count * nz, nrhs), gy = ((nrhs + 7) / 8 + ng - 1) / ng;
    if (nrhs == 1) launch_k(k_bwd_update<T, 1>, dim3(count, 1, nz), dim3(256), 0, st, s, tiles, P, Y, ldy, nrhs, 1);
    else launch_k(k_bwd_update<T, 8>, dim3(count, gy, nz), dim3(256), 0, st, s, tiles, P, Y, ldy, nrhs, ng);
}
template <typename T>
void launch_diag_scale(const DevStruct &s, int cblknbr, const T *L, T *Y, int ldy, int nrhs, cudaStream_t st) {
    if (cblknbr <= 0) return;
    launch_k(k_diag_scale<T>, dim3(cblknbr), dim3(128), 0, st, s, L, Y, ldy, nrhs);
}
// Shared-memory opt-in of the solve kernels on the current device.
template <typename T>
static cudaError_t solve_attrs_of() {
    cudaError_t e = cudaSuccess;
    for (auto k : {k_diag_inv<T, 1, true>, k_diag_inv<T, 1, false>, k_diag_inv<T, 8, true>, k_diag_inv<T, 8, false>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SD_SMEM);
    return e;
}
cudaError_t set_solve_attrs() {
    const cudaError_t e = solve_attrs_of<double>();
    return e == cudaSuccess ? solve_attrs_of<float>() : e;
}
int solve_rows_per_tile() { return ST_R; }

#define PGPU_INST_SOLVE(T)                                                                                       \
    template void launch_fwd_diag<T>(const DevStruct &, const int *, int, int, const T *, int, T *, int, int,     \
                                     cudaStream_t);                                                              \
    template void launch_bwd_diag<T>(const DevStruct &, const int *, int, int, const T *, int, T *, int, int,     \
                                     cudaStream_t);                                                              \
    template void launch_fwd_diag_inv<T>(const DevStruct &, const int *, int, int, const T *, const T *, int,     \
                                         int, const T *, T *, int, int, const float *, const int64_t *, int,     \
                                         cudaStream_t);                                                          \
    template void launch_bwd_diag_inv<T>(const DevStruct &, const int *, int, int, const T *, const T *, int,     \
                                         int, const T *, T *, int, int, const float *, const int64_t *, int,     \
                                         cudaStream_t);                                                          \
    template void launch_fwd_update<T>(const DevStruct &, const RowTile *, int, int, const T *, T *, int, int,    \
                                       cudaStream_t);                                                            \
    template void launch_bwd_update<T>(const DevStruct &, const RowTile *, int, int, const T *, T *, int, int,    \
                                       cudaStream_t);                                                            \
    template void launch_diag_scale<T>(const DevStruct &, int, const T *, T *, int, int, cudaStream_t);

PGPU_INST_SOLVE(double)
PGPU_INST_SOLVE(float)

}  // namespace pgpu
