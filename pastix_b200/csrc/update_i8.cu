// FP64 updates on the 5th-generation tensor cores through exact integer slices
// (tcgen05.mma kind::i8, 32-bit integer accumulators in tensor memory).
//
// The product C -= A B^T of an update task is formed from fixed-point operands
// (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms
// 59, 2012, with a common exponent per row): k_split_i8 scales every panel row
// by a power of two, rounds it to 63 fractional bits below the row's largest
// entry and cuts the integer into eight signed 8-bit digits (balanced base
// 256).  Products of digits and their sums over up to I8_MAX_K columns are
// exact in 32 bits; the digit products i, j with i + j <= 7 are kept (36 of
// 64).  What is lost, with a and b the scales of the two rows (the powers of two
// above their largest entries):
//   entries smaller than 2^-10 a are rounded at 2^-64 a, the others are exact;
//   the dropped digit products come to about 2^-60 a b for 128 columns of equal
//   size (at most 2^-61 a b for each column); the sums i + j >= 4 are rounded at
//   2^-60 a b, and the whole sum once to FP64.
// So the error is bounded against a b, not against the sum of the |a_c b_c| that
// bounds FP64 accumulation: for Cholesky a b <= 4 sqrt(A_ii A_jj), the bound that
// its FP64 rounding has, with 2^-60 in place of K 2^-53.  Rows with a non-finite
// entry carry a NaN scale, so that it reaches the target.
// Measured against the factor in 64-bit mantissas (full 520 x 520 kernel matrix
// with shuffled rows, panels of 64): FP64 on DMMA 3.3e-14, here 1.8e-14; seven
// digits with the low sums rounded at 2^-51 a b gave 2.4e-13.
// Rounding relative to the row's largest entry asks for columns of like size:
// the rows of a Cholesky factor are bounded by the diagonal of A, those of L in
// LDL^T and LU are not (a small pivot makes a large column).  There column c is
// scaled by h_c = 2^(half the exponent of the pivot), exactly: (L h)(L D / h)^T
// and (L h)(U / h), the balance that Cholesky has.  LDL^T keeps the bound with
// f_i = sum_c |l_ic d_c l_ic|, which bounds its FP64 rounding at (i, i), in place of
// A_ii: a^2 <= 16 f_i by construction.  In LU that holds only while L and U share
// their scaling; a matrix with rows or columns scaled on one side does not.  So
// k_split_i8 checks every row: the squares of its largest entries in L h and U / h
// are at most I8_OVER = 64 times max(|A_ii|, f_i), f_i = sum_c |l_ic u_ci|.  The error at
// (i, j) is then at most 2^-52 sqrt(g_i g_j) (g: that maximum).  A source with a row that fails (or with one beyond the range of the
// scales, or not finite) is flagged and updated by DMMA instead
// (launch_update_flagged), whose FP64 products such scalings leave unchanged.
// Flagged, of the 132 sources of a 32^3 convection-diffusion: none, nor with 30 to 80 %
// of the off-diagonal entries dropped at random or scaled over 8 decades each; 6 with
// one direction's cut to 10^-8; 129 with every other row and column in other units
// (2^40, 2^30).
//
// Why: the FP64 tensor cores (DMMA) multiply 64 x 2 flops per clock and SM, the
// 8-bit ones 8192 x 2; 36 digit products per FP64 product are 3.6 times fewer
// tensor-core cycles.  Rates measured are given at k_update_i8.
//
// Image of cblk k (bytes from i8_off[k]): digit p (0 the leading one), K block
// kb of 32 columns, row group g of 8 panel rows at ((p * nkb + kb) * ng + g) *
// I8_GROUP; inside a group the two 8 x 16-byte core matrices of the tensor
// cores' K-major, no-swizzle layout.  ng = ceil(stride / 8) + 16, so that a
// window of 16 row groups from any group of the panel stays inside the image.
#include "device.cuh"
#include "tcgen05.cuh"

#include <climits>

namespace pgpu {

constexpr int I8_S = 8;                    // digits
constexpr int I8_BITS = 8 * I8_S - 1;      // fractional bits below a row's largest entry
constexpr int I8_KB = 32;                  // columns per K block (one MMA step)
constexpr int I8_GROUP = 256;              // bytes of 8 rows x 32 columns of one digit
constexpr int I8_PIECE = 16 * I8_GROUP;    // one digit of a 128-row operand block
constexpr int I8_STAGE = 2 * I8_S * I8_PIECE;
constexpr int I8_STAGES = 3;
constexpr size_t I8_SMEM = (size_t)I8_STAGES * I8_STAGE;
constexpr int I8_THREADS = 320;            // 8 epilogue warps, producer, MMA issuer
constexpr int I8_EPI = 256;
constexpr int I8_BN = 128;
constexpr int I8_TQ = 4;                   // tile-index ring
constexpr int FAR_TILES_I8 = 6;            // tiles of a CTA of the far updates, about 80 us: 60^3 Laplacian,
                                           // factorization 15.7 -> 13.9 ms against one stream (far_grid)
constexpr double I8_OVER = 64.0;           // LU: bound on the square of a row's largest entry over its diagonal's scale
constexpr int I8_MAX_K = 512;              // widest source: the sums i + j >= 4 stay within 2^50

__host__ __device__ inline int i8_nkb(int nc) { return (nc + I8_KB - 1) / I8_KB; }
__host__ __device__ inline int i8_ng(int st) { return (st + 7) / 8 + 16; }

int far_grid(int count, int quota);  // factor.cu

long long i8_image_bytes(int nc, int st) { return (long long)I8_S * i8_nkb(nc) * i8_ng(st) * I8_GROUP; }
int i8_max_k() { return I8_MAX_K; }

// ---------------------------------------------------------------------------
// Digits of 32-row slabs (blockIdx.y) of 128-row panel slabs, of both operands
// (LDL^T: L h and L D / h; LU: L h and U / h).  A lane holds a row; the warps
// share its 16-column chunks.  The first pass finds the row's largest magnitudes
// and for LU the sum_c |l_c u_c|, the second (the slab is in L1 / L2 by then)
// writes the digits, 16 bytes per digit and chunk.  Bound by HBM: 8 bytes read
// and 8 written per entry.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double i8_pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

template <int FACT>
__global__ void __launch_bounds__(256) k_split_i8(DevStruct s, const SplitSlab *__restrict__ slabs, const double *L,
                                                  const double *U, const int64_t *__restrict__ i8_off,
                                                  unsigned char *img0, unsigned char *img1, double *__restrict__ sc0,
                                                  double *__restrict__ sc1, const double *__restrict__ val,
                                                  const int *__restrict__ diag_pos, int *flag, int *level_flag,
                                                  int *flagged) {
    constexpr int SIDES = FACT == FACT_POTRF ? 1 : 2;
    constexpr bool LU = FACT == FACT_GETRF;
    __shared__ double red[SIDES][8][32], fsum[LU ? 8 : 1][32];
    __shared__ int badw[8][32];
    __shared__ double colf[SIDES][I8_MAX_K];
    const SplitSlab sl = slabs[blockIdx.x];
    const int k = sl.cblk;
    const int nc = s.cb_lcol[k] - s.cb_fcol[k] + 1;
    const int st = s.cb_stride[k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pr = sl.r0 + 32 * blockIdx.y + lane;
    if (sl.r0 + 32 * (int)blockIdx.y >= st) return;  // whole CTA
    const int nkb = i8_nkb(nc), ng = i8_ng(st), nch = 2 * nkb;
    const double *AL = L + s.cb_coef[k] + pr, *AU = LU ? U + s.cb_coef[k] + pr : AL;
    auto load = [&](int side, int ch, double (&v)[16]) {
        const double *A = side ? AU : AL;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int c = 16 * ch + j;
            v[j] = (pr < st && c < nc) ? A[(size_t)c * st] : 0.0;
        }
        if (FACT != FACT_POTRF) {
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const int c = 16 * ch + j;
                if (c < nc) v[j] *= colf[side][c];
            }
        }
    };
    if (FACT != FACT_POTRF) {
        for (int c = threadIdx.x; c < nc; c += 256) {
            const double d = L[s.cb_coef[k] + c + (size_t)c * st];
            const int e = (__double2hiint(d) >> 20) & 0x7ff;
            const int h = (e == 0 || e == 0x7ff) ? 0 : (e - 1023) / 2;  // zero and non-finite pivots: none
            colf[0][c] = i8_pow2(h);
            colf[SIDES - 1][c] = LU ? i8_pow2(-h) : d * i8_pow2(-h);
        }
        __syncthreads();
    }
    double m[SIDES], f = 0.0;
    int bad = 0;
#pragma unroll
    for (int q = 0; q < SIDES; q++) m[q] = 0.0;
    for (int ch = warp; ch < nch; ch += 8) {
        double v[SIDES][16];
#pragma unroll
        for (int q = 0; q < SIDES; q++) load(q, ch, v[q]);
#pragma unroll
        for (int j = 0; j < 16; j++) {
#pragma unroll
            for (int q = 0; q < SIDES; q++) {
                const double a = fabs(v[q][j]);
                m[q] = a > m[q] ? a : m[q];
                bad |= !(a <= 1.7976931348623157e308) << q;
            }
            if (LU) f += fabs(v[0][j] * v[SIDES - 1][j]);
        }
    }
#pragma unroll
    for (int q = 0; q < SIDES; q++) red[q][warp][lane] = m[q];
    badw[warp][lane] = bad;
    if (LU) fsum[warp][lane] = f;
    __syncthreads();
    f = 0.0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
#pragma unroll
        for (int q = 0; q < SIDES; q++) m[q] = red[q][w][lane] > m[q] ? red[q][w][lane] : m[q];
        bad |= badw[w][lane];
        if (LU) f += fsum[w][lane];
    }
    if (LU && warp == 0) {
        // rows that the integer products cannot take: see the head of this file.  A
        // scaled entry that left the range of FP64 is among them (bad), and so is a
        // non-finite one, which DMMA carries on.
        const bool off = pr >= nc && pr < st;
        const int dp = off ? diag_pos[s.rowidx[s.cb_rowidx[k] + pr]] : -1;
        const double aii = dp >= 0 ? fabs(val[dp]) : 0.0, g = I8_OVER * (aii > f ? aii : f);
        auto fits = [&](double x) { return x == 0.0 || (x >= 0x1p-500 && x <= 0x1p500 && x * x <= g); };
        const bool fails = bad || !fits(m[0]) || !fits(m[SIDES - 1]);
        if (__any_sync(0xffffffffu, off && fails) && lane == 0) {
            *level_flag = 1;
            if (atomicExch(flag + k, 1) == 0) atomicAdd(flagged, 1);
        }
    }
#pragma unroll
    for (int q = 0; q < SIDES; q++) {
        // row exponent: |a| < 127.375 / 128 * 2^ex, so that the leading digit fits 8
        // bits after the carries of the balanced digits (at most 0.502 of it)
        const bool nan = (bad >> q) & 1;
        const int mhi = __double2hiint(m[q]);
        int ex = ((mhi >> 20) & 0x7ff) - 1022;
        if ((mhi & 0xfffff) >= 0xfd800) ex++;  // mantissa of 2 * 127.375 / 128
        if (ex < -958) ex = -958;              // smaller rows: rounded at 2^-1021, as subnormal numbers are
        const double mult = nan ? 0.0 : i8_pow2(I8_BITS - ex);
        if (warp == 0 && pr < st)
            (q ? sc1 : sc0)[s.cb_rowidx[k] + pr] = nan ? __longlong_as_double(0x7ff8000000000000LL) : i8_pow2(ex - 19);
        if (pr >= 8 * ((st + 7) / 8)) continue;
        unsigned char *out = (q ? img1 : img0) + i8_off[k] + (size_t)(pr >> 3) * I8_GROUP + (pr & 7) * 16;
        for (int ch = warp; ch < nch; ch += 8) {
            double v[16];
            load(q, ch, v);
            uint32_t w[I8_S][4];
#pragma unroll
            for (int g = 0; g < 4; g++) {
                uint32_t lo[4], hi[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const long long i = nan ? 0 : __double2ll_rn(v[4 * g + j] * mult);
                    const unsigned long long t = (unsigned long long)i + 0x80808080808080ULL;
                    lo[j] = (uint32_t)t;
                    hi[j] = (uint32_t)(t >> 32);
                }
                // byte b of the four values, by 4 x 4 byte transposes
                const uint32_t l01a = __byte_perm(lo[0], lo[1], 0x5140), l23a = __byte_perm(lo[2], lo[3], 0x5140);
                const uint32_t l01b = __byte_perm(lo[0], lo[1], 0x7362), l23b = __byte_perm(lo[2], lo[3], 0x7362);
                const uint32_t h01a = __byte_perm(hi[0], hi[1], 0x5140), h23a = __byte_perm(hi[2], hi[3], 0x5140);
                const uint32_t h01b = __byte_perm(hi[0], hi[1], 0x7362), h23b = __byte_perm(hi[2], hi[3], 0x7362);
                w[7][g] = __byte_perm(l01a, l23a, 0x5410) ^ 0x80808080u;
                w[6][g] = __byte_perm(l01a, l23a, 0x7632) ^ 0x80808080u;
                w[5][g] = __byte_perm(l01b, l23b, 0x5410) ^ 0x80808080u;
                w[4][g] = __byte_perm(l01b, l23b, 0x7632) ^ 0x80808080u;
                w[3][g] = __byte_perm(h01a, h23a, 0x5410) ^ 0x80808080u;
                w[2][g] = __byte_perm(h01a, h23a, 0x7632) ^ 0x80808080u;
                w[1][g] = __byte_perm(h01b, h23b, 0x5410) ^ 0x80808080u;
                w[0][g] = __byte_perm(h01b, h23b, 0x7632);
            }
            unsigned char *o = out + (size_t)(ch >> 1) * ng * I8_GROUP + (ch & 1) * 128;
#pragma unroll
            for (int p = 0; p < I8_S; p++)
                *reinterpret_cast<uint4 *>(o + (size_t)p * nkb * ng * I8_GROUP) =
                    make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
        }
    }
}

// ---------------------------------------------------------------------------
// The tile kernel: persistent, warp specialized, tiles from a device work queue
// as in the FP32 engine.  128 x 128 tiles; the eight digit sums d = i + j do not
// fit the 512 tensor-memory columns at once, so that a tile takes two passes
// over K: first d = 4..7 (26 digit products, eight digits of each operand), kept
// by the epilogue threads as 40-bit integers, then d = 0..3 (10 products, four
// digits), added and scattered into the facing panel.  N = 128 rather than 64
// with all sums resident: at N = 64 the tensor cores read shared memory faster
// than it delivers (192 bytes a clock).
// 100^3 Laplacian, B200, all updates of an FP64 factorization: 264 ms on DMMA
// (k_update_dmma, 23 Tflop/s), 118 ms here (52 Tflop/s; 112 with seven digits).
// 80^3: 33.8 ms.  Bounds there, with seven digits (whole kernel 31.8): copies
// alone 22.9 ms (L2 to shared memory, 35 bytes a clock and SM), products and
// hand-offs alone 22.2 (tensor pipe 14.3), both without epilogue 24.0.
// Slower: 16 or 8 epilogue warps that release the accumulators before
// they scatter (33.1, 37.2: the registers spill), one polling lane per warp (34.7).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t i8_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(I8_GROUP >> 4) << 32) |
           (1ull << 46);
}
// S8 x S8 -> S32, both operands K-major, M = 128, N = n
__device__ __forceinline__ uint32_t i8_idesc(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void i8_mma(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
// The four digit sums of 8 columns, a[d] = accumulator d: sum of a[d] 2^(24 - 8 d)
__device__ __forceinline__ void i8_load4(uint32_t taddr, long long (&z)[8]) {
    int a[4][8];
#pragma unroll
    for (int d = 0; d < 4; d++) tmem_ld8(taddr + I8_BN * d, a[d]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; j++)
        z[j] = (((long long)a[0][j] * 256 + a[1][j]) << 16) + ((long long)a[2][j] * 256 + a[3][j]);
}
__device__ __forceinline__ int i8_bar_or(int pred) {  // OR over the epilogue threads, which it also orders
    int r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.red.or.pred q, 1, 256, p;\n\t"
        "selp.b32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"(pred)
        : "memory");
    return r;
}

template <int FACT>
__global__ void __launch_bounds__(I8_THREADS, 1)
    k_update_i8(DevStruct s, const UpdTile *__restrict__ tiles, int count, int quota, double *L, double *U,
                const unsigned char *img0, const unsigned char *img1, const double *__restrict__ sc0,
                const double *__restrict__ sc1, const int64_t *__restrict__ i8_off, const int *flag,
                const int *level_flag, int *queue, int *status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[I8_STAGES], empty[I8_STAGES], tfull, tempty, tq_full[I8_TQ], tq_empty[I8_TQ];
    __shared__ __align__(8) uint64_t drained;
    __shared__ uint32_t tmem_sh;
    __shared__ int ctab[2][I8_BN];
    __shared__ double csc[2][I8_BN];
    __shared__ int tq[I8_TQ];
    if (*(volatile int *)status != 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(4 * I8_BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < I8_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&tfull, 1);
        mbar_init(&tempty, I8_EPI);
        mbar_init(&drained, 1);
        for (int i = 0; i < I8_TQ; i++) {
            mbar_init(&tq_full[i], 1);
            mbar_init(&tq_empty[i], 1 + I8_EPI);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_sh;
    int late = 0;
    uint32_t g = 0;  // producer, MMA issuer: K blocks so far
    if (warp == 8) {
        if (lane == 0) {  // producer: claims tiles, loads their operands
            int next = atomicAdd(queue, 1);  // claimed one tile ahead
            // LU: tiles of flagged sources are left to DMMA
            const bool any = FACT == FACT_GETRF && *level_flag != 0;
            auto skipped = [&](int t) { return any && t < count && flag[s.tasks[tiles[t].task].src] != 0; };
            for (int j = 0; !late; j++) {
                const int slot = j % I8_TQ;
                if (j >= I8_TQ && !mbar_wait(&tq_empty[slot], ((j / I8_TQ) - 1) & 1)) {
                    late = 1;
                    break;
                }
                int t = j < quota ? next : count;  // `quota`: tiles of this CTA
                while (skipped(t)) t = atomicAdd(queue, 1);
                if (t >= count) t = -1;
                else if (j + 1 < quota) next = atomicAdd(queue, 1);
                tq[slot] = t;
                mbar_arrive(&tq_full[slot]);
                if (t < 0) break;
                const UpdTile tl = tiles[t];
                const TaskDev tk = s.tasks[tl.task];
                const int k = tk.src, K = s.cb_lcol[k] - s.cb_fcol[k] + 1, st = s.cb_stride[k];
                const int nkb = i8_nkb(K), ng = i8_ng(st);
                const int ga = ((tk.row0 + (tl.side ? tk.n : 0)) >> 3) + 16 * tl.mt, gb = (tk.row0 >> 3) + 16 * tl.nt;
                const int nmma = (min(I8_BN, tk.row0 + tk.n - 8 * gb) + 15) & ~15;
                const bool swap = (FACT == FACT_GETRF && tl.side == 1);
                const unsigned char *iA = (swap ? img1 : img0) + i8_off[k];
                const unsigned char *iB = ((FACT == FACT_POTRF) ? img0 : (swap ? img0 : img1)) + i8_off[k];
                const size_t digit = (size_t)nkb * ng * I8_GROUP;
                const uint32_t bbytes = (uint32_t)(nmma / 8) * I8_GROUP;
                for (int pass = 0; pass < 2 && !late; pass++) {
                    const int nd = pass ? 4 : I8_S;
                    for (int kb = 0; kb < nkb; kb++, g++) {
                        const int sidx = g % I8_STAGES;
                        if (g >= I8_STAGES && !mbar_wait(&empty[sidx], ((g / I8_STAGES) - 1) & 1)) {
                            late = 1;
                            break;
                        }
                        unsigned char *sp = smem_raw + (size_t)sidx * I8_STAGE;
                        mbar_expect_tx(&full[sidx], (uint32_t)nd * (I8_PIECE + bbytes));
                        for (int p = 0; p < nd; p++) {
                            bulk_g2s(sp + p * I8_PIECE, iA + p * digit + ((size_t)kb * ng + ga) * I8_GROUP, I8_PIECE,
                                     &full[sidx]);
                            bulk_g2s(sp + (I8_S + p) * I8_PIECE, iB + p * digit + ((size_t)kb * ng + gb) * I8_GROUP,
                                     bbytes, &full[sidx]);
                        }
                    }
                }
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {  // MMA issuer
            const uint32_t sbase = smem_u32(smem_raw);
            uint32_t ph = 0;
            for (int i = 0; !late; i++) {
                const int slot = i % I8_TQ;
                if (!mbar_wait(&tq_full[slot], (i / I8_TQ) & 1)) {
                    late = 1;
                    break;
                }
                const int t = tq[slot];
                mbar_arrive(&tq_empty[slot]);
                if (t < 0) break;
                const UpdTile tl = tiles[t];
                const TaskDev tk = s.tasks[tl.task];
                const int nkb = i8_nkb(s.cb_lcol[tk.src] - s.cb_fcol[tk.src] + 1);
                const int gb = (tk.row0 >> 3) + 16 * tl.nt;
                const uint32_t idesc = i8_idesc((min(I8_BN, tk.row0 + tk.n - 8 * gb) + 15) & ~15);
                for (int pass = 0; pass < 2 && !late; pass++, ph++) {
                    if (ph > 0 && !mbar_wait(&tempty, (ph - 1) & 1)) {  // accumulators drained
                        late = 1;
                        break;
                    }
                    tc_fence_after();
                    for (int kb = 0; kb < nkb; kb++, g++) {
                        const int sidx = g % I8_STAGES;
                        if (!mbar_wait(&full[sidx], (g / I8_STAGES) & 1)) {
                            late = 1;
                            break;
                        }
                        tc_fence_after();
                        const uint64_t da = i8_desc(sbase + sidx * I8_STAGE);
                        const uint64_t db = i8_desc(sbase + sidx * I8_STAGE + I8_S * I8_PIECE);
                        if (pass == 0) {
#pragma unroll
                            for (int d = 4; d < 8; d++)
#pragma unroll
                                for (int p = 0; p <= d; p++)
                                    i8_mma(tmem + I8_BN * (d - 4), da + p * (I8_PIECE >> 4), db + (d - p) * (I8_PIECE >> 4),
                                           idesc, kb > 0 || p > 0);
                        } else {
#pragma unroll
                            for (int d = 0; d < 4; d++)
#pragma unroll
                                for (int p = 0; p <= d; p++)
                                    i8_mma(tmem + I8_BN * d, da + p * (I8_PIECE >> 4), db + (d - p) * (I8_PIECE >> 4), idesc,
                                           kb > 0 || p > 0);
                        }
                        tc_commit(&empty[sidx]);
                    }
                    if (!late) tc_commit(&tfull);
                }
            }
        }
    } else {  // epilogue: warps w and w + 4 share 32 tile rows, 64 columns each
        const int row = 32 * (warp & 3) + lane, cbase = 64 * (warp >> 2);
        uint32_t ph = 0;
        for (int i = 0;; i++) {
            const int slot = i % I8_TQ;
            if (i8_bar_or(!mbar_wait(&tq_full[slot], (i / I8_TQ) & 1))) {
                late = 1;
                break;
            }
            const int t = tq[slot];
            mbar_arrive(&tq_empty[slot]);
            if (t < 0) break;
            const UpdTile tl = tiles[t];
            const TaskDev tk = s.tasks[tl.task];
            const int k = tk.src, f = tk.dst, b = i & 1;
            const bool swap = (FACT == FACT_GETRF && tl.side == 1);
            const double *scA = (swap ? sc1 : sc0) + s.cb_rowidx[k];
            const double *scB = ((FACT == FACT_POTRF) ? sc0 : (swap ? sc0 : sc1)) + s.cb_rowidx[k];
            const int *ridx = s.rowidx + s.cb_rowidx[k];
            const int ra = tk.row0 + (tl.side ? tk.n : 0);
            const int pr = 8 * ((ra >> 3) + 16 * tl.mt) + row, gb = (tk.row0 >> 3) + 16 * tl.nt;
            const int nmma = (min(I8_BN, tk.row0 + tk.n - 8 * gb) + 15) & ~15;
            if (tid < I8_BN) {  // target columns and their scales
                const int pc = 8 * gb + tid;
                const bool in = pc >= tk.row0 && pc < tk.row0 + tk.n;
                ctab[b][tid] = in ? ridx[pc] - s.cb_fcol[f] : -1;
                csc[b][tid] = in ? scB[pc] : 0.0;
            }
            int rr = -1;  // target row in the facing panel
            double rs = 0.0;
            if (pr >= ra && pr < tk.row0 + tk.m) {
                const int g = ridx[pr];
                int lo = s.cb_fblok[f], hi = s.cb_fblok[f + 1] - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (s.bk_frow[mid] <= g) lo = mid;
                    else hi = mid - 1;
                }
                rr = s.bk_rowoff[lo] + (g - s.bk_frow[lo]);
                rs = -scA[pr];
            }
            const uint32_t taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)cbase;
            if (i8_bar_or(!mbar_wait(&tfull, ph & 1))) {
                late = 1;
                break;
            }
            tc_fence_after();
            ph++;
            // the sums d = 4..7 in units of 2^11 of the last digit's, 40 bits: upper 32 and lower 8
            int low[64];
            uint32_t lob[16];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                if (cbase + 8 * q < nmma) {
                    long long z[8];
                    i8_load4(taddr + 8 * q, z);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const long long r = (z[j] + (1 << 10)) >> 11;
                        low[8 * q + j] = (int)(r >> 8);
                        uint32_t &w = lob[2 * q + (j >> 2)];
                        w = (j & 3) ? w | ((uint32_t)r & 255u) << 8 * (j & 3) : (uint32_t)r & 255u;
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(&tempty);
            if (i8_bar_or(!mbar_wait(&tfull, ph & 1))) {
                late = 1;
                break;
            }
            tc_fence_after();
            ph++;
            double *Cp = (swap ? U : L) + s.cb_coef[f] + (rr >= 0 ? rr : 0);
            const int stf = s.cb_stride[f];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                if (cbase + 8 * q < nmma) {
                    long long z[8];
                    i8_load4(taddr + 8 * q, z);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        // both integers to FP64 exactly (|z| < 2^51) by the offset of their magic exponents
                        const double h = __longlong_as_double(z[j] + 0x4338000000000000LL) - 6755399441055744.0;
                        const long long r = (long long)low[8 * q + j] * 256 + ((lob[2 * q + (j >> 2)] >> 8 * (j & 3)) & 255u);
                        const double l = __longlong_as_double(r + 0x4338000000000000LL) - 6755399441055744.0;
                        const int cc = ctab[b][cbase + 8 * q + j];
                        const double v = fma(l, 0x1p-21, h) * (rs * csc[b][cbase + 8 * q + j]);
                        if (rr >= 0 && cc >= 0) atomicAdd(Cp + (size_t)cc * stf, v);
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(&tempty);
        }
    }
    __syncwarp();
    const int aborted = __syncthreads_or(late);
    if (aborted) {  // nothing of this CTA may be in flight when it ends
        if (tid == 0) atomicExch(status, PGPU_STATUS_TIMEOUT);
        if (warp == 8 && lane == 0) drain_loads(full, I8_STAGES, g);
        if (warp == 9 && lane == 0) drain_mmas(&drained);
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(4 * I8_BN));
}

// ---------------------------------------------------------------------------
template <int FACT>
void launch_split_i8(const DevStruct &s, const SplitSlab *slabs, int count, const double *L, const double *U,
                     const int64_t *i8_off, unsigned char *img0, unsigned char *img1, double *sc0, double *sc1,
                     const double *val, const int *diag_pos, int *flag, int *level_flag, int *flagged,
                     cudaStream_t st) {
    if (count <= 0) return;
    k_split_i8<FACT><<<dim3(count, 4), 256, 0, st>>>(s, slabs, L, U, i8_off, img0, img1, sc0, sc1, val, diag_pos, flag,
                                                     level_flag, flagged);
}
template <int FACT>
void launch_update_i8(const DevStruct &s, const UpdTile *tiles, int count, double *L, double *U,
                      const unsigned char *img0, const unsigned char *img1, const double *sc0, const double *sc1,
                      const int64_t *i8_off, const int *flag, const int *level_flag, int *queue, int *status, bool far,
                      cudaStream_t st) {
    if (count <= 0) return;
    const int quota = far ? FAR_TILES_I8 : INT_MAX;
    k_update_i8<FACT><<<far_grid(count, quota), I8_THREADS, I8_SMEM, st>>>(s, tiles, count, quota, L, U, img0, img1, sc0,
                                                                           sc1, i8_off, flag, level_flag, queue, status);
}
cudaError_t set_i8_attrs() {
    cudaError_t e = cudaSuccess;
    for (auto k : {k_update_i8<FACT_POTRF>, k_update_i8<FACT_SYTRF>, k_update_i8<FACT_GETRF>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)I8_SMEM);
    return e;
}
#define PGPU_INST_I8(F)                                                                                               \
    template void launch_split_i8<F>(const DevStruct &, const SplitSlab *, int, const double *, const double *,       \
                                     const int64_t *, unsigned char *, unsigned char *, double *, double *,           \
                                     const double *, const int *, int *, int *, int *, cudaStream_t);                 \
    template void launch_update_i8<F>(const DevStruct &, const UpdTile *, int, double *, double *,                    \
                                      const unsigned char *, const unsigned char *, const double *, const double *,   \
                                      const int64_t *, const int *, const int *, int *, int *, bool, cudaStream_t);
PGPU_INST_I8(FACT_POTRF)
PGPU_INST_I8(FACT_SYTRF)
PGPU_INST_I8(FACT_GETRF)

}  // namespace pgpu
