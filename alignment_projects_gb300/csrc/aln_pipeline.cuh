// aln_pipeline.cuh -- the batched CorrPatches kernels built on the
// register-resident FFT (aln_fft_reg.cuh).  Included by aln_corr.cu, after
// the device helpers (load_px, sat slots, lag rows, r_int, best_merge).
//
//   k3_sat    per 32-column band: warp-local column prefix sums of v, v^2,
//             (v != 0) at the needed rows, per-warp offsets, column totals
//   k3_satp   the same for 8-bit pairs whose sums pack into 64 bits, in bands
//             of 64 columns copied to shared memory asynchronously
//   k2_sat2w  per needed row: add the warp offset, x-prefix -> SAT row; the
//             column totals -> mu
//   k2_rowfft<L>   rows: (v - mu), zero pad, real FFT of length 2L, [kx][y]
//   k2_corrcol<Ny> per column kx: FFT of b's column (or the cached spectrum),
//             FFT of a's column, X2 * conj(X1), inverse FFT, the window's
//             lag rows -> Q[kx][j].  Nothing else leaves the SM.
//   k2_corrseg<NS> the same with the column cut into segments of a's rows
//             (CorrPatches): per segment two NS-point FFTs and the product,
//             summed per column, one inverse
//   k2_lagrow<L>   per lag row: inverse real FFT -> the lag image
//   k2_lagscan     per lag row: r per lag, row argmax
//   k2_imgscan     the same for CorrImagesR (bounded in FP32, FP64 where it counts)
//   k2_lagimg / k2_lagss / k2_lagp2i, k_final_img / k_makef / k_fpeak / k_final_p2i:
//             the CorrImages and CorrPatchToImage ends of the pipeline
#pragma once

#include "aln_fft_reg.cuh"
#include "aln_row_layout.cuh"

__device__ __forceinline__ bool int_pixels(int dt) { return dt == ALN_U8 || dt == ALN_U16; }

// The table pointer as if new: the next transform loads its twiddles again.
// Without it the compiler kept up to 60 registers of them from one transform
// to the next of the radix-16 column kernels and spilled as much (k2_corrcol
// 2.38 -> 2.13 ms and k2_corrseg 1.30 -> 1.16 ms per 3000 uneven pairs,
// k2_corrcol of the coarse scan of 48 thumbnail pairs 7.83 -> 7.22 ms; the
// radix-8 segments ran 2 % slower with it).
__device__ __forceinline__ void fresh(const float2 *__restrict__ &tw)
{
    asm volatile("" : "+l"(tw));
}

// Loads of what an earlier kernel of the chain wrote (grid_dep) and this one
// only reads: coherent, which __ldg is not, but free to move, where a plain load
// waits for the stores before it.  Their addresses come out of the job's
// descriptor, which is read after the wait.
__device__ __forceinline__ float ld_chain(const float *a)
{
    float v;
    asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(a));
    return v;
}
__device__ __forceinline__ double2 ld_chain(const double2 *a)
{
    double2 v;
    asm("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(a));
    return v;
}
__device__ __forceinline__ longlong2 ld_chain(const longlong2 *a)
{
    longlong2 v;
    asm("ld.global.v2.s64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(a));
    return v;
}
__device__ __forceinline__ ulonglong2 ld_chain(const ulonglong2 *a)
{
    ulonglong2 v;
    asm("ld.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(a));
    return v;
}

// asynchronous copies, global -> shared without registers
__device__ __forceinline__ void cp_async8(void *dst_shared, const void *src_global)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_shared);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src_global) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// s + e += x with the rounding error of the sum kept in e (Knuth's TwoSum;
// explicit round-to-nearest operations, so nothing is contracted or reordered)
__device__ __forceinline__ void two_sum_acc(float &s, float &e, float x)
{
    const float t = __fadd_rn(s, x);
    const float bp = __fsub_rn(t, s);
    const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(x, bp));
    e = __fadd_rn(e, err);
    s = t;
}

// Column prefix sums of v, v^2 and (v != 0) at the rows the lag window needs
// (IntegrateImage's sums, 0_GEN/Correlation.cpp:49-105, restricted to the
// rows IntegralTable will read).  The count table is written for every job
// (zeros without a count rule): skipping its stores changed this walk's
// code and made it 1.7x slower on the montage strips.  grid (ceil(w/32),
// 2*npairs), block (32, SAT_WARPS): each CTA owns 32 columns of one image;
// warp ty owns the rows of segment ty (sat_seg_start) and walks them once, storing its
// local column prefix at the needed rows.  The warps' exclusive offsets per
// column go to segoff[ty][c]; k2_sat2w adds them.  Exact int64 for 8/16-bit
// pixels, FP64 otherwise.  Also writes the column totals (mean shift).
#define SAT_WARPS 16

// Row segments of the column walk, balanced by work: a row costs 1, a row
// the lag window needs (stored) costs 1 + sat_need_cost, and segment g holds
// the rows whose cost position falls in [g, g + 1) * total / SAT_WARPS.  The
// needed rows sit at both ends of the image, so for uint8 pixels equal row
// counts left the first and last warps of a CTA twice as long as the rest,
// which waited at the CTA barrier (stall "barrier" 8.0 per issue on the
// montage strips; weight 2: k3_sat 4.19 -> 3.83 ms per step).  Wider pixels
// sum in 64 bits, so a stored row costs relatively less: weight 2 made the
// uint16 uneven batch's k3_sat 20 % slower, and they keep equal row counts.
// k3_sat and k2_sat2w compute the same map.  A segment spans at most
// 3 h / 16 rows (cost <= 3 h).
__device__ __forceinline__ int sat_need_cost(const PairDev &p, int i)
{
    return p.dt[i] == ALN_U8 ? 2 : 0;
}

__device__ __forceinline__ int sat_cost(const PairDev &p, int i, int y)
{
    const int k = sat_need_cost(p, i);
    int c = y;
    const int lo0 = p.need_lo[i][0], hi0 = p.need_hi[i][0];
    const int lo1 = p.need_lo[i][1], hi1 = p.need_hi[i][1];
    if (hi0 >= lo0)
        c += k * min(max(y - lo0, 0), hi0 - lo0 + 1);
    if (hi1 >= lo1)
        c += k * min(max(y - lo1, 0), hi1 - lo1 + 1);
    return c;
}

// segment of row y (0 <= y < h)
__device__ __forceinline__ int sat_seg_of(const PairDev &p, int i, int y)
{
    const long long total = sat_cost(p, i, p.h[i]);
    return (int)((long long)sat_cost(p, i, y) * SAT_WARPS / max(total, 1LL));
}

// first row of segment g (g = SAT_WARPS: h): the least y with
// cost(y) * SAT_WARPS >= g * total.  need_rows() makes the two needed
// intervals disjoint and ordered (or the second empty), so cost is linear
// with slope 1 before, between and after them and 1 + k inside them, and
// the least y with cost(y) >= C follows piece by piece.  (A binary search
// here -- some 14 dependent steps per warp -- cost the uneven batch's small
// images a fifth of their walk.)
__device__ __forceinline__ int sat_seg_start(const PairDev &p, int i, int g)
{
    const int h = p.h[i], k = sat_need_cost(p, i);
    const long long total = sat_cost(p, i, h);
    const int C = (int)(((long long)g * total + SAT_WARPS - 1) / SAT_WARPS);
    int y;
    if (k == 0) {
        y = C;
    } else {
        const int lo0 = p.need_lo[i][0], lo1 = p.need_lo[i][1];
        const int len0 = max(0, p.need_hi[i][0] - lo0 + 1);
        const int len1 = max(0, p.need_hi[i][1] - lo1 + 1);
        const int k1 = k + 1;
        if (len0 == 0 || C <= lo0)
            y = C;   // (len0 == 0: no needed row at all)
        else if (C <= lo0 + k1 * len0)
            y = lo0 + (C - lo0 + k) / k1;
        else if (len1 == 0 || C <= lo1 + k * len0)
            y = C - k * len0;
        else if (C <= lo1 + k * len0 + k1 * len1)
            y = lo1 + (C - lo1 - k * len0 + k) / k1;
        else
            y = C - k * (len0 + len1);
    }
    return min(max(y, 0), h);
}

// Accumulator of a warp's segment-local sums: 32-bit for uint8 pixels (a
// segment is at most 1536 rows -- h <= 8192 -- so the sums of v and v^2 stay
// below 2^27), the table type otherwise.
// a table entry: (sum v, sum v^2)
template <typename TA>
struct SatPair;
template <>
struct SatPair<long long> {
    typedef longlong2 type;
    __device__ __forceinline__ static longlong2 of(long long s, long long q)
    {
        return make_longlong2(s, q);
    }
};
template <>
struct SatPair<double> {
    typedef double2 type;
    __device__ __forceinline__ static double2 of(double s, double q) { return make_double2(s, q); }
};

template <typename TA, typename PIX>
struct SatAcc {
    typedef TA type;
};
template <>
struct SatAcc<long long, uint8_t> {
    typedef unsigned type;
};

template <typename TA, typename PIX, bool SQ = true>
__device__ __forceinline__ void sat_cols(const PairDev &p, int i, TA *shS, TA *shQ, int *shN)
{
    typedef typename SatAcc<TA, PIX>::type AC;
    const int w = p.w[i];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int c = blockIdx.x * 32 + tx;
    const bool cok = c < w;
    const int y0 = sat_seg_start(p, i, ty), y1 = sat_seg_start(p, i, ty + 1);
    const PIX *img = (const PIX *)p.img[i];
    const long long st = p.stride[i];
    const int lo0 = p.need_lo[i][0], hi0 = p.need_hi[i][0];
    const int lo1 = p.need_lo[i][1], hi1 = p.need_hi[i][1];
    const int len0 = hi0 - lo0 + 1;
    const bool want_n = p.cnt_kind == ALN_CNT_GT;
    typename SatPair<TA>::type *__restrict__ S = (typename SatPair<TA>::type *)p.sat[i];
    int *__restrict__ N = p.satN[i];
    AC s = 0, q = 0;
    int n = 0;
    if (cok) {
        const PIX *__restrict__ col = img + c;
        // walk [y0, y1) as store-free runs (loads batch freely) separated by
        // the needed rows, where the running prefix is stored
        int y = y0;
        while (y < y1) {
            int stop = y1;   // next needed row at or after y
            if (hi0 >= lo0 && hi0 >= y)
                stop = min(stop, max(lo0, y));
            if (hi1 >= lo1 && hi1 >= y)
                stop = min(stop, max(lo1, y));
#pragma unroll 8
            for (; y < stop; ++y) {
                const AC v = (AC)__ldg(&col[y * st]);
                if (SQ) {
                    s += v;
                    q += v * v;
                }
                if (want_n)
                    n += (v != 0);
            }
            if (y >= y1)
                break;
            // needed run: rows y .. end of its interval (within the warp's rows)
            const bool first = y >= lo0 && y <= hi0;
            const int rend = min(y1 - 1, first ? hi0 : hi1);
            const long long base = first ? (long long)(y - lo0) : (long long)(len0 + y - lo1);
            for (long long o = base * p.sp[i] + c; y <= rend; ++y, o += p.sp[i]) {
                const AC v = (AC)__ldg(&col[y * st]);
                if (SQ) {
                    s += v;
                    q += v * v;
                    S[o] = SatPair<TA>::of((TA)s, (TA)q);
                }
                if (want_n)
                    n += (v != 0);
                N[o] = n;
            }
        }
    }
    shS[ty * 32 + tx] = (TA)s;
    shQ[ty * 32 + tx] = (TA)q;
    shN[ty * 32 + tx] = n;
    __syncthreads();
    if (!cok)
        return;
    TA os = 0, oq = 0;
    int on = 0;
    for (int g = 0; g < ty; ++g) {
        os += shS[g * 32 + tx];
        oq += shQ[g * 32 + tx];
        on += shN[g * 32 + tx];
    }
    if (SQ) {
        ((typename SatPair<TA>::type *)p.seg[i])[ty * p.sp[i] + c] = SatPair<TA>::of(os, oq);
        if (ty == SAT_WARPS - 1)
            p.colsum[i][c] = (double)(os + (TA)s);
    }
    p.segN[i][ty * p.sp[i] + c] = on;
}

// The walk for packed tables (uint8): two columns per thread, 64 per CTA.
// Each warp copies its rows to shared memory SATP_ROWS at a time with
// asynchronous 16-byte copies, the next block's in flight while this one is
// summed: the walk through registers kept 16 rows of 64 bytes per warp in
// flight and waited on them (stall "long scoreboard" 13.6 per issue, 23 % of
// issue slots).  Four rows at a time are turned into one word per column and
// summed by dot products: about 2 instructions per pixel where the general
// walk takes 5, and a stored row is one 16-byte store per thread of whole
// sectors.
#define SATP_ROWS 32
#define SATP_PITCH 80   // 64 bytes of a row in 16-byte blocks, any start

__host__ __device__ constexpr int satp_smem() { return SAT_WARPS * 2 * SATP_ROWS * SATP_PITCH; }

__device__ __forceinline__ void cp_async16(unsigned dst_shared, const void *src_global)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_shared), "l"(src_global)
                 : "memory");
}

template <bool COUNT>
__device__ __forceinline__ void sat_cols_packed(const PairDev &p, int i, unsigned char *stage,
                                                unsigned long long *shP, int *shN)
{
    typedef unsigned long long u64;
    const int w = p.w[i], h = p.h[i], sp = p.sp[i];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int c0 = blockIdx.x * 64, c = c0 + 2 * tx;
    const bool cok = c < w, two = c + 1 < w;
    const int y0 = sat_seg_start(p, i, ty), y1 = sat_seg_start(p, i, ty + 1);
    const long long st = p.stride[i];
    const unsigned char *band = (const unsigned char *)p.img[i] + c0;
    const int nb = min(64, w - c0);   // bytes of the band's rows
    const int lo0 = p.need_lo[i][0], hi0 = p.need_hi[i][0];
    const int lo1 = p.need_lo[i][1], hi1 = p.need_hi[i][1];
    const int len0 = hi0 - lo0 + 1;
    u64 *__restrict__ S = (u64 *)p.sat[i];
    int *__restrict__ N = p.satN[i];
    unsigned s0 = 0, s1 = 0, q0 = 0, q1 = 0;
    int n0 = 0, n1 = 0;
    unsigned char *mine = stage + ty * (2 * SATP_ROWS * SATP_PITCH);
    const unsigned mine_s = (unsigned)__cvta_generic_to_shared(mine);
    // rows [y, y + SATP_ROWS) of the segment -> buffer b, each from the 16-byte
    // boundary at or below its first byte (a block that holds a byte of the row
    // never leaves the row's allocation)
    auto fetch = [&](int y, int b) {
        const int rows = min(SATP_ROWS, y1 - y);
        for (int e = tx; e < 5 * rows; e += 32) {
            const int r = e / 5, k = e - 5 * r;
            const unsigned char *a = band + (y + r) * st;
            const int off = (int)((uintptr_t)a & 15);
            if (16 * k < off + nb)
                cp_async16(mine_s + (b * SATP_ROWS + r) * SATP_PITCH + 16 * k, a - off + 16 * k);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (y0 < y1)
        fetch(y0, 0);
    int buf = 0;
    for (int yb = y0; yb < y1; yb += SATP_ROWS, buf ^= 1) {
        if (yb + SATP_ROWS < y1) {
            fetch(yb + SATP_ROWS, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        const unsigned char *src = mine + buf * SATP_ROWS * SATP_PITCH;
        // the bytes of columns c, c + 1 in row y of the block
        auto load2 = [&](int y) -> unsigned {
            const unsigned at = ((unsigned)(uintptr_t)band + (unsigned)(y * st) & 15u) + 2 * tx;
            const unsigned odd = at & 1u;
            const unsigned short *b =
                (const unsigned short *)(src + (y - yb) * SATP_PITCH + (at - odd));
            const unsigned lo = b[0], hi = odd && two ? (unsigned)b[1] : 0u;
            return (lo | hi << 16) >> (8 * odd);
        };
        const int ye = min(y1, yb + SATP_ROWS);
        int y = cok ? yb : ye;
        while (y < ye) {
            int stop = ye;   // next needed row at or after y
            if (hi0 >= lo0 && hi0 >= y)
                stop = min(stop, max(lo0, y));
            if (hi1 >= lo1 && hi1 >= y)
                stop = min(stop, max(lo1, y));
#pragma unroll 2
            for (; y + 4 <= stop; y += 4) {
                const unsigned r0 = load2(y), r1 = load2(y + 1), r2 = load2(y + 2),
                               r3 = load2(y + 3);
                const unsigned a = __byte_perm(r0, r1, 0x5140), b = __byte_perm(r2, r3, 0x5140);
                const unsigned t0 = __byte_perm(a, b, 0x5410), t1 = __byte_perm(a, b, 0x7632);
                s0 = __dp4a(t0, 0x01010101u, s0);
                s1 = __dp4a(t1, 0x01010101u, s1);
                q0 = __dp4a(t0, t0, q0);
                q1 = __dp4a(t1, t1, q1);
                if (COUNT) {
                    n0 += __popc(__vcmpne4(t0, 0u)) >> 3;
                    n1 += __popc(__vcmpne4(t1, 0u)) >> 3;
                }
            }
            for (; y < stop; ++y) {
                const unsigned v = load2(y), a = v & 0xffu, b = v >> 8 & 0xffu;
                s0 += a;
                s1 += b;
                q0 += a * a;
                q1 += b * b;
                if (COUNT) {
                    n0 += a != 0;
                    n1 += b != 0;
                }
            }
            if (y >= ye)
                break;
            // needed run: rows y .. end of its interval (within the block)
            const bool first = y >= lo0 && y <= hi0;
            const int rend = min(ye - 1, first ? hi0 : hi1);
            const long long base = first ? (long long)(y - lo0) : (long long)(len0 + y - lo1);
#pragma unroll 4
            for (long long o = base * sp + c; y <= rend; ++y, o += sp) {
                const unsigned v = load2(y), a = v & 0xffu, b = v >> 8 & 0xffu;
                s0 += a;
                s1 += b;
                q0 += a * a;
                q1 += b * b;
                // sums of u = v - 128 over the m rows so far
                const int m = y - y0 + 1;
                ulonglong2 e;
                e.x = sat_pack((int)s0 - 128 * m, q0 - 256u * s0 + 16384u * m);
                e.y = sat_pack((int)s1 - 128 * m, q1 - 256u * s1 + 16384u * m);
                *(ulonglong2 *)(S + o) = e;   // sp is even: aligned, inside the row
                if (COUNT) {
                    n0 += a != 0;
                    n1 += b != 0;
                    *(int2 *)(N + o) = make_int2(n0, n1);
                }
            }
        }
        __syncwarp();   // this buffer is copied into again two blocks on
    }
    const int m = y1 - y0;
    shP[ty * 64 + 2 * tx] = sat_pack((int)s0 - 128 * m, q0 - 256u * s0 + 16384u * m);
    shP[ty * 64 + 2 * tx + 1] = sat_pack((int)s1 - 128 * m, q1 - 256u * s1 + 16384u * m);
    if (COUNT) {
        shN[ty * 64 + 2 * tx] = n0;
        shN[ty * 64 + 2 * tx + 1] = n1;
    }
    __syncthreads();
    if (!cok)
        return;
    ulonglong2 os = make_ulonglong2(0, 0);
    int2 on = make_int2(0, 0);
    for (int g = 0; g < ty; ++g) {
        os.x += shP[g * 64 + 2 * tx];
        os.y += shP[g * 64 + 2 * tx + 1];
        if (COUNT) {
            on.x += shN[g * 64 + 2 * tx];
            on.y += shN[g * 64 + 2 * tx + 1];
        }
    }
    *(ulonglong2 *)((u64 *)p.seg[i] + (long long)ty * sp + c) = os;
    if (COUNT)
        *(int2 *)(p.segN[i] + (long long)ty * sp + c) = on;
    if (ty == SAT_WARPS - 1) {   // column totals of v
        p.colsum[i][c] =
            (double)(sat_pack_s(os.x + shP[ty * 64 + 2 * tx]) + 128 * h);
        if (two)
            p.colsum[i][c + 1] =
                (double)(sat_pack_s(os.y + shP[ty * 64 + 2 * tx + 1]) + 128 * h);
    }
}

// The jobs with packed tables: grid (ceil(max w / 64), 2 * npairs), satp_smem()
// bytes of dynamic shared memory.
__global__ void __launch_bounds__(32 * SAT_WARPS, 2) k3_satp(PairDev *pairs)
{
    grid_dep();
    extern __shared__ __align__(16) unsigned char satp_stage[];
    __shared__ unsigned long long shP[64 * SAT_WARPS];
    __shared__ int shN[64 * SAT_WARPS];
    const PairDev &p = pairs[blockIdx.y >> 1];
    const int i = blockIdx.y & 1;
    if (p.status != 0 || !p.sat_packed || blockIdx.x * 64 >= p.w[i])
        return;
    if (p.cnt_kind == ALN_CNT_GT)
        sat_cols_packed<true>(p, i, satp_stage, shP, shN);
    else
        sat_cols_packed<false>(p, i, satp_stage, shP, shN);
}

__global__ void k3_sat(PairDev *pairs)
{
    grid_dep();
    __shared__ long long shS[32 * SAT_WARPS], shQ[32 * SAT_WARPS];
    __shared__ int shN[32 * SAT_WARPS];
    const PairDev &p = pairs[blockIdx.y >> 1];
    const int i = blockIdx.y & 1;
    if (p.status != 0 || p.sat_packed || blockIdx.x * 32 >= p.w[i] || (i == 1 && p.sat_shared))
        return;
    if (p.sat_nonly) {   // counts only (CorrImagesS without a mincor)
        if (p.cnt_kind != ALN_CNT_GT)
            return;
        switch (p.dt[i]) {
        case ALN_U8: sat_cols<long long, uint8_t, false>(p, i, shS, shQ, shN); break;
        case ALN_U16: sat_cols<long long, uint16_t, false>(p, i, shS, shQ, shN); break;
        case ALN_F32: sat_cols<double, float, false>(p, i, (double *)shS, (double *)shQ, shN); break;
        default: sat_cols<double, double, false>(p, i, (double *)shS, (double *)shQ, shN); break;
        }
        return;
    }
    switch (p.dt[i]) {
    case ALN_U8:
        sat_cols<long long, uint8_t>(p, i, shS, shQ, shN);
        break;
    case ALN_U16:
        sat_cols<long long, uint16_t>(p, i, shS, shQ, shN);
        break;
    case ALN_F32:
        sat_cols<double, float>(p, i, (double *)shS, (double *)shQ, shN);
        break;
    default:
        sat_cols<double, double>(p, i, (double *)shS, (double *)shQ, shN);
        break;
    }
}

// ---------------------------------------------------------------------------
// transposed copies of wide images (jobs solved in the transposed frame)
// ---------------------------------------------------------------------------

__device__ __forceinline__ unsigned long long load_bits(const char *p, int es, long long idx)
{
    switch (es) {
    case 1: return ((const uint8_t *)p)[idx];
    case 2: return ((const uint16_t *)p)[idx];
    case 4: return ((const uint32_t *)p)[idx];
    default: return ((const unsigned long long *)p)[idx];
    }
}

__device__ __forceinline__ void store_bits(char *p, int es, long long idx, unsigned long long v)
{
    switch (es) {
    case 1: ((uint8_t *)p)[idx] = (uint8_t)v; break;
    case 2: ((uint16_t *)p)[idx] = (uint16_t)v; break;
    case 4: ((uint32_t *)p)[idx] = (uint32_t)v; break;
    default: ((unsigned long long *)p)[idx] = v; break;
    }
}

// grid (ceil(max caller w / (32 TR_TILES)), ceil(max caller h / 32),
// 2*npairs), block (32, 8): frame pixel (xf, yf) = caller pixel (yf, xf).
// uint8 images use 32 x 128 tiles (blockIdx.x then counts 128 TR_TILES
// columns; a launch whose transposed images are all uint8 has grid x =
// ceil(max caller w / (128 TR_TILES))).  Each CTA moves TR_TILES tiles side
// by side: a 4 KB tile per CTA left the montage strips' transposes bound by
// block scheduling (hundreds of thousands of CTAs per step).
#define TR_TILES 4
#define TR_WORDS (3 * 296 + 9 * 32)   // words of a turned uint8 tile
__global__ void __launch_bounds__(256) k_transpose(PairDev *pairs)
{
    grid_dep();
    __shared__ __align__(16) unsigned long long tile[37][32];
    static_assert(sizeof tile >= 2 * TR_WORDS * 4 && sizeof tile >= 32 * 33 * 8, "tile buffers");
    PairDev &p = pairs[blockIdx.z >> 1];
    const int i = blockIdx.z & 1;
    if (p.status != 0 || !p.transposed)
        return;
    const int sw = p.h[i], sh = p.w[i];   // caller's width and height
    const int y0 = blockIdx.y * 32;
    if (y0 >= sh)
        return;
    const int es = p.dt[i] == ALN_U8 ? 1 : p.dt[i] == ALN_U16 ? 2 : p.dt[i] == ALN_F32 ? 4 : 8;
    const char *src = (const char *)p.src_img[i];
    const long long sst = p.src_stride[i];
    if (es == 1) {
        // uint8: 32 x 128 tiles, a 4 x 4 block per thread: four words (of four
        // rows) turned in registers into four (of four columns), which change
        // threads through shared memory so that eight threads store a column's
        // 32 bytes.  All the tiles' words are loaded first.  (Byte by byte out
        // of shared memory, a tile's loads after the last one's stores, 4096
        // strips took 1.61 ms, now 1.12.)
        unsigned *turned = (unsigned *)tile;   // two buffers of TR_WORDS
        unsigned char *dst = (unsigned char *)p.img[i];
        const long long dstr = p.stride[i];
        const int c = threadIdx.x, g = threadIdx.y;   // columns 4c.., rows 4g..
        // 4-byte loads where the caller's rows allow them (4-byte aligned
        // base and stride, the whole word inside the row)
        const bool vec = (((uintptr_t)src | (uintptr_t)sst) & 3) == 0;
        unsigned wd[TR_TILES][4];
#pragma unroll
        for (int kt = 0; kt < TR_TILES; ++kt) {
            const int xq = (blockIdx.x * TR_TILES + kt) * 128 + 4 * c;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int yy = y0 + 4 * g + m;
                unsigned v = 0;
                if (yy < sh && xq < sw) {
                    const unsigned char *a = (const unsigned char *)src + yy * sst + xq;
                    if (vec && xq + 3 < sw)
                        v = __ldg((const unsigned *)a);
                    else
                        for (int k = 0; k < 4 && xq + k < sw; ++k)
                            v |= (unsigned)a[k] << (8 * k);
                }
                wd[kt][m] = v;
            }
        }
#pragma unroll
        for (int kt = 0; kt < TR_TILES; ++kt) {
            const int xb0 = (blockIdx.x * TR_TILES + kt) * 128;
            if (xb0 >= sw)
                break;   // uniform over the CTA
            unsigned *t = turned + (kt & 1) * TR_WORDS;
            const unsigned a = __byte_perm(wd[kt][0], wd[kt][1], 0x5140);
            const unsigned b = __byte_perm(wd[kt][2], wd[kt][3], 0x5140);
            const unsigned d = __byte_perm(wd[kt][0], wd[kt][1], 0x7362);
            const unsigned e = __byte_perm(wd[kt][2], wd[kt][3], 0x7362);
            // column 4c + k of the tile at k 296 + 9c + g: both accesses fall on
            // 32 banks
            t[0 * 296 + 9 * c + g] = __byte_perm(a, b, 0x5410);
            t[1 * 296 + 9 * c + g] = __byte_perm(a, b, 0x7632);
            t[2 * 296 + 9 * c + g] = __byte_perm(d, e, 0x5410);
            t[3 * 296 + 9 * c + g] = __byte_perm(d, e, 0x7632);
            __syncthreads();   // (and this buffer's reads two tiles ago are done)
            const int tid = threadIdx.y * 32 + threadIdx.x;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = (tid + 256 * q) >> 3, wq = tid & 7;
                const int xs = xb0 + j, ys = y0 + 4 * wq;
                if (xs >= sw || ys >= sh)
                    continue;
                const unsigned word = t[(j & 3) * 296 + 9 * (j >> 2) + wq];
                if (ys + 3 < sh && (dstr & 3) == 0) {
                    *(unsigned int *)(dst + xs * dstr + ys) = word;
                } else {
                    for (int m = 0; m < 4 && ys + m < sh; ++m)
                        dst[xs * dstr + ys + m] = (unsigned char)(word >> (8 * m));
                }
            }
        }
        return;
    }
    char *dst = (char *)p.img[i];
    const long long dstr = p.stride[i];
    unsigned long long(*wide)[33] = (unsigned long long(*)[33])tile;
    for (int kt = 0; kt < TR_TILES; ++kt) {
        const int x0 = (blockIdx.x * TR_TILES + kt) * 32;
        if (x0 >= sw)
            break;   // uniform over the CTA
        if (kt > 0)
            __syncthreads();
        for (int yy = threadIdx.y; yy < 32; yy += 8) {
            const int y = y0 + yy, x = x0 + threadIdx.x;
            if (y < sh && x < sw)
                wide[yy][threadIdx.x] = load_bits(src, es, y * sst + x);
        }
        __syncthreads();
        for (int xx = threadIdx.y; xx < 32; xx += 8) {
            const int x = x0 + xx, y = y0 + threadIdx.x;
            if (x < sw && y < sh)
                store_bits(dst, es, x * dstr + y, wide[threadIdx.x][xx]);
        }
    }
}

// An FP64 number as FP32, toward zero, in integer instructions (conversions
// share the narrow FP64 pipe).  Out of FP32's normal range: 0, or infinity (NaN
// too).
__device__ __forceinline__ float d2f_trunc(double v)
{
    const int hi = __double2hiint(v), m = (hi & 0x7fffffff) - 0x38000000;
    const unsigned lo = (unsigned)__double2loint(v);
    const unsigned b = m < 0x00100000 ? 0u : m > 0x0fdfffff ? 0x7f800000u
                                            : __funnelshift_l(lo, (unsigned)m, 3);
    return __uint_as_float(b | ((unsigned)hi & 0x80000000u));
}
// An FP64 number rounded to FP32 as the conversion does, in integer
// instructions where the result is a normal number.
__device__ __forceinline__ float d2f_rn(double v)
{
    const int hi = __double2hiint(v), m = (hi & 0x7fffffff) - 0x38000000;
    const unsigned lo = (unsigned)__double2loint(v);
    if (m < 0x00100000 || m > 0x0fdfffff)
        return (float)v;
    const unsigned b = __funnelshift_l(lo, (unsigned)m, 3), rem = lo << 3;   // the 29 bits cut
    const unsigned up = rem > 0x80000000u || (rem == 0x80000000u && (b & 1u));
    return __uint_as_float((b + up) | ((unsigned)hi & 0x80000000u));
}

// The row pass of the summed-area tables: per needed row, add the warp
// segment offsets of k3_sat and take the x-prefix.  One warp per row (no
// block-wide synchronisation, so a CTA carries eight rows and small images
// do not pay one CTA per row); the warp walks the row a few columns per lane
// at a time, with an inclusive shuffle scan per step and a carry between them.
// (On the uneven uint16 batch a CTA-per-row scan on the rows wider than 512
// columns took nearly twice as long.)

template <typename TA>
__device__ __forceinline__ TA warp_incl_scan(TA v, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const TA u = __shfl_up_sync(0xffffffff, v, o);
        if (lane >= o)
            v += u;
    }
    return v;
}

// Four consecutive columns per lane: three additions, then one scan of the
// lanes' totals per 128 columns (a scan is ten 64-bit shuffles, and on FP64
// tables ten additions on the narrow FP64 pipe: 199 -> 148 us for 24 pairs of
// FP64 images, where one column per lane took a scan per 32 columns).
template <typename TA>
__device__ __forceinline__ void sat2_row_any(const PairDev &p, int i, int slot, int y, int lane)
{
    typedef SatPair<TA> SP;
    constexpr int K = 4;
    const int w = p.w[i];
    const int seg = sat_seg_of(p, i, y);
    const typename SP::type *__restrict__ o =
        (const typename SP::type *)p.seg[i] + (long long)seg * p.sp[i];
    typename SP::type *__restrict__ r = (typename SP::type *)p.sat[i] + (long long)slot * p.sp[i];
    float2 *__restrict__ rf = p.satf[i] ? p.satf[i] + (long long)slot * p.sp[i] : nullptr;
    TA cs = 0, cq = 0;
    for (int c0 = 0; c0 < w; c0 += 32 * K) {
        const int c = c0 + K * lane;
        TA s[K], q[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            s[k] = q[k] = 0;
            if (c + k < w) {
                const typename SP::type a = r[c + k], b = ld_chain(o + c + k);
                s[k] = a.x + b.x;
                q[k] = a.y + b.y;
            }
        }
#pragma unroll
        for (int k = 1; k < K; ++k) {
            s[k] += s[k - 1];
            q[k] += q[k - 1];
        }
        const TA ts = warp_incl_scan(s[K - 1], lane), tq = warp_incl_scan(q[K - 1], lane);
        TA bs = __shfl_up_sync(0xffffffff, ts, 1), bq = __shfl_up_sync(0xffffffff, tq, 1);
        bs = lane ? bs + cs : cs;
        bq = lane ? bq + cq : cq;
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (c + k < w) {
                const typename SP::type e = SP::of(s[k] + bs, q[k] + bq);
                r[c + k] = e;
                if (rf)
                    rf[c + k] = make_float2(d2f_trunc((double)e.x), d2f_trunc((double)e.y));
            }
        cs += __shfl_sync(0xffffffff, ts, 31);
        cq += __shfl_sync(0xffffffff, tq, 31);
    }
}

// Packed tables: two entries (16 bytes) per lane, one scan per 64 columns.
__device__ __forceinline__ void sat2_row_packed(const PairDev &p, int i, int slot, int y, int lane)
{
    typedef unsigned long long u64;
    const int w = p.w[i], sp = p.sp[i];
    const ulonglong2 *__restrict__ o =
        (const ulonglong2 *)((const u64 *)p.seg[i] + (long long)sat_seg_of(p, i, y) * sp);
    ulonglong2 *__restrict__ r = (ulonglong2 *)((u64 *)p.sat[i] + (long long)slot * sp);
    u64 carry = 0;
    constexpr int K = 4;   // steps whose loads are in flight together
    for (int c0 = 0; c0 < sp; c0 += 64 * K) {
        ulonglong2 e[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int c = c0 + 64 * k + 2 * lane;
            e[k] = make_ulonglong2(0, 0);
            if (c < sp) {
                const ulonglong2 a = r[c >> 1], b = ld_chain(o + (c >> 1));
                e[k].x = a.x + b.x;
                e[k].y = c + 1 < w ? a.y + b.y : 0;
            }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (c0 + 64 * k >= sp)
                break;   // uniform over the warp
            const int c = c0 + 64 * k + 2 * lane;
            const u64 t = warp_incl_scan(e[k].x + e[k].y, lane) + carry;
            const u64 x = t - e[k].y;   // modulo 2^64: exact
            carry = __shfl_sync(0xffffffff, t, 31);
            if (c < sp)
                r[c >> 1] = make_ulonglong2(x, t);
        }
    }
}

// Counts-only form (CorrImagesS without a mincor): K rounds of 32 columns
// per pass, their loads issued together (one memory latency per pass), then
// scanned in registers in column order.  (Measured on the thumbnail sweep:
// 52 ms per 1024-pair step against 132 ms one round at a time; the same
// batching of the int64 S and Q tables needed 91 registers and ran slower.)
__device__ __forceinline__ void sat2_row_counts(const PairDev &p, int i, int slot, int y,
                                                int lane)
{
    constexpr int K = 8;
    const int w = p.w[i];
    const int seg = sat_seg_of(p, i, y);
    const int *__restrict__ oN = p.segN[i] + (long long)seg * p.sp[i];
    int *__restrict__ rN = p.satN[i] + (long long)slot * p.sp[i];
    int cn = 0;
    for (int cb = 0; cb < w; cb += 32 * K) {
        int vn[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int c = cb + 32 * k + lane;
            vn[k] = c < w ? rN[c] + oN[c] : 0;
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (cb + 32 * k >= w)
                break;   // uniform over the warp
            vn[k] = warp_incl_scan(vn[k], lane) + cn;
            cn = __shfl_sync(0xffffffff, vn[k], 31);
            const int c = cb + 32 * k + lane;
            if (c < w)
                rN[c] = vn[k];
        }
    }
}

// grid (ceil(maxslots / 8), 2, npairs), block 256: warp k takes slot 8*bx + k;
// an image's first block also makes its mean shift (a launch of its own for two
// sums took 7 of a single pair's 105 us).  CorrImagesS without a mincor has no
// value sums and correlates unshifted images: its mu stays 0.
// NONLY: the form launched for chunks of counts-only jobs (its registers are
// not sized for the int64 tables).
template <bool NONLY>
__global__ void k2_sat2w(PairDev *pairs)
{
    grid_dep();
    PairDev &p = pairs[blockIdx.z];
    const int i = blockIdx.y;
    const int slot = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (p.status != 0)
        return;
    if (!NONLY && blockIdx.x == 0 && !p.sat_nonly)
        mean_shift(p, i);
    if (slot >= nslots(p, i) || (i == 1 && p.sat_shared))
        return;
    const int len0 = p.need_hi[i][0] - p.need_lo[i][0] + 1;
    const int y = slot < len0 ? p.need_lo[i][0] + slot : p.need_lo[i][1] + slot - len0;
    const int lane = threadIdx.x & 31;
    if (p.cnt_kind == ALN_CNT_GT)   // the count table only where a count rule reads it
        sat2_row_counts(p, i, slot, y, lane);
    if (NONLY || p.sat_nonly)
        return;
    if (p.sat_packed)
        sat2_row_packed(p, i, slot, y, lane);
    else if (int_pixels(p.dt[i]))
        sat2_row_any<long long>(p, i, slot, y, lane);
    else
        sat2_row_any<double>(p, i, slot, y, lane);
}

// ---------------------------------------------------------------------------
// forward rows
// ---------------------------------------------------------------------------

// launch shape and shared-memory layout: aln_row_layout.cuh

// Each team of T threads (rowfft_T<L>()) transforms one row.  G =
// blockDim.x / T rows per CTA.
template <int L>
__global__ void __launch_bounds__(rowfft_threads(rowfft_T<L>()), rowfft_minb<L>())
k2_rowfft(PairDev *pairs, const float2 *__restrict__ tw, int only_img, const int *sel)
{
    grid_dep();
    using F = RowFFT<L>;
    constexpr int V = F::V, T = F::T;
    constexpr int G = rowfft_threads(T) / T;
    extern __shared__ float2 smem[];
    // sel: the jobs of this launch are pairs[sel[z]] (spectrum-cache fills)
    PairDev &p = pairs[sel ? sel[blockIdx.z] : blockIdx.z];
    const int i = only_img >= 0 ? only_img : blockIdx.y;
    if (p.status != 0 || (i == 1 && p.b_cached && !sel))
        return;
    const int team = threadIdx.x / T, t = threadIdx.x - team * T;
    const int h = p.h[i], w = p.w[i], dt = p.dt[i];
    const int y0 = blockIdx.x * G;
    if (y0 >= h)
        return;
    const int y = y0 + team;
    float2 *sm = smem + rowfft_base<L>(team);
    const void *img = p.img[i];
    const long long st = p.stride[i];
    float2 v[V];
    if (dt == ALN_U8 || dt == ALN_U16) {
        // integer pixels, integer shift: exact before the conversion.  The
        // row is staged in shared memory with 16-byte loads from its
        // 16-byte-aligned start (an aligned 16-byte block that holds a byte
        // of the row never leaves the row's allocation page).
        const int es = dt == ALN_U8 ? 1 : 2;
        const int mu = (int)p.mu[i];
        // the region's first 16-byte boundary (at most 8 bytes in): the row's
        // <= 4L + 30 staged bytes end inside the region (rowfft_pitch)
        unsigned char *sb = (unsigned char *)(((uintptr_t)sm + 15) & ~(uintptr_t)15);
        int at = 0;   // the staged row's first byte
        if (y < h) {
            const unsigned char *base = (const unsigned char *)img + (long long)y * st * es;
            const uintptr_t a0 = (uintptr_t)base & ~(uintptr_t)15;
            const int off = (int)((uintptr_t)base - a0), nb = w * es;
            const int nvec = (off + nb + 15) >> 4;
            const uint4 *src = (const uint4 *)a0;
            // a thread reads its pixel pairs as one 2- or 4-byte word: a row that
            // starts between such words is staged shifted onto one
            const int odd = off & (2 * es - 1);
            at = off - odd;
            if (odd == 0) {
                for (int k = t; k < nvec; k += T)
                    ((uint4 *)sb)[k] = src[k];
            } else {
                for (int k = t; k < nvec; k += T) {
                    const uint4 v4 = src[k];
                    const unsigned nx = k + 1 < nvec ? *(const unsigned *)(src + k + 1) : 0u;
                    ((uint4 *)sb)[k] = make_uint4(__funnelshift_r(v4.x, v4.y, 8 * odd),
                                                  __funnelshift_r(v4.y, v4.z, 8 * odd),
                                                  __funnelshift_r(v4.z, v4.w, 8 * odd),
                                                  __funnelshift_r(v4.w, nx, 8 * odd));
                }
            }
        }
        team_sync<T>(team);
        if (y < h) {   // the padding holds mu, which becomes 0
            if (es == 1)
                for (int k = w + t; k < 2 * L; k += T)
                    sb[at + k] = (unsigned char)mu;
            else
                for (int k = w + t; k < 2 * L; k += T)
                    *(unsigned short *)(sb + at + 2 * k) = (unsigned short)mu;
        }
        team_sync<T>(team);   // each team reads back its own row only
        // (rows past the image read what is there: their bins are not stored)
        const unsigned char *row = sb + at;
        // 2^23 + pixel is the float with the pixel as its last bits: less 2^23 + mu
        // it is the shifted pixel, exactly, without a conversion
        const float bias = 8388608.0f + (float)mu;
        if (es == 1) {
#pragma unroll
            for (int q = 0; q < V; ++q) {
                const unsigned d = *(const unsigned short *)(row + 2 * F::in_idx(t, q));
                v[q].x = __uint_as_float(__byte_perm(d, 0x4b000000u, 0x7440)) - bias;
                v[q].y = __uint_as_float(__byte_perm(d, 0x4b000000u, 0x7441)) - bias;
            }
        } else {
#pragma unroll
            for (int q = 0; q < V; ++q) {
                const unsigned d = *(const unsigned *)(row + 4 * F::in_idx(t, q));
                v[q].x = __uint_as_float(__byte_perm(d, 0x4b000000u, 0x7410)) - bias;
                v[q].y = __uint_as_float(__byte_perm(d, 0x4b000000u, 0x7432)) - bias;
            }
        }
    } else if (dt == ALN_F32) {
        // the shift is an FP32 number (mean_shift), and the FP64 difference of two
        // FP32 numbers rounds to FP32 as the FP32 difference does: no FP64
        // instruction (they held this kernel's sweep rows at 50 % of that pipe)
        const float mu = (float)p.mu[i];
        const float *row = (const float *)img + y * st;
#pragma unroll
        for (int q = 0; q < V; ++q) {
            const int xa = 2 * F::in_idx(t, q), xb = xa + 1;
            float2 z = make_float2(0.f, 0.f);
            if (y < h) {
                if (xa < w)
                    z.x = __fsub_rn(__ldg(row + xa), mu);
                if (xb < w)
                    z.y = __fsub_rn(__ldg(row + xb), mu);
            }
            v[q] = z;
        }
    } else {
        const double mu = p.mu[i];
        const double *row = (const double *)img + y * st;
#pragma unroll
        for (int q = 0; q < V; ++q) {
            const int xa = 2 * F::in_idx(t, q), xb = xa + 1;
            float2 z = make_float2(0.f, 0.f);
            if (y < h) {
                if (xa < w)
                    z.x = d2f_rn(__dsub_rn(__ldg(row + xa), mu));
                if (xb < w)
                    z.y = d2f_rn(__dsub_rn(__ldg(row + xb), mu));
            }
            v[q] = z;
        }
    }
    F::run_team(v, sm, t, tw, team);
    // split the half-length transform into the N/2+1 bins of the real row
    __syncthreads();
#pragma unroll
    for (int q = 0; q < V; ++q)
        sm[F::out_idx(t, q)] = v[q];
    __syncthreads();
    // bins for (kx, row) with row fastest: coalesced [kx][y] stores.  Bin kx
    // needs Z[kx] and conj(Z[L - kx]) (indices mod L), bin L - kx the same
    // two values swapped: one item makes both (kx = 0..L/2; L is even).  The
    // CTA has G * T threads, so thread x always takes row x % G and bins
    // kx = x / G + m T: its row's region and store pointers are set once.
    constexpr int THR = G * T;
    const int rr = threadIdx.x % G;
    if (rr >= min(G, h - y0))
        return;
    const float2 *Z = smem + rowfft_base<L>(rr);
    const long long Ts = p.Ts[i];
    const int kx0 = threadIdx.x / G;
    float2 *lo = p.T[i] + y0 + rr + kx0 * Ts;          // bin kx
    float2 *hi = p.T[i] + y0 + rr + (L - kx0) * Ts;    // bin L - kx
    const float2 *twk = tw + tw_base(2 * L) + 2 * L;   // exp(-2 pi i k / 2L) at twk[k]
    // With A = Z[kx], B = Z[L - kx], e the even and d the odd part's spectrum at
    // kx, both bins need one product t = -i d w(kx): bin kx is e + t, and bin
    // L - kx, where w(L - kx) = -conj(w(kx)), is conj(e - t).
    for (int kx = kx0; kx <= L / 2; kx += THR / G, lo += (THR / G) * Ts, hi -= (THR / G) * Ts) {
        const float2 A = Z[kx];
        const float2 B = Z[kx == 0 ? 0 : L - kx];
        const float2 ev = make_float2(0.5f * (A.x + B.x), 0.5f * (A.y - B.y));
        const float2 dd = make_float2(0.5f * (A.x - B.x), 0.5f * (A.y + B.y));
        const float2 o = make_float2(dd.y, -dd.x);
        const float2 tt = cmul(o, __ldg(&twk[kx]));
        *lo = cadd(ev, tt);
        if (kx != L / 2)
            *hi = make_float2(ev.x - tt.x, tt.y - ev.y);
    }
}

// ---------------------------------------------------------------------------
// columns: forward b and a, product, inverse, window rows
// ---------------------------------------------------------------------------

// VAR: 1 = CorrPatches chunks (plain inverse only, no low-pass, no
// whitening), 2 = CorrImagesS without a mincor (whitened inverse only), 3 = the
// same where every job's b is a cached spectrum, read from global memory at the
// product instead of parked in shared memory (which bounds this kernel: a fifth
// of its wavefronts, and half of its allocation), 0 = any job; the specialised forms are compiled without the other jobs'
// branches.
// Per-thread radix of the column FFTs, per kernel form.  (Measured on the
// montage batch: 8 points per thread at 4096 -- twice the threads per
// column -- ran 45% slower than 16, so every form uses fft_radix.)
template <int NY, int VAR>
__host__ __device__ constexpr int corrcol_radix()
{
    return fft_radix(NY);
}

template <int NY, int VAR>
__host__ __device__ constexpr int corrcol_threads()
{
    return NY / corrcol_radix<NY, VAR>() >= 256 ? NY / corrcol_radix<NY, VAR>() : 256;
}

// Occupancy: the CorrPatches form keeps 2 CTAs per SM; the S-only form runs
// 3 (80 registers, small spills, faster).
template <int NY, int VAR>
__global__ void __launch_bounds__(corrcol_threads<NY, VAR>(),
                                  (NY >= 8192 || corrcol_threads<NY, VAR>() > 256) ? 1
                                                                                 : (VAR >= 2 ? 3 : 2))
k2_corrcol(PairDev *pairs, const float2 *__restrict__ tw, int use_cached_b)
{
    grid_dep();
    constexpr bool PLAIN = VAR == 1, SONLY = VAR >= 2, DIRECT = VAR == 3;
    using FF = RegFFT<NY, -1, corrcol_radix<NY, VAR>()>;
    using FI = RegFFT<NY, +1, corrcol_radix<NY, VAR>()>;
    static_assert(FI::SMEM <= FF::SMEM, "the inverse runs in the forward transform's buffer");
    constexpr int R = FF::R, T = FF::T;
    extern __shared__ float2 smem[];
    PairDev &p = pairs[blockIdx.y];
    if (p.status != 0)
        return;
    const int L1 = (p.Nx >> 1) + 1;
    const int G = blockDim.x / T;
    const int team = threadIdx.x / T, t = threadIdx.x - team * T;
    const int kx = blockIdx.x * G + team;
    const bool live = kx < L1;
    if (blockIdx.x * G >= L1)
        return;
    float2 *sm = smem + team * FF::SMEM;
    float2 *sb = smem + G * FF::SMEM + team * NY;   // b's spectrum, this team's own slots
    const int kxc = live ? kx : L1 - 1;   // idle teams compute a copy, store nothing
    float2 va[R];
    if constexpr (!DIRECT) {
        float2 vb[R];
        if (use_cached_b || p.b_cached) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                vb[r] = p.X2[(long long)kxc * NY + t + r * T];
        } else {
            const float2 *Tb = p.T[1] + (long long)kxc * p.Ts[1];
            const int hb = p.h[1];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int y = t + r * T;
                vb[r] = y < hb ? Tb[y] : make_float2(0.f, 0.f);
            }
            FF::run_team(vb, sm, t, tw, team);
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            sb[r * T + t] = vb[r];
    }
    {
        const float2 *Ta = p.T[0] + (long long)kxc * p.Ts[0];
        const int ha = p.h[0];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int y = t + r * T;
            va[r] = y < ha ? Ta[y] : make_float2(0.f, 0.f);
        }
    }
    fresh(tw);
    FF::run_team(va, sm, t, tw, team);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float2 x2 = DIRECT ? __ldg(&p.X2[(long long)kxc * NY + t + r * T]) : sb[r * T + t];
        va[r] = cmulc(x2, va[r]);   // X2 * conj(X1)
    }
    const bool is_p2i = VAR == 0 && p.mode == JOB_P2I;
    if (is_p2i && p.p2i_filter) {
        // CorrPatchToImage's low-pass (0_GEN/Correlation.cpp:1255-1283): the
        // reference names the row index "x" (wrapped) and the column "y"
#pragma unroll
        for (int r = 0; r < R; ++r) {
            int x = t + r * T;
            if (x >= NY / 2)
                x -= NY;
            const double rad2 = ((double)x * x + (double)kxc * kxc) / 10000.0;
            const float filt = rad2 > 10.0 ? 0.f : (float)exp(-rad2);
            va[r] = make_float2(va[r].x * filt, va[r].y * filt);
        }
    }
    // CorrPatches / CorrImagesR need the plain inverse; CorrImagesS the inverse
    // of the whitened product P / sqrt(|P|) (0_GEN/Correlation.cpp:2311-2317)
    // (always so for the plain form: as a run-time condition it keeps the inverse's
    // twiddle loads out of the forward transform, where they cost 150 bytes of
    // spills)
    const bool want_r = PLAIN ? p.mode == JOB_PATCHES : (!SONLY && (p.mode == JOB_PATCHES || is_p2i || p.want_r));
    const bool want_s = SONLY || (!PLAIN && p.want_s != 0);
    if (want_r && want_s) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            sb[r * T + t] = va[r];
    }
    if (want_r) {
        fresh(tw);
        FI::run_team(va, sm, t, tw, team);
        if (live && is_p2i) {   // every storage row, in storage order
            float2 *Q = p.Q + (long long)kx * NY;
#pragma unroll
            for (int r = 0; r < R; ++r)
                Q[t + r * T] = va[r];
        } else if (live) {
            const int ylo = p.ylo, Wy = p.yhi - ylo + 1, nnegy = p.h[0] - 1;
            float2 *Q = p.Q + (long long)kx * Wy;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int ys = t + r * T;
                const int j = (ys >= NY - nnegy ? ys - NY : ys) - ylo;
                if ((unsigned)j < (unsigned)Wy)
                    Q[j] = va[r];
            }
        }
    }
    if (want_s) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float2 v = want_r ? sb[r * T + t] : va[r];
            const float m = hypotf(v.x, v.y);
            if (m > 1e-10f) {
                const float q = 1.0f / sqrtf(m);
                v = make_float2(v.x * q, v.y * q);
            }
            va[r] = v;
        }
        fresh(tw);
        FI::run_team(va, sm, t, tw, team);
        if (live) {
            const int ylo = p.ylo, Wy = p.yhi - ylo + 1, nnegy = p.h[0] - 1;
            float2 *Q = (want_r ? p.Q2 : p.Q) + (long long)kx * Wy;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int ys = t + r * T;
                const int j = (ys >= NY - nnegy ? ys - NY : ys) - ylo;
                if ((unsigned)j < (unsigned)Wy)
                    Q[j] = va[r];
            }
        }
    }
}

// CorrPatches columns with the long axis cut into segments.  Only the Wy lag
// rows [ylo, yhi] are read, so for column kx
//   C[ylo + e] = sum_y conj(A[y]) B[y + ylo + e],   e in [0, Wy),
// splits over segments of a's rows, y = s*seg_len + j (j < seg_len): segment
// s pairs a's rows [s*seg_len, +seg_len) with b's rows [s*seg_len + ylo,
// +seg_len + Wy - 1), and NS >= seg_len + Wy - 1 makes its circular
// correlation on NS points the linear one at e in [0, Wy).  The segments'
// spectral products are summed (one accumulator per column) and inverted
// once: 2 nseg + 1 transforms of NS points instead of 3 of Ny.  Each thread
// keeps its accumulator and parked a-spectrum points to itself, in
// registers or its own shared-memory slots (corrseg_regs; no exchange).
// Output: Q[kx][e], as k2_corrcol; the column transform length the lag
// kernel normalises by is NS (p.Ny).
// Per-thread radix of the segment transforms.  Measured on the montage
// strips (6 segments of 512 points, accumulator then in shared memory):
// radix 8 at 3 CTAs per SM ran 25% faster than radix 16 at 2 (spills, low
// occupancy); at 1024 and 2048 points radix 16 stays ahead.
template <int NS>
__host__ __device__ constexpr int corrseg_radix()
{
    return NS == 512 ? 8 : fft_radix(NS);
}

// Where a thread keeps its a-spectrum points and the column's accumulated
// product: registers at radix <= 8 (each thread owns the same R points
// throughout; a third fewer shared-memory wavefronts than parking them in
// shared memory, 2 CTAs per SM at 128 registers instead of 3 at 80:
// k2_corrseg<512> 10.18 -> 9.84 ms per montage step), shared memory at
// radix 16 (32 more points per thread spilled 260-280 bytes).
template <int NS>
__host__ __device__ constexpr bool corrseg_regs()
{
    return corrseg_radix<NS>() <= 8;
}

template <int NS>
__global__ void __launch_bounds__(256, 2)
k2_corrseg(PairDev *pairs, const float2 *__restrict__ tw)
{
    grid_dep();
    using FF = RegFFT<NS, -1, corrseg_radix<NS>()>;
    using FI = RegFFT<NS, +1, corrseg_radix<NS>()>;
    static_assert(FI::SMEM <= FF::SMEM, "the inverse runs in the forward transform's buffer");
    constexpr int R = FF::R, T = FF::T;
    extern __shared__ float2 smem[];
    const PairDev &p = pairs[blockIdx.y];
    if (p.status != 0)
        return;
    const int L1 = (p.Nx >> 1) + 1;
    const int G = blockDim.x / T;
    const int team = threadIdx.x / T, t = threadIdx.x - team * T;
    const int kx = blockIdx.x * G + team;
    if (blockIdx.x * G >= L1)
        return;
    const bool live = kx < L1;
    const int kxc = live ? kx : L1 - 1;   // idle teams compute a copy, store nothing
    float2 *sm = smem + team * FF::SMEM;
    constexpr bool REGS = corrseg_regs<NS>();
    float2 accr[REGS ? R : 1];
    float2 *park = REGS ? nullptr : smem + G * FF::SMEM + team * (2 * NS);
    float2 *acc = REGS ? nullptr : park + NS;
    const float2 *Ta = p.T[0] + (long long)kxc * p.Ts[0];
    const float2 *Tb = p.T[1] + (long long)kxc * p.Ts[1];
    const int ha = p.h[0], hb = p.h[1];
    const int B = p.seg_len, nseg = p.nseg, ylo = p.ylo;
    const int Wy = p.yhi - p.ylo + 1;
    const int lb = B + Wy - 1;
    auto load_a = [&](int s, float2 *v) {
        const int y0 = s * B, n = min(B, ha - y0);
        const float2 *src = Ta + y0 + t;
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = t + r * T < n ? src[r * T] : make_float2(0.f, 0.f);
    };
    auto load_b = [&](int s, float2 *v) {
        const int y0 = s * B + ylo, lo = max(0, -y0);
        const unsigned n = (unsigned)max(0, min(lb, hb - y0) - lo);
        const float2 *src = Tb + y0 + t;
#pragma unroll
        for (int r = 0; r < R; ++r)
            v[r] = (unsigned)(t + r * T - lo) < n ? src[r * T] : make_float2(0.f, 0.f);
    };
    float2 va[R], vb[R];
    if constexpr (REGS)
        load_a(0, va);
    for (int s = 0; s < nseg; ++s) {
        if constexpr (REGS) {
            // b's loads are in flight while a is transformed, the next segment's
            // a while b is (waiting for each load in turn left the warps on the
            // long scoreboard, 2.7 stalled per issue: 4096 strips 9.50 -> 8.12 ms)
            load_b(s, vb);
            FF::run_team(va, sm, t, tw, team);
            float2 na[R];
            load_a(s + 1 < nseg ? s + 1 : s, na);
            FF::run_team(vb, sm, t, tw, team);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float2 q = cmulc(vb[r], va[r]);   // X2 * conj(X1)
                accr[r] = s == 0 ? q : cadd(accr[r], q);
                va[r] = na[r];
            }
        } else {
            load_a(s, va);
            fresh(tw);
            FF::run_team(va, sm, t, tw, team);
#pragma unroll
            for (int r = 0; r < R; ++r)
                park[r * T + t] = va[r];
            load_b(s, vb);
            fresh(tw);
            FF::run_team(vb, sm, t, tw, team);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float2 q = cmulc(vb[r], park[r * T + t]);
                acc[r * T + t] = s == 0 ? q : cadd(acc[r * T + t], q);
            }
        }
    }
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if constexpr (REGS)
            v[r] = accr[r];
        else
            v[r] = acc[r * T + t];
    }
    if constexpr (!REGS)
        fresh(tw);
    FI::run_team(v, sm, t, tw, team);
    if (live) {
        float2 *Q = p.Q + (long long)kx * Wy;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int e = t + r * T;
            if (e < Wy)
                Q[e] = v[r];
        }
    }
}

// Spectrum of image b alone into X2 (a cache entry): per column kx, the
// column FFT of b's row-pass output, stored as k2_corrcol reads a cached
// spectrum.  The same RegFFT code as the fused path, so the cached and the
// recomputed spectra are the same numbers.  grid (ceil((L+1)/G), nsel): the
// jobs are pairs[sel[y]].
// RAD: the per-thread radix of the column kernel that reads the entry (the
// same FFT code, so the cached and the recomputed spectra are the same
// numbers).
template <int NY, int RAD>
__global__ void __launch_bounds__(NY / RAD >= 256 ? NY / RAD : 256)
k2_colspec(PairDev *pairs, const float2 *__restrict__ tw, const int *sel)
{
    grid_dep();
    using FF = RegFFT<NY, -1, RAD>;
    constexpr int R = FF::R, T = FF::T;
    extern __shared__ float2 smem[];
    PairDev &p = pairs[sel[blockIdx.y]];
    if (p.status != 0)
        return;
    const int L1 = (p.Nx >> 1) + 1;
    const int G = blockDim.x / T;
    const int team = threadIdx.x / T, t = threadIdx.x - team * T;
    const int kx = blockIdx.x * G + team;
    if (blockIdx.x * G >= L1)
        return;
    float2 *sm = smem + team * FF::SMEM;
    const int kxc = kx < L1 ? kx : L1 - 1;
    const float2 *Tb = p.T[1] + (long long)kxc * p.Ts[1];
    const int hb = p.h[1];
    float2 vb[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int y = t + r * T;
        vb[r] = y < hb ? Tb[y] : make_float2(0.f, 0.f);
    }
    FF::run(vb, sm, t, tw);
    if (kx < L1) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            p.X2[(long long)kx * NY + t + r * T] = vb[r];
    }
}

// ---------------------------------------------------------------------------
// lag rows
// ---------------------------------------------------------------------------
// The job's descriptor in shared memory: the lag scans read many of its
// fields inside loops that also store through its pointers; from global
// memory each read would be a fresh L1 round trip (the compiler cannot keep
// them across the stores).  All threads of the CTA must call this.
__device__ __forceinline__ const PairDev &stage_job(const PairDev *pairs, int j, PairDev &sp)
{
    const int *src = (const int *)(pairs + j);
    int *dst = (int *)&sp;
    for (int i = threadIdx.x; i < (int)(sizeof(PairDev) / sizeof(int)); i += blockDim.x)
        dst[i] = src[i];
    __syncthreads();
    return sp;
}


// The L+1 spectrum bins of the CTA's G lag rows j0 .. j0+G-1 (Q is [kx][j],
// stride Wy; rows past Wy repeat the last one) into the teams' shared rows
// (team g at base + g * stride), loaded by the whole CTA so that a warp's
// loads cover whole 8-row segments of Q (G consecutive j per kx); four loads
// per thread are in flight before their stores.
// G: rows per CTA (blockDim.x / T).  The copies are asynchronous
// (cp.async, 8 bytes each, global -> shared without registers), so every
// element a thread moves is in flight at once; the loads through registers
// this replaces kept four per thread in flight, and the lag kernels waited on
// them (long-scoreboard stalls, k2_lagimg 33 % warps active).  The caller's
// __syncthreads after the call publishes the rows to the CTA.
template <int L, int T, int G = (T >= 256 ? T : 256) / T>
__device__ __forceinline__ void load_lag_rows(float2 *base, int stride,
                                              const float2 *__restrict__ Q, int Wy, int j0)
{
    constexpr int TOT = (L + 1) * G;
    for (int e = threadIdx.x; e < TOT; e += blockDim.x) {
        const int kx = e / G, g = e - kx * G;
        cp_async8(&base[g * stride + padi(kx)], &Q[(long long)kx * Wy + min(j0 + g, Wy - 1)]);
    }
    cp_async_wait_all();
}

// Threads per CTA of k2_lagrow: eight lag rows per CTA for teams smaller
// than a warp (the split lengths' 8-thread teams would otherwise take 32 rows
// per CTA, and a 129-row disc window 160 team-rows), at least one whole warp
// (the row reduction shuffles over full warps), 256 threads for larger teams.
__host__ __device__ constexpr int lagrow_threads(int T)
{
    return T < 32 ? (8 * T < 32 ? 32 : 8 * T) : (T >= 256 ? T : 256);
}

template <int L>
__global__ void __launch_bounds__(lagrow_threads(FFTOf<L, +1>::T))
k2_lagrow(PairDev *pairs, const float2 *__restrict__ tw)
{
    grid_dep();
    using F = FFTOf<L, +1>;   // RegFFT, or MixFFT for L = 3 * 2^k, 5 * 2^k
    static_assert(F::SMEM <= lag_pitch<L>(), "the exchange buffer fits the team's row region");
    constexpr int V = F::V, T = F::T;
    constexpr int PITCH = lag_pitch<L>();   // holds the L+1 bins
    extern __shared__ float2 smem[];
    const PairDev &p = pairs[blockIdx.y];
    if (p.status != 0)
        return;
    const int xlo = p.xlo, xhi = p.xhi, Wx = xhi - xlo + 1, Wy = p.yhi - p.ylo + 1;
    const int G = blockDim.x / T;
    const int team = threadIdx.x / T, t = threadIdx.x - team * T;
    const int j0 = blockIdx.x * G;
    if (j0 >= Wy)
        return;
    const int j = j0 + team;
    const bool live = j < Wy;
    float2 *sm = smem + team * PITCH;
    // spectrum bins of the CTA's lag rows
    load_lag_rows<L, T, lagrow_threads(T) / T>(smem, PITCH, p.Q, Wy, j0);
    __syncthreads();
    float2 v[V];
#pragma unroll
    for (int q = 0; q < V; ++q) {
        const int k = F::in_idx(t, q);
        float2 a = sm[padi(k)];
        float2 b = cconj(sm[padi(L - k)]);
        if (k == 0) {
            a.y = 0.f;
            b.y = 0.f;
        }
        const float2 e = cadd(a, b);
        const float2 dd = csub(a, b);
        const float2 wv = twn<2 * L, +1>(tw, k);   // W^{-k}
        const float2 o = cmul(dd, wv);
        v[q] = make_float2(e.x - o.y, e.y + o.x);
    }
    // the teams' rows are their own from here on: team barriers only
    F::run_team(v, sm, t, tw, team);
    if (!live)
        return;
    // storage index xs holds lag xs (xs <= xhi) or xs - Nx; the window's lags
    // go to the row of the lag image
    float *row = (float *)p.rr + (long long)j * Wx - xlo;
#pragma unroll
    for (int q = 0; q < V; ++q) {
        const int xs = 2 * F::out_idx(t, q);
        const int xa = xs > xhi ? xs - 2 * L : xs, xb = xs + 1 > xhi ? xs + 1 - 2 * L : xs + 1;
        if (xa >= xlo && xa <= xhi)
            row[xa] = v[q].x;
        if (xb >= xlo && xb <= xhi)
            row[xb] = v[q].y;
    }
}

// r per lag and each lag row's best, from the lag image k2_lagrow wrote: one
// warp per lag row, lanes on consecutive lags.  Apart from the transforms,
// because a row's transform has few threads (8 for the 160- and 192-point
// rows), and its lags then ran one after another on them: 16 per thread on
// a 129-lag row, each a chain of table loads.  The row's table rows, box
// height and disc span are set once per warp (LagRow); r itself is not
// stored, k_final computes the four it needs again.  Transform and scan
// together, before (one kernel) and now: one 235 x 2048 pair 45 -> 22 us, 3000
// uneven pairs 7.3 -> 4.7 ms, 48 pairs of 512^2 over all lags 1120 -> 752 us.
#define LAGSCAN_ROWS 8

// The lags xa + lane, xa + lane + 32, ... <= xb of one row of an integer pair:
// the best FP32 r and its storage index.  KIND: 0 packed tables, 1 int64
// pairs with sums below 2^31, 2 int64 pairs, 3 those whose overlaps may be
// int_wide (uint16 600^2 over all lags: 137 us as KIND 2, 138 as 3); CHECK: a
// legality table or a
// count rule is looked up too.  The body has no branch and reads past the
// row's end at xb again, so that the unrolled loop's loads are in flight
// together: with a branch per lag the scan waited for them one lag at a time.
template <int KIND, bool CHECK>
__device__ __forceinline__ void scan_row_int(const PairDev &p, const LagRow &q, int xa, int xb,
                                             int y, long long in, int key0, float &br, int &bk)
{
    typedef unsigned long long u64;
    const int lane = threadIdx.x & 31, ox = p.ox, Nx = p.Nx;
    const int m1 = (int)p.mu[0] - (KIND == 0 ? 128 : 0), m2 = (int)p.mu[1] - (KIND == 0 ? 128 : 0);
    // 1 / (Nx Ny): exact for power-of-two grids; on the split lengths one
    // more FP32 rounding, below the transform's own error
    const float invf = 1.0f / ((float)Nx * (float)p.Ny);
    const float *__restrict__ row =
        (const float *)p.rr + (long long)(y - p.ylo) * (p.xhi - p.xlo + 1) - p.xlo;
    const void *t1 = p.sat[0], *t2 = p.sat[1];
#pragma unroll 2
    for (int x0 = xa; x0 <= xb; x0 += 32) {
        const int x = min(x0 + lane, xb);
        const int L2 = max(0, x), R2 = max(min(q.w2 - 1, x + q.w1 - 1), L2);
        const int olw = R2 - L2 + 1, n = olw * q.olh;
        const float cs = ld_chain(row + x) * invf;
        float r;
        if (KIND == 0) {
            const u64 a = row_box_p((const u64 *)t1, q.oT[0], q.oB[0], L2 - x, R2 - x);
            const u64 b = row_box_p((const u64 *)t2, q.oT[1], q.oB[1], L2, R2);
            const int s1 = sat_pack_s(a), s2 = sat_pack_s(b);
            r = r_int32(n, cs, s1, sat_pack_q(a, s1), s2, sat_pack_q(b, s2), m1, m2);
        } else {
            const longlong2 a = row_box2((const longlong2 *)t1, q.oT[0], q.oB[0], L2 - x, R2 - x);
            const longlong2 b = row_box2((const longlong2 *)t2, q.oT[1], q.oB[1], L2, R2);
            r = KIND == 1 ? r_int32(n, cs, (int)a.x, a.y, (int)b.x, b.y, m1, m2)
                          : r_int(n, cs, a.x, a.y, b.x, b.y, m1, m2, KIND == 3);
        }
        const int dx = x - ox;
        bool ok = olw >= q.omin && olw <= q.omax && (long long)dx * dx <= in;
        if (CHECK && ok) {
            int l, h;
            ok = lag_row_legal(p, q, x, l, h);
        }
        const int k = key0 + (x < 0 ? x + Nx : x);
        if (ok && (r > br || (r == br && k < bk))) {
            br = r;
            bk = k;
        }
    }
}

// grid (ceil(max Wy / LAGSCAN_ROWS), npairs), block 32 * LAGSCAN_ROWS
__global__ void __launch_bounds__(32 * LAGSCAN_ROWS) k2_lagscan(PairDev *pairs)
{
    grid_dep();
    const PairDev &p = pairs[blockIdx.y];
    if (p.status != 0 || !(p.fin & 4))
        return;
    const int j = blockIdx.x * LAGSCAN_ROWS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= p.yhi - p.ylo + 1)
        return;
    const int Nx = p.Nx, Ny = p.Ny;
    const int y = p.ylo + j, ox = p.ox;
    const long long dy = y - p.oy, in = p.rsqr - dy * dy;   // disc: dx^2 <= in
    // the row's span of the disc, a little wide; the lag's own test is exact
    // (an FP64 square root per row cost more than the test).  Where the span
    // reaches 2^15 px to each side, the whole row: the centre may be far off
    int xa = p.xlo, xb = in < 0 ? xa - 1 : p.xhi;
    if (in >= 0 && in < 1ll << 30) {
        const int xr = (int)sqrtf(__int2float_rn((int)in)) + 2;
        xa = max(xa, ox - xr);
        xb = min(xb, ox + xr);
    }
    const LagRow q = lag_row(p, y);
    const int key0 = (y < 0 ? y + Ny : y) * Nx;   // storage indices are < 2^26
    const int nmax = min(q.w1, q.w2) * q.olh;     // largest overlap of the row
    if (r_int_ok(p, nmax)) {
        // every lag of the row takes r_int: FP32 keys
        const bool check = q.tbl || q.cnt;
        const bool narrow = nmax < (1 << 15) ||
                            (p.dt[0] == ALN_U8 && p.dt[1] == ALN_U8 && nmax < (1 << 23));
        float br = -1.0e30f;
        int bk = 0x7fffffff;
        if (p.sat_packed) {
            if (check)
                scan_row_int<0, true>(p, q, xa, xb, y, in, key0, br, bk);
            else
                scan_row_int<0, false>(p, q, xa, xb, y, in, key0, br, bk);
        } else if (check) {
            scan_row_int<3, true>(p, q, xa, xb, y, in, key0, br, bk);
        } else if (narrow) {
            scan_row_int<1, false>(p, q, xa, xb, y, in, key0, br, bk);
        } else if (int_wide(p, nmax)) {
            scan_row_int<3, false>(p, q, xa, xb, y, in, key0, br, bk);
        } else {
            scan_row_int<2, false>(p, q, xa, xb, y, in, key0, br, bk);
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float r2 = __shfl_down_sync(0xffffffff, br, o);
            const int k2 = __shfl_down_sync(0xffffffff, bk, o);
            if (r2 > br || (r2 == br && k2 < bk)) {
                br = r2;
                bk = k2;
            }
        }
        if (lane == 0) {
            p.rb[j].r = (double)br;
            p.rb[j].key = bk;
        }
        return;
    }
    const float invf = 1.0f / ((float)Nx * (float)Ny);
    const float *__restrict__ row =
        (const float *)p.rr + (long long)j * (p.xhi - p.xlo + 1) - p.xlo;
    double br = -1.0e30;
    long long bk = 0x7fffffffffffffffLL;
    for (int x = xa + lane; x <= xb; x += 32) {
        const long long dx = x - ox;
        double rv;
        if (dx * dx <= in && lag_row_r(p, q, x, ld_chain(row + x) * invf, rv))
            best_merge(br, bk, rv, key0 + (x < 0 ? x + Nx : x));
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double r2 = __shfl_down_sync(0xffffffff, br, o);
        const long long k2 = __shfl_down_sync(0xffffffff, bk, o);
        best_merge(br, bk, r2, k2);
    }
    if (lane == 0) {
        p.rb[j].r = br;
        p.rb[j].key = bk;
    }
}

// ---------------------------------------------------------------------------
// CorrImagesR/S lag images (CCorImg::MakeRandA / MakeSandRandA + OrderF +
// SimpleMax, 0_GEN/Correlation.cpp:2060-2380,2509-2569,2939-2948)
// ---------------------------------------------------------------------------

// Per lag row: inverse real FFT of the S rows (whitened product) and/or the
// R rows (plain product), S and R per lag, A = legality & oval (& R > mincor),
// the row's best candidate (key S or R; ties -> smallest R-image index) and
// the row's S sums.
// (S-key jobs without a mincor, the sweep's correlator, have k2_lagss.)
template <int L>
__global__ void __launch_bounds__(256, 2) k2_lagimg(PairDev *pairs, const float2 *__restrict__ tw)
{
    grid_dep();
    using F = RegFFT<L, +1>;
    static_assert(F::SMEM <= lag_pitch<L>(), "the exchange buffer fits the team's row region");
    constexpr int R = F::R, T = F::T;
    constexpr int PITCH = lag_pitch<L>();
    extern __shared__ float2 smem[];
    __shared__ double red_r[32], red_s[32], red_s2[32];
    __shared__ long long red_k[32];
    __shared__ PairDev sp;
    const PairDev &p = stage_job(pairs, blockIdx.y, sp);
    if (p.status != 0)
        return;
    const int Wy = p.yhi - p.ylo + 1, Wx = p.xhi - p.xlo + 1;
    const int G = blockDim.x / T;
    const int team = threadIdx.x / T, t = threadIdx.x - team * T;
    const int j0 = blockIdx.x * G;
    if (j0 >= Wy)
        return;
    const int j = j0 + team;
    const bool live = j < Wy;
    const bool want_r = p.want_r != 0, want_s = p.want_s != 0;
    const bool both = want_r && want_s;
    float2 *sm = smem + team * PITCH * (both ? 2 : 1);
    const int Nx = p.Nx, Ny = p.Ny;
    const float *CS = nullptr, *CR = nullptr;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        const bool doS = pass == 0;
        if ((doS && !want_s) || (!doS && !want_r))
            continue;
        const float2 *Qs = doS ? (both ? p.Q2 : p.Q) : p.Q;
        float2 *reg = sm + ((both && !doS) ? PITCH : 0);
        __syncthreads();
        load_lag_rows<L, T>(smem + ((both && !doS) ? PITCH : 0), PITCH * (both ? 2 : 1), Qs,
                            Wy, j0);
        __syncthreads();
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int k = t + r * T;
            float2 a = reg[padi(k)];
            float2 b = cconj(reg[padi(L - k)]);
            if (k == 0) {
                a.y = 0.f;
                b.y = 0.f;
            }
            const float2 e = cadd(a, b);
            const float2 dd = csub(a, b);
            float2 wv = __ldg(&tw[2 * L + k]);
            wv.y = -wv.y;
            const float2 o = cmul(dd, wv);
            v[r] = make_float2(e.x - o.y, e.y + o.x);
        }
        F::run_team(v, reg, t, tw, team);   // the team's own row
        __syncthreads();
        float *C = (float *)reg;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int n = t + r * T;
            C[2 * n] = v[r].x;
            C[2 * n + 1] = v[r].y;
        }
        if (doS)
            CS = C;
        else
            CR = C;
    }
    __syncthreads();
    const double inv = 1.0 / ((double)Nx * (double)Ny);
    double br = -1.0e30, ss = 0.0, ss2 = 0.0;
    long long bk = 0x7fffffffffffffffLL;
    if (live) {
        const int y = p.ylo + j, iy = y + p.cy;
        const bool keyS = p.mode == JOB_IMAGES_S;
        const LagRow lr = lag_row(p, y);
        for (int x = p.xlo + t; x <= p.xhi; x += T) {
            const int xs = x < 0 ? x + Nx : x;
            double S = 0.0, rv = 0.0;
            if (want_s) {
                S = (double)CS[xs] * inv;
                ss += S;
                ss2 += S * S;
            }
            const bool legal = lag_eval(p, lr, x, want_r ? (double)CR[xs] * inv : 0.0, want_r, rv);
            const double key = keyS ? S : rv;
            const long long o = (long long)j * Wx + (x - p.xlo);
            p.rr[o] = key;
            if (keyS && want_r)
                p.rr2[o] = rv;
            const int ix = x + p.cx;
            const bool cand = legal && oval_ok(p, ix, iy) && (p.mincor <= 0.0 || rv > p.mincor);
            if (p.mode == JOB_IMAGES_F)   // OrderF's candidates (A, R > mincor)
                p.fst[o] = cand ? 4 : 0;
            if (cand)
                best_merge(br, bk, key, (long long)iy * p.wR + ix);
        }
    }
    const int lane = threadIdx.x & 31;
    for (int o = 16; o > 0; o >>= 1) {
        const double r2 = __shfl_down_sync(0xffffffff, br, o);
        const long long k2 = __shfl_down_sync(0xffffffff, bk, o);
        const double a2 = __shfl_down_sync(0xffffffff, ss, o);
        const double b2 = __shfl_down_sync(0xffffffff, ss2, o);
        if (lane + o < 32 && (lane + o) / T == lane / T) {
            best_merge(br, bk, r2, k2);
            ss += a2;
            ss2 += b2;
        }
    }
    if (T <= 32) {
        if (live && t == 0) {
            p.rb[j].r = br;
            p.rb[j].key = bk;
            p.rb[j].ssum = ss;
            p.rb[j].ssum2 = ss2;
        }
        return;
    }
    const int wid = threadIdx.x >> 5;
    if (lane == 0) {
        red_r[wid] = br;
        red_k[wid] = bk;
        red_s[wid] = ss;
        red_s2[wid] = ss2;
    }
    __syncthreads();
    if (live && t == 0) {
        const int w0 = team * (T / 32);
        for (int q = 1; q < T / 32; ++q) {
            best_merge(br, bk, red_r[w0 + q], red_k[w0 + q]);
            ss += red_s[w0 + q];
            ss2 += red_s2[w0 + q];
        }
        p.rb[j].r = br;
        p.rb[j].key = bk;
        p.rb[j].ssum = ss;
        p.rb[j].ssum2 = ss2;
    }
}

// The lags x of image row iy (lag row y) whose overlap's box and oval are
// legal, as one interval (empty: lo > hi): the box width is min(w1, w2, x + w1,
// w2 - x), so widths >= omin are an interval of x, and so is a row of the
// oval.  Exact when span_exact.
#define OVAL_SPAN 46340   // squares up to here are ints, as oval_ok's
__device__ __forceinline__ bool span_exact(const PairDev &p, const LagRow &q)
{
    return !q.tbl && q.omax == 0x7fffffff && !(p.oval_on && p.orx > OVAL_SPAN);
}
__device__ __forceinline__ void legal_span(const PairDev &p, const LagRow &q, int iy, int &lo,
                                           int &hi)
{
    lo = p.xlo;
    hi = p.xhi;
    if (q.omin > min(q.w1, q.w2)) {
        hi = lo - 1;
        return;
    }
    lo = max(lo, q.omin - q.w1);
    hi = min(hi, q.w2 - q.omin);
    if (!p.oval_on || p.orx > OVAL_SPAN)
        return;
    if (iy < p.ocy - p.ory || iy > p.ocy + p.ory) {
        hi = lo - 1;
        return;
    }
    const int y = iy - p.ocy;
    const double base = p.oasq * y * y;   // oval_ok's terms
    const int dmax = p.orx;
    auto in = [&](int d) { return d <= dmax && !((double)(d * d) + base > p.orx2); };
    int d = min(dmax, (int)sqrtf(fmaxf((float)(p.orx2 - base), 0.f)));
    while (d >= 0 && !in(d))
        --d;
    while (in(d + 1))
        ++d;
    lo = max(lo, p.ocx - d - p.cx);
    hi = min(hi, p.ocx + d - p.cx);
}

__device__ __forceinline__ bool key_better(float a, int ka, float b, int kb)
{
    return a > b || (a == b && ka < kb);
}

// Lag rows of S-key jobs without a mincor (the sweep's correlator): one inverse
// per row; S = c / (Nx Ny) is strictly increasing in the FP32 inverse value c,
// so the scan compares c itself (same argmax, same ties); the S statistics
// are compensated FP32 sums of c and c^2.
// A CTA takes row groups blockIdx.x, blockIdx.x + gridDim.x, ... of its job, the
// next group's spectrum rows in flight (second buffer) while it transforms and
// scans this one: with one group per CTA the warps waited for descriptor and
// rows at a third of the SM's occupancy.  A row's legal lags are an interval, so
// the scan compares c inside it and looks the point counts up once, at the
// row's best lag (and lag by lag only where that one fails): looked up at
// every lag that beat the thread's best so far, in nearly every step some
// lane of the warp did (4340 instructions per warp and row, of which the
// transform is a fifth).  Measured on the 1024 x 1024 transforms of 256^2
// thumbnails: 3.35 -> 2.30 us per correlator call in a large batch, 22.9 -> 16.8 us
// for one call.
template <int L>
__global__ void __launch_bounds__(256, 3) k2_lagss(PairDev *pairs, const float2 *__restrict__ tw)
{
    grid_dep();
    using F = RegFFT<L, +1>;
    static_assert(F::SMEM <= lag_pitch<L>(), "the exchange buffer fits the team's row region");
    constexpr int R = F::R, T = F::T, G = 256 / T, W = T < 32 ? T : 32;
    constexpr int PITCH = lag_pitch<L>();
    extern __shared__ float2 smem[];   // two buffers of G rows
    __shared__ float red_c[8];
    __shared__ int red_k[8];
    __shared__ double red_s[8], red_s2[8];
    const PairDev &p = pairs[blockIdx.y];
    if (p.status != 0)
        return;
    const int xlo = p.xlo, xhi = p.xhi, ylo = p.ylo, Nx = p.Nx;
    const int Wy = p.yhi - ylo + 1, Wx = xhi - xlo + 1;
    const int team = threadIdx.x / T, t = threadIdx.x - team * T;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const float2 *__restrict__ Q = p.Q;
    const int step = gridDim.x * G;
    auto fetch = [&](int j0, int b) {
        float2 *base = smem + b * (G * PITCH);
        for (int e = threadIdx.x; e < (L + 1) * G; e += 256) {
            const int kx = e / G, g = e - kx * G;
            cp_async8(&base[g * PITCH + padi(kx)], &Q[(long long)kx * Wy + min(j0 + g, Wy - 1)]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int j0 = blockIdx.x * G, buf = 0;
    if (j0 >= Wy)
        return;
    fetch(j0, 0);
    for (; j0 < Wy; j0 += step, buf ^= 1) {
        if (j0 + step < Wy) {
            fetch(j0 + step, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const int j = j0 + team;
        const bool live = j < Wy;
        float2 *reg = smem + (buf * G + team) * PITCH;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int k = t + r * T;
            float2 a = reg[padi(k)];
            float2 b = cconj(reg[padi(L - k)]);
            if (k == 0) {
                a.y = 0.f;
                b.y = 0.f;
            }
            const float2 e = cadd(a, b);
            const float2 dd = csub(a, b);
            float2 wv = __ldg(&tw[2 * L + k]);
            wv.y = -wv.y;
            const float2 o = cmul(dd, wv);
            v[r] = make_float2(e.x - o.y, e.y + o.x);
        }
        F::run_team(v, reg, t, tw, team);   // the team's own row
        team_sync<T>(team);
        float *C = (float *)reg;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int n = t + r * T;
            *(float2 *)(C + 2 * n) = v[r];
        }
        team_sync<T>(team);
        float bc = 0.f;
        int bk = 0x7fffffff;   // none
        double ss = 0.0, ss2 = 0.0;
        const int y = ylo + j, iy = y + p.cy;
        const int key0 = iy * p.wR + p.cx;   // key of lag x: key0 + x
        LagRow q;
        int xl = 0, xr = -1;
        bool slow = false;
        if (live) {
            q = lag_row(p, y);
            slow = !span_exact(p, q);
            if (!slow)
                legal_span(p, q, iy, xl, xr);
            float fs = 0.f, fe = 0.f, fq = 0.f, fqe = 0.f;
            float *rf = (float *)p.rr + (long long)j * Wx - xlo;
            for (int x = xlo + t; x <= xhi; x += T) {
                const float c = C[x < 0 ? x + Nx : x];
                two_sum_acc(fs, fe, c);
                const float c2 = __fmul_rn(c, c);
                two_sum_acc(fq, fqe, c2);
                fqe = __fadd_rn(fqe, __fmaf_rn(c, c, -c2));
                rf[x] = c;
                // this thread's lags come in increasing key order: a tie never wins
                if (x >= xl && x <= xr && (bk == 0x7fffffff || c > bc)) {
                    bc = c;
                    bk = key0 + x;
                }
            }
            ss = (double)fs + (double)fe;
            ss2 = (double)fq + (double)fqe;
        }
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) {
            const float c2 = __shfl_xor_sync(0xffffffff, bc, o);
            const int k2 = __shfl_xor_sync(0xffffffff, bk, o);
            if (k2 != 0x7fffffff && (bk == 0x7fffffff || key_better(c2, k2, bc, bk))) {
                bc = c2;
                bk = k2;
            }
            ss += __shfl_xor_sync(0xffffffff, ss, o);
            ss2 += __shfl_xor_sync(0xffffffff, ss2, o);
        }
        // the group's best lag (all its lanes hold it) against the count rule
        if (live && !slow && q.cnt && bk != 0x7fffffff) {
            int l, h;
            slow = !lag_row_legal(p, q, bk - key0, l, h);
        }
        if (__any_sync(0xffffffff, slow)) {
            if (slow) {
                bk = 0x7fffffff;
                for (int x = xlo + t; x <= xhi; x += T) {
                    const float c = C[x < 0 ? x + Nx : x];
                    double rv;
                    if ((bk == 0x7fffffff || c > bc) && lag_eval(p, q, x, 0.0, false, rv) &&
                        oval_ok(p, x + p.cx, iy)) {
                        bc = c;
                        bk = key0 + x;
                    }
                }
            }
#pragma unroll
            for (int o = W / 2; o > 0; o >>= 1) {
                const float c2 = __shfl_xor_sync(0xffffffff, bc, o);
                const int k2 = __shfl_xor_sync(0xffffffff, bk, o);
                if (k2 != 0x7fffffff && (bk == 0x7fffffff || key_better(c2, k2, bc, bk))) {
                    bc = c2;
                    bk = k2;
                }
            }
        }
        if constexpr (T > 32) {
            if (lane == 0) {
                red_c[wid] = bc;
                red_k[wid] = bk;
                red_s[wid] = ss;
                red_s2[wid] = ss2;
            }
            __syncthreads();
            if (t == 0) {
                const int w0 = team * (T / 32);
                for (int m = 1; m < T / 32; ++m) {
                    const float c2 = red_c[w0 + m];
                    const int k2 = red_k[w0 + m];
                    if (k2 != 0x7fffffff && (bk == 0x7fffffff || key_better(c2, k2, bc, bk))) {
                        bc = c2;
                        bk = k2;
                    }
                    ss += red_s[w0 + m];
                    ss2 += red_s2[w0 + m];
                }
            }
        }
        if (live && t == 0) {
            RowBest rb;
            rb.r = bk == 0x7fffffff ? -1.0e30 : (double)bc;
            rb.key = bk == 0x7fffffff ? 0x7fffffffffffffffLL : (long long)bk;
            rb.ssum = ss;
            rb.ssum2 = ss2;
            p.rb[j] = rb;
        }
        __syncthreads();   // the buffer is copied into again, red_* written again
    }
}

// an FP32 number as an integer that orders the same way, and back
__host__ __device__ __forceinline__ int ord_float(float f)
{
#ifdef __CUDA_ARCH__
    const int b = __float_as_int(f);
#else
    int b;
    memcpy(&b, &f, 4);
#endif
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float from_ord_float(int o)
{
    return __int_as_float(o ^ ((o >> 31) & 0x7fffffff));
}

// R of a lag of the lag image (CorrImagesR: the value the R image holds there,
// legal or not), FP64 as RCalc::CalcR.
__device__ __forceinline__ double img_r(const PairDev &p, int ix, int iy)
{
    const float c = ((const float *)p.rr)[(long long)iy * p.wR + ix];
    double r;
    lag_eval(p, lag_row(p, iy - p.cy), ix - p.cx,
             (double)c * (1.0 / ((double)p.Nx * (double)p.Ny)), true, r);
    return r;
}

// An upper bound of R at a lag, FP32: box sums of the FP32 tables, with the
// error that their truncation (2^-23 of each corner) and the FP32 arithmetic
// can have made.  Infinite or NaN where the bound says nothing.
__device__ __forceinline__ float4 row_box_f(const float2 *__restrict__ t, int oT, int oB, int L,
                                            int R)
{
    // sums S, Q and the errors they may carry
    float2 r = __ldg(t + oT + R);
    float as = fabsf(r.x);
    const float top = r.y;   // sum v^2 grows along both axes: the largest corner
    if (L > 0) {
        const float2 a = __ldg(t + oT + L - 1);
        r.x -= a.x;
        r.y -= a.y;
        as += fabsf(a.x);
    }
    if (oB >= 0) {
        const float2 b = __ldg(t + oB + R);
        r.x -= b.x;
        r.y -= b.y;
        as += fabsf(b.x);
        if (L > 0) {
            const float2 c = __ldg(t + oB + L - 1);
            r.x += c.x;
            r.y += c.y;
            as += fabsf(c.x);
        }
    }
    // per corner 2^-23, per difference 2^-24 of an operand: 2^-21 of the sum of
    // magnitudes covers both with room
    return make_float4(r.x, r.y, 4.8e-7f * as, 1.9e-6f * top);
}

__device__ __forceinline__ float r_bound(float n, float cs, const float4 &A, const float4 &B,
                                         float mu1, float mu2)
{
    const float EPS = 4.8e-7f;   // a few FP32 roundings of a term
    const float a = A.x - n * mu1, b = B.x - n * mu2;
    const float ea = A.z + EPS * (fabsf(A.x) + fabsf(n * mu1));
    const float eb = B.z + EPS * (fabsf(B.x) + fabsf(n * mu2));
    const float d1 = n * A.y - A.x * A.x, d2 = n * B.y - B.x * B.x;
    const float e1 = n * A.w + (2.0f * fabsf(A.x) + A.z) * A.z + EPS * (n * A.y + A.x * A.x);
    const float e2 = n * B.w + (2.0f * fabsf(B.x) + B.z) * B.z + EPS * (n * B.y + B.x * B.x);
    const float num = n * cs - a * b + (fabsf(a) + ea) * eb + fabsf(b) * ea +
                      EPS * (fabsf(n * cs) + fabsf(a * b));
    const float lo1 = d1 - e1, lo2 = d2 - e2;
    if (!(lo1 > 1e-30f && lo2 > 1e-30f && lo1 < 1e30f && lo2 < 1e30f))
        return __int_as_float(0x7f800000);
    // (num < 0: the larger denominator would bound it; 0 does)
    return fmaxf(num, 0.0f) * (rsqrtf(lo1) * rsqrtf(lo2)) * (1.0f + 1.0e-6f) + 1.0e-6f;
}

// The same bound for integer pixels, whose box sums are exact.  FP32 rounds n cs
// and a b, and where an overlap lies far from the image's mean they cancel:
// 100 grey levels off with a deviation of 0.5, the rounded R is 2e-3 off and
// more.  So their magnitudes enter, as in r_bound.  FP64 itself rounds n Q and
// S^2: e64 n^2 is more than that, e64 being 2^-51 times the largest pixel value
// squared.  (n Q - S^2 of 16-bit pixels may pass 2^64; what is left of it then is
// less, and bounds R too.)  Infinite where the flat-overlap guard may hold.
__device__ __forceinline__ float r_bound_int(int n, float cs, const longlong2 &A,
                                             const longlong2 &B, int m1, int m2, float e64)
{
    typedef unsigned long long u64;
    const float EPS = 4.8e-7f;   // a few FP32 roundings of a term
    const float f1 = u64_to_float((u64)n * (u64)A.y - (u64)A.x * (u64)A.x);
    const float f2 = u64_to_float((u64)n * (u64)B.y - (u64)B.x * (u64)B.x);
    const float fn = __int2float_rn(n), nc = fn * cs;
    const float ab = i64_to_float(A.x - (long long)n * m1) * i64_to_float(B.x - (long long)n * m2);
    if (!(f1 * f2 > fn * fn * 1.001e-9f))
        return __int_as_float(0x7f800000);
    const float i1 = rsqrtf(f1), i2 = rsqrtf(f2);
    const float num = fmaxf(nc - ab, 0.0f) + EPS * (fabsf(nc) + fabsf(ab));
    return num * (i1 * i2) * (1.0f + 1.0e-6f) + fn * fn * e64 * (i1 * i1 + i2 * i2) + 1.0e-6f;
}

// CorrImagesR's scan of the lag image k2_lagrow wrote: one warp per lag row.
// R itself is FP64 (RCalc::CalcR, clamped to (-1, 1)), and this GPU computes
// FP64 two lanes per clock and SM: with R, its box sums, conversions and
// comparisons in FP64 at every lag the scan took 1063 of 1543 us for 24 pairs
// of 300 x 421.  So each lag's R is first bounded from above without FP64 --
// integer images from their exact sums, others from FP32 copies of the tables
// -- and the FP64 R, the counts and the exact comparison are made where the
// bound reaches the best R that any row of the job has found so far (p.reach;
// what is skipped lies below that one, so the result does not depend on the
// rows' order): 234 us.  grid (ceil(max Wy / LAGSCAN_ROWS), njobs), block
// 32 * LAGSCAN_ROWS.
template <bool INT>
__device__ __forceinline__ void scan_row_img(const PairDev &p, const LagRow &q, int j, int lo,
                                             int hi, bool check, int *job_reach, double &br,
                                             int &bk)
{
    const int lane = threadIdx.x & 31, y = p.ylo + j, iy = y + p.cy;
    const float *__restrict__ row =
        (const float *)p.rr + (long long)j * (p.xhi - p.xlo + 1) - p.xlo;
    // 1 / (Nx Ny): CorrImages grids are powers of two
    const double inv = __hiloint2double((1023 - p.logNx - p.logNy) << 20, 0);
    const double mincor = p.mincor;
    const float invf = (float)inv;
    const int key0 = iy * p.wR + p.cx;   // key of lag x: key0 + x
    const float mu1 = (float)p.mu[0], mu2 = (float)p.mu[1];
    const int m1 = INT ? (int)p.mu[0] : 0, m2 = INT ? (int)p.mu[1] : 0;
    const float e64 = p.dt[0] == ALN_U8 && p.dt[1] == ALN_U8 ? 2.9e-11f : 1.91e-6f;
    float reach = from_ord_float(*(volatile int *)job_reach);   // R below it cannot win
#pragma unroll 2
    for (int x0 = lo; x0 <= hi; x0 += 32) {
        const int x = min(x0 + lane, hi);
        const int L2 = max(0, x), R2 = max(min(q.w2 - 1, x + q.w1 - 1), L2);
        const int n = (R2 - L2 + 1) * q.olh;
        const float c = ld_chain(row + x);
        float top;
        if (INT) {
            const longlong2 A = row_box_i(p, q, 0, n, L2 - x, R2 - x);
            const longlong2 B = row_box_i(p, q, 1, n, L2, R2);
            top = r_bound_int(n, c * invf, A, B, m1, m2, e64);
        } else {
            top = r_bound((float)n, c * invf,
                          row_box_f(p.satf[0], q.oT[0], q.oB[0], L2 - x, R2 - x),
                          row_box_f(p.satf[1], q.oT[1], q.oB[1], L2, R2), mu1, mu2);
        }
        const bool cand = x0 + lane <= hi && !(top < reach);   // (NaN: look closer)
        if (__any_sync(0xffffffff, cand)) {
            if (cand) {
                double rv;
                bool ok = lag_eval(p, q, x, (double)c * inv, true, rv);
                if (check)
                    ok = ok && oval_ok(p, x + p.cx, iy);
                if (ok && (mincor <= 0.0 || rv > mincor) &&
                    (rv > br || (rv == br && key0 + x < bk))) {
                    br = rv;
                    bk = key0 + x;
                }
            }
            const int m = __reduce_max_sync(
                0xffffffff, ord_float(bk == 0x7fffffff ? -2.0f : __double2float_rd(br)));
            reach = fmaxf(reach, from_ord_float(m));
            if (lane == 0 && m > *(volatile int *)job_reach)
                reach = fmaxf(reach, from_ord_float(atomicMax(job_reach, m)));
            reach = __shfl_sync(0xffffffff, reach, 0);
        }
    }
}

__global__ void __launch_bounds__(32 * LAGSCAN_ROWS) k2_imgscan(PairDev *pairs)
{
    grid_dep();
    const PairDev &p = pairs[blockIdx.y];
    if (p.status != 0)
        return;
    const int j = blockIdx.x * LAGSCAN_ROWS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= p.yhi - p.ylo + 1)
        return;
    const int y = p.ylo + j;
    const LagRow q = lag_row(p, y);
    const bool check = !span_exact(p, q);
    int lo, hi;
    legal_span(p, q, y + p.cy, lo, hi);
    double br = -1.0e30;
    int bk = 0x7fffffff;
    // (16-bit rows of 2^20 pixels and more take the FP64 R at each lag)
    if (!p.satf[0] && r_int_ok(p, (long long)min(q.w1, q.w2) * q.olh)) {
        scan_row_img<true>(p, q, j, lo, hi, check, &pairs[blockIdx.y].reach, br, bk);
    } else if (p.satf[0]) {
        scan_row_img<false>(p, q, j, lo, hi, check, &pairs[blockIdx.y].reach, br, bk);
    } else {
        const double inv = __hiloint2double((1023 - p.logNx - p.logNy) << 20, 0);
        const float *row = (const float *)p.rr + (long long)j * (p.xhi - p.xlo + 1) - p.xlo;
        for (int x = lo + lane; x <= hi; x += 32) {
            double rv;
            if (lag_eval(p, q, x, (double)row[x] * inv, true, rv) &&
                (!check || oval_ok(p, x + p.cx, y + p.cy)) &&
                (p.mincor <= 0.0 || rv > p.mincor) && (bk == 0x7fffffff || rv > br)) {
                br = rv;
                bk = (y + p.cy) * p.wR + p.cx + x;
            }
        }
    }
    long long k = bk == 0x7fffffff ? 0x7fffffffffffffffLL : bk;
    for (int o = 16; o > 0; o >>= 1) {
        const double r2 = __shfl_down_sync(0xffffffff, br, o);
        const long long k2 = __shfl_down_sync(0xffffffff, k, o);
        best_merge(br, k, r2, k2);
    }
    if (lane == 0) {
        RowBest rb;
        rb.r = br;
        rb.key = k;
        rb.ssum = rb.ssum2 = 0.0;
        p.rb[j] = rb;
    }
}

// The key image (the window is the whole R image) at R-image pixel (rx, ry),
// k = 0, or its neighbour k = 1..4 (0 outside the image).
__device__ double img_near(const PairDev &p, int rx, int ry, int k)
{
    const int x = rx + (k == 1 ? -1 : k == 2 ? 1 : 0), y = ry + (k == 3 ? -1 : k == 4 ? 1 : 0);
    if (x < 0 || y < 0 || x >= p.wR || y >= p.hR)
        return 0.0;
    if (p.fin & 4)   // CorrImagesR: R from the lag image
        return img_r(p, x, y);
    const long long o = (long long)y * p.wR + x;
    return p.s_float ? (double)((const float *)p.rr)[o] : p.rr[o];
}

// ParabPeak on the key image at R-image pixel (rx, ry) (neighbours must be
// > 0, 0_GEN/Correlation.cpp:2975-3010), ReturnR's offsets (:3016-3043); the
// S score 10 (S - mean) / (sd sqrt(nR)) with the sample sd for CorrImagesS
// (:3285-3289).  Writes the job's result.
__device__ void img_result(PairDev &p, int rx, int ry, double ss, double ss2, const double *v,
                           ResultDev &o)
{
    // v: the key image at the peak, left, right, below, above (img_near); the
    // FP32 c when s_float: ParabPeak's ratios and the S score are the same in
    // c units
    const int wR = p.wR, hR = p.hR;
    double xpk = rx, ypk = ry;
    const double z1 = v[0];
    double z0, z2;
    if (rx - 1 >= 0 && rx + 1 < wR && (z0 = v[1]) > 0.0 && (z2 = v[2]) > 0.0) {
        z0 = (z0 - z2) / (2 * (z0 + z2 - z1 - z1));
        if (fabs(z0) <= 8)
            xpk += z0;
    }
    if (ry - 1 >= 0 && ry + 1 < hR && (z0 = v[3]) > 0.0 && (z2 = v[4]) > 0.0) {
        z0 = (z0 - z2) / (2 * (z0 + z2 - z1 - z1));
        if (fabs(z0) <= 8)
            ypk += z0;
    }
    double r = z1;
    if (p.mode == JOB_IMAGES_S) {
        const double n = (double)wR * hR;
        const double mn = ss / n;
        const double sd = sqrt(fmax(ss2 - n * mn * mn, 0.0) / (n - 1.0));
        r = 10.0 * (z1 - mn) / (sd * sqrt(n));
    }
    p.r = r;
    p.dx = xpk + (p.x0[1] - p.x0[0]) - p.cx;
    p.dy = ypk + (p.y0[1] - p.y0[0]) - p.cy;
    p.px = rx - p.cx;
    p.py = ry - p.cy;
    p.status = ALN_OK;
    o.r = p.r;
    o.dx = p.dx;
    o.dy = p.dy;
    o.status = ALN_OK;
    o.px = p.px;
    o.py = p.py;
}

// grid (npairs), block 256: argmax over rows, ParabPeak on the key image
// (neighbours must be > 0, 0_GEN/Correlation.cpp:2975-3010), ReturnR's
// offsets (:3016-3043); CorrImagesS returns 10 (S - mean) / (sd sqrt(nR))
// with the sample sd over the whole S image (:3285-3289).
__global__ void k_final_img(PairDev *pairs, ResultDev *res)
{
    grid_dep();
    __shared__ double red_r[32], red_s[32], red_s2[32];
    __shared__ long long red_k[32];
    PairDev &p = pairs[blockIdx.x];
    if (p.status != 0)
        return;
    const int Wy = p.yhi - p.ylo + 1;
    double br = -1.0e30, ss = 0.0, ss2 = 0.0;
    long long bk = 0x7fffffffffffffffLL;
    for (int j = threadIdx.x; j < Wy; j += blockDim.x) {
        best_merge(br, bk, p.rb[j].r, p.rb[j].key);
        ss += p.rb[j].ssum;
        ss2 += p.rb[j].ssum2;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double r2 = __shfl_down_sync(0xffffffff, br, o);
        const long long k2 = __shfl_down_sync(0xffffffff, bk, o);
        const double a2 = __shfl_down_sync(0xffffffff, ss, o);
        const double b2 = __shfl_down_sync(0xffffffff, ss2, o);
        best_merge(br, bk, r2, k2);
        ss += a2;
        ss2 += b2;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        red_r[wid] = br;
        red_k[wid] = bk;
        red_s[wid] = ss;
        red_s2[wid] = ss2;
    }
    __syncthreads();
    if (threadIdx.x >= 5)
        return;
    // five threads: each finds the peak and fetches one value of the key image
    __shared__ double near[5];
    br = red_r[0];
    bk = red_k[0];
    ss = red_s[0];
    ss2 = red_s2[0];
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
        best_merge(br, bk, red_r[q], red_k[q]);
        ss += red_s[q];
        ss2 += red_s2[q];
    }
    ResultDev &o = res[blockIdx.x];
    if (bk == 0x7fffffffffffffffLL) {   // no candidate lag
        if (threadIdx.x == 0) {
            p.status = ALN_NO_PEAK;
            o.r = o.dx = o.dy = 0.0;
            o.status = ALN_NO_PEAK;
            o.px = o.py = 0;
        }
        return;
    }
    const int ry = (int)(bk / p.wR), rx = (int)(bk - (long long)ry * p.wR);
    near[threadIdx.x] = img_near(p, rx, ry, threadIdx.x);
    __syncwarp(0x1f);
    if (threadIdx.x == 0)
        img_result(p, rx, ry, ss, ss2, near, o);
}

// ---------------------------------------------------------------------------
// CorrImagesF (0_GEN/Correlation.cpp:3066-3122): F = the R image filtered by
// the 3 x 3 kernel {-1 x 8, 9} (MakeF, :2412-2492), the best isolated F peak
// (FPeak, :2580-2767), ParabPeak and ReturnR on R there
// ---------------------------------------------------------------------------

// grid (ceil(wR/32), ceil(hR/8), njobs), block (32, 8).  MakeF convolves R
// over a frame of CeilPow2(wR) x CeilPow2(hR) and then clears a guard band of
// 2 pixels (F and the candidate flags); inside the band every tap lies in R,
// so the filter is the plain 3 x 3 stencil.  F keeps its positive part; the
// reference's division by the maximum is left out: every FPeak test compares
// F values with multiples of a peak's F, so a common positive scale changes
// no decision.
__global__ void k_makef(PairDev *pairs)
{
    PairDev &p = pairs[blockIdx.z];
    if (p.status != 0 || p.mode != JOB_IMAGES_F)
        return;
    const int wR = p.wR, hR = p.hR;
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    if (x >= wR || y >= hR)
        return;
    const long long k = (long long)y * wR + x;
    const int grd = 2;
    if (x < grd || x >= wR - grd || y < grd || y >= hR - grd) {
        p.fimg[k] = 0.0;
        p.fst[k] = 0;
        return;
    }
    const double *R = p.rr;
    double f = 9.0 * R[k];
    for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx)
            if (dx || dy)
                f -= R[k + (long long)dy * wR + dx];
    p.fimg[k] = f > 0.0 ? f : 0.0;
}

// FPeak, one CTA of 1024 threads per job.  Candidates in OrderF's order (F
// descending; equal F: smaller index first) are taken one at a time: each
// thread keeps the best live candidate of its own pixels (k = t mod 1024)
// and rescans only when that one is visited or masked; a block argmax
// picks the next.  The candidate's tests run on the whole block: the four
// scans for the half-height radius ri (one warp each, 32 pixels per
// ballot), the guard-band bounds, the core mask, and the ring between ri and
// 3 ri for a neighbour above nbmaxht x peak.  The first candidate that passes
// is the peak.
#define FPK_THREADS 1024

__device__ __forceinline__ bool fpk_better(double a, long long ia, double b, long long ib)
{
    return a > b || (a == b && ia < ib);
}

__global__ void __launch_bounds__(FPK_THREADS) k_fpeak(PairDev *pairs, ResultDev *res)
{
    __shared__ double s_v[32];
    __shared__ long long s_i[32];
    __shared__ int s_dist[4];
    __shared__ long long s_pick;
    PairDev &p = pairs[blockIdx.x];
    if (p.status != 0 || p.mode != JOB_IMAGES_F)
        return;
    ResultDev &o = res[blockIdx.x];
    const int wR = p.wR, hR = p.hR;
    const long long nR = (long long)wR * hR;
    const double *F = p.fimg;
    unsigned char *st = p.fst;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double lv = -1.0;
    long long li = -1;   // this thread's best live candidate (-1: rescan)
    for (;;) {
        if (li >= 0 && (st[li] & 3))
            li = -1;
        if (li < 0) {
            lv = -1.0;
            for (long long k = tid; k < nR; k += FPK_THREADS)
                if ((st[k] & 7) == 4 && (li < 0 || fpk_better(F[k], k, lv, li))) {
                    lv = F[k];
                    li = k;
                }
        }
        // block argmax (value desc, index asc); li < 0 never wins
        double bv = li >= 0 ? lv : -2.0;
        long long bi = li >= 0 ? li : 0x7fffffffffffffffLL;
        for (int off = 16; off > 0; off >>= 1) {
            const double v2 = __shfl_down_sync(0xffffffff, bv, off);
            const long long i2 = __shfl_down_sync(0xffffffff, bi, off);
            if (fpk_better(v2, i2, bv, bi)) {
                bv = v2;
                bi = i2;
            }
        }
        if (lane == 0) {
            s_v[wid] = bv;
            s_i[wid] = bi;
        }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < FPK_THREADS / 32; ++w)
                if (fpk_better(s_v[w], s_i[w], bv, bi)) {
                    bv = s_v[w];
                    bi = s_i[w];
                }
            s_pick = bv > -1.5 ? bi : -1;
        }
        __syncthreads();
        const long long k = s_pick;
        if (k < 0)
            break;   // every candidate tried
        const double fpk = F[k], half = 0.5 * fpk, tol = p.nbmaxht * fpk;
        const int ry = (int)(k / wR), rx = (int)(k - (long long)ry * wR);
        // ri: first pixel at or below half height up, down, left, right
        if (wid < 4) {
            const int dx = wid == 2 ? -1 : (wid == 3 ? 1 : 0);
            const int dy = wid == 0 ? -1 : (wid == 1 ? 1 : 0);
            const int lim = wid == 0 ? ry : wid == 1 ? hR - 1 - ry : wid == 2 ? rx : wR - 1 - rx;
            int found = -1;
            for (int d0 = 1; d0 <= lim && found < 0; d0 += 32) {
                const int d = d0 + lane;
                bool hit = false;
                if (d <= lim)
                    hit = F[(long long)(ry + dy * d) * wR + (rx + dx * d)] <= half;
                const unsigned b = __ballot_sync(0xffffffff, hit);
                if (b)
                    found = d0 + __ffs(b) - 1;
            }
            if (lane == 0)
                s_dist[wid] = found;
        }
        __syncthreads();
        if (tid == 0) {
            int ri = 1 << 30, ok = 1;
            for (int w = 0; w < 4; ++w) {
                if (s_dist[w] < 0)
                    ok = 0;   // Ri_edge
                else
                    ri = min(ri, s_dist[w]);
            }
            if (ok && ri <= 1 && p.rr[k] < 0.1)
                ok = 0;   // Micropk
            const int ro = 3 * ri;
            if (ok && (ry - ro < 0 || ry + ro >= hR || rx - ro < 0 || rx + ro >= wR))
                ok = 0;   // Ro_edge
            st[k] |= 2;   // visited
            s_dist[0] = ok ? ri : -1;
        }
        __syncthreads();
        const int ri = s_dist[0];
        if (ri >= 0) {
            const int ro = 3 * ri, rm = max(1, ri / 3);
            // mask the core peak region
            const int mw = 2 * rm + 1;
            for (int e = tid; e < mw * mw; e += FPK_THREADS) {
                const int yy = ry - rm + e / mw, xx = rx - rm + e % mw;
                st[(long long)yy * wR + xx] |= 1;
            }
            // any pixel above tol in the ring between ri and ro
            const int ow = 2 * ro + 1;
            const long long tot = (long long)ow * ow;
            int hi = 0;
            for (long long e = tid; e < tot && !hi; e += FPK_THREADS) {
                const int yy = ry - ro + (int)(e / ow), xx = rx - ro + (int)(e % ow);
                if (yy >= ry - ri && yy <= ry + ri && xx >= rx - ri && xx <= rx + ri)
                    continue;
                hi = F[(long long)yy * wR + xx] > tol;
            }
            hi = __syncthreads_or(hi);
            if (!hi) {
                if (tid == 0) {
                    double v[5];
                    for (int m = 0; m < 5; ++m)
                        v[m] = img_near(p, rx, ry, m);
                    img_result(p, rx, ry, 0.0, 0.0, v, o);
                }
                return;
            }
        }
        __syncthreads();
    }
    if (tid == 0) {   // All peaks rejected / no candidates
        p.status = ALN_NO_PEAK;
        o.r = o.dx = o.dy = 0.0;
        o.status = ALN_NO_PEAK;
        o.px = o.py = 0;
    }
}

// ---------------------------------------------------------------------------
// CorrPatchToImage (0_GEN/Correlation.cpp:1186-1355): raw correlation over an
// N x N frame, its own lag zones, ParabPeakFFT on the raw inverse
// ---------------------------------------------------------------------------

// Per storage row: inverse real FFT -> raw values (kept for the neighbour
// look-ups), the row's best lag by the reference's zone rules:
// y > N - h1 negative, else y >= h2 dead (likewise x), disc on (x, y).
template <int L>
__global__ void k2_lagp2i(PairDev *pairs, const float2 *__restrict__ tw)
{
    using F = RegFFT<L, +1>;
    static_assert(F::SMEM <= lag_pitch<L>(), "the exchange buffer fits the team's row region");
    constexpr int R = F::R, T = F::T;
    constexpr int PITCH = lag_pitch<L>();
    extern __shared__ float2 smem[];
    __shared__ double red_r[32];
    __shared__ long long red_k[32];
    PairDev &p = pairs[blockIdx.y];
    if (p.status != 0)
        return;
    const int N = p.Nx, Wy = p.Ny;
    const int G = blockDim.x / T;
    const int team = threadIdx.x / T, t = threadIdx.x - team * T;
    const int j0 = blockIdx.x * G;
    if (j0 >= Wy)
        return;
    const int j = j0 + team;
    const bool live = j < Wy;
    float2 *sm = smem + team * PITCH;
    load_lag_rows<L, T>(smem, PITCH, p.Q, Wy, j0);
    __syncthreads();
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int k = t + r * T;
        float2 a = sm[padi(k)];
        float2 b = cconj(sm[padi(L - k)]);
        if (k == 0) {
            a.y = 0.f;
            b.y = 0.f;
        }
        const float2 e = cadd(a, b);
        const float2 dd = csub(a, b);
        float2 wv = __ldg(&tw[2 * L + k]);
        wv.y = -wv.y;
        const float2 o = cmul(dd, wv);
        v[r] = make_float2(e.x - o.y, e.y + o.x);
    }
    F::run_team(v, sm, t, tw, team);   // the team's own row
    double br = -1.0e30;
    long long bk = 0x7fffffffffffffffLL;
    if (live) {
        // storage row j; its lag row by the reference's rule
        int y = j;
        bool ydead = false;
        if (y > N - p.p2i_h1)
            y -= N;
        else if (y >= p.p2i_h2)
            ydead = true;
        const long long dy = y - p.oy;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int n = t + r * T;
            for (int h = 0; h < 2; ++h) {
                const int xs = 2 * n + h;
                const double val = h ? (double)v[r].y : (double)v[r].x;
                p.rr[(long long)j * N + xs] = val;
                if (ydead)
                    continue;
                int x = xs;
                if (x > N - p.p2i_w1)
                    x -= N;
                else if (x >= p.p2i_w2)
                    continue;
                const long long dx = x - p.ox;
                if (dx * dx + dy * dy > p.rsqr)
                    continue;
                best_merge(br, bk, val, (long long)j * N + xs);
            }
        }
    }
    const int lane = threadIdx.x & 31;
    for (int o = 16; o > 0; o >>= 1) {
        const double r2 = __shfl_down_sync(0xffffffff, br, o);
        const long long k2 = __shfl_down_sync(0xffffffff, bk, o);
        if (lane + o < 32 && (lane + o) / T == lane / T)
            best_merge(br, bk, r2, k2);
    }
    if (T <= 32) {
        if (live && t == 0) {
            p.rb[j].r = br;
            p.rb[j].key = bk;
        }
        return;
    }
    const int wid = threadIdx.x >> 5;
    if (lane == 0) {
        red_r[wid] = br;
        red_k[wid] = bk;
    }
    __syncthreads();
    if (live && t == 0) {
        const int w0 = team * (T / 32);
        for (int q = 1; q < T / 32; ++q)
            best_merge(br, bk, red_r[w0 + q], red_k[w0 + q]);
        p.rb[j].r = br;
        p.rb[j].key = bk;
    }
}

__global__ void k_final_p2i(PairDev *pairs, ResultDev *res)
{
    __shared__ double red_r[32];
    __shared__ long long red_k[32];
    PairDev &p = pairs[blockIdx.x];
    if (p.status != 0)
        return;
    const int N = p.Nx;
    double br = -1.0e30;
    long long bk = 0x7fffffffffffffffLL;
    for (int j = threadIdx.x; j < N; j += blockDim.x)
        best_merge(br, bk, p.rb[j].r, p.rb[j].key);
    for (int o = 16; o > 0; o >>= 1) {
        const double r2 = __shfl_down_sync(0xffffffff, br, o);
        const long long k2 = __shfl_down_sync(0xffffffff, bk, o);
        best_merge(br, bk, r2, k2);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        red_r[wid] = br;
        red_k[wid] = bk;
    }
    __syncthreads();
    if (threadIdx.x != 0)
        return;
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q)
        best_merge(br, bk, red_r[q], red_k[q]);
    ResultDev &o = res[blockIdx.x];
    int bigx = -1, bigy = -1;
    double biggest = -1.0E30;
    if (br > -1.0e30) {
        const int ys = (int)(bk / N), xs = (int)(bk - (long long)ys * N);
        bigy = ys > N - p.p2i_h1 ? ys - N : ys;
        bigx = xs > N - p.p2i_w1 ? xs - N : xs;
        biggest = br;
    }
    biggest /= p.p2i_norm;
    // ParabPeakFFT, d = 1, LkFFT on the raw inverse (0_GEN/Correlation.cpp:268-298,482-517)
    const double *I = p.rr;
    auto lk = [&](int x, int y) {
        if (x < 0)
            x += N;
        if (y < 0)
            y += N;
        return I[x + (long long)N * y];
    };
    double xpk = bigx, ypk = bigy;
    const int ix = bigx, iy = bigy;
    if (ix > -N && iy > -N) {
        const double z1 = lk(ix, iy);
        double z0, z2;
        if (ix - 1 >= 0 && ix + 1 < N && (z0 = lk(ix - 1, iy)) != 0.0 &&
            (z2 = lk(ix + 1, iy)) != 0.0) {
            z0 = (z0 - z2) / (2 * (z0 + z2 - z1 - z1));
            if (fabs(z0) <= 8)
                xpk += z0;
        }
        if (iy - 1 >= 0 && iy + 1 < N && (z0 = lk(ix, iy - 1)) != 0.0 &&
            (z2 = lk(ix, iy + 1)) != 0.0) {
            z0 = (z0 - z2) / (2 * (z0 + z2 - z1 - z1));
            if (fabs(z0) <= 8)
                ypk += z0;
        }
    }
    p.r = biggest;
    p.dx = xpk;
    p.dy = ypk;
    p.px = bigx;
    p.py = bigy;
    // the reference exits (44) on a normalised peak above 1.0001
    p.status = biggest > 1.0001 ? ALN_NO_PEAK : ALN_OK;
    o.r = p.r;
    o.dx = p.dx;
    o.dy = p.dy;
    o.status = p.status;
    o.px = bigx;
    o.py = bigy;
}
