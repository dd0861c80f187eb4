// stencil.cuh -- row kernels over stencil-indexed rows (sm_100a).
//
// On a grid the rows of a level take their columns from one short list of offsets (the stencil: 7
// or 27 of them), each row a subset of it, and few subsets occur (27 boundary types). The stencil
// form (build_stencil, setup.cu) keeps that list, ascending, as a kernel argument, and one byte per
// row naming the row's form: the bit mask of the offsets it has and, when the values repeat too
// (constant coefficients), the values themselves, from a table in shared memory. Otherwise the
// values are stored by slices of 32 rows, entry k of the 32 rows side by side (zero where a row has
// no entry k). No column is read: the address of entry k is the row's plus an offset that is the
// same for every row, so the loads of a row wait for nothing but its form byte, and they are
// consecutive over the lanes. One lane owns a row and adds its entries in CSR order with the same
// multiply-adds as k_rowop<1>; an offset that a row lacks is not loaded and adds a zero product, so
// the results equal k_rowop<1>'s bit for bit.
#pragma once

#include "rowops.cuh"

namespace bcmgx {

constexpr int kStThreads = 256;

template <typename T> struct StVec4;
template <> struct StVec4<float> {
    float4 u;
    __device__ __forceinline__ void lds(const float* p) { u = *(const float4*)p; }
    __device__ __forceinline__ float get(int i) const { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; }
};
template <> struct StVec4<double> {
    double2 a, b;
    __device__ __forceinline__ void lds(const double* p)
    {
        a = *(const double2*)p;
        b = *((const double2*)p + 1);
    }
    __device__ __forceinline__ double get(int i) const { return i == 0 ? a.x : i == 1 ? a.y : i == 2 ? b.x : b.y; }
};

extern __shared__ __align__(128) unsigned char st_smem[];

// y = alpha A x + beta y, y = f - A x, or one l1-Jacobi sweep (the operations of k_rowop). With stored
// values HBM bounds it: one FP32 sweep of the 7-point 256^3 diffusion level streams 755 MB instead of
// 1.27 GB and takes 142 us (5.3 TB/s) instead of 224 with int32 columns. With the table the loads of x
// do: 7-point 100^3 7.0 us instead of 10.6 with pattern-indexed slices, 27-point 160^3 47.9 instead of
// 70.6 (k_rowop_box27 below: 26.9). u: the offsets of the stencil, stencil_blocks(u) == NB. TAB: vals is the table of the forms' values (nform
// rows of 4 NB, dynamic shared memory holds it); else the stored values.
template <int OP, int NB, bool TAB, typename T, typename XT, typename FT, typename MT, typename YT>
__global__ void __launch_bounds__(kStThreads) k_rowop_stencil(int n, int u, StencilOffs so,
    const unsigned char* __restrict__ form, const unsigned* __restrict__ fmask, int nform, const T* __restrict__ vals,
    const XT* __restrict__ x, const FT* __restrict__ f, const MT* __restrict__ M, YT* __restrict__ y, double alpha,
    double beta, const int* __restrict__ skip)
{
    using AT = typename Acc<T>::type;
    constexpr int UP = 4 * NB;
    constexpr int UMIN = NB == 2 ? 1 : NB == 4 ? 9 : NB == 7 ? 17 : 29;   // the least u of this NB
    __shared__ unsigned mask_s[256];
    T* tab_s = (T*)st_smem;
    for (int i = threadIdx.x; i < nform; i += kStThreads) mask_s[i] = __ldg(fmask + i);
    if constexpr (TAB)
        for (int i = threadIdx.x; i < nform * UP; i += kStThreads) tab_s[i] = __ldg(vals + i);
    // the tables above are written during set-up only; vectors are read after the wait
    dep_wait();
    dep_release();
    if (skip && *skip) return;
    __syncthreads();
    const unsigned full = u == 32 ? 0xffffffffu : (1u << u) - 1u;
    const int lane = threadIdx.x & 31;
    const long nt = ((long)n + kStThreads - 1) / kStThreads;
    for (long t = blockIdx.x; t < nt; t += gridDim.x) {
        const int r = (int)(t * kStThreads) + (int)threadIdx.x;
        const bool live = r < n;
        const int rr = live ? r : n - 1;
        const int id = __ldg(form + rr);
        const T* vp = nullptr;
        if constexpr (!TAB) vp = vals + (long)(r >> 5) * (32L * u) + lane;
        T v[UP];
        if constexpr (!TAB) {
#pragma unroll
            for (int k = 0; k < UP; k++) v[k] = (k < UMIN || k < u) && live ? ld_stream(vp + 32 * k) : T(0);
        }
        AT o1 = 0, o2 = 0, o3 = 0;
        if (live) {
            if (OP == OP_AXPBY) {
                if (beta != 0.0) o1 = (AT)y[r];
            } else if (OP == OP_RESID) {
                o1 = (AT)ld_stream(f + r);
            } else {
                o1 = (AT)ld_stream(f + r);
                o2 = (AT)ld_stream(M + r);
                o3 = (AT)ld_ro(x + r);
            }
        }
        const unsigned m = mask_s[id];
        XT xv[UP];
        if (__all_sync(0xffffffffu, m == full)) {
#pragma unroll
            for (int k = 0; k < UP; k++)
                xv[k] = (k < UMIN || k < u) ? ld_ro(x + (rr + so.o[k])) : XT(0);
        } else {
#pragma unroll
            for (int k = 0; k < UP; k++) xv[k] = ((m >> k) & 1u) ? ld_ro(x + (rr + so.o[k])) : XT(0);
        }
        AT s = 0;
        if constexpr (TAB) {
            const T* tp = tab_s + id * UP;
#pragma unroll
            for (int q = 0; q < NB; q++) {
                StVec4<T> c;
                c.lds(tp + 4 * q);
#pragma unroll
                for (int i = 0; i < 4; i++) s += (AT)c.get(i) * (AT)xv[4 * q + i];
            }
        } else {
#pragma unroll
            for (int k = 0; k < UP; k++) s += (AT)v[k] * (AT)xv[k];
        }
        if (live) {
            if (OP == OP_AXPBY) {
                AT o = (AT)alpha * s;
                if (beta != 0.0) o += (AT)beta * o1;
                y[r] = (YT)o;
            } else if (OP == OP_RESID) {
                y[r] = (YT)(o1 - s);
            } else {
                y[r] = (YT)(((-s + o1) / o2) + o3);
            }
        }
    }
}

// The same operations on a 27-point box with a table of values: the offsets are those of three
// planes of three lines, pl[a] + (b - 1) s + (c - 1) for entry 9 a + 3 b + c (stencil_box checks it;
// pl[1] = 0). A lane takes P rows s apart, the same place on P consecutive lines: the three lines
// that a row reads in a plane are shared with its neighbours', so P rows load 9 (P + 2) values of x
// instead of 27 P, from addresses that the three entries of a line share. A warp whose rows are
// all of one form with every offset (the inside of the box) takes the values as broadcasts and tests
// nothing; in any other, a value is loaded when one of the P rows has its column and added to the
// rows that have it. Rows q P s + p s + t (t < s, p < P) of a lane: the last group may pass n.
// Measured at 160^3 (FP32 sweep): k_rowop_stencil 47.9 us (240 warp instructions per 32 rows), P = 2
// 28.9, P = 4 26.9 us: 2.6 TB/s on its 70 MB of vectors and form bytes, most of them in L2, bound by the
// loads of x and by issue. An FP64 product and its dots 78.7 -> 61.9 us (P = 2). launch_box chooses P.
template <int OP, int P, typename T, typename XT, typename FT, typename MT, typename YT>
__global__ void __launch_bounds__(kStThreads) k_rowop_box27(int n, int s, int pl0, int pl2,
    const unsigned char* __restrict__ form, const unsigned* __restrict__ fmask, int nform, const T* __restrict__ vals,
    const XT* __restrict__ x, const FT* __restrict__ f, const MT* __restrict__ M, YT* __restrict__ y, double alpha,
    double beta, const int* __restrict__ skip)
{
    using AT = typename Acc<T>::type;
    constexpr unsigned kFull = (1u << 27) - 1u;
    constexpr int W = 36;   // table row: three planes of 9 values and 3 of padding
    __shared__ unsigned mask_s[256];
    T* tab_s = (T*)st_smem;
    for (int i = threadIdx.x; i < nform; i += kStThreads) mask_s[i] = __ldg(fmask + i);
    for (int i = threadIdx.x; i < nform * W; i += kStThreads) {
        const int id = i / W, w = i % W;
        tab_s[i] = w % 12 < 9 ? __ldg(vals + id * 28 + (w / 12) * 9 + w % 12) : T(0);
    }
    // the tables above are written during set-up only; vectors are read after the wait
    dep_wait();
    dep_release();
    if (skip && *skip) return;
    __syncthreads();
    const long items = ((long)n + (long)P * s - 1) / ((long)P * s) * s;
    const long stride = (long)gridDim.x * kStThreads;
    const int dq = (int)(stride / s), dt = (int)(stride % s);
    const long i0 = (long)blockIdx.x * kStThreads + threadIdx.x;
    int q = (int)(i0 / s), t = (int)(i0 % s);
    for (long i = i0 - threadIdx.x; i < items; i += stride) {
        const long base = (long)q * P * s + t;   // rows of lanes past the last group are all >= n
        int id[P];
        unsigned m[P];
        AT o1[P], o2[P], o3[P];
        bool one = true;
#pragma unroll
        for (int p = 0; p < P; p++) {
            const long r = base + (long)p * s;
            id[p] = r < n ? (int)__ldg(form + r) : -1;
            o1[p] = o2[p] = o3[p] = 0;
            if (r < n) {
                if (OP == OP_AXPBY) {
                    if (beta != 0.0) o1[p] = (AT)y[r];
                } else {
                    o1[p] = (AT)ld_stream(f + r);
                    if (OP == OP_JACOBI) o2[p] = (AT)ld_stream(M + r);
                }
            }
        }
#pragma unroll
        for (int p = 0; p < P; p++) {
            m[p] = id[p] >= 0 ? mask_s[id[p]] : 0u;
            one = one && id[p] == id[0];
        }
        const int id0 = __shfl_sync(0xffffffffu, id[0], 0);   // by every lane, whatever its rows
        one = one && m[0] == kFull && id[0] == id0;
        AT acc[P];
#pragma unroll
        for (int p = 0; p < P; p++) acc[p] = 0;
        const XT* xb = x + base;
        if (__all_sync(0xffffffffu, one)) {
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const XT* xl = xb + ((a == 0 ? pl0 : a == 1 ? 0 : pl2) - s);
                XT xv[P + 2][3];
#pragma unroll
                for (int l = 0; l < P + 2; l++, xl += s)
#pragma unroll
                    for (int c = 0; c < 3; c++) xv[l][c] = ld_ro(xl + (c - 1));
                StVec4<T> cv[3];
#pragma unroll
                for (int k = 0; k < 3; k++) cv[k].lds(tab_s + id[0] * W + 12 * a + 4 * k);
#pragma unroll
                for (int p = 0; p < P; p++) {
#pragma unroll
                    for (int k = 0; k < 9; k++) acc[p] += (AT)cv[k / 4].get(k % 4) * (AT)xv[p + k / 3][k % 3];
                    if (OP == OP_JACOBI && a == 1) o3[p] = (AT)xv[p + 1][1];
                }
            }
        } else {
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const XT* xl = xb + ((a == 0 ? pl0 : a == 1 ? 0 : pl2) - s);
                unsigned need = 0u;   // bit 3 l + c: the columns of line l that some row has
#pragma unroll
                for (int p = 0; p < P; p++) need |= ((m[p] >> (9 * a)) & 511u) << (3 * p);
                XT xv[P + 2][3];
#pragma unroll
                for (int l = 0; l < P + 2; l++, xl += s)
#pragma unroll
                    for (int c = 0; c < 3; c++) xv[l][c] = ((need >> (3 * l + c)) & 1u) ? ld_ro(xl + (c - 1)) : XT(0);
#pragma unroll
                for (int p = 0; p < P; p++) {
                    StVec4<T> cv[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) cv[k].lds(tab_s + max(id[p], 0) * W + 12 * a + 4 * k);
#pragma unroll
                    for (int k = 0; k < 9; k++)
                        if ((m[p] >> (9 * a + k)) & 1u) acc[p] += (AT)cv[k / 4].get(k % 4) * (AT)xv[p + k / 3][k % 3];
                }
            }
            if (OP == OP_JACOBI)
#pragma unroll
                for (int p = 0; p < P; p++)
                    if (id[p] >= 0) o3[p] = (AT)ld_ro(xb + (long)p * s);
        }
#pragma unroll
        for (int p = 0; p < P; p++) {
            const long r = base + (long)p * s;
            if (r < n) {
                if (OP == OP_AXPBY) {
                    AT o = (AT)alpha * acc[p];
                    if (beta != 0.0) o += (AT)beta * o1[p];
                    y[r] = (YT)o;
                } else if (OP == OP_RESID) {
                    y[r] = (YT)(o1[p] - acc[p]);
                } else {
                    y[r] = (YT)(((-acc[p] + o1[p]) / o2[p]) + o3[p]);
                }
            }
        }
        q += dq;
        t += dt;
        if (t >= s) {
            t -= s;
            q++;
        }
    }
}

}  // namespace bcmgx
