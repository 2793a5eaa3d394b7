// Diagonal-format SpMV kernels: DIA and BDIA (banded DIA).
//
// Layout (matrix_storage.h:27-94): diagonal d of `len` rows at data[d*len + row],
// x index row + offset.  Out-of-range columns hold 0 in the data and are skipped
// here by a predicated load instead of the reference's zero-extended copy of x
// (spmv_cocktail.cpp:253 cpy_vec_extended), so no extended vector has to be kept
// in sync with x.
#pragma once

#include "common.cuh"

namespace csp {
namespace dev {

constexpr int kDiaThreads = 256;

__device__ __forceinline__ float ldx_guarded(const float* __restrict__ x, int c, int n)
{
    return (c >= 0 && c < n) ? __ldg(x + c) : 0.0f;
}

// DIA, ROWS rows per thread strided by the CTA width: coalesced 4-byte loads of every
// diagonal, offsets staged in shared memory (spmv_dia.cl gpu_dia).
template <class V, int ROWS>
__global__ void __launch_bounds__(kDiaThreads) dia_kernel(const int* __restrict__ offsets, const V* __restrict__ data,
                                                          const float* __restrict__ x, float* __restrict__ y,
                                                          int m, int n, int ndia, int len)
{
    extern __shared__ int s_off[];
    for (int i = threadIdx.x; i < ndia; i += kDiaThreads) s_off[i] = __ldg(offsets + i);
    __syncthreads();
    const int base = blockIdx.x * (kDiaThreads * ROWS) + threadIdx.x;
    float acc[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; q++) acc[q] = 0.0f;
    for (int d = 0; d < ndia; d++) {
        const int o = s_off[d];
        const V* dd = data + (size_t)d * len;
#pragma unroll
        for (int q = 0; q < ROWS; q++) {
            const int r = base + q * kDiaThreads;
            if (r < m) acc[q] += Val<V>::ld(dd + r) * ldx_guarded(x, r + o, n);
        }
    }
#pragma unroll
    for (int q = 0; q < ROWS; q++) {
        const int r = base + q * kDiaThreads;
        if (r < m) y[r] += acc[q];
    }
}

// DIA and BDIA, four consecutive rows per thread with 128-bit copies of the diagonals
// (spmv_dia.cl gpu_dia_v4, spmv_bdia.cl gpu_bdia_v4_nlvec; len is a multiple of 4):
// yout = yin + A x.  The host cuts the diagonals, in their stored order, into groups of at
// most kDiaGroup with consecutive offsets (groups[g] = {first offset, diagonals}).
//
// HBM bounds it once enough bytes are in flight.  Values held in registers ahead of their
// use cost the occupancy they were to make up for (5 diagonals ahead 81 us on the 160^3
// stencil, 9 ahead 84, 14 ahead 90; BF16 slower than one at a time), so every thread
// copies its own four rows of the next kDiaStages - 1 groups into shared memory with
// cp.async and reads them back itself: no barrier, no registers.  A group reads its x once, as
// the two or three aligned 128-bit vectors around its 4 + (diagonals - 1) entries, picked
// by the offset's residue, which is the same for the whole CTA.  CTAs whose rows leave the
// matrix for some offset (omin .. omax) take guarded scalar loads of x.  x and y of any
// 4-byte alignment are taken (the adjoint's vectors are the caller's).
// Measured on one B200 (27 diagonals, before: a scalar guarded x load per entry, or for
// BDIA x staged per band between two barriers): 160^3 FP32 BDIA 94.5 -> 80.5 us (6.1 TB/s),
// 97^3 FP32 DIA 33.5 -> 20.8, 150^3 BF16 70 -> 53.  FP32 also requests the next group's
// window ahead (97^3: 22.8 us without) and does best at 3 CTAs an SM; BF16 keeps 5 CTAs
// resident instead (53 us against 66).
//
// The first groups are requested before grid_dependency(), so that they overlap the previous
// step of csp_iterate.
constexpr int kDiaRowsThreads = 256;
constexpr int kDiaGroup = 3;   // 3 + 4 + (kDiaGroup - 1) floats: at most three vectors
template <class V> struct DiaStages { static constexpr int n = sizeof(V) == 4 ? 2 : 4; };   // powers of two: the same bytes in flight

// acc += a[k] * x[S + k ..], the window v starting S floats before the group's first entry
template <int S>
__device__ __forceinline__ void dia_fma(float4& acc, const float4 (&a)[kDiaGroup], const float (&v)[12], int w)
{
#pragma unroll
    for (int k = 0; k < kDiaGroup; k++) {
        if (k >= w) break;
        acc.x += a[k].x * v[S + k];
        acc.y += a[k].y * v[S + k + 1];
        acc.z += a[k].z * v[S + k + 2];
        acc.w += a[k].w * v[S + k + 3];
    }
}

template <class V>
__global__ void __launch_bounds__(kDiaRowsThreads, sizeof(V) == 4 ? 3 : 5) dia_rows_kernel(const int2* __restrict__ groups, const V* __restrict__ data,
                                                                   const float* x, const float* yin, float* yout, int m, int n,
                                                                   int ng, int len, int omin, int omax)
{
    constexpr bool kAhead = sizeof(V) == 4;   // the next group's window is in flight
    constexpr int NS = DiaStages<V>::n, ES = 4 * sizeof(V);   // bytes of a thread's four values
    __shared__ __align__(16) unsigned char s_val[NS * kDiaGroup][kDiaRowsThreads * ES];
    const int rb = blockIdx.x * (kDiaRowsThreads * 4);
    const int r0 = rb + 4 * threadIdx.x;
    if (r0 >= m) return;
    const V* __restrict__ p = data + r0;
    unsigned char* own = s_val[0] + threadIdx.x * ES;
    const unsigned own_addr = (unsigned)__cvta_generic_to_shared(own);
    auto issue = [&](int g) {
        if (g < ng) {
            const int w = __ldg(&groups[g].y);
            const unsigned dst = own_addr + (g & (NS - 1)) * (kDiaGroup * kDiaRowsThreads * ES);
#pragma unroll
            for (int k = 0; k < kDiaGroup; k++)
                if (k < w) {
                    if (ES == 16)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + k * kDiaRowsThreads * ES), "l"(p + (size_t)k * len));
                    else
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst + k * kDiaRowsThreads * ES), "l"(p + (size_t)k * len));
                }
            p += (size_t)w * len;
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
#pragma unroll
    for (int g = 0; g < NS - 1; g++) issue(g);
    grid_dependency();
    const bool yvec = ((reinterpret_cast<uintptr_t>(yin) | reinterpret_cast<uintptr_t>(yout)) & 15) == 0 && r0 + 3 < m;
    float4 yo = make_float4(0.f, 0.f, 0.f, 0.f);
    if (yvec) {
        yo = *reinterpret_cast<const float4*>(yin + r0);
    } else {
        yo.x = yin[r0];
        if (r0 + 1 < m) yo.y = yin[r0 + 1];
        if (r0 + 2 < m) yo.z = yin[r0 + 2];
        if (r0 + 3 < m) yo.w = yin[r0 + 3];
    }
    const int e = (int)((reinterpret_cast<uintptr_t>(x) >> 2) & 3);   // floats x lies past a 16-byte boundary
    const float* xa = x - e;
    const bool interior = (long long)rb + omin - 3 >= 0 && (long long)rb + 4 * (kDiaRowsThreads - 1) + omax + 12 <= n;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    // the window of x of one group, s floats before its first entry
    auto window = [&](int off, int w, int s, float (&v)[12]) {
        const int c = r0 + off;
        if (interior) {
            const float4* q = reinterpret_cast<const float4*>(xa + (c + e - s));
            const float4 v0 = q[0];
            float4 v1 = v0, v2 = v0;
            if (s + w > 1) v1 = q[1];
            if (s + w > 5) v2 = q[2];
            v[0] = v0.x; v[1] = v0.y; v[2] = v0.z; v[3] = v0.w;
            v[4] = v1.x; v[5] = v1.y; v[6] = v1.z; v[7] = v1.w;
            v[8] = v2.x; v[9] = v2.y; v[10] = v2.z; v[11] = v2.w;
        } else {
#pragma unroll
            for (int k = 0; k < 12; k++) v[k] = 0.0f;
#pragma unroll
            for (int k = 0; k < kDiaGroup + 3; k++)
                if (k < w + 3 && c + k >= 0 && c + k < n) v[k] = x[c + k];
        }
    };
    float v[12], vn[12];
    int2 gd = ng ? __ldg(groups) : make_int2(0, 0);
    int s = interior ? (gd.x + e) & 3 : 0;   // uniform: rows come in fours
    if (kAhead && ng) window(gd.x, gd.y, s, v);
    for (int g = 0; g < ng; g++) {
        const int w = gd.y, sc = s;
        if (!kAhead) window(gd.x, w, s, v);
        issue(g + NS - 1);
        if (g + 1 < ng) {
            gd = __ldg(groups + g + 1);
            s = interior ? (gd.x + e) & 3 : 0;
            if (kAhead) window(gd.x, gd.y, s, vn);
        }
        asm volatile("cp.async.wait_group %0;\n" ::"n"(NS - 1) : "memory");
        const unsigned char* src = own + (g & (NS - 1)) * (kDiaGroup * kDiaRowsThreads * ES);
        float4 a[kDiaGroup];
#pragma unroll
        for (int k = 0; k < kDiaGroup; k++)
            if (k < w) a[k] = Val<V>::lds4(reinterpret_cast<const V*>(src + k * kDiaRowsThreads * ES));
        switch (sc) {
        case 0: dia_fma<0>(acc, a, v, w); break;
        case 1: dia_fma<1>(acc, a, v, w); break;
        case 2: dia_fma<2>(acc, a, v, w); break;
        default: dia_fma<3>(acc, a, v, w); break;
        }
        if (kAhead) {
#pragma unroll
            for (int k = 0; k < 12; k++) v[k] = vn[k];
        }
    }
    if (yvec) {
        *reinterpret_cast<float4*>(yout + r0) = make_float4(yo.x + acc.x, yo.y + acc.y, yo.z + acc.z, yo.w + acc.w);
    } else {
        yout[r0] = yo.x + acc.x;
        if (r0 + 1 < m) yout[r0 + 1] = yo.y + acc.y;
        if (r0 + 2 < m) yout[r0 + 2] = yo.z + acc.z;
        if (r0 + 3 < m) yout[r0 + 3] = yo.w + acc.w;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// The same for diagonals that mostly stand alone (the host's groups are one diagonal each): the
// values of a diagonal come as one 128-bit load and its four x entries as guarded loads, and
// the compiler keeps four diagonals in flight.  HBM bounds it on large matrices (4.9 TB/s at 27
// diagonals of 2 M rows FP32), the L2 and the chain of loads on small ones.  The offsets are staged in shared
// memory before grid_dependency(); read one by one in the loop they cost 64 diagonals of
// 200,000 rows in BF16 24.4 us instead of 17.6.
constexpr int kDiaEachMax = 12000;   // their offsets in shared memory

template <class V>
__global__ void __launch_bounds__(kDiaThreads) dia_each_kernel(const int2* __restrict__ groups, const V* __restrict__ data, const float* x,
                                                               const float* yin, float* yout, int m, int n, int nd, int len)
{
    extern __shared__ int s_off[];
    for (int i = threadIdx.x; i < nd; i += kDiaThreads) s_off[i] = __ldg(&groups[i].x);
    __syncthreads();
    const int r0 = (blockIdx.x * kDiaThreads + threadIdx.x) * 4;
    if (r0 >= m) return;
    grid_dependency();
    float yo[4];
#pragma unroll
    for (int q = 0; q < 4; q++) yo[q] = r0 + q < m ? yin[r0 + q] : 0.0f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    auto at = [&](int c) { return c >= 0 && c < n ? x[c] : 0.0f; };
    for (int d = 0; d < nd; d++) {
        const int c = r0 + s_off[d];
        const float4 a = Val<V>::ld4(data + (size_t)d * len + r0);
        acc.x += a.x * at(c);
        acc.y += a.y * at(c + 1);
        acc.z += a.z * at(c + 2);
        acc.w += a.w * at(c + 3);
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (r0 + q < m) yout[r0 + q] = yo[q] + (q == 0 ? acc.x : q == 1 ? acc.y : q == 2 ? acc.z : acc.w);
}

constexpr int kBdiaStagedMax = 8000;   // widest band whose window fits 48 KB of shared memory

// BDIA with the band's window of x staged in shared memory (spmv_bdia.cl gpu_bdia:
// one staged window per band, reused by the band's adjacent diagonals).  The CTA
// covers kDiaThreads*ROWS rows, thread t owning rows t, t+256, ... so shared-memory
// reads are conflict-free and global loads coalesced.  Dynamic shared memory holds
// kDiaThreads*ROWS + max_band_width - 1 floats.
template <class V, int ROWS>
__global__ void __launch_bounds__(kDiaThreads) bdia_staged_kernel(const int* __restrict__ offsets, const int* __restrict__ bptr,
                                                                  const V* __restrict__ data, const float* __restrict__ x,
                                                                  float* __restrict__ y, int m, int n, int nbands, int len)
{
    extern __shared__ float s_x[];
    constexpr int RB = kDiaThreads * ROWS;
    const int rbase = blockIdx.x * RB;
    float acc[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; q++) acc[q] = 0.0f;
    for (int b = 0; b < nbands; b++) {
        const int o = __ldg(offsets + b);
        const int d0 = __ldg(bptr + b), w = __ldg(bptr + b + 1) - d0;
        __syncthreads();
        for (int i = threadIdx.x; i < RB + w - 1; i += kDiaThreads) s_x[i] = ldx_guarded(x, rbase + o + i, n);
        __syncthreads();
        for (int k = 0; k < w; k++) {
            const V* dd = data + (size_t)(d0 + k) * len + rbase;
#pragma unroll
            for (int q = 0; q < ROWS; q++) {
                const int lr = threadIdx.x + q * kDiaThreads;
                if (rbase + lr < m) acc[q] += Val<V>::ld(dd + lr) * s_x[lr + k];
            }
        }
    }
#pragma unroll
    for (int q = 0; q < ROWS; q++) {
        const int r = rbase + threadIdx.x + q * kDiaThreads;
        if (r < m) y[r] += acc[q];
    }
}

}  // namespace dev
}  // namespace csp
