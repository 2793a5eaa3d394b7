// Multiple right-hand sides: Y += A * X with X (n x k) and Y (m x k) row-major, so
// the k values of one column index are contiguous and every gather is a coalesced
// row segment.  A lane group of G = min(k, 32) lanes serves one (block) row, lane l
// owning right-hand sides l, l + G, ...; the group's entries are staged in shared
// memory by coalesced loads and read back as broadcasts.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace csp {
namespace dev {

constexpr int kSpmmThreads = 256;

// CSR: one group per row.
template <class V, int G>
__global__ void __launch_bounds__(kSpmmThreads) csr_spmm_kernel(const int* __restrict__ rp, const int* __restrict__ col,
                                                                const V* __restrict__ val, const float* __restrict__ x,
                                                                float* __restrict__ y, int m, int k)
{
    __shared__ int s_col[kSpmmThreads];
    __shared__ float s_val[kSpmmThreads];
    const int lane = threadIdx.x % G;
    const int gbase = threadIdx.x - lane;   // this group's slice of the staging arrays
    // groups of one warp run different trip counts: each synchronises only its own lanes
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) - lane));
    const int row = (int)(((long long)blockIdx.x * kSpmmThreads + threadIdx.x) / G);
    const bool valid = row < m;
    const int s = valid ? __ldg(rp + row) : 0, e = valid ? __ldg(rp + row + 1) : 0;
    for (int c0 = 0; c0 < k; c0 += G) {
        const int c = c0 + lane;
        float acc = 0.0f;
        for (int j0 = s; j0 < e; j0 += G) {
            const int n = min(G, e - j0);
            __syncwarp(gmask);
            if (lane < n) {
                s_col[gbase + lane] = __ldg(col + j0 + lane);
                s_val[gbase + lane] = Val<V>::ld(val + j0 + lane);
            }
            __syncwarp(gmask);
            if (c < k)
                for (int t = 0; t < n; t++) acc += s_val[gbase + t] * __ldg(x + (size_t)s_col[gbase + t] * k + c);
        }
        if (valid && c < k) y[(size_t)row * k + c] += acc;
    }
}

// Generic BCSR (block-element-major data[e * aligned + block]): one group per block row.
// The staged block values take kSpmmThreads * BH * BW floats of shared memory, so
// blocks are limited to 36 elements (6 x 6).
template <class V, int BH, int BW, int G>
__global__ void __launch_bounds__(kSpmmThreads) bcsr_spmm_kernel(const int* __restrict__ rp, const int* __restrict__ col,
                                                                 const V* __restrict__ data, const float* __restrict__ x,
                                                                 float* __restrict__ y, int nbr, int aligned, int m, int n,
                                                                 int k)
{
    constexpr int BS = BH * BW;
    __shared__ float s_val[kSpmmThreads * BS];
    __shared__ int s_col[kSpmmThreads];
    const int lane = threadIdx.x % G;
    const int gbase = threadIdx.x - lane;
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) - lane));
    const int br = (int)(((long long)blockIdx.x * kSpmmThreads + threadIdx.x) / G);
    const bool valid = br < nbr;
    const int s = valid ? __ldg(rp + br) : 0, e = valid ? __ldg(rp + br + 1) : 0;
    for (int c0 = 0; c0 < k; c0 += G) {
        const int c = c0 + lane;
        float acc[BH];
#pragma unroll
        for (int h = 0; h < BH; h++) acc[h] = 0.0f;
        for (int j0 = s; j0 < e; j0 += G) {
            const int nb = min(G, e - j0);
            __syncwarp(gmask);
            if (lane < nb) {
                s_col[gbase + lane] = __ldg(col + j0 + lane);
#pragma unroll
                for (int q = 0; q < BS; q++) s_val[(gbase + lane) * BS + q] = Val<V>::ld(data + (size_t)q * aligned + j0 + lane);
            }
            __syncwarp(gmask);
            if (c < k) {
                for (int t = 0; t < nb; t++) {
                    const int bc = s_col[gbase + t];
                    const float* bv = s_val + (gbase + t) * BS;
                    float xv[BW];
#pragma unroll
                    for (int w = 0; w < BW; w++) xv[w] = (bc + w < n) ? __ldg(x + (size_t)(bc + w) * k + c) : 0.0f;
#pragma unroll
                    for (int h = 0; h < BH; h++)
#pragma unroll
                        for (int w = 0; w < BW; w++) acc[h] += bv[h * BW + w] * xv[w];
                }
            }
        }
        if (valid && c < k) {
#pragma unroll
            for (int h = 0; h < BH; h++) {
                const int r = br * BH + h;
                if (r < m) y[(size_t)r * k + c] += acc[h];
            }
        }
    }
}

// Generic BCSR with k a multiple of 4, on a layout of its own: block j is BlockRec<V, BS>
// words -- its BS values in row-major order (two per word in BF16), then the index of
// its first X row in float4s -- so a run of blocks is one contiguous stream.  A warp is
// cut into groups of GL = 4 CW lanes; a group takes `rows` consecutive block rows, or those of the
// host's list `groups` where some rows are long, one after the other and copies their blocks through a ring of four chunks in shared memory
// with 16-byte cp.async, two chunks ahead.  Per step a group takes 4 U blocks of its
// current row: lane (cw, sub) owns right-hand sides 4 cw .. 4 cw + 3 of blocks sub,
// sub + 4, ..., whose X loads are all in flight together.  At the end of a row the four
// lanes of a column are summed by two shuffle steps that also split the four right-hand
// sides over them, so Y is read (when the row begins) and written by whole segments of
// consecutive lanes.
//
// What bounds it: the X rows.  Every block reads BW * k floats of X from L2 (384 bytes at
// 3x3, k = 32; the band of a FEM matrix is too wide for L1), so the floor is the L2 -> SM
// path and the L1 tag rate (BW lines a block at a line a clock), not HBM; next to it, issue
// slots: BH * BW * 4 FMAs per lane and block, and as few other instructions as possible --
// no predicated loads (lanes past the row's end read X row 0 and skip the products).
// Measured (500,000 block rows, 10 M 3x3 blocks, one B200): k = 32 FP32 615 -> 342 us, k = 16
// 530 -> 271, k = 8 BF16 250 -> 187, k = 4 FP32 245 -> 182 (before: blocks staged row by row
// from the element planes, one barrier pair per 32 blocks, ~880 instructions a block row at
// k = 32; now ~580).  The X gathers alone take 192 us at k = 32.  Also measured at k = 32:
// one round of X loads in flight (U = 1) 406 us, 24 warps an SM 403, 48 warps with U = 1 482;
// X rows copied to shared memory by cp.async.bulk 250 us for the gathers alone; a block's
// three X rows read as one request over 6 lanes, 227 us at k = 8 (three FMA sets for one).
template <class V, int BS> struct BlockRec {
    static constexpr int value_words = sizeof(V) == 4 ? BS : (BS + 1) / 2;
    static constexpr int align = value_words >= 8 ? 4 : 2;    // words of one shared-memory read
    static constexpr int words = (value_words + align) / align * align;
    static constexpr int xrow_word = words - 1;
};
// BlockRec<V, bs>::words
inline size_t record_words(int bs, bool bf16)
{
    const int value_words = bf16 ? (bs + 1) / 2 : bs, align = value_words >= 8 ? 4 : 2;
    return (size_t)(value_words + align) / align * align;
}

// Records of n blocks from their columns and element planes (plane q at q * stride
// elements); set-up only.  x_units: float4s per X row.
__global__ void __launch_bounds__(256) block_records_kernel(const int* __restrict__ col, const void* __restrict__ planes,
                                                            unsigned* __restrict__ rec, int n, int stride, int bs, bool bf16,
                                                            int x_units)
{
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= n) return;
    const int value_words = bf16 ? (bs + 1) / 2 : bs, align = value_words >= 8 ? 4 : 2;
    const int words = (value_words + align) / align * align;
    unsigned* r = rec + (size_t)j * words;
    for (int i = 0; i < words - 1; i++) {
        unsigned v = 0u;
        if (i < value_words) {
            if (bf16) {
                const unsigned short* s = static_cast<const unsigned short*>(planes);
                v = s[(size_t)(2 * i) * stride + j];
                if (2 * i + 1 < bs) v |= (unsigned)s[(size_t)(2 * i + 1) * stride + j] << 16;
            } else {
                v = static_cast<const unsigned*>(planes)[(size_t)i * stride + j];
            }
        }
        r[i] = v;
    }
    r[words - 1] = (unsigned)col[j] * (unsigned)x_units;
}

constexpr int kSpmmPadBlocks = 32;   // zero records behind the last block: a chunk may be copied past its end

// values of a block record in shared memory
template <class V, int BS>
__device__ __forceinline__ void read_block(const unsigned* s, float (&a)[BS])
{
    using Rec = BlockRec<V, BS>;
    unsigned wd[(Rec::value_words + 3) / 4 * 4];
    if (Rec::align == 4) {
#pragma unroll
        for (int i = 0; i < (Rec::value_words + 3) / 4; i++) {
            const uint4 u = *reinterpret_cast<const uint4*>(s + 4 * i);
            wd[4 * i] = u.x;
            wd[4 * i + 1] = u.y;
            wd[4 * i + 2] = u.z;
            wd[4 * i + 3] = u.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < (Rec::value_words + 1) / 2; i++) {
            const uint2 u = *reinterpret_cast<const uint2*>(s + 2 * i);
            wd[2 * i] = u.x;
            wd[2 * i + 1] = u.y;
        }
    }
#pragma unroll
    for (int q = 0; q < BS; q++) {
        if (sizeof(V) == 4) a[q] = __uint_as_float(wd[q]);
        else a[q] = __uint_as_float(q % 2 ? wd[q / 2] & 0xffff0000u : wd[q / 2] << 16);
    }
}

// Whether a shape has a second kernel, for rows of many blocks (MANY below).
constexpr bool spmm_has_many(int bw, int cw) { return (bw == 1 && cw != 2) || (bw == 2 && cw == 1); }

// The lane split for CW float4 columns a pass.
template <class V_, int BH_, int BW_, int CW_, bool MANY = false> struct SpmmShape {
    using V = V_;
    static constexpr int BH = BH_, BW = BW_, CW = CW_, BS = BH * BW;
    static constexpr int GL = 4 * CW, groups = 32 / GL;
    // rounds of X loads in flight: two, where 64 registers hold them; at one float4 column
    // (k = 4) one, which halves the ring and keeps more warps resident (3x3: 197 -> 182 us).  Small
    // blocks of rows with many (MANY): four for 1x1, whose rounds are one load a lane, two for 2x2 at k = 4.
    // 1x1, 200,000 rows, one B200, few / MANY: 3 entries a row, k = 32 24.6 / 33.7 us (rounds past a row's
    // end are loads for nothing), 10 entries 39.4 / 37.7, k = 16 27.3 / 23.1; 100,000 rows of 10 to 30, k = 4
    // 24.3 / 17.1; 120,000 Zipf rows, bound by the longest, k = 4 420 / 118.  At k = 8 MANY gains nothing
    // (20,000 rows of 48: 8.9 / 11.1).  2x2, k = 4: 30,000 block rows of 10 to 30 13.0 / 10.5, 800,000 of 3 47.4 / 55.8
    static constexpr int U = MANY ? (BW == 1 ? 4 : 2) : (BW > 4 || CW == 1 ? 1 : 2);
    static constexpr int chunk = 4 * U > 2 * CW ? 4 * U : 2 * CW;               // blocks; a step spans at most two
    static constexpr int ring_words = 4 * chunk * BlockRec<V, BS>::words;       // per group
    static constexpr int warp_bytes = groups * ring_words * 4;
    static constexpr int warps = warp_bytes * 8 <= 48 * 1024 ? 8 : (warp_bytes * 4 <= 48 * 1024 ? 4 : (warp_bytes * 2 <= 48 * 1024 ? 2 : 1));
    static constexpr int threads = 32 * warps;
    // consecutive block rows per group, at most: a warp per row needs eight to hide the start of its ring
    static constexpr int max_rows = groups == 1 ? 8 : 4;
    // per SM: by registers, and by the rings in its 228 KB of shared memory (1 KB a CTA is the system's).
    // 4x4 blocks and larger at 16 warps (128 registers): at 24 the 4x4 FP32 kernel that takes any k had no
    // room for its X loads (30,000 block rows, one B200: k = 64 112 -> 91.6 us, k = 20 51.8 -> 43.7)
    static constexpr int reg_ctas = (BS <= 9 ? 32 : 16) / warps;
    static constexpr int smem_ctas = 228 * 1024 / (warps * warp_bytes + 1024);
    static constexpr int ctas = reg_ctas < smem_ctas ? reg_ctas : smem_ctas;
};

// K: the number of right-hand sides where it is known (0: `k_arg`).  An instance of its own for k = 32
// gains 4 to 12 % on 3x3 and 4x4 blocks over the one that takes any k above 16.
template <class Sh, int K>
__global__ void __launch_bounds__(Sh::threads, Sh::ctas)
    bcsr_spmm_stream_kernel(const int4* __restrict__ groups, int ngroups, int rows, const int* __restrict__ rp,
                            const unsigned* __restrict__ rec, const float* x, float* y, int nbr, int m, int k_arg)
{
    using V = typename Sh::V;
    constexpr int BH = Sh::BH, BW = Sh::BW, CW = Sh::CW;
    using Rec = BlockRec<V, BH * BW>;
    constexpr int BS = BH * BW, GL = Sh::GL, U = Sh::U, CH = Sh::chunk, NW = Rec::words;
    constexpr int RM = 4 * CH - 1;   // ring index mask
    static_assert((CH & (CH - 1)) == 0 && CH * NW % 4 == 0, "ring of a power of two blocks, whole 16-byte copies");
    static_assert(Sh::ctas >= 1 && Sh::ctas * (Sh::warps * Sh::warp_bytes + 1024) <= 228 * 1024, "the CTAs that a wave counts on fit an SM");
    __shared__ __align__(16) unsigned s_ring[32 * Sh::warps / GL][Sh::ring_words];
    const int k = K ? K : k_arg;
    const int lane = threadIdx.x % GL;                       // in the group
    unsigned* ring = s_ring[threadIdx.x / GL];
    const unsigned ring_addr = (unsigned)__cvta_generic_to_shared(ring);
    const int gid = (int)(((long long)blockIdx.x * Sh::threads + threadIdx.x) / GL);
    // block rows [r0, r1) with blocks [sb, eb)
    int r0, r1, sb, eb;
    if (groups) {
        const int4 gr = gid < ngroups ? __ldg(groups + gid) : make_int4(0, 0, 0, 0);
        r0 = gr.x, r1 = gr.y, sb = gr.z, eb = gr.w;
    } else {
        r0 = (int)min((long long)gid * rows, (long long)nbr), r1 = min(r0 + rows, nbr);
        sb = __ldg(rp + r0), eb = __ldg(rp + r1);
    }
    const int cw = lane % CW, sub = lane / CW;
    const int rend = __ldg(rp + min(r0 + 1 + lane, r1));     // rows <= GL: the ends of the group's rows
    const int base = sb & ~1;                                // chunks start on 16 bytes
    // the right-hand side of this lane's results: c + comp
    const int comp = ((lane & CW) ? 2 : 0) + ((lane & (2 * CW)) ? 1 : 0);
    const size_t kb = (size_t)k * 4;

    // chunk q of the group's blocks into ring slot q % 4
    auto issue = [&](int q) {
        const int j = base + q * CH;
        if (j < eb) {
            const char* src = reinterpret_cast<const char*>(rec + (size_t)j * NW);
            const unsigned dst = ring_addr + (q & 3) * (CH * NW * 4);
#pragma unroll
            for (int i = 0; i < CH * NW / 4; i += GL)
                if (i + lane < CH * NW / 4)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16 * (i + lane)),
                                 "l"(src + 16 * (i + lane)));
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };

    for (int c0 = 0; c0 < k; c0 += 4 * CW) {
        const int c = c0 + 4 * cw;
        const bool writer = c < k;
        const char* xc = reinterpret_cast<const char*>(x + (c < k ? c : 0));
        float* yp = y + (size_t)r0 * BH * k + c + comp;   // this lane's Y entry of the row's first line
        issue(0);
        issue(1);
        if (c0 == 0) grid_dependency();
        int next = 0;               // chunks 0 .. next - 1 have landed
        int j = sb, r = r0, re = sb;
        float4 acc[BH];
        float yv[BH];
        auto begin_row = [&](int end) {
            re = end;
#pragma unroll
            for (int h = 0; h < BH; h++) {
                acc[h] = make_float4(0.f, 0.f, 0.f, 0.f);
                yv[h] = (writer && r * BH + h < m) ? yp[(size_t)h * k] : 0.0f;
            }
        };
        const int end0 = __shfl_sync(0xffffffffu, rend, 0, GL);
        if (r < r1) begin_row(end0);
        while (__any_sync(0xffffffffu, r < r1)) {
            // the blocks of this step: [j, min(j + 4 U, re)), all landed
            const int jn = min(j + 4 * U, re);
            bool need = j < re && jn > base + next * CH;
            while (__any_sync(0xffffffffu, need)) {
                __syncwarp();       // the slot about to be filled is no longer read
                if (need) {
                    issue(next + 2);
                    asm volatile("cp.async.wait_group 2;\n" ::);
                    next++;
                    need = jn > base + next * CH;
                }
                __syncwarp();
            }
            const unsigned* bk[U];
            float4 xv[U][BW];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int t = j + 4 * u + sub;
                bk[u] = ring + ((t - base) & RM) * NW;
                const unsigned off = t < re ? bk[u][Rec::xrow_word] : 0u;
                const char* xp = xc + (size_t)off * 16;
#pragma unroll
                for (int w = 0; w < BW; w++) xv[u][w] = *reinterpret_cast<const float4*>(xp + w * kb);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (j + 4 * u + sub >= re) continue;
                float a[BS];
                read_block<V, BS>(bk[u], a);
#pragma unroll
                for (int w = 0; w < BW; w++)
#pragma unroll
                    for (int h = 0; h < BH; h++) {
                        acc[h].x += a[h * BW + w] * xv[u][w].x;
                        acc[h].y += a[h * BW + w] * xv[u][w].y;
                        acc[h].z += a[h * BW + w] * xv[u][w].z;
                        acc[h].w += a[h * BW + w] * xv[u][w].w;
                    }
            }
            j = jn;
            const bool done = r < r1 && j == re;
            if (__any_sync(0xffffffffu, done)) {
                const bool up = lane & CW, up2 = lane & (2 * CW);
                const int end = __shfl_sync(0xffffffffu, rend, min(r + 1 - r0, GL - 1), GL);
                float out[BH];
#pragma unroll
                for (int h = 0; h < BH; h++) {
                    float a = up ? acc[h].z : acc[h].x, b = up ? acc[h].w : acc[h].y;
                    a += __shfl_xor_sync(0xffffffffu, up ? acc[h].x : acc[h].z, CW);
                    b += __shfl_xor_sync(0xffffffffu, up ? acc[h].y : acc[h].w, CW);
                    out[h] = (up2 ? b : a) + __shfl_xor_sync(0xffffffffu, up2 ? a : b, 2 * CW);
                }
                if (done) {
#pragma unroll
                    for (int h = 0; h < BH; h++)
                        if (writer && r * BH + h < m) yp[(size_t)h * k] = yv[h] + out[h];
                    r++;
                    yp += (size_t)BH * k;
                    if (r < r1) begin_row(end);
                }
            }
        }
        // the chunks issued ahead land before the ring is used again
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncwarp();
    }
}

}  // namespace dev
}  // namespace csp

namespace csp {
namespace dev {

// ---------------------------------------------------------------------------
// Generic BCSR SpMM on tensor cores: k a multiple of 32, blocks of BH <= 8 rows and
// BW <= 4 columns (mma.sync.m16n8k8, TF32 operands, FP32 accumulation).
//
// One warp per block row.  For each panel of 32 right-hand sides the block row's
// BH x 32 output is two 16 x 8 MMA tiles D[m][n]: M = 16 right-hand sides, N = the
// block row's rows (BH of 8), K = the columns of two blocks per step, each block's BW
// columns padded to 4.  Lane (g, t) = (lane / 4, lane % 4) feeds
//   A (16 x 8, X^T):  X[col(t)][rhs(g)], X[col(t)][rhs(g + 8)], and the same at t + 4,
//   B (8 x 8, A^T):   A[row g][col t] of the step's first and second block,
// and the right-hand sides are numbered so that tile tau's rows g and g + 8 are
// right-hand sides 4g + 2tau and 4g + 2tau + 1: one 128-bit load of X[col][4g .. 4g + 3]
// gives a lane both tiles' A entries of one column, and lane t's outputs (rows 2t and
// 2t + 1) are two 128-bit Y rows segments.  Padding columns (t >= BW) and rows
// (g >= BH) contribute zeros; they cost no loads.
//
// FP32 accuracy from TF32 operands: every operand v is split into vh = tf32(v) (round
// to nearest) and the exact remainder vl = v - vh, and a * x is taken as
// ah*xh + (ah*xl + al*xh) -- three MMAs, the two small terms in their own accumulator
// so they do not perturb the large one's rounding (the dropped al*xl is below 2^-22 of
// |a x|).  BF16 values are exact in TF32 (al = 0): two MMAs.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mma_tf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// High and low TF32 parts of v: hi = v rounded to nearest (ties away from zero) at
// TF32's 10 fraction bits -- half a TF32 ulp (bit 12) added to the magnitude bits, the
// 13 low bits cleared -- and the exact remainder lo = v - hi, passed as raw FP32 bits
// (the MMA reads its top 19).  Finite |v| below 2^128 (1 - 2^-11) only.
__device__ __forceinline__ void tf32_split(float v, uint32_t& hi, uint32_t& lo)
{
    hi = (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(v - __uint_as_float(hi));
}

constexpr int kMmaThreads = 256;   // 8 warps, one block row each

template <class V, int BH, int BW, int KS>
__global__ void __launch_bounds__(kMmaThreads) bcsr_spmm_mma_kernel(const int* __restrict__ rp, const int* __restrict__ col,
                                                                    const V* __restrict__ data, const float* __restrict__ x,
                                                                    float* __restrict__ y, int nbr, int aligned, int m,
                                                                    int n, int k)
{
    static_assert(BH >= 1 && BH <= 8 && BW >= 1 && BW <= 4, "block shape");
    constexpr bool kExactA = !std::is_same<V, float>::value;   // BF16 values: exact in TF32
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int br = (int)(((long long)blockIdx.x * kMmaThreads + threadIdx.x) >> 5);
    if (br >= nbr) return;   // the whole warp leaves together
    const int s = __ldg(rp + br), e = __ldg(rp + br + 1);
    const bool xlane = t < BW;                // lanes whose column is a real one
    const bool alane = xlane && g < BH;       // lanes holding a matrix value
    const V* __restrict__ plane = data + (size_t)(alane ? g * BW + t : 0) * aligned;
    // lane t's output rows 2t and 2t + 1
    const int r0 = br * BH + 2 * t, r1 = r0 + 1;
    const bool w0 = 2 * t < BH && r0 < m, w1 = 2 * t + 1 < BH && r1 < m;
    for (int c0 = 0; c0 < k; c0 += 32) {
        const int cx = c0 + 4 * g;
        // the Y rows this lane updates, requested before the block loads and X gathers
        float4 y0 = w0 ? *reinterpret_cast<const float4*>(y + (size_t)r0 * k + cx) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 y1 = w1 ? *reinterpret_cast<const float4*>(y + (size_t)r1 * k + cx) : make_float4(0.f, 0.f, 0.f, 0.f);
        float big[2][4], small[2][4];
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int q = 0; q < 4; q++) big[u][q] = small[u][q] = 0.0f;
        for (int j0 = s; j0 < e; j0 += 2 * KS) {
            // every load of KS steps (2 KS blocks) first
            float4 xv[KS][2];
            float av[KS][2];
#pragma unroll
            for (int u = 0; u < KS; u++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int j = j0 + 2 * u + h;
                    const bool vj = j < e;
                    const int bc = vj ? __ldg(col + j) : 0;
                    xv[u][h] = (vj && xlane && bc + t < n)
                                   ? __ldg(reinterpret_cast<const float4*>(x + (size_t)(bc + t) * k + cx))
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
                    av[u][h] = (vj && alane) ? Val<V>::ld(plane + j) : 0.0f;
                }
#pragma unroll
            for (int u = 0; u < KS; u++) {
                if (j0 + 2 * u >= e) break;
                uint32_t xh[2][4], xl[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    tf32_split(xv[u][h].x, xh[h][0], xl[h][0]);
                    tf32_split(xv[u][h].y, xh[h][1], xl[h][1]);
                    tf32_split(xv[u][h].z, xh[h][2], xl[h][2]);
                    tf32_split(xv[u][h].w, xh[h][3], xl[h][3]);
                }
                uint32_t ah0, ah1, al0 = 0, al1 = 0;
                if (kExactA) {
                    ah0 = __float_as_uint(av[u][0]);
                    ah1 = __float_as_uint(av[u][1]);
                } else {
                    tf32_split(av[u][0], ah0, al0);
                    tf32_split(av[u][1], ah1, al1);
                }
                // tile 0: right-hand sides 4g, 4g + 1 (x, y components); tile 1: 4g + 2, 4g + 3 (z, w)
#pragma unroll
                for (int tau = 0; tau < 2; tau++) {
                    const int p = 2 * tau, q = 2 * tau + 1;
                    mma_tf32(small[tau], xl[0][p], xl[0][q], xl[1][p], xl[1][q], ah0, ah1);
                    if (!kExactA) mma_tf32(small[tau], xh[0][p], xh[0][q], xh[1][p], xh[1][q], al0, al1);
                    mma_tf32(big[tau], xh[0][p], xh[0][q], xh[1][p], xh[1][q], ah0, ah1);
                }
            }
        }
        // D[m][n] fragments: d[0] = (g, 2t), d[1] = (g, 2t + 1), d[2] = (g + 8, 2t), d[3] = (g + 8, 2t + 1)
        float d[2][4];
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int q = 0; q < 4; q++) d[u][q] = big[u][q] + small[u][q];
        if (w0) {
            y0.x += d[0][0];
            y0.y += d[0][2];
            y0.z += d[1][0];
            y0.w += d[1][2];
            *reinterpret_cast<float4*>(y + (size_t)r0 * k + cx) = y0;
        }
        if (w1) {
            y1.x += d[0][1];
            y1.y += d[0][3];
            y1.z += d[1][1];
            y1.w += d[1][3];
            *reinterpret_cast<float4*>(y + (size_t)r1 * k + cx) = y1;
        }
    }
}

}  // namespace dev
}  // namespace csp
