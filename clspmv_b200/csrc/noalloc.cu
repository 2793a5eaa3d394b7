// COO SpMV for callers that cannot allocate device memory.
//
// Some callers of this library must not call the CUDA allocator at all: code that
// runs inside a framework whose caching allocator has already reserved the device's
// memory, real-time solver loops where cudaMalloc/cudaFree (which can synchronize the
// whole device and take milliseconds) are forbidden, and embedders that hand the
// library only the buffers they own.  csp_coo_spmv_noalloc serves them: it computes
// y += A*x for a row-sorted COO matrix whose arrays the caller already holds in device
// memory, and allocates nothing.  The per-warp partial sums that the segmented
// reduction needs live in g_noalloc_scratch, a fixed array in this library's device
// image (CSP_NOALLOC_SCRATCH_BYTES = 1 MiB): every GPU that loads the library holds it
// until the process exits.  It bounds the matrix to CSP_NOALLOC_MAX_NNZ entries.
//
// The kernels restate the COO segmented reduction of kernels/flat.cuh
// (coo_segment_kernel) for unpadded caller arrays, with a fix-up pass: the last tile
// is read with masked scalar loads, and every row/column index is range-checked so a
// malformed matrix gives a wrong result instead of an out-of-bounds access.
#include <cuda_runtime.h>
#include <mutex>

#include "csp/clspmv.h"
#include "internal.h"
#include "engine.h"
#include "launch.h"
#include "kernels/common.cuh"

namespace csp {

constexpr int kNoAllocChunk = 512;                                        // entries per warp, at most
constexpr int kNoAllocMaxWarps = CSP_NOALLOC_MAX_NNZ / kNoAllocChunk;     // 65,536
static_assert(CSP_NOALLOC_SCRATCH_BYTES == 2 * kNoAllocMaxWarps * (4 + 4), "scratch holds 2 (row, sum) pairs per warp");

// Scratch of the no-allocation entry point: rows of the 2 * warps (row, partial) pairs,
// then their partial sums.  Shared by every call on a device.
static __device__ __align__(256) unsigned char g_noalloc_scratch[CSP_NOALLOC_SCRATCH_BYTES];

namespace {

__device__ __forceinline__ void load_entry(const int* rowid, const int* colid, const float* val, int j, int nnz, int last_row,
                                           int& r, int& c, float& v)
{
    if (j < nnz) {
        r = rowid[j];
        c = colid[j];
        v = val[j];
    } else {   // padding past the caller's arrays: extends the last row by zeros
        r = last_row;
        c = 0;
        v = 0.0f;
    }
}

__device__ __forceinline__ float x_at(const float* x, int c, int width)
{
    return (c >= 0 && c < width) ? x[c] : 0.0f;
}

__device__ __forceinline__ float y_at(const float* y, int r, int height)
{
    return (r >= 0 && r < height) ? y[r] : 0.0f;
}

// One tile of 128 entries, four consecutive ones per lane.
struct Tile {
    int4 r, c;
    float4 a;
};

// Each warp reduces `chunk` entries (two or four tiles), tile by tile.  Latency is what bounds it (a few
// thousand warps, three dependent steps a tile), so the steps overlap: while tile t is
// reduced, the gathers of x and y for tile t + 1 and the entries of tile t + 2 are in
// flight.  Past that the L1's gather rate (a line a clock) is the limit.  300,007 Zipf rows,
// 1.9 M entries, one B200: 31 us a call (segment 16, fix-up 8, and the launches) -> 24.  A row closed inside the chunk is written by the lane that closes it; the
// chunk's first and last row go to the scratch pairs.
__global__ void __launch_bounds__(256) coo_noalloc_segment(const int* rowid, const int* colid, const float* val, const float* x,
                                                           float* y, int nnz, int height, int width, int nwarps, int chunk,
                                                           int* part_row, float* part_val)
{
    dev::grid_dependency();   // the caller's arrays may be written by the operation before
    const int lane = threadIdx.x & 31;
    const int w = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (w >= nwarps) return;
    const int last_row = rowid[nnz - 1];
    const int nnz_tiles = (nnz + 127) / 128 * 128;
    const int base = w * chunk;
    const int end = min(base + chunk, nnz_tiles);
    const int head_row = rowid[base];
    bool head_open = true;
    int carry_row = head_row;
    float carry_val = 0.0f, carry_y = 0.0f;
    auto load = [&](int t, Tile& q) {
        const int j = t + 4 * lane;
        if (t + 128 <= nnz) {
            q.r = *reinterpret_cast<const int4*>(rowid + j);
            q.c = *reinterpret_cast<const int4*>(colid + j);
            q.a = *reinterpret_cast<const float4*>(val + j);
        } else {
            load_entry(rowid, colid, val, j + 0, nnz, last_row, q.r.x, q.c.x, q.a.x);
            load_entry(rowid, colid, val, j + 1, nnz, last_row, q.r.y, q.c.y, q.a.y);
            load_entry(rowid, colid, val, j + 2, nnz, last_row, q.r.z, q.c.z, q.a.z);
            load_entry(rowid, colid, val, j + 3, nnz, last_row, q.r.w, q.c.w, q.a.w);
        }
    };
    auto gather = [&](const Tile& q, float4& xv, float4& yv) {
        xv = make_float4(x_at(x, q.c.x, width), x_at(x, q.c.y, width), x_at(x, q.c.z, width), x_at(x, q.c.w, width));
        yv = make_float4(y_at(y, q.r.x, height), y_at(y, q.r.y, height), y_at(y, q.r.z, height), y_at(y, q.r.w, height));
    };
    Tile cur, nxt;
    float4 xv, yv;
    load(base, cur);
    if (base + 128 < end) load(base + 128, nxt);
    gather(cur, xv, yv);
    for (int t = base; t < end; t += 128) {
        const int4 r = cur.r;
        const float p0 = cur.a.x * xv.x, p1 = cur.a.y * xv.y, p2 = cur.a.z * xv.z, p3 = cur.a.w * xv.w;
        const float4 y4 = yv;
        if (t + 128 < end) {
            cur = nxt;
            if (t + 256 < end) load(t + 256, nxt);
            gather(cur, xv, yv);
        }
        const int tile_first = __shfl_sync(0xffffffffu, r.x, 0);
        if (tile_first != carry_row) {
            if (lane == 0) {
                if (head_open && carry_row == head_row) {
                    part_row[2 * w] = carry_row;
                    part_val[2 * w] = carry_val;
                } else if (carry_row >= 0 && carry_row < height) {
                    y[carry_row] = carry_y + carry_val;
                }
            }
            if (head_open && carry_row == head_row) head_open = false;
            carry_row = tile_first;
            carry_val = 0.0f;
        }
        float tail = p3;
        if (r.z == r.w) { tail += p2; if (r.y == r.w) { tail += p1; if (r.x == r.w) tail += p0; } }
        float scan = tail;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float o = __shfl_up_sync(0xffffffffu, scan, d);
            const int ok = __shfl_up_sync(0xffffffffu, r.w, d);
            if (lane >= d && ok == r.w) scan += o;
        }
        const float prev_scan = __shfl_up_sync(0xffffffffu, scan, 1);
        const int prev_key = __shfl_up_sync(0xffffffffu, r.w, 1);
        const int next_first = __shfl_down_sync(0xffffffffu, r.x, 1);
        float run = (lane > 0 && prev_key == r.x) ? prev_scan : 0.0f;
        if (r.x == carry_row) run += carry_val;
        bool closed_head = false;
        const int rr[4] = {r.x, r.y, r.z, r.w};
        const float pp[4] = {p0, p1, p2, p3};
        const float yy[4] = {y4.x, y4.y, y4.z, y4.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            run += pp[k];
            const int nx = (k == 3) ? next_first : rr[k + 1];
            const bool closes = (k < 3) ? (nx != rr[k]) : (lane < 31 && nx != rr[k]);
            if (closes) {
                if (head_open && rr[k] == head_row) {
                    part_row[2 * w] = rr[k];
                    part_val[2 * w] = run;
                    closed_head = true;
                } else if (rr[k] >= 0 && rr[k] < height) {
                    y[rr[k]] = yy[k] + run;
                }
                run = 0.0f;
            }
        }
        carry_row = __shfl_sync(0xffffffffu, r.w, 31);
        carry_val = __shfl_sync(0xffffffffu, run, 31);
        carry_y = __shfl_sync(0xffffffffu, y4.w, 31);
        if (__any_sync(0xffffffffu, closed_head)) head_open = false;
    }
    if (lane == 0) {
        if (head_open) {
            part_row[2 * w] = carry_row;
            part_val[2 * w] = carry_val;
            part_row[2 * w + 1] = carry_row;
            part_val[2 * w + 1] = 0.0f;
        } else {
            part_row[2 * w + 1] = carry_row;
            part_val[2 * w + 1] = carry_val;
        }
    }
}

// Adds each row's consecutive scratch pairs to y.  A warp takes 32 pairs: a keyed scan over
// the lanes sums the runs that start in it, and the run that reaches its last lane is
// followed through the next pairs 32 at a time (a row of 10,000 entries has 40 pairs: one
// thread per run read them one after the other, 8 us of a 300,007-row Zipf product).  Runs
// that start in an earlier warp's pairs are that warp's.
__global__ void __launch_bounds__(256) coo_noalloc_fixup(const int* part_row, const float* part_val,
                                                         int nparts, int height, float* y)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int lane = threadIdx.x & 31, first = i - lane;
    dev::grid_dependency();
    if (first >= nparts) return;   // the whole warp leaves together
    // plain loads: the pairs are written within the life of this waiting kernel
    const volatile int* prow = part_row;
    const volatile float* pval = part_val;
    const bool valid = i < nparts;
    const int r = valid ? prow[i] : 0;
    const float v = valid ? pval[i] : 0.0f;
    const float y0 = valid ? y_at(y, r, height) : 0.0f;
    const int before = lane == 0 && i > 0 ? prow[i - 1] : 0;
    const int up = __shfl_up_sync(0xffffffffu, r, 1);
    const bool head = valid && (i == 0 || (lane == 0 ? before : up) != r);
    const unsigned heads = __ballot_sync(0xffffffffu, head), valids = __ballot_sync(0xffffffffu, valid);
    if (!heads) return;
    // this lane's run starts at lane `start` (none: it starts in an earlier warp)
    const unsigned below = heads & (0xffffffffu >> (31 - lane));
    const int start = below ? 31 - __clz(below) : -1;
    float sum = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float o = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane - d >= max(start, 0)) sum += o;
    }
    const bool last = valid && (lane == 31 || ((heads >> (lane + 1)) & 1u) || !((valids >> (lane + 1)) & 1u));
    if ((valids >> 31) & 1u) {
        // the run of lane 31 may go on
        const int row = __shfl_sync(0xffffffffu, r, 31);
        float more = 0.0f;
        for (int j0 = first + 32; j0 < nparts; j0 += 32) {
            const int j = j0 + lane;
            const bool same = j < nparts && prow[j] == row;
            const unsigned mism = __ballot_sync(0xffffffffu, !same);
            const int n = mism ? __ffs(mism) - 1 : 32;
            float t = lane < n ? pval[j] : 0.0f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            more += t;
            if (mism) break;
        }
        if (lane == 31) sum += more;
    }
    if (last && start >= 0 && r >= 0 && r < height) y[r] = y0 + sum;
}

// Device address of g_noalloc_scratch, looked up once per device with that device
// current and kept for the process (a cudaDeviceReset afterwards is not supported).
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
void* g_scratch_addr[kMaxDevices];

int scratch_for_current_device(void** out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) return set_error(CSP_EUNSUP, "device %d beyond the %d the no-allocation path tracks", dev, kMaxDevices);
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_error(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return CSP_OK;
}

}  // namespace
}  // namespace csp

extern "C" int csp_coo_spmv_noalloc(int height, int width, int nnz, const int* d_row, const int* d_col, const float* d_val,
                                    const float* d_x, float* d_y, void* stream)
{
    using namespace csp;
    if (height < 0 || width < 0 || nnz < 0) return set_error(CSP_EINVAL, "coo_spmv_noalloc: negative size");
    if (nnz > CSP_NOALLOC_MAX_NNZ)
        return set_error(CSP_EINVAL, "coo_spmv_noalloc: %d entries exceed the no-allocation limit of %d (use csp_init_mat_kernels)",
                         nnz, CSP_NOALLOC_MAX_NNZ);
    if (nnz == 0) return CSP_OK;
    if (!d_row || !d_col || !d_val || !d_x || !d_y) return set_error(CSP_EINVAL, "coo_spmv_noalloc: null device pointer");
    {
        // x is read while y is written: the arrays must not overlap
        const uintptr_t x0 = (uintptr_t)d_x, x1 = x0 + sizeof(float) * (size_t)width;
        const uintptr_t y0 = (uintptr_t)d_y, y1 = y0 + sizeof(float) * (size_t)height;
        if (x0 < y1 && y0 < x1 && width > 0 && height > 0)
            return set_error(CSP_EINVAL, "coo_spmv_noalloc: x and y overlap");
    }
    if (((uintptr_t)d_row | (uintptr_t)d_col | (uintptr_t)d_val) & 15)
        return set_error(CSP_EINVAL, "coo_spmv_noalloc: row, column and value arrays must be 16-byte aligned");
    void* scratch = nullptr;
    int rc = scratch_for_current_device(&scratch);
    if (rc) return rc;
    int* part_row = static_cast<int*>(scratch);
    float* part_val = reinterpret_cast<float*>(static_cast<char*>(scratch) + CSP_NOALLOC_SCRATCH_BYTES / 2);
    // two tiles a warp where that fills the chip's 148 x 32 warps at most once (100,000 Zipf rows:
    // 13.4 us a call against 15.0 with four), four beyond (1 M rows: 47.3 against 48.0)
    const int chunk = nnz <= 148 * 32 * kNoAllocChunk / 2 ? kNoAllocChunk / 2 : kNoAllocChunk;
    const int nwarps = (nnz + chunk - 1) / chunk;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    launch_chained(coo_noalloc_segment, (nwarps * 32 + 255) / 256, 256, 0, st, d_row, d_col, d_val, d_x, d_y, nnz, height, width,
                   nwarps, chunk, part_row, part_val);
    launch_chained(coo_noalloc_fixup, (2 * nwarps + 255) / 256, 256, 0, st, part_row, part_val, 2 * nwarps, height, d_y);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CSP_OK : cuda_error(e, "coo_spmv_noalloc launch");
}
