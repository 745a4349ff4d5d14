// Learned surrogate of the particle step (include/sdem_surrogate.h), sm_103a.
//
// Kernels:
//   k_graph_bin, scan, k_graph_scatter, k_graph_order, k_graph_count,
//   k_graph_fill                    cell-grid neighbour graph at radius
//                                   1.5 d_max, CSR by receiver, deterministic
//                                   order (neighbour cell, then sphere index);
//   k_cells / k_edges<count|fill>   the same step by step;
//   k_node_feat                     node features (velocity frames, spin,
//                                   size, plane distances) as bf16;
//   k_mlp                           both layers of one MLP of the forward pass, with
//                                   residual and message sums, on tcgen05;
//   k_gemm_rows, k_gemm_wgrad       the network's layers on tcgen05, forward and
//                                   backward: C = A . B^T over operands that may be
//                                   row-gathered, split in column segments
//                                   (concatenated edge/node inputs) and read
//                                   transposed (weight gradients), with a
//                                   fused bias/ReLU/mask/residual epilogue;
//   k_gemm_tc, k_gemm               the same for other shapes: tcgen05 with B read
//                                   per tile, and mma.sync for every form;
//   k_split_reduce, k_colsum*       deterministic reductions (split-K weight
//                                   gradients, bias gradients);
//   k_segsum, k_gather_add          message aggregation and its adjoints;
//   k_sphere_grad, k_gather_add_sum
//                                   the same fused for rows of 128;
//   k_mse, k_adam, k_to_bf16,
//   k_advance                       loss, optimiser, casts, one stride.
//
// Every element of a product is summed in steps of 16 in the order of the
// reduction, whichever kernel takes it, so results are the same bits between the
// kernels and from run to run.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <algorithm>
#include <stdint.h>

#include "../../include/sdem_surrogate.h"
#include "fp64_int.cuh"
#include "scan.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 32, LDS = BK + 8, GT = 128;
constexpr int kColsumBlocks = 160;

__device__ __forceinline__ uint16_t bf16_bits(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }

__device__ __forceinline__ bool bf16_positive(uint16_t b) { return (b & 0x8000u) == 0 && (b & 0x7fffu) != 0; }

// ------------------------------------------------------------------ graph

__global__ void k_cells(int n, const double* __restrict__ posR, sdem_sg_grid g, int* __restrict__ cell) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double q = (posR[4 * (size_t)i + a] - g.lo[a]) / g.cell;
        c[a] = (q >= 0.0) ? (q < (double)g.dim[a] ? (int)q : g.dim[a] - 1) : 0;
    }
    cell[i] = (c[2] * g.dim[1] + c[1]) * g.dim[0] + c[0];
}

template <bool kFill>
__global__ void k_edges(int n, const double* __restrict__ posR, sdem_sg_grid g, const int* __restrict__ cell,
                        const int* __restrict__ cell_start, const int* __restrict__ sorted, int* __restrict__ degree,
                        const int* __restrict__ row_off, int* __restrict__ dst, int* __restrict__ src,
                        uint16_t* __restrict__ efeat) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double xi = posR[4 * (size_t)i], yi = posR[4 * (size_t)i + 1], zi = posR[4 * (size_t)i + 2];
    const double ri = posR[4 * (size_t)i + 3];
    const int c = cell[i];
    const int cx = c % g.dim[0], cy = (c / g.dim[0]) % g.dim[1], cz = c / (g.dim[0] * g.dim[1]);
    const double rc2 = g.cutoff * g.cutoff;
    int cnt = 0;
    const int base = kFill ? row_off[i] : 0;
    for (int dz = -1; dz <= 1; ++dz) {
        const int z = cz + dz;
        if (z < 0 || z >= g.dim[2]) continue;
        for (int dy = -1; dy <= 1; ++dy) {
            const int y = cy + dy;
            if (y < 0 || y >= g.dim[1]) continue;
            for (int dx = -1; dx <= 1; ++dx) {
                const int x = cx + dx;
                if (x < 0 || x >= g.dim[0]) continue;
                const int cc = (z * g.dim[1] + y) * g.dim[0] + x;
                const int s1 = cell_start[cc + 1];
                for (int s = cell_start[cc]; s < s1; ++s) {
                    const int j = sorted[s];
                    if (j == i) continue;
                    const double ex = posR[4 * (size_t)j] - xi, ey = posR[4 * (size_t)j + 1] - yi,
                                 ez = posR[4 * (size_t)j + 2] - zi;
                    const double d2 = ex * ex + ey * ey + ez * ez;
                    if (!(d2 < rc2)) continue;
                    if (kFill) {
                        const size_t e = (size_t)base + cnt;
                        dst[e] = i;
                        src[e] = j;
                        const double d = sqrt(d2);
                        const double ov = fmax(ri + posR[4 * (size_t)j + 3] - d, 0.0);
                        __align__(16) uint16_t f[8];
                        f[0] = bf16_bits((float)(ex / g.scale));
                        f[1] = bf16_bits((float)(ey / g.scale));
                        f[2] = bf16_bits((float)(ez / g.scale));
                        f[3] = bf16_bits((float)(d / g.scale));
                        f[4] = bf16_bits((float)(100.0 * ov / g.scale));
                        f[5] = f[6] = f[7] = 0;
                        uint4* o = reinterpret_cast<uint4*>(efeat + e * 16);
                        o[0] = *reinterpret_cast<const uint4*>(f);
                        o[1] = make_uint4(0u, 0u, 0u, 0u);
                    }
                    ++cnt;
                }
            }
        }
    }
    if (!kFill) degree[i] = cnt;
}

// ---- the whole graph build on the device (sdem_sg_graph_count / _fill)
// Counting sort of the spheres by cell, then by index; one thread per sorted
// sphere lists its neighbours; a block writes the edges of 64 of them.  The
// candidates are tested in single precision on coordinates relative to their
// cell's corner; only those within a margin of the cutoff take the exact FP64
// test (which k_edges runs for every candidate, twice, on GB300's two FP64
// operations per SM per clock).  Square roots and divisions of the features run
// on the integer pipes (fp64_int.cuh), bit-identical to the hardware's.
// 200k spheres, 3.9M edges: 7.0 ms as k_edges twice with torch's sorts and
// prefix sums in between, 0.31 ms here (111 us until the edges are counted, 146 to
// write them, bound by the FP64 pipe; the rest is the count on its way to the host).
constexpr int GR_CAP = 96;    // neighbours kept per sphere between the two calls; longer lists are searched again
constexpr int GR_T = 256;

struct __align__(32) Rec4 {
    double x, y, z, r;
};

struct GraphWork {
    unsigned long long* total;   // edges
    int* status;
    scan::ScanCtl *cctl, *rctl;
    unsigned long long *cwords, *rwords;
    int* cell_cnt;
    size_t clear;                // bytes from the start that begin as zeros
    int *cell_start, *cell, *rank, *tmp, *sorted, *degree, *nbr;
    float4* rec;                 // (x, y, z relative to the cell's corner, index), sorted; x is NaN outside the grid
    Rec4* pos;                   // sorted
    size_t bytes;
};

GraphWork graph_work(void* base, int n, long long ncell) {
    GraphWork w;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? static_cast<char*>(base) + off : nullptr;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    char* head = take(256);
    w.total = reinterpret_cast<unsigned long long*>(head);
    w.status = reinterpret_cast<int*>(head + 8);
    w.cctl = reinterpret_cast<scan::ScanCtl*>(head + 32);
    w.rctl = reinterpret_cast<scan::ScanCtl*>(head + 64);
    w.cwords = reinterpret_cast<unsigned long long*>(take(8 * scan::scan_words(ncell)));
    w.rwords = reinterpret_cast<unsigned long long*>(take(8 * scan::scan_words(n)));
    w.cell_cnt = reinterpret_cast<int*>(take(4 * (size_t)ncell));
    w.clear = off;
    w.cell_start = reinterpret_cast<int*>(take(4 * ((size_t)ncell + 1)));
    int** per[5] = {&w.cell, &w.rank, &w.tmp, &w.sorted, &w.degree};
    for (int** p : per) *p = reinterpret_cast<int*>(take(4 * (size_t)n));
    w.rec = reinterpret_cast<float4*>(take(16 * (size_t)n));
    w.pos = reinterpret_cast<Rec4*>(take(32 * (size_t)n));
    w.nbr = reinterpret_cast<int*>(take(4 * (size_t)n * GR_CAP));
    w.bytes = off;
    return w;
}

struct GridDiv {
    fpi::Divisor cell, scale;
};

__global__ void __launch_bounds__(GR_T) k_graph_bin(int n, const double* __restrict__ posR, sdem_sg_grid g, GridDiv dv,
                                                    GraphWork w) {
    const int i = blockIdx.x * GR_T + threadIdx.x;
    if (i >= n) return;
    int c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {   // as k_cells
        const double q = fpi::div_by(posR[4 * (size_t)i + a] - g.lo[a], dv.cell);
        c[a] = (q >= 0.0) ? (q < (double)g.dim[a] ? (int)q : g.dim[a] - 1) : 0;
    }
    const int k = (c[2] * g.dim[1] + c[1]) * g.dim[0] + c[0];
    w.cell[i] = k;
    w.rank[i] = atomicAdd(&w.cell_cnt[k], 1);
}

__global__ void __launch_bounds__(GR_T) k_graph_scatter(int n, GraphWork w) {
    const int i = blockIdx.x * GR_T + threadIdx.x;
    if (i < n) w.tmp[w.cell_start[w.cell[i]] + w.rank[i]] = i;
}

// by index inside a cell, and the sorted copies
__global__ void __launch_bounds__(GR_T) k_graph_order(int n, const double* __restrict__ posR, sdem_sg_grid g, GraphWork w) {
    const int i = blockIdx.x * GR_T + threadIdx.x;
    if (i >= n) return;
    const int k = w.cell[i], a = w.cell_start[k], b = w.cell_start[k + 1];
    int s = a;
    for (int t = a; t < b; ++t) s += w.tmp[t] < i;
    Rec4 P;
    P.x = posR[4 * (size_t)i];
    P.y = posR[4 * (size_t)i + 1];
    P.z = posR[4 * (size_t)i + 2];
    P.r = posR[4 * (size_t)i + 3];
    w.sorted[s] = i;
    w.pos[s] = P;
    const int cx = k % g.dim[0], cy = (k / g.dim[0]) % g.dim[1], cz = k / (g.dim[0] * g.dim[1]);
    const float fx = (float)(P.x - (g.lo[0] + cx * g.cell)), fy = (float)(P.y - (g.lo[1] + cy * g.cell)),
                fz = (float)(P.z - (g.lo[2] + cz * g.cell));
    // a sphere outside the grid sits in a border cell with offsets of any size:
    // its pairs take the exact test
    const float lo = -0.001f * (float)g.cell, hi = 1.001f * (float)g.cell;
    const bool in = fx >= lo && fx <= hi && fy >= lo && fy <= hi && fz >= lo && fz <= hi;
    w.rec[s] = make_float4(in ? fx : __int_as_float(0x7fffffff), fy, fz, __int_as_float(i));
}

// Calls hit(t) for every neighbour of the sphere at sort position s, in the
// edges' order: rows of three cells along x are runs of the sort.
template <class Hit>
__device__ __forceinline__ void graph_neighbours(int s, const sdem_sg_grid& g, const GraphWork& w, float margin,
                                                 const Hit& hit) {
    const float4 me = w.rec[s];
    const int k = w.cell[__float_as_int(me.w)];
    const int cx = k % g.dim[0], cy = (k / g.dim[0]) % g.dim[1], cz = k / (g.dim[0] * g.dim[1]);
    const float cell = (float)g.cell, cut = (float)g.cutoff;
    const float near = fmaxf(cut - margin, 0.f), far2 = (cut + margin) * (cut + margin), near2 = near * near;
    const double rc2 = g.cutoff * g.cutoff;
    for (int dz = -1; dz <= 1; ++dz) {
        const int z = cz + dz;
        if (z < 0 || z >= g.dim[2]) continue;
        const float oz = me.z - (float)dz * cell;
        for (int dy = -1; dy <= 1; ++dy) {
            const int y = cy + dy;
            if (y < 0 || y >= g.dim[1]) continue;
            const float oy = me.y - (float)dy * cell;
            const int row = (z * g.dim[1] + y) * g.dim[0] + cx;
            const int b1 = __ldg(w.cell_start + row), b2 = __ldg(w.cell_start + row + 1);
            const int b0 = cx > 0 ? __ldg(w.cell_start + row - 1) : b1, b3 = cx + 1 < g.dim[0] ? __ldg(w.cell_start + row + 2) : b2;
            for (int t = b0; t < b3; ++t) {
                const float4 q = w.rec[t];
                const float ex = q.x - (me.x + (t < b1 ? cell : (t < b2 ? 0.f : -cell))), ey = q.y - oy, ez = q.z - oz;
                const float d2 = ex * ex + ey * ey + ez * ez;
                if (d2 > far2 || t == s) continue;
                if (!(d2 < near2)) {   // near the cutoff, or NaN
                    const Rec4 A = w.pos[s], B = w.pos[t];
                    const double fx = B.x - A.x, fy = B.y - A.y, fz = B.z - A.z;
                    if (!(fx * fx + fy * fy + fz * fz < rc2)) continue;
                }
                hit(t);
            }
        }
    }
}

__global__ void __launch_bounds__(GR_T) k_graph_count(int n, sdem_sg_grid g, float margin, GraphWork w) {
    const int s = blockIdx.x * GR_T + threadIdx.x;
    int cnt = 0;
    if (s < n) {
        int* list = w.nbr + (size_t)s * GR_CAP;
        graph_neighbours(s, g, w, margin, [&](int t) {
            if (cnt < GR_CAP) list[cnt] = t;
            ++cnt;
        });
        w.degree[w.sorted[s]] = cnt;
    }
    unsigned long long all = (unsigned long long)cnt;
    for (int o = 16; o > 0; o >>= 1) all += __shfl_down_sync(0xffffffffu, all, o);
    if ((threadIdx.x & 31) == 0 && all) atomicAdd(w.total, all);
}

__device__ __forceinline__ void graph_edge(const sdem_sg_grid& g, const GridDiv& dv, const GraphWork& w, const Rec4& A,
                                           int i, int t, size_t e, int* __restrict__ dst, int* __restrict__ src,
                                           uint16_t* __restrict__ efeat) {
    const Rec4 B = w.pos[t];
    const double ex = B.x - A.x, ey = B.y - A.y, ez = B.z - A.z;
    const double d = fpi::sqrt_rn(ex * ex + ey * ey + ez * ez);
    dst[e] = i;
    src[e] = w.sorted[t];
    auto h = [&](double q) { return (uint32_t)bf16_bits(fpi::to_float_rn(q)); };
    const double v[4] = {ex, ey, ez, d};
    double q[4];
    fpi::div_many(v, dv.scale, q);
    // 100 max(r_i + r_j - d, 0) / scale: the difference of unequal doubles is not 0
    const double reach = A.r + B.r;
    const uint32_t ov = fpi::gt(reach, d) ? h(fpi::div_by(100.0 * (reach - d), dv.scale)) : 0u;
    uint4* o = reinterpret_cast<uint4*>(efeat + e * 16);
    o[0] = make_uint4(h(q[0]) | h(q[1]) << 16, h(q[2]) | h(q[3]) << 16, ov, 0u);
    o[1] = make_uint4(0u, 0u, 0u, 0u);
}

// A block writes the edges of 64 spheres, a thread an edge, so that no lane idles
// while the FP64 pipe works (with eight lanes a sphere a quarter did): a graph of
// 200k spheres and 3.9M edges takes 314 us instead of 335.
constexpr int GF_S = 64;
__global__ void __launch_bounds__(GR_T) k_graph_fill(int n, sdem_sg_grid g, GridDiv dv, float margin, GraphWork w,
                                                     const int* __restrict__ row_off, int* __restrict__ dst,
                                                     int* __restrict__ src, uint16_t* __restrict__ efeat) {
    __shared__ int start[GF_S + 1], base[GF_S], who[GF_S];
    __shared__ Rec4 at[GF_S];
    const int s0 = blockIdx.x * GF_S, t = threadIdx.x, lane = t & 31;
    static_assert(GF_S == 64, "two spheres per lane of one warp");
    if (t < 32) {   // the spheres' places in the block's edges
        int c[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = 2 * lane + h, s = s0 + j;
            c[h] = 0;
            if (s < n) {
                const int i = w.sorted[s];
                who[j] = i;
                base[j] = row_off[i];
                at[j] = w.pos[s];
                c[h] = min(row_off[i + 1] - base[j], GR_CAP);
            }
        }
        int incl = c[0] + c[1];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        start[2 * lane] = incl - c[0] - c[1];
        start[2 * lane + 1] = incl - c[1];
        if (lane == 31) start[GF_S] = incl;
    }
    __syncthreads();
    for (int e = t; e < start[GF_S]; e += GR_T) {
        int j = 0;   // the last sphere that starts at or before e
#pragma unroll
        for (int o = GF_S / 2; o > 0; o >>= 1)
            if (start[j + o] <= e) j += o;
        const int k = e - start[j];
        graph_edge(g, dv, w, at[j], who[j], w.nbr[(size_t)(s0 + j) * GR_CAP + k], (size_t)base[j] + k, dst, src, efeat);
    }
    const int s = s0 + t;
    if (t < GF_S && s < n && row_off[who[t] + 1] - base[t] > GR_CAP) {   // a longer list is searched again
        int k = 0;
        graph_neighbours(s, g, w, margin, [&](int q) {
            if (k >= GR_CAP) graph_edge(g, dv, w, at[t], who[t], q, (size_t)base[t] + k, dst, src, efeat);
            ++k;
        });
    }
}

__global__ void k_node_feat(int n, const double* __restrict__ posR, const double* __restrict__ vel,
                            const double* __restrict__ omega, int nw, const double* __restrict__ planes, double scale,
                            double vscale, double dclip, uint16_t* __restrict__ nf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    __align__(16) uint16_t f[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) f[k] = 0;
#pragma unroll
    for (int fr = 0; fr < 3; ++fr)
#pragma unroll
        for (int a = 0; a < 3; ++a) f[fr * 3 + a] = bf16_bits((float)(vel[((size_t)fr * n + i) * 3 + a] / vscale));
    const double x = posR[4 * (size_t)i], y = posR[4 * (size_t)i + 1], z = posR[4 * (size_t)i + 2];
    const double r = posR[4 * (size_t)i + 3];
#pragma unroll
    for (int a = 0; a < 3; ++a) f[9 + a] = bf16_bits((float)(omega[3 * (size_t)i + a] * r / vscale));
    f[12] = bf16_bits((float)(2.0 * r / scale));
    for (int w = 0; w < nw && w < 5; ++w) {
        const double dist = planes[4 * w] * x + planes[4 * w + 1] * y + planes[4 * w + 2] * z + planes[4 * w + 3];
        const double q = fmin(fmax(dist / scale, -dclip), dclip);
        f[13 + w] = bf16_bits((float)(q / dclip));
    }
    uint4* o = reinterpret_cast<uint4*>(nf + (size_t)i * 32);
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = reinterpret_cast<const uint4*>(f)[k];
}

// ------------------------------------------------------------------- GEMM

struct Operand {
    const uint16_t* ptr[3];
    const int* idx[3];
    int ld[3];
    int c0[3];
    int nseg;
    int trans;
};

// Address of the 8 elements (row, col..col+7) of an operand.  The segment
// fields are picked with selects, not by a runtime array index, so the
// kernel parameters stay in the constant bank (no local-memory copy).
__device__ __forceinline__ const uint4* chunk_addr(const Operand& op, int row, int col) {
    const bool s1 = op.nseg > 1 && col >= op.c0[1];
    const bool s2 = op.nseg > 2 && col >= op.c0[2];
    const uint16_t* p = s2 ? op.ptr[2] : (s1 ? op.ptr[1] : op.ptr[0]);
    const int* ix = s2 ? op.idx[2] : (s1 ? op.idx[1] : op.idx[0]);
    const int ld = s2 ? op.ld[2] : (s1 ? op.ld[1] : op.ld[0]);
    const int c0 = s2 ? op.c0[2] : (s1 ? op.c0[1] : op.c0[0]);
    const size_t r = ix ? (size_t)ix[row] : (size_t)row;
    return reinterpret_cast<const uint4*>(p + r * ld + (col - c0));
}

// Stages the 64 x 32 tile (dim rows d0.., reduction r0..) of an operand into
// S[d][r].  Elements outside [0, ndim) x [r0, rend) are zero.
__device__ __forceinline__ void load_tile(uint16_t (*S)[LDS], const Operand& op, int d0, int ndim, int r0,
                                          int rend) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int c = tid + q * GT;  // 256 chunks of 8 elements
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (op.trans == 0) {
            const int d = c >> 2, rc = (c & 3) * 8;
            const int gd = d0 + d, gr = r0 + rc;
            if (gd < ndim && gr < rend) v = __ldg(chunk_addr(op, gd, gr));
            *reinterpret_cast<uint4*>(&S[d][rc]) = v;
        } else {
            const int r = c >> 3, dc = (c & 7) * 8;
            const int gr = r0 + r, gd = d0 + dc;
            if (gr < rend && gd < ndim) v = __ldg(chunk_addr(op, gr, gd));
            const uint16_t* e = reinterpret_cast<const uint16_t*>(&v);
#pragma unroll
            for (int k = 0; k < 8; ++k) S[dc + k][r] = e[k];
        }
    }
}

__device__ __forceinline__ uint32_t lds32(const uint16_t* p) { return *reinterpret_cast<const uint32_t*>(p); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// mma.sync, for every form: 128 threads (4 warps) per 64x64 output tile, 32-deep
// slices of the reduction staged in padded shared memory (row stride 40 bf16 = 20
// words, so the 8x4 fragment reads of a warp hit 32 distinct banks), each
// warp a 32x32 sub-tile of 2x4 mma.m16n8k16 (bf16 in, fp32 accumulate).
__global__ void __launch_bounds__(GT) k_gemm(int I, int J, int R, Operand A, Operand B, sdem_sg_epilogue ep,
                                             int rchunk, float* __restrict__ partial) {
    __shared__ __align__(16) uint16_t As[BM][LDS];
    __shared__ __align__(16) uint16_t Bs[BN][LDS];
    const int i0 = blockIdx.x * BM, j0 = blockIdx.y * BN;
    const int rb = blockIdx.z * rchunk;
    const int re = min(R, rb + rchunk);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
    float acc[2][4][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;

    for (int r0 = rb; r0 < re; r0 += BK) {
        load_tile(As, A, i0, I, r0, re);
        load_tile(Bs, B, j0, J, r0, re);
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk += 16) {
            uint32_t af[2][4], bfr[4][2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const int row = wm + mt * 16 + g;
                af[mt][0] = lds32(&As[row][kk + 2 * t]);
                af[mt][1] = lds32(&As[row + 8][kk + 2 * t]);
                af[mt][2] = lds32(&As[row][kk + 2 * t + 8]);
                af[mt][3] = lds32(&As[row + 8][kk + 2 * t + 8]);
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int col = wn + nt * 8 + g;
                bfr[nt][0] = lds32(&Bs[col][kk + 2 * t]);
                bfr[nt][1] = lds32(&Bs[col][kk + 2 * t + 8]);
            }
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) mma_bf16(acc[mt][nt], af[mt], bfr[nt]);
        }
        __syncthreads();
    }

#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int gi = i0 + wm + mt * 16 + g + h * 8;
                    const int gj = j0 + wn + nt * 8 + 2 * t + q;
                    if (gi >= I || gj >= J) continue;
                    float v = acc[mt][nt][h * 2 + q];
                    if (partial) {
                        partial[((size_t)blockIdx.z * I + gi) * J + gj] = v;
                        continue;
                    }
                    if (ep.bias) v += ep.bias[gj];
                    if (ep.relu) v = fmaxf(v, 0.f);
                    if (ep.mask && !bf16_positive(ep.mask[(size_t)gi * ep.ld_mask + gj])) v = 0.f;
                    if (ep.out) {
                        float* o = ep.out + (size_t)gi * ep.ld_out + gj;
                        *o = ep.accumulate ? *o + v : v;
                    }
                    if (ep.out_bf) ep.out_bf[(size_t)gi * ep.ld_out_bf + gj] = bf16_bits(v);
                    if (ep.resid) {
                        const float w = ep.resid[(size_t)gi * ep.ld_resid + gj] + v;
                        if (ep.res_out) ep.res_out[(size_t)gi * ep.ld_res_out + gj] = w;
                        if (ep.res_out_bf) ep.res_out_bf[(size_t)gi * ep.ld_res_out_bf + gj] = bf16_bits(w);
                    }
                }
}

// ------------------------------------------------------ tcgen05 GEMM
// The same C = A . B^T with the fused epilogue on the 5th-generation tensor
// cores, for the forms without transposed operands or split reductions (the
// forward layers): one CTA of 256 threads per 128 x 128 output tile.
//
// Operand slices (128 rows x 32 reduction elements of A and of B) are
// copied from global memory into shared memory with cp.async -- each 16-byte
// chunk from its own row, so gathered rows and column segments need no
// staging pass -- into the UMMA K-major layout without swizzle: core
// matrices of 8 rows x 16 bytes, (row group, k group) at
// k group * 2048 + row group * 128 bytes, i.e. the descriptor's leading (K)
// byte offset 2048 and stride (M/N) byte offset 128.  Four slice buffers
// form a ring: while the tensor cores work on slice c, the copies of slices
// c+1..c+3 are in flight.  One thread issues tcgen05.mma (kind::f16, bf16 x
// bf16 -> fp32, M = N = 128, K = 16, two per slice) into a 128-column fp32
// accumulator in tensor memory, and tcgen05.commit arrives on the slice
// buffer's mbarrier, which gates the buffer's next copy.  After the last
// slice the accumulator goes through shared memory (tcgen05.ld by lane
// quarter, then whole rows per warp) to a coalesced epilogue.
//
// Every mbarrier wait of the tensor-core kernels is bounded.  After one that ran
// out its role overwrites no slice, issues no product and hands nothing over, so
// that what the others meet is complete or does not come, and their waits run out
// in turn.  Products not read by then count as zero, and the CTA is counted once
// (sdem_sg_tensor_timeouts).  What was issued is drained, with a limit of its own,
// before the accumulators are freed.
constexpr int TC_M = 128, TC_N = 128, TC_K = 32, TC_T = 256, TC_STAGES = 4;
constexpr int TC_TILE = TC_M * TC_K * 2;          // bytes of one operand slice (8 KB)
constexpr int TC_SMEM = TC_STAGES * 2 * TC_TILE;  // 64 KB: A and B slices of every stage
#ifndef SDEM_SG_WAIT_LIMIT
#define SDEM_SG_WAIT_LIMIT (1 << 22)   // polls of one wait (each suspends the thread for a while)
#endif
constexpr int TC_WAIT_LIMIT = SDEM_SG_WAIT_LIMIT, TC_DRAIN_LIMIT = 1 << 22;
constexpr uint32_t TC_IDESC = (1u << 4)                        // D: fp32
                              | (1u << 7) | (1u << 10)         // A, B: bf16
                              | ((uint32_t)(TC_N >> 3) << 17)  // N / 8
                              | ((uint32_t)(TC_M >> 4) << 24); // M / 16; both operands K-major
__device__ unsigned int g_tc_timeouts = 0;
int g_tc_enabled = 1;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    const uint64_t lbo = 2048, sbo = 128;
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((lbo >> 4) << 16) | ((sbo >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred P;\n mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n selp.u32 %0, 1, 0, P;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// false, and `failed` set, where the wait ran out
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int& failed) {
    for (int it = 0; it < TC_WAIT_LIMIT; ++it) {
        if (mbar_try(bar, parity)) return true;
    }
    failed = 1;
    return false;
}
// until the products behind a commit are done
__device__ __forceinline__ bool mbar_drain(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < TC_DRAIN_LIMIT; ++it)
        if (mbar_try(bar, parity)) return true;
    return false;
}

// cp.async of 16 bytes; src_bytes = 0 fills the chunk with zeros (nothing is read)
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// rows d0.. (128) x reduction r0..r0+31 of an operand into the core-matrix layout
__device__ __forceinline__ void tc_copy(uint32_t S, const Operand& op, int d0, int ndim, int r0, int rend) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int c = threadIdx.x + q * TC_T;   // 512 chunks of 8 elements
        const int d = c >> 2, kg = c & 3;
        const int gd = d0 + d, gr = r0 + kg * 8;
        const bool in = gd < ndim && gr < rend;
        const void* src = in ? (const void*)chunk_addr(op, gd, gr) : (const void*)op.ptr[0];
        cp16(S + kg * 2048 + (d >> 3) * 128 + (d & 7) * 16, src, in ? 16u : 0u);
    }
}

__global__ void __launch_bounds__(TC_T, 1) k_gemm_tc(int I, int J, int R, Operand A, Operand B,
                                                      sdem_sg_epilogue ep) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    __shared__ __align__(8) uint64_t mbar[TC_STAGES];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    const uint32_t As0 = smem_u32(tc_smem), Bs0 = As0 + TC_STAGES * TC_TILE;
    const int i0 = blockIdx.x * TC_M, j0 = blockIdx.y * TC_N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                     "r"(TC_N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        failed = 0;
        for (int k = 0; k < TC_STAGES; ++k)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&mbar[k])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int nch = (R + TC_K - 1) / TC_K;
    bool ok = true;
    int issued = 0;   // slices
    // prologue: slices 0 .. STAGES-2 in flight (one commit group each, empty past the end)
#pragma unroll
    for (int k = 0; k < TC_STAGES - 1; ++k) {
        if (k < nch) {
            tc_copy(As0 + k * TC_TILE, A, i0, I, k * TC_K, R);
            tc_copy(Bs0 + k * TC_TILE, B, j0, J, k * TC_K, R);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int c = 0; c < nch; ++c) {
        const int b = c % TC_STAGES;
        // this thread's copies of slice c have landed; make every thread's
        // visible to the tensor cores
        asm volatile("cp.async.wait_group %0;\n" ::"n"(TC_STAGES - 2) : "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        if (__syncthreads_or(!ok)) break;
        issued = c + 1;
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int kk = 0; kk < TC_K / 16; ++kk) {
                const uint64_t ad = umma_desc(As0 + b * TC_TILE + kk * 2 * 2048);
                const uint64_t bd = umma_desc(Bs0 + b * TC_TILE + kk * 2 * 2048);
                const uint32_t acc = (c > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(TC_IDESC), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smem_u32(&mbar[b]))
                         : "memory");
        }
        // slice c + STAGES - 1 goes into the buffer slice c - 1 used: wait
        // for that slice's MMAs first
        const int nx = c + TC_STAGES - 1;
        if (nx < nch) {
            const int bx = nx % TC_STAGES;
            if (c >= 1 && ok) ok = mbar_wait(smem_u32(&mbar[bx]), ((c - 1) / TC_STAGES) & 1, failed);
            if (ok) {
                tc_copy(As0 + bx * TC_TILE, A, i0, I, nx * TC_K, R);
                tc_copy(Bs0 + bx * TC_TILE, B, j0, J, nx * TC_K, R);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (issued > 0 && !mbar_drain(smem_u32(&mbar[(issued - 1) % TC_STAGES]), ((issued - 1) / TC_STAGES) & 1)) ok = false;
    ok = !__syncthreads_or(!ok || issued < nch);
    if (!ok && threadIdx.x == 0) atomicAdd(&g_tc_timeouts, 1u);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    // Epilogue in two column halves through shared memory (the slice buffers
    // are free now): warp w moves accumulator rows 32 (w mod 4).. and columns
    // 32 (w / 4).. of the half from tensor memory into a padded row-major
    // tile, then every warp writes whole rows, so that the epilogue's global
    // loads and stores are coalesced along j.
    float* T = reinterpret_cast<float*>(tc_smem);   // 128 rows x 65 floats (33 KB)
    const int quarter = warp & 3, sub = warp >> 2;
    const bool valid = nch > 0 && ok;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        const int col = half * 64 + sub * 32;
        uint32_t r[32];
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)col;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        const int row = quarter * 32 + lane;
#pragma unroll
        for (int q = 0; q < 32; ++q) T[row * 65 + sub * 32 + q] = valid ? __uint_as_float(r[q]) : 0.f;
        __syncthreads();
        // 128 rows x 64 columns: warp w writes rows w, w+8, ...; lane l columns l and l+32
#pragma unroll 1
        for (int rr = warp; rr < TC_M; rr += TC_T / 32) {
            const int gi = i0 + rr;
            if (gi >= I) break;
#pragma unroll
            for (int h2 = 0; h2 < 2; ++h2) {
                const int cj = h2 * 32 + lane;
                const int gj = j0 + half * 64 + cj;
                if (gj >= J) continue;
                float v = T[rr * 65 + cj];
                if (ep.bias) v += ep.bias[gj];
                if (ep.relu) v = fmaxf(v, 0.f);
                if (ep.mask && !bf16_positive(ep.mask[(size_t)gi * ep.ld_mask + gj])) v = 0.f;
                if (ep.out) {
                    float* o = ep.out + (size_t)gi * ep.ld_out + gj;
                    *o = ep.accumulate ? *o + v : v;
                }
                if (ep.out_bf) ep.out_bf[(size_t)gi * ep.ld_out_bf + gj] = bf16_bits(v);
                if (ep.resid) {
                    const float w = ep.resid[(size_t)gi * ep.ld_resid + gj] + v;
                    if (ep.res_out) ep.res_out[(size_t)gi * ep.ld_res_out + gj] = w;
                    if (ep.res_out_bf) ep.res_out_bf[(size_t)gi * ep.ld_res_out_bf + gj] = bf16_bits(w);
                }
            }
        }
        __syncthreads();
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TC_N) : "memory");
}

// ------------------------------------------- tcgen05, weight kept in shared memory
// The forms whose B fits in shared memory whole (every layer of the network:
// forward C = [gathered rows] . W^T and input gradient C = dY . W): one
// persistent CTA per SM keeps B there, K-major, for all its 128-row tiles, so
// that a tile moves its A rows and nothing else (k_gemm_tc, which reads B anew
// for every tile, moves twice as much).  Roles: warps 4-7 copy A slices of 64
// reduction elements with cp.async into a ring of six (four to five in flight); one
// thread of warp 8 issues the tcgen05.mma's into a ring of four 128-column
// accumulators in tensor memory; warps 0-3 drain them, each thread one row,
// with 32-byte global accesses straight from registers, while the next
// accumulators fill.  Shared-memory operands are K-major with the 128-byte
// swizzle: element (row, k) of a 64-wide slice at row * 128 bytes + ((k / 8) xor
// (row mod 8)) * 16.  The reduction runs in the same order and steps of 16 as
// in k_gemm_tc and k_gemm, and the results are the same bits.
// Bound by L2 on the gathered forward form (600k rows, R = 384: 108 us, 6.4 TB/s
// of L2; k_gemm_tc 328 us) and by HBM on the input gradient (J = 384, fp32 out:
// 183 us, 5.8 TB/s; k_gemm 1150 us).
// An epilogue that reads a mask or a residual (kReads) has eight warps, two to a
// row quarter, and requests what it reads before it waits for the products: with
// four warps that read behind the wait, a residual update of 330k rows took 140 us
// (85 here; 62 for its bytes), a masked gradient 104 (92).  Without reads four warps
// are better (600k rows, both forms above together: 317 against 405 us with eight;
// the copying warps lose registers to the others).
constexpr int RW_M = 128, RW_K = 64, RW_STAGES = 6, RW_LAG = 5, RW_ACC = 4, RW_T = 288, RW_T_READS = 416;
constexpr int RW_SLICE = RW_M * RW_K * 2;              // 16 KB
constexpr int RW_B_MAX = 98304;                        // bytes of B kept
constexpr int RW_J_MAX = 384;

__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mbar_init(uint64_t* b, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(b))
                 : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u)
        : "memory");
}
// the same with A in tensor memory (K-major, two 16-bit elements a column)
__device__ __forceinline__ void tc_mma_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u)
        : "memory");
}
// 16 columns of this warp's lane quarter
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
// 32 accumulator columns of this warp's lane quarter
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
// 32-byte global accesses (one sector a thread)
__device__ __forceinline__ void st8(void* p, const uint32_t* v) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void ld8(const void* p, uint32_t* v) {
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    return (uint32_t)bf16_bits(lo) | (uint32_t)bf16_bits(hi) << 16;
}

// The epilogue of 32 columns gj0.. of row gi, held by one thread.  `wide`: every
// pointer and leading dimension allows 32-byte accesses, and all 32 columns exist.
// kPre (wide only): pre holds the residual (32 floats) where ep.resid is given,
// else the mask (32 bf16 in its first half), read before the accumulator was ready.
template <bool kPre>
__device__ __forceinline__ void epilogue32(const sdem_sg_epilogue& ep, bool wide, const float* __restrict__ bias,
                                           int gi, int gj0, int J, uint32_t (&r)[32], const uint32_t (&pre)[32]) {
    if (wide) {
        if (ep.bias) {
#pragma unroll
            for (int q = 0; q < 32; ++q) r[q] = __float_as_uint(__uint_as_float(r[q]) + bias[gj0 + q]);
        }
        if (ep.relu) {
#pragma unroll
            for (int q = 0; q < 32; ++q) r[q] = __float_as_uint(fmaxf(__uint_as_float(r[q]), 0.f));
        }
        if (ep.mask) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t m[8];
                if (!kPre || ep.resid) {
                    ld8(ep.mask + (size_t)gi * ep.ld_mask + gj0 + 16 * h, m);
                } else {
#pragma unroll
                    for (int q = 0; q < 8; ++q) m[q] = pre[8 * h + q];
                }
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    if (!bf16_positive((uint16_t)(m[q >> 1] >> (16 * (q & 1))))) r[16 * h + q] = 0u;
            }
        }
        if (ep.out) {
            float* o = ep.out + (size_t)gi * ep.ld_out + gj0;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (ep.accumulate) {
                    uint32_t a[8];
                    ld8(o + 8 * h, a);
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        a[q] = __float_as_uint(__uint_as_float(a[q]) + __uint_as_float(r[8 * h + q]));
                    st8(o + 8 * h, a);
                } else {
                    st8(o + 8 * h, r + 8 * h);
                }
            }
        }
        if (ep.out_bf) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t b[8];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    b[q] = bf16_pair(__uint_as_float(r[16 * h + 2 * q]), __uint_as_float(r[16 * h + 2 * q + 1]));
                st8(ep.out_bf + (size_t)gi * ep.ld_out_bf + gj0 + 16 * h, b);
            }
        }
        if (ep.resid) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                uint32_t a[8];
                if (!kPre) ld8(ep.resid + (size_t)gi * ep.ld_resid + gj0 + 8 * h, a);
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    r[8 * h + q] = __float_as_uint(__uint_as_float(kPre ? pre[8 * h + q] : a[q]) + __uint_as_float(r[8 * h + q]));
                if (ep.res_out) st8(ep.res_out + (size_t)gi * ep.ld_res_out + gj0 + 8 * h, r + 8 * h);
            }
            if (ep.res_out_bf) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t b[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        b[q] = bf16_pair(__uint_as_float(r[16 * h + 2 * q]), __uint_as_float(r[16 * h + 2 * q + 1]));
                    st8(ep.res_out_bf + (size_t)gi * ep.ld_res_out_bf + gj0 + 16 * h, b);
                }
            }
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < 32; ++q) {
        const int gj = gj0 + q;
        if (gj >= J) continue;
        float v = __uint_as_float(r[q]);
        if (ep.bias) v += bias[gj];
        if (ep.relu) v = fmaxf(v, 0.f);
        if (ep.mask && !bf16_positive(ep.mask[(size_t)gi * ep.ld_mask + gj])) v = 0.f;
        if (ep.out) {
            float* o = ep.out + (size_t)gi * ep.ld_out + gj;
            *o = ep.accumulate ? *o + v : v;
        }
        if (ep.out_bf) ep.out_bf[(size_t)gi * ep.ld_out_bf + gj] = bf16_bits(v);
        if (ep.resid) {
            const float w = ep.resid[(size_t)gi * ep.ld_resid + gj] + v;
            if (ep.res_out) ep.res_out[(size_t)gi * ep.ld_res_out + gj] = w;
            if (ep.res_out_bf) ep.res_out_bf[(size_t)gi * ep.ld_res_out_bf + gj] = bf16_bits(w);
        }
    }
}

// B (J x R) into shared memory: 64-wide slices of jpad rows, 128-byte swizzle; zeros beyond J and R
// K-major B goes there by cp.async, all chunks in flight.  For a transposed B the
// threads' order is what counts: with consecutive threads on consecutive columns
// all 2-byte stores of a warp met in one bank, 3 us of a 17 us product of 16k rows
// and 12 of 27 with J = 256.
__device__ __forceinline__ void stage_b(uint8_t* Bs, const Operand& B, int J, int jpad, int R, int kslices) {
    if (B.trans == 0) {
        const uint32_t dst = smem_u32(Bs);
        for (int c = threadIdx.x; c < jpad * kslices * 8; c += blockDim.x) {
            const int j = c / (kslices * 8), kc = c % (kslices * 8);
            const bool in = j < J && kc * 8 < R;
            cp16(dst + (kc >> 3) * jpad * 128 + j * 128 + (((kc & 7) ^ (j & 7)) << 4),
                 in ? (const void*)chunk_addr(B, j, kc * 8) : (const void*)B.ptr[0], in ? 16u : 0u);
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    } else {
        // consecutive threads take consecutive reduction rows: their 2-byte stores
        // fall into different banks (eight columns further they would share one)
        const int rows = kslices * RW_K, chunks = rows * (jpad / 8), step = blockDim.x;
        for (int c0 = threadIdx.x; c0 < chunks; c0 += 4 * step) {
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = c0 + u * step, r = c % rows, j0 = c / rows * 8;
                v[u] = make_uint4(0u, 0u, 0u, 0u);
                if (c < chunks && r < R && j0 < J) v[u] = __ldg(chunk_addr(B, r, j0));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = c0 + u * step, r = c % rows, j0 = c / rows * 8;
                if (c >= chunks) break;
                const uint16_t* e = reinterpret_cast<const uint16_t*>(&v[u]);
                uint8_t* row = Bs + (size_t)(r >> 6) * jpad * 128 + j0 * 128 + (r & 7) * 2;
#pragma unroll
                for (int k = 0; k < 8; ++k)   // j0 is a multiple of eight
                    *reinterpret_cast<uint16_t*>(row + k * 128 + ((((r >> 3) & 7) ^ k) << 4)) = e[k];
            }
        }
    }
}

template <bool kReads>
__global__ void __launch_bounds__(kReads ? RW_T_READS : RW_T, 1) k_gemm_rows(int I, int J, int R, Operand A, Operand B,
                                                                             sdem_sg_epilogue ep, int wide) {
    extern __shared__ __align__(1024) uint8_t rw_smem[];
    __shared__ __align__(8) uint64_t full[RW_STAGES], empty[RW_STAGES], accf[RW_ACC], acce[RW_ACC], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    __shared__ float bias_s[RW_J_MAX];
    const int jpad = (J + 15) / 16 * 16, kslices = (R + RW_K - 1) / RW_K, nb = (jpad + 127) / 128;
    const int tiles = (I + RW_M - 1) / RW_M;
    const bool by_segment = (A.nseg < 2 || A.c0[1] % RW_K == 0) && (A.nseg < 3 || A.c0[2] % RW_K == 0);
    uint8_t* Bs = rw_smem;
    const uint32_t Bs0 = smem_u32(Bs), As0 = Bs0 + (uint32_t)(kslices * jpad * 128);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                     "r"(RW_ACC * 128)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < RW_STAGES; ++k) {
            mbar_init(&full[k], 128);
            mbar_init(&empty[k], 1);
        }
        for (int k = 0; k < RW_ACC; ++k) {
            mbar_init(&accf[k], 1);
            mbar_init(&acce[k], kReads ? 256 : 128);
        }
        mbar_init(&drain, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    for (int j = threadIdx.x; j < RW_J_MAX; j += blockDim.x) bias_s[j] = ep.bias && j < J ? ep.bias[j] : 0.f;
    stage_b(Bs, B, J, jpad, R, kslices);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int mine = tiles > (int)blockIdx.x ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;   // this CTA's tiles
    const int slices = mine * kslices;
    if (warp >= 4 && warp < 8) {
        // ---- copies: thread = (row mod 16, 16-byte chunk of the row's 128 bytes)
        const int pt = threadIdx.x - 128, kc = pt & 7, r0 = pt >> 3;
        bool ok = true;
        int t = 0;   // slices issued
        const uint32_t dst0 = As0 + r0 * 128 + ((kc ^ (r0 & 7)) << 4);
        auto begin = [&]() -> uint32_t {   // the ring slot of slice t, free again
            const int st = t % RW_STAGES, use = t / RW_STAGES;
            if (use > 0) ok = mbar_wait(smem_u32(&empty[st]), (use - 1) & 1, failed);
            return dst0 + st * RW_SLICE;
        };
        auto finish = [&]() {
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            if (t >= RW_LAG - 1) {   // the slice of RW_LAG - 1 rounds ago has landed: hand it to the tensor cores
                asm volatile("cp.async.wait_group %0;\n" ::"n"(RW_LAG - 1) : "memory");
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                if (t - (RW_LAG - 1) < slices) mbar_arrive(&full[(t - (RW_LAG - 1)) % RW_STAGES]);
            }
            ++t;
        };
        if (by_segment) {
            // Whole slices lie in one segment: the rows' addresses are made once
            // per segment, from indices that were requested a tile earlier (as a
            // load beside each copy, their latency held every slice up: 342 us
            // instead of 117 at 600k rows of 384).
            int nxt[3][8];
            auto fetch = [&](int m) {
                const int i0 = ((int)blockIdx.x + m * (int)gridDim.x) * RW_M;
#pragma unroll
                for (int s = 0; s < 3; ++s)
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int gd = i0 + r0 + 16 * q;
                        nxt[s][q] = -1;
                        if (s < A.nseg && m < mine && gd < I) nxt[s][q] = A.idx[s] ? __ldg(A.idx[s] + gd) : gd;
                    }
            };
            fetch(0);
            for (int m = 0; m < mine && ok; ++m) {
                int cur[3][8];
#pragma unroll
                for (int s = 0; s < 3; ++s)
#pragma unroll
                    for (int q = 0; q < 8; ++q) cur[s][q] = nxt[s][q];
                fetch(m + 1);
#pragma unroll
                for (int s = 0; s < 3; ++s) {
                    if (s >= A.nseg || !ok) break;
                    const int w = (s + 1 < A.nseg ? A.c0[s + 1] : R) - A.c0[s];
                    for (int c = 0; c < w; c += RW_K) {
                        const uint32_t dst = begin();
                        if (!ok) break;
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const bool in = cur[s][q] >= 0 && c + kc * 8 < w;
                            cp16(dst + q * 2048,
                                 in ? A.ptr[s] + (size_t)cur[s][q] * A.ld[s] + c + kc * 8 : A.ptr[0], in ? 16u : 0u);
                        }
                        finish();
                    }
                }
            }
        } else {
            while (ok && t < slices) {
                const int i0 = ((int)blockIdx.x + (t / kslices) * (int)gridDim.x) * RW_M;
                const int gr = (t % kslices) * RW_K + kc * 8;
                const uint32_t dst = begin();
                if (!ok) break;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int gd = i0 + r0 + 16 * q;
                    const bool in = gd < I && gr < R;
                    cp16(dst + q * 2048, in ? (const void*)chunk_addr(A, gd, gr) : (const void*)A.ptr[0], in ? 16u : 0u);
                }
                finish();
            }
        }
        while (ok && t < slices + RW_LAG - 1) finish();
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    } else if (warp == 8) {
        if (lane == 0) {
            bool ok = true, issued = false;
            for (int m = 0; m < mine && ok; ++m)
                for (int n = 0; n < nb && ok; ++n) {
                    const int u = m * nb + n, buf = u % RW_ACC, use = u / RW_ACC;
                    if (use > 0) ok = mbar_wait(smem_u32(&acce[buf]), (use - 1) & 1, failed);
                    const int cols = min(128, jpad - n * 128);
                    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(cols >> 3) << 17) |
                                           ((uint32_t)(RW_M >> 4) << 24);
                    for (int ks = 0; ks < kslices && ok; ++ks) {
                        const int t = m * kslices + ks, st = t % RW_STAGES;
                        if (n == 0) ok = mbar_wait(smem_u32(&full[st]), (t / RW_STAGES) & 1, failed);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                        const int steps = (min(RW_K, R - ks * RW_K) + 15) / 16;
                        issued = true;
                        for (int k = 0; k < steps; ++k)
                            tc_mma(tmem + buf * 128,
                                   umma_desc_sw128(As0 + st * RW_SLICE + k * 32, 16, 1024),
                                   umma_desc_sw128(Bs0 + ks * jpad * 128 + n * 16384 + k * 32, 16, 1024), idesc,
                                   ks > 0 || k > 0);
                        if (n == nb - 1) tc_commit(&empty[st]);
                    }
                    if (ok) tc_commit(&accf[buf]);
                }
            if (issued) {   // nothing is in flight when the CTA ends
                tc_commit(&drain);
                if (!mbar_drain(smem_u32(&drain), 0)) failed = 1;
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue: a warp holds rows 32 (w mod 4).. of the tile; kReads: warps 0-3
        // the first 64 of a block's columns, 9-12 the others
        constexpr int kChunks = kReads ? 2 : 4;
        const int quarter = warp & 3, half = warp > 8 ? 64 : 0;
        bool ok = true;
        for (int m = 0; m < mine; ++m) {
            const int gi = ((int)blockIdx.x + m * (int)gridDim.x) * RW_M + quarter * 32 + lane;
            for (int n = 0; n < nb; ++n) {
                const int u = m * nb + n, buf = u % RW_ACC;
                const int cols = min(128, jpad - n * 128);
                // what the epilogue reads does not wait for the products
                uint32_t pre[kChunks][32];
                if (kReads && gi < I) {
#pragma unroll
                    for (int c = 0; c < kChunks; ++c) {
                        const int gj = n * 128 + half + 32 * c;
                        if (half + 32 * c < cols) {
                            if (ep.resid) {
#pragma unroll
                                for (int h = 0; h < 4; ++h) ld8(ep.resid + (size_t)gi * ep.ld_resid + gj + 8 * h, pre[c] + 8 * h);
                            } else {
#pragma unroll
                                for (int h = 0; h < 2; ++h) ld8(ep.mask + (size_t)gi * ep.ld_mask + gj + 16 * h, pre[c] + 8 * h);
                            }
                        }
                    }
                }
                if (ok) ok = mbar_wait(smem_u32(&accf[buf]), (u / RW_ACC) & 1, failed);
                ok = __all_sync(0xffffffffu, ok);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll (kReads ? 2 : 1)
                for (int c = 0; c < kChunks; ++c) {
                    const int col = half + 32 * c;
                    if (col >= cols) continue;
                    uint32_t r[32];
                    tc_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + buf * 128 + col, r);
                    if (!ok) {
#pragma unroll
                        for (int q = 0; q < 32; ++q) r[q] = 0u;
                    }
                    if (gi < I) epilogue32<kReads>(ep, wide != 0, bias_s, gi, n * 128 + col, J, r, pre[c]);
                    __syncwarp();   // tcgen05.ld takes whole warps
                }
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                if (ok) mbar_arrive(&acce[buf]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (threadIdx.x == 0 && failed) atomicAdd(&g_tc_timeouts, 1u);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(RW_ACC * 128) : "memory");
}

// ------------------------------------------------ tcgen05, both operands transposed
// The weight gradients: C (I x J) = sum over rows r of A(r, i) B(r, j), rows of
// B gathered, the reduction split over blocks.  One CTA per (128 x 128 tile of
// C, split); slices of 64 rows of both operands go to shared memory as they lie
// in global memory, M- and N-major with the 128-byte swizzle -- element (r, i)
// at (i / 64) * 8192 + (r / 8) * 1024 + (r mod 8) * 128 + ((i / 8 mod 8) xor (r mod
// 8)) * 16 bytes -- where k_gemm transposed them element by element.  A ring of
// six slices, five in flight, gated by the mbarriers that tcgen05.commit
// arrives on.  Split boundaries, order and steps of the reduction are k_gemm's,
// and the results are the same bits.
// L2 bound: 600k rows, 128 x 384, 50 splits: 229 us (4.9 TB/s of L2; k_gemm 1150
// us, the transposing 2-byte stores to shared memory).
constexpr int WG_T = 256, WG_K = 64, WG_STAGES = 6;
constexpr int WG_TILE = WG_K * 128 * 2;                   // 16 KB of one operand
constexpr int WG_SMEM = WG_STAGES * 2 * WG_TILE;

// The copies of one operand by one CTA: 16 threads a row (256 bytes), four rows a
// thread.  Where the tile's columns lie in one segment, the rows' indices are
// requested one slice ahead of their copies.
struct WgSource {
    const uint16_t* p;
    const int* ix;
    int ld, nxt[4];
    bool one, in;
    __device__ __forceinline__ void init(const Operand& op, int d0, int ndim) {
        const int gd = d0 + (threadIdx.x & 15) * 8, last = min(d0 + 128, ndim) - 1;
        const int s0 = (op.nseg > 2 && d0 >= op.c0[2]) ? 2 : (op.nseg > 1 && d0 >= op.c0[1]) ? 1 : 0;
        const int s1 = (op.nseg > 2 && last >= op.c0[2]) ? 2 : (op.nseg > 1 && last >= op.c0[1]) ? 1 : 0;
        one = s0 == s1;
        in = gd < ndim;
        p = (s0 == 2 ? op.ptr[2] : s0 == 1 ? op.ptr[1] : op.ptr[0]);
        ix = (s0 == 2 ? op.idx[2] : s0 == 1 ? op.idx[1] : op.idx[0]);
        ld = (s0 == 2 ? op.ld[2] : s0 == 1 ? op.ld[1] : op.ld[0]);
        const int c0 = (s0 == 2 ? op.c0[2] : s0 == 1 ? op.c0[1] : 0);
        if (in) p += gd - c0;
    }
    __device__ __forceinline__ void fetch(int r0, int rend) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int gr = r0 + (int)(threadIdx.x >> 4) + 16 * q;
            nxt[q] = -1;
            if (in && gr < rend) nxt[q] = ix ? __ldg(ix + gr) : gr;
        }
    }
    __device__ __forceinline__ void copy(uint32_t S, const Operand& op, int d0, int r0, int rend) {
        const int mc = threadIdx.x & 15, rr = threadIdx.x >> 4;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = rr + 16 * q;
            const uint32_t dst = S + (mc >> 3) * 8192 + (r >> 3) * 1024 + (r & 7) * 128 + (((mc & 7) ^ (r & 7)) << 4);
            const bool ok = nxt[q] >= 0;
            const void* src = !ok ? (const void*)op.ptr[0]
                              : one ? (const void*)(p + (size_t)nxt[q] * ld)
                                    : (const void*)chunk_addr(op, r0 + r, d0 + mc * 8);
            cp16(dst, src, ok ? 16u : 0u);
        }
        fetch(r0 + WG_K, rend);
    }
};

__global__ void __launch_bounds__(WG_T, 1) k_gemm_wgrad(int I, int J, int R, Operand A, Operand B, float* __restrict__ out,
                                                        int ld_out, int accumulate, int rchunk,
                                                        float* __restrict__ partial) {
    extern __shared__ __align__(1024) uint8_t wg_smem[];
    __shared__ __align__(8) uint64_t done[WG_STAGES];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    const uint32_t As0 = smem_u32(wg_smem), Bs0 = As0 + WG_STAGES * WG_TILE;
    const int i0 = blockIdx.x * 128, j0 = blockIdx.y * 128;
    const int rb = blockIdx.z * rchunk, re = min(R, rb + rchunk);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cols = min(128, (J - j0 + 15) / 16 * 16);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                     "r"(128)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < WG_STAGES; ++k) mbar_init(&done[k], 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int nch = re > rb ? (re - rb + WG_K - 1) / WG_K : 0;
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |   // both operands MN-major
                           ((uint32_t)(cols >> 3) << 17) | (8u << 24);
    bool ok = true;
    int issued = 0;   // slices
    WgSource sa, sb;
    sa.init(A, i0, I);
    sb.init(B, j0, J);
    sa.fetch(rb, re);
    sb.fetch(rb, re);
#pragma unroll
    for (int k = 0; k < WG_STAGES - 1; ++k) {
        if (k < nch) {
            sa.copy(As0 + k * WG_TILE, A, i0, rb + k * WG_K, re);
            sb.copy(Bs0 + k * WG_TILE, B, j0, rb + k * WG_K, re);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int c = 0; c < nch; ++c) {
        const int b = c % WG_STAGES;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(WG_STAGES - 2) : "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        if (__syncthreads_or(!ok)) break;
        issued = c + 1;
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int steps = (min(WG_K, re - rb - c * WG_K) + 15) / 16;
            for (int k = 0; k < steps; ++k)
                tc_mma(tmem, umma_desc_sw128(As0 + b * WG_TILE + k * 2048, 8192, 1024),
                       umma_desc_sw128(Bs0 + b * WG_TILE + k * 2048, 8192, 1024), idesc, c > 0 || k > 0);
            tc_commit(&done[b]);
        }
        // slice c + STAGES - 1 goes where slice c - 1 was: wait for its MMAs
        const int nx = c + WG_STAGES - 1;
        if (nx < nch) {
            const int bx = nx % WG_STAGES;
            if (c >= 1 && ok) ok = mbar_wait(smem_u32(&done[bx]), ((c - 1) / WG_STAGES) & 1, failed);
            if (ok) {
                sa.copy(As0 + bx * WG_TILE, A, i0, rb + nx * WG_K, re);
                sb.copy(Bs0 + bx * WG_TILE, B, j0, rb + nx * WG_K, re);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (issued > 0 && !mbar_drain(smem_u32(&done[(issued - 1) % WG_STAGES]), ((issued - 1) / WG_STAGES) & 1)) ok = false;
    ok = !__syncthreads_or(!ok || issued < nch);
    if (!ok && threadIdx.x == 0) atomicAdd(&g_tc_timeouts, 1u);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const int gi = i0 + (warp & 3) * 32 + lane;   // warps w and w + 4 hold the same rows, alternate column groups
    for (int c = (warp >> 2) * 32; c < cols; c += 64) {
        uint32_t r[32];
        tc_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c, r);
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            const int gj = j0 + c + q;
            if (gi >= I || gj >= J) continue;
            const float v = nch > 0 && ok ? __uint_as_float(r[q]) : 0.f;
            if (partial) {
                partial[((size_t)blockIdx.z * I + gi) * J + gj] = v;
            } else {
                float* o = out + (size_t)gi * ld_out + gj;
                *o = accumulate ? *o + v : v;
            }
        }
        __syncwarp();   // tcgen05.ld takes whole warps
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(128) : "memory");
}

// ------------------------------------------------------- two layers in one kernel
// One MLP of the network: z = relu(A W1^T + b1) (128 wide), v = z W2^T + b2, with
// an optional residual and an optional sum of v over the rows of each receiver
// (the messages of an edge block).  Both weights stay in shared memory; z goes
// from tensor memory through registers back into tensor memory as the second
// product's operand, and v through shared memory to its place, so that of the
// intermediate values only what the caller asks for reaches HBM.  As separate
// kernels an edge block moved 3 KB of HBM an edge (z twice, the messages twice,
// the residual stream in two precisions); here it moves 1.5 KB.
//
// A CTA owns a contiguous range of rows, cut at receivers when there are sums,
// and walks it in tiles of 128 rows.  Warps 12-15 copy A (ring of slices as in
// k_gemm_rows), one thread of warp 16 issues the products -- the second layer of
// tile m, then the first of tile m+1 -- warps 4-7 make z, warps 8-11 put v into
// strips of 32 columns in shared memory and sum the rows of each receiver there,
// one after another in row order (as k_segsum's), and warps 0-3 store the strips
// with their residuals.  The receiver that a tile leaves open carries its sums to
// the next tile.  All results are the bits of the separate kernels.
// Tensor memory (512 columns): one accumulator of the first layer, two of the
// second, whose readers are the slower ones, and two of z.
// Two things bound it, measured on an edge block of 974k edges (331 us, 367 with z
// kept; its HBM bytes would take 230): the sums (250 us alone) and the copies (255
// for a bf16 result alone; 164 at R = 128).  A thread per row storing 32 bytes of
// 32 rows at a time instead of strips, which make whole lines: 473.  z in shared
// memory, which leaves room for a ring of three slices instead of five: 373.
// Slices are handed over two behind the copies (3 behind: 346, 1: 355).
// The forward pass of 50k spheres went from 5.84 ms of separate kernels to 2.42.
constexpr int ML_T = 544, ML_LAG = 3, ML_MAX_STAGES = 6, ML_STRIP = 32;
constexpr int ML_STRIP_BYTES = 128 * ML_STRIP * 4;   // 16-byte chunk q of a row at q xor (row mod 8)
constexpr int ML_SMEM_MAX = 232448 - 3072;   // dynamic part beside the static arrays (below 3 KB)

struct MlpArgs {
    int M, R, J;
    const uint16_t *w1, *w2;
    const float *b1, *b2;
    uint16_t* z;
    const float* resid;
    float* out;
    uint16_t* out_bf;
    int nagg;
    const int *row_off, *dst;
    uint16_t* agg;
    int stages;
};

// first r in [0, n] with off[r] >= target (off ascending, off[n] >= target); one warp
__device__ __forceinline__ int lower_bound32(const int* __restrict__ off, int n, int target) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;
    while (hi > lo) {
        const int step = (hi - lo + 31) / 32, p = lo + lane * step;
        const int c = __popc(__ballot_sync(0xffffffffu, p < hi && __ldg(off + p) < target));
        if (c == 0) break;
        hi = min(hi, lo + c * step);
        lo = lo + (c - 1) * step + 1;
    }
    return lo;
}

__device__ __forceinline__ void bar_sums() { asm volatile("bar.sync 1, 128;\n" ::: "memory"); }
// the strip between its writers (warps 8-11) and the warps that store v (0-3): each
// side arrives where it has nothing to wait for
__device__ __forceinline__ void bar_strip_full(bool writer) {
    if (writer) asm volatile("bar.arrive 2, 256;\n" ::: "memory");
    else asm volatile("bar.sync 2, 256;\n" ::: "memory");
}
__device__ __forceinline__ void bar_strip_free(bool writer) {
    if (writer) asm volatile("bar.sync 3, 256;\n" ::: "memory");
    else asm volatile("bar.arrive 3, 256;\n" ::: "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }

__global__ void __launch_bounds__(ML_T, 1) k_mlp(Operand A, MlpArgs g) {
    extern __shared__ __align__(1024) uint8_t ml_smem[];
    __shared__ __align__(8) uint64_t full[ML_MAX_STAGES], empty[ML_MAX_STAGES], a1f, a1e, a2f[2], a2e[2], zf[2], ze[2], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    __shared__ __align__(16) float b1s[128], b2s[128], carry[2][128];   // carry: sums of the open receiver, by tile parity
    __shared__ int range[2], s_dst[128], s_after;
    __shared__ uint8_t s_seg[132];   // rows where receivers start in the tile
    __shared__ unsigned s_head[4];
    const int kslices = (g.R + RW_K - 1) / RW_K, jpad = (g.J + 15) / 16 * 16;
    const uint32_t W1 = smem_u32(ml_smem), W2 = W1 + kslices * 16384, ring = W2 + 2 * jpad * 128;
    float* strip = reinterpret_cast<float*>(ml_smem + kslices * 16384 + 2 * jpad * 128 + g.stages * RW_SLICE);
    const bool stored = g.out || g.out_bf;              // v goes to HBM
    const int strips = g.J > ML_STRIP ? g.J / ML_STRIP : 1;   // a tile's
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < ML_MAX_STAGES; ++k) {
            mbar_init(&full[k], 128);
            mbar_init(&empty[k], 1);
        }
        failed = 0;
        mbar_init(&drain, 1);
        mbar_init(&a1f, 1);
        mbar_init(&a1e, 128);
        for (int k = 0; k < 2; ++k) {
            mbar_init(&a2f[k], 1);
            mbar_init(&a2e[k], 128);
            mbar_init(&zf[k], 128);
            mbar_init(&ze[k], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1 || warp == 2) {   // this CTA's rows
        const int b = (int)blockIdx.x + (warp - 1), G = (int)gridDim.x;
        int at;
        if (g.agg) {
            const int target = (int)((long long)g.M * b / G);
            at = b == G ? g.M : g.row_off[lower_bound32(g.row_off, g.nagg, target)];
        } else {
            const long long tiles = (g.M + 127) / 128;
            at = (int)min((long long)g.M, tiles * b / G * 128);
        }
        if (lane == 0) range[warp - 1] = at;
    }
    if (threadIdx.x < 128) {
        b1s[threadIdx.x] = g.b1[threadIdx.x];
        b2s[threadIdx.x] = (int)threadIdx.x < g.J ? g.b2[threadIdx.x] : 0.f;
    }
    {
        Operand w;
        w.ptr[0] = g.w1; w.ptr[1] = w.ptr[2] = nullptr;
        w.idx[0] = w.idx[1] = w.idx[2] = nullptr;
        w.ld[0] = g.R; w.ld[1] = w.ld[2] = 0;
        w.c0[0] = 0; w.c0[1] = w.c0[2] = 1 << 30;
        w.nseg = 1;
        w.trans = 0;
        stage_b(ml_smem, w, 128, 128, g.R, kslices);
        w.ptr[0] = g.w2;
        w.ld[0] = 128;
        stage_b(ml_smem + kslices * 16384, w, g.J, jpad, 128, 2);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int lo = range[0], hi = range[1];
    const int mine = (hi - lo + 127) / 128, slices = mine * kslices;
    bool ok = true;
    if (warp >= 12 && warp < 16) {
        // ---- copies of A
        const int pt = threadIdx.x - 384, kc = pt & 7, r0 = pt >> 3, S = g.stages;
        int t = 0, slot = 0, round = 0;
        const uint32_t dst0 = ring + r0 * 128 + ((kc ^ (r0 & 7)) << 4);
        int hand = 0;   // ring slot handed over next
        auto finish = [&]() {
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            if (t >= ML_LAG - 1) {
                asm volatile("cp.async.wait_group %0;\n" ::"n"(ML_LAG - 1) : "memory");
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                if (t - (ML_LAG - 1) < slices) mbar_arrive(&full[hand]);
                hand = hand + 1 == S ? 0 : hand + 1;
            }
            ++t;
            if (++slot == S) {
                slot = 0;
                ++round;
            }
        };
        int nxt[3][8];
        auto fetch = [&](int m) {
#pragma unroll
            for (int s = 0; s < 3; ++s)
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int gd = lo + m * 128 + r0 + 16 * q;
                    nxt[s][q] = -1;
                    if (s < A.nseg && gd < hi) nxt[s][q] = A.idx[s] ? __ldg(A.idx[s] + gd) : gd;
                }
        };
        fetch(0);
        for (int m = 0; m < mine; ++m) {
            int cur[3][8];
#pragma unroll
            for (int s = 0; s < 3; ++s)
#pragma unroll
                for (int q = 0; q < 8; ++q) cur[s][q] = nxt[s][q];
            fetch(m + 1);
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                if (s >= A.nseg) break;
                const int w = (s + 1 < A.nseg ? A.c0[s + 1] : g.R) - A.c0[s];
                for (int c = 0; c < w; c += RW_K) {
                    // a way out of the loop here, or a condition on the copies, keeps their
                    // addresses from being made during the wait: 50k spheres' forward pass
                    // 2,588 and 2,480 us instead of 2,464
                    if (round > 0 && !mbar_wait(smem_u32(&empty[slot]), (round - 1) & 1, failed))
                        asm volatile("cp.async.wait_all;\nexit;\n" ::: "memory");
                    const uint32_t dst = dst0 + slot * RW_SLICE;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const bool in = cur[s][q] >= 0 && c + kc * 8 < w;
                        cp16(dst + q * 2048, in ? A.ptr[s] + (size_t)cur[s][q] * A.ld[s] + c + kc * 8 : A.ptr[0],
                             in ? 16u : 0u);
                    }
                    finish();
                }
            }
        }
        while (t < slices + ML_LAG - 1) finish();
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    } else if (warp == 16) {
        if (lane == 0) {
            const uint32_t id1 = (1u << 4) | (1u << 7) | (1u << 10) | (16u << 17) | (8u << 24);
            const uint32_t id2 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(jpad >> 3) << 17) | (8u << 24);
            int slot = 0, round = 0;
            bool issued = false;
            auto first = [&](int m) {
                if (m >= 1 && ok) ok = mbar_wait(smem_u32(&a1e), (m - 1) & 1, failed);
                for (int ks = 0; ks < kslices && ok; ++ks) {
                    ok = mbar_wait(smem_u32(&full[slot]), round & 1, failed);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const int steps = (min(RW_K, g.R - ks * RW_K) + 15) / 16;
                    issued = true;
                    for (int k = 0; k < steps; ++k)
                        tc_mma(tmem, umma_desc_sw128(ring + slot * RW_SLICE + k * 32, 16, 1024),
                               umma_desc_sw128(W1 + ks * 16384 + k * 32, 16, 1024), id1, ks > 0 || k > 0);
                    tc_commit(&empty[slot]);
                    if (++slot == g.stages) {
                        slot = 0;
                        ++round;
                    }
                }
                if (ok) tc_commit(&a1f);
            };
            if (mine > 0) first(0);
            for (int m = 0; m < mine && ok; ++m) {
                const int b = m & 1;
                if (m >= 2 && ok) ok = mbar_wait(smem_u32(&a2e[b]), ((m >> 1) - 1) & 1, failed);
                if (ok) ok = mbar_wait(smem_u32(&zf[b]), (m >> 1) & 1, failed);
                if (ok) {
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    for (int k = 0; k < 8; ++k)
                        tc_mma_ta(tmem + 128 + b * 128, tmem + 384 + b * 64 + k * 8,
                                  umma_desc_sw128(W2 + (k >> 2) * jpad * 128 + (k & 3) * 32, 16, 1024), id2, k > 0);
                    tc_commit(&ze[b]);
                }
                if (ok) tc_commit(&a2f[b]);
                if (m + 1 < mine) first(m + 1);
            }
            if (issued) {   // nothing is in flight when the CTA ends
                tc_commit(&drain);
                if (!mbar_drain(smem_u32(&drain), 0)) failed = 1;
            }
        }
        __syncwarp();
    } else if (warp >= 8) {
        // ---- strips and sums: warp w holds rows 32 (w mod 4).. of the tile
        const int w4 = warp & 3, row = w4 * 32 + lane;
        // receivers of this tile and the next, requested two tiles ahead
        int d0 = lo + row < hi && g.agg ? __ldg(g.dst + lo + row) : -1;
        int d1 = lo + 128 + row < hi && g.agg ? __ldg(g.dst + lo + 128 + row) : -1;
        for (int m = 0; m < mine; ++m) {
            const int b = m & 1, e0 = lo + m * 128, gi = e0 + row, rows = min(128, hi - e0);
            int nseg = 0;
            bool open_first = false, open_last = false;
            if (g.agg) {
                const int before = s_dst[127];   // the tile before's last receiver
                const int mydst = d0;
                d0 = d1;
                bar_sums();
                s_dst[row] = mydst;
                if (row == 0) s_after = d0;
                d1 = gi + 256 < hi ? __ldg(g.dst + gi + 256) : -1;
                int prev = __shfl_up_sync(0xffffffffu, mydst, 1);
                bar_sums();
                if (lane == 0 && row > 0) prev = s_dst[row - 1];
                const bool head = gi < hi && (row == 0 || mydst != prev);
                const unsigned hb = __ballot_sync(0xffffffffu, head);
                if (lane == 0) s_head[w4] = hb;
                bar_sums();
                int rank = __popc(hb & ((1u << lane) - 1u));
                for (int w = 0; w < 4; ++w) {
                    if (w < w4) rank += __popc(s_head[w]);
                    nseg += __popc(s_head[w]);
                }
                if (head) s_seg[rank] = (uint8_t)row;
                if (row == 0) s_seg[nseg] = (uint8_t)rows;   // (the barrier before the first strip is read orders s_seg)
                // the first receiver goes on from the tile before, the last into the next
                open_first = m > 0 && s_dst[0] == before;
                open_last = rows == 128 && e0 + 128 < hi && s_after == s_dst[127];
            }
            if (ok) ok = mbar_wait(smem_u32(&a2f[b]), (m >> 1) & 1, failed);
            ok = __all_sync(0xffffffffu, ok);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll 1
            for (int p = 0; p < strips; ++p) {
                const int c = p * ML_STRIP;
                uint32_t r[32];
                tc_ld32(tmem + 128 + ((uint32_t)(w4 * 32) << 16) + b * 128 + c, r);
                // the strip before has been read
                if (m > 0 || p > 0) {
                    if (stored) bar_strip_free(true);
                    else bar_sums();
                }
#pragma unroll
                for (int q = 0; q < ML_STRIP / 4; ++q) {
                    const float4 bias = *reinterpret_cast<const float4*>(&b2s[c + 4 * q]);
                    float4 v = make_float4(__uint_as_float(r[4 * q]) + bias.x, __uint_as_float(r[4 * q + 1]) + bias.y,
                                           __uint_as_float(r[4 * q + 2]) + bias.z, __uint_as_float(r[4 * q + 3]) + bias.w);
                    if (!ok) v = make_float4(0.f, 0.f, 0.f, 0.f);
                    *reinterpret_cast<float4*>(strip + row * ML_STRIP + ((q ^ (row & 7)) << 2)) = v;
                }
                if (p == strips - 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    mbar_arrive(&a2e[b]);
                }
                if (stored) bar_strip_full(true);
                if (!g.agg) continue;
                bar_sums();
                // a warp per receiver, a lane per column
                const int j = c + lane;
                for (int k = w4; k < nseg; k += 4) {
                    const int r0 = s_seg[k];
                    int left = s_seg[k + 1] - r0;
                    const int to = s_dst[r0];
                    float sum = k == 0 && open_first ? carry[b][j] : 0.f;
                    // where this column lies in eight rows on end; eight rows further it is the same
                    const float* x[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = strip + (r0 + i) * ML_STRIP + (lane ^ (((r0 + i) & 7) << 2));
                    int at = 0;
                    for (; left >= 8; left -= 8, at += 8 * ML_STRIP) {
                        float v[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[i] = x[i][at];
#pragma unroll
                        for (int i = 0; i < 8; ++i) sum += v[i];
                    }
                    if (left > 0) {   // past the end +0, which leaves the sum (never -0) as it is
                        float v[7];
#pragma unroll
                        for (int i = 0; i < 7; ++i) v[i] = i < left ? x[i][at] : 0.f;
#pragma unroll
                        for (int i = 0; i < 7; ++i) sum += v[i];
                    }
                    if (k == nseg - 1 && open_last) carry[b ^ 1][j] = sum;
                    else g.agg[(size_t)to * 128 + j] = bf16_bits(sum);
                }
                __syncwarp();   // tcgen05.ld and the barrier take whole warps
            }
        }
    } else if (warp >= 4) {
        // ---- z: warp w holds rows 32 (w mod 4).. of the tile
        const int row = (warp & 3) * 32 + lane;
        const uint32_t quarter = (uint32_t)((warp & 3) * 32) << 16;
        int m = 0;
        for (; m < mine; ++m) {
            const int b = m & 1, gi = lo + m * 128 + row;
            const bool ready = (m < 2 || mbar_wait(smem_u32(&ze[b]), ((m >> 1) - 1) & 1, failed)) &&
                               mbar_wait(smem_u32(&a1f), m & 1, failed);
            if (!__all_sync(0xffffffffu, ready)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int c = 0; c < 128; c += 32) {
                uint32_t r[32], h[16];
                tc_ld32(tmem + quarter + c, r);
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    h[q] = bf16_pair(fmaxf(__uint_as_float(r[2 * q]) + b1s[c + 2 * q], 0.f),
                                     fmaxf(__uint_as_float(r[2 * q + 1]) + b1s[c + 2 * q + 1], 0.f));
                tc_st16(tmem + 384 + quarter + b * 64 + c / 2, h);
                if (g.z && gi < hi) {
                    st8(g.z + (size_t)gi * 128 + c, h);
                    st8(g.z + (size_t)gi * 128 + c + 16, h + 8);
                }
                __syncwarp();
            }
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            mbar_arrive(&a1e);
            mbar_arrive(&zf[b]);
        }
        if (g.z)   // after a wait that ran out
            for (int gi = lo + m * 128 + row; gi < hi; gi += 128)
                for (int c = 0; c < 16; ++c) reinterpret_cast<uint4*>(g.z + (size_t)gi * 128)[c] = make_uint4(0u, 0u, 0u, 0u);
    } else {
        // ---- v: warp w stores rows 32 w.. of the tile from the strips, eight lanes a
        // row (whole lines), four columns a lane
        const int q = lane & 7, J = g.J, total = stored ? mine * strips : 0;
        // row of this lane's k-th four columns of strip P, and its place in v
        auto gi_of = [&](int P, int k) { return lo + P / strips * 128 + warp * 32 + 4 * k + (lane >> 3); };
        auto col_of = [&](int P) { return P % strips * ML_STRIP + 4 * q; };
        float4 r[8];   // residual of the strip to come
        auto load_res = [&](int P) {
            if (!g.resid || P >= total) return;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (gi_of(P, k) < hi) r[k] = __ldcs(reinterpret_cast<const float4*>(g.resid + (size_t)gi_of(P, k) * 128 + col_of(P)));
        };
        auto finish = [&](int P) {
            __syncwarp();   // the barriers take whole warps
            bar_strip_full(false);
            float4 v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int row = warp * 32 + 4 * k + (lane >> 3);
                v[k] = *reinterpret_cast<const float4*>(strip + row * ML_STRIP + ((q ^ (row & 7)) << 2));
            }
            __syncwarp();
            if (P + 1 < total) bar_strip_free(false);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (g.resid) v[k] = make_float4(r[k].x + v[k].x, r[k].y + v[k].y, r[k].z + v[k].z, r[k].w + v[k].w);
            load_res(P + 1);
            if (col_of(P) < J) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int gi = gi_of(P, k);
                    if (gi >= hi) continue;
                    if (g.out) *reinterpret_cast<float4*>(g.out + (size_t)gi * J + col_of(P)) = v[k];
                    if (g.out_bf)
                        *reinterpret_cast<uint2*>(g.out_bf + (size_t)gi * J + col_of(P)) =
                            make_uint2(bf16_pair(v[k].x, v[k].y), bf16_pair(v[k].z, v[k].w));
                }
            }
        };
        load_res(0);
#pragma unroll 1
        for (int P = 0; P < total; ++P) {
            if (g.resid && P % strips == 0) {   // the next tile's residual on its way to L2
                const int gi = lo + (P / strips + 1) * 128 + warp * 32 + lane;
                if (gi < hi) {
#pragma unroll
                    for (int h = 0; h < 4; ++h) prefetch_l2(g.resid + (size_t)gi * 128 + 32 * h);
                }
            }
            finish(P);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (threadIdx.x == 0 && failed) atomicAdd(&g_tc_timeouts, 1u);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
}

// Partial products of a split reduction (or column sums by chunk), added in order.  A block stages
// SR_SPLITS splits of 32 outputs in shared memory, all loads in flight, and one
// warp adds them.  One thread per output left 64 blocks with a thread's 152 loads
// in rounds of latency (11 us a weight gradient of the network's edges, 7 here).
constexpr int SR_SPLITS = 160;
__global__ void __launch_bounds__(256) k_split_reduce(int I, int J, int splits, const float* __restrict__ partial,
                                                      float* __restrict__ out, int ld_out, int accumulate) {
    __shared__ float tile[SR_SPLITS][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const size_t IJ = (size_t)I * J, k = (size_t)blockIdx.x * 32 + lane;
    float s = 0.f;
    for (int z0 = 0; z0 < splits; z0 += SR_SPLITS) {
        const int m = min(SR_SPLITS, splits - z0);
        __syncthreads();
        if (k < IJ) {
#pragma unroll 20
            for (int z = g; z < m; z += 8) tile[z][lane] = partial[(z0 + z) * IJ + k];
        }
        __syncthreads();
        if (g == 0) {
#pragma unroll 32
            for (int z = 0; z < m; ++z) s += tile[z][lane];
        }
    }
    if (g > 0 || k >= IJ) return;
    const int i = (int)(k / J), j = (int)(k % J);
    float* o = out + (size_t)i * ld_out + j;
    *o = accumulate ? *o + s : s;
}

// ------------------------------------------------------- reductions, misc

__global__ void k_segsum(int nrows, int J, const int* __restrict__ row_off, const int* __restrict__ perm,
                         const float* __restrict__ x, int ldx, float* __restrict__ out, int ld_out, int accumulate,
                         uint16_t* __restrict__ out_bf, int ld_out_bf) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= nrows) return;
    const int row = (int)w;
    const int e0 = row_off[row], e1 = row_off[row + 1];
    for (int j = lane; j < J; j += 32) {
        float s = (accumulate && out) ? out[(size_t)row * ld_out + j] : 0.f;
        for (int e = e0; e < e1; ++e) {
            const size_t sr = perm ? (size_t)perm[e] : (size_t)e;
            s += x[sr * ldx + j];
        }
        if (out) out[(size_t)row * ld_out + j] = s;
        if (out_bf) out_bf[(size_t)row * ld_out_bf + j] = bf16_bits(s);
    }
}

// The gradient of h of every sphere (rows of 128): out[i] = y[i] + x[i], then the
// rows off0[i] .. of d (columns 0..127) and the rows perm1[off1[i]] .. (columns
// 128..255) added in list order, and its bf16 copy: the additions of
// sdem_sg_gather_add and two sdem_sg_segsum calls, in their order.
// Bound by HBM (d, 1 KB an edge, once).  k_segsum keeps one row in flight a warp;
// here four (with eight, and with 16, too few warps fit: 78 and 93 us against 68):
// 330k edges of 16k spheres 65 us in a training step (5.1 TB/s), 108 in three kernels.
__global__ void __launch_bounds__(256) k_sphere_grad(int n, const int* __restrict__ off0, const int* __restrict__ off1,
                                                     const int* __restrict__ perm1, const float* __restrict__ x, int ldx,
                                                     const float* __restrict__ y, const float* __restrict__ d,
                                                     float* __restrict__ out, uint16_t* __restrict__ out_bf) {
    const int i = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= n) return;
    const float4 a = *reinterpret_cast<const float4*>(x + (size_t)i * ldx + lane * 4);
    const float4 u = *reinterpret_cast<const float4*>(y + (size_t)i * 128 + lane * 4);
    float4 s = make_float4(u.x + a.x, u.y + a.y, u.z + a.z, u.w + a.w);
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const int* __restrict__ off = side ? off1 : off0;
        const int e0 = off[i], e1 = off[i + 1];
        const float* __restrict__ dc = d + side * 128 + lane * 4;
        for (int b = e0; b < e1; b += 32) {
            const int mine = b + lane < e1 ? (side ? perm1[b + lane] : b + lane) : 0, m = min(32, e1 - b);
            for (int k = 0; k < m; k += 4) {
                float4 v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int row = __shfl_sync(0xffffffffu, mine, (k + q) & 31);
                    if (k + q < m) v[q] = __ldcs(reinterpret_cast<const float4*>(dc + (size_t)row * 256));
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (k + q < m) s = make_float4(s.x + v[q].x, s.y + v[q].y, s.z + v[q].z, s.w + v[q].w);
            }
        }
    }
    *reinterpret_cast<float4*>(out + (size_t)i * 128 + lane * 4) = s;
    *reinterpret_cast<uint2*>(out_bf + (size_t)i * 128 + lane * 4) = make_uint2(bf16_pair(s.x, s.y), bf16_pair(s.z, s.w));
}

// rows of whole float4s, eight columns a thread (k_gather_add: one; 337k rows of
// 128 columns with a gather, an addend and a bf16 copy: 210 us, 67 here at 6.5 TB/s
// of HBM)
__global__ void k_gather_add8(int rows, int J8, const int* __restrict__ idx, const float* __restrict__ x, int ldx,
                              const float* __restrict__ y, int ldy, float* __restrict__ out, int ld_out,
                              uint16_t* __restrict__ out_bf, int ld_out_bf) {
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (size_t)rows * J8) return;
    const size_t e = k / J8;
    const int j = (int)(k % J8) * 8;
    const size_t xr = idx ? (size_t)__ldg(idx + e) : e;
    float4 v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        v[h] = *reinterpret_cast<const float4*>(x + xr * ldx + j + 4 * h);
        if (y) {
            const float4 u = *reinterpret_cast<const float4*>(y + e * ldy + j + 4 * h);
            v[h] = make_float4(u.x + v[h].x, u.y + v[h].y, u.z + v[h].z, u.w + v[h].w);
        }
        if (out) *reinterpret_cast<float4*>(out + e * ld_out + j + 4 * h) = v[h];
    }
    if (out_bf)
        *reinterpret_cast<uint4*>(out_bf + e * ld_out_bf + j) =
            make_uint4(bf16_pair(v[0].x, v[0].y), bf16_pair(v[0].z, v[0].w), bf16_pair(v[1].x, v[1].y),
                       bf16_pair(v[1].z, v[1].w));
}

__global__ void k_gather_add(int rows, int J, const int* __restrict__ idx, const float* __restrict__ x, int ldx,
                             const float* __restrict__ y, int ldy, float* __restrict__ out, int ld_out,
                             uint16_t* __restrict__ out_bf, int ld_out_bf) {
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (size_t)rows * J) return;
    const size_t e = k / J;
    const int j = (int)(k % J);
    const size_t xr = idx ? (size_t)idx[e] : e;
    float v = x[xr * ldx + j];
    if (y) v = y[e * ldy + j] + v;
    if (out) out[e * ld_out + j] = v;
    if (out_bf) out_bf[e * ld_out_bf + j] = bf16_bits(v);
}

__global__ void k_colsum_part(int M, int J, const float* __restrict__ x, int ldx, float* __restrict__ partial) {
    const int b = blockIdx.x;
    const int chunk = (M + kColsumBlocks - 1) / kColsumBlocks;
    const int r0 = b * chunk, r1 = min(M, r0 + chunk);
    for (int j = threadIdx.x; j < J; j += blockDim.x) {
        float s = 0.f;
        for (int r = r0; r < r1; ++r) s += x[(size_t)r * ldx + j];
        partial[(size_t)b * J + j] = s;
    }
}

// The same chunks and order of additions for rows of 128 floats: a block takes
// half the columns of a chunk, whose rows come through shared memory, three tiles
// of 64 in flight (cp.async), where one thread per column left one load in flight
// at a time (330k rows: 148 us; 36 with whole rows a block, 29 here).
constexpr int CS_ROWS = 64, CS_COLS = 64, CS_STAGES = 4;
__global__ void __launch_bounds__(256) k_colsum_part128(int M, const float* __restrict__ x, int ldx,
                                                        float* __restrict__ partial) {
    extern __shared__ __align__(16) float cs_tile[];   // CS_STAGES x CS_ROWS x CS_COLS
    const int chunk = (M + kColsumBlocks - 1) / kColsumBlocks;
    const int r0 = blockIdx.x * chunk, r1 = min(M, r0 + chunk);
    const int tiles = r1 > r0 ? (r1 - r0 + CS_ROWS - 1) / CS_ROWS : 0;
    constexpr int kLanes = CS_COLS / 4;
    x += blockIdx.y * CS_COLS;
    auto copy = [&](int t) {
        if (t < tiles) {
            const uint32_t dst = smem_u32(cs_tile + (t % CS_STAGES) * CS_ROWS * CS_COLS);
#pragma unroll
            for (int q = 0; q < CS_ROWS * kLanes / 256; ++q) {
                const int c = threadIdx.x + q * 256, r = r0 + t * CS_ROWS + c / kLanes;
                cp16(dst + c * 16, r < r1 ? x + (size_t)r * ldx + (c & (kLanes - 1)) * 4 : x, r < r1 ? 16u : 0u);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int t = 0; t < CS_STAGES - 1; ++t) copy(t);
    float s = 0.f;
    for (int t = 0; t < tiles; ++t) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(CS_STAGES - 2) : "memory");
        __syncthreads();
        copy(t + CS_STAGES - 1);   // into the tile read in the last round
        if (threadIdx.x < CS_COLS) {
            const float* v = cs_tile + (t % CS_STAGES) * CS_ROWS * CS_COLS + threadIdx.x;
            const int rows = min(CS_ROWS, r1 - r0 - t * CS_ROWS);
            if (rows == CS_ROWS) {
#pragma unroll
                for (int r = 0; r < CS_ROWS; ++r) s += v[r * CS_COLS];
            } else {
                for (int r = 0; r < rows; ++r) s += v[r * CS_COLS];
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (threadIdx.x < CS_COLS) partial[(size_t)blockIdx.x * 128 + blockIdx.y * CS_COLS + threadIdx.x] = s;
}

// out_bf[e] = bf16(v), v = y[e] + x[idx[e]] (rows of 128), and the column sums of v
// in k_colsum_part128's chunks and order, so that v is neither written nor read
// back for the bias gradient.  A block takes tiles of 64 half rows of its chunk: the
// next tile's rows are on their way while this one's go to shared memory, where
// 64 threads add them.  Bound by HBM (768 B a row).  330k rows: 45 us (5.6 TB/s; 55
// with all columns in one block) instead of 67 and 36 in two kernels; with the
// gather's indices loaded beside the rows they point to, 83.
constexpr int GS_ROWS = 64, GS_COLS = 64, GS_T = 512;
constexpr int GS_SMEM = 2 * GS_ROWS * GS_COLS * 4;
__global__ void __launch_bounds__(GS_T) k_gather_add_sum(int M, const int* __restrict__ idx, const float* __restrict__ x,
                                                         int ldx, const float* __restrict__ y, uint16_t* __restrict__ out_bf,
                                                         float* __restrict__ partial) {
    extern __shared__ __align__(16) float gs_tile[];   // two of GS_ROWS x GS_COLS
    const int chunk = (M + kColsumBlocks - 1) / kColsumBlocks;
    const int r0 = blockIdx.x * chunk, r1 = min(M, r0 + chunk);
    const int tiles = r1 > r0 ? (r1 - r0 + GS_ROWS - 1) / GS_ROWS : 0;
    // 16 consecutive threads take half a row, four columns each; two rows a thread
    constexpr int kLanes = GS_COLS / 4, kRows = GS_T / kLanes, kPer = GS_ROWS / kRows;
    const int jt = (threadIdx.x & (kLanes - 1)) * 4, j = blockIdx.y * GS_COLS + jt, g = threadIdx.x / kLanes;
    float4 a[kPer], u[kPer];
    int ids[kPer];   // of the tile after the one in a and u
    auto load_ids = [&](int t) {
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int e = r0 + t * GS_ROWS + q * kRows + g;
            ids[q] = e < r1 ? __ldg(idx + e) : 0;
        }
    };
    auto load = [&](int t) {
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int e = r0 + t * GS_ROWS + q * kRows + g;
            if (e < r1) {
                u[q] = __ldcs(reinterpret_cast<const float4*>(y + (size_t)e * 128 + j));
                a[q] = *reinterpret_cast<const float4*>(x + (size_t)ids[q] * ldx + j);
            }
        }
        load_ids(t + 1);
    };
    load_ids(0);
    load(0);
    float s = 0.f;
    for (int t = 0; t < tiles; ++t) {
        float* tile = gs_tile + (t & 1) * GS_ROWS * GS_COLS;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int r = q * kRows + g, e = r0 + t * GS_ROWS + r;
            if (e < r1) {
                const float4 v = make_float4(u[q].x + a[q].x, u[q].y + a[q].y, u[q].z + a[q].z, u[q].w + a[q].w);
                *reinterpret_cast<float4*>(tile + r * GS_COLS + jt) = v;
                *reinterpret_cast<uint2*>(out_bf + (size_t)e * 128 + j) = make_uint2(bf16_pair(v.x, v.y), bf16_pair(v.z, v.w));
            }
        }
        load(t + 1);
        __syncthreads();   // the tile is whole; the other one is read no more
        if (threadIdx.x < GS_COLS) {
            const float* v = tile + threadIdx.x;
            const int rows = min(GS_ROWS, r1 - r0 - t * GS_ROWS);
            if (rows == GS_ROWS) {
#pragma unroll
                for (int r = 0; r < GS_ROWS; ++r) s += v[r * GS_COLS];
            } else {
                for (int r = 0; r < rows; ++r) s += v[r * GS_COLS];
            }
        }
    }
    if (threadIdx.x < GS_COLS) partial[(size_t)blockIdx.x * 128 + blockIdx.y * GS_COLS + threadIdx.x] = s;
}

__global__ void k_mse(int n, int K, const float* __restrict__ pred, int ldp, const float* __restrict__ target,
                      float* __restrict__ rowerr, float* __restrict__ dpred, uint16_t* __restrict__ dpred_bf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float inv = 2.0f / ((float)n * (float)K);
    float e = 0.f;
    for (int k = 0; k < ldp; ++k) {
        float d = 0.f;
        if (k < K) {
            const float r = pred[(size_t)i * ldp + k] - target[(size_t)i * K + k];
            e += r * r;
            d = r * inv;
        }
        if (dpred) dpred[(size_t)i * ldp + k] = d;
        if (dpred_bf) dpred_bf[(size_t)i * ldp + k] = bf16_bits(d);
    }
    if (rowerr) rowerr[i] = e;
}

__global__ void k_adam(long long n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, uint16_t* __restrict__ p_bf, float lr, float b1, float b2, float eps,
                       float wd, float c1, float c2) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float gk = g[k];
    const float mk = b1 * m[k] + (1.f - b1) * gk;
    const float vk = b2 * v[k] + (1.f - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    const float mh = mk / c1, vh = vk / c2;
    const float pk = p[k] - lr * (mh / (sqrtf(vh) + eps) + wd * p[k]);
    p[k] = pk;
    if (p_bf) p_bf[k] = bf16_bits(pk);
}

__global__ void k_to_bf16(long long n, const float* __restrict__ x, uint16_t* __restrict__ y) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) y[k] = bf16_bits(x[k]);
}

__global__ void k_advance(int n, const float* __restrict__ pred, int ldp, double ascale, double gx, double gy,
                          double gz, double h, sdem_sg_box box, double* __restrict__ posR, double* __restrict__ vel,
                          double* __restrict__ omega) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double g[3] = {gx, gy, gz};
    const double r = posR[4 * (size_t)i + 3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double acc = ascale * (double)pred[(size_t)i * ldp + a] + g[a];
        const double v0 = vel[(size_t)i * 3 + a];
        double vn = v0 + acc * h;
        double x = posR[4 * (size_t)i + a] + vn * h;
        const double lo = box.lo[a] + r, hi = box.hi[a] - r;
        if (x < lo) {
            x = lo;
            vn = fmax(vn, 0.0);
        } else if (x > hi) {
            x = hi;
            vn = fmin(vn, 0.0);
        }
        vel[((size_t)2 * n + i) * 3 + a] = vel[((size_t)n + i) * 3 + a];
        vel[((size_t)n + i) * 3 + a] = v0;
        vel[(size_t)i * 3 + a] = vn;
        posR[4 * (size_t)i + a] = x;
        const double al = ascale * (double)pred[(size_t)i * ldp + 3 + a] / r;
        omega[(size_t)i * 3 + a] += al * h;
    }
}

// ------------------------------------------------------------------- host

inline cudaStream_t st(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline int launched() { return cudaGetLastError() == cudaSuccess ? SDEM_SG_OK : SDEM_SG_E_CUDA; }

inline unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

inline bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

// The opt-in of a kernel to large dynamic shared memory, per device (idempotent,
// a host-side attribute: cheap enough to set at every call).
inline bool set_smem(const void* f, int bytes) {
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

inline int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    return n;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Checks an operand against the dimension its columns cover (total width)
// and converts it to the device form.
bool make_operand(const sdem_sg_operand* in, int cover, Operand* out) {
    if (!in || in->nseg < 1 || in->nseg > 3 || (in->trans != 0 && in->trans != 1)) return false;
    int col = 0;
    for (int s = 0; s < 3; ++s) {
        if (s < in->nseg) {
            if (!in->ptr[s] || !aligned16(in->ptr[s]) || in->width[s] <= 0 || in->width[s] % 8 || in->ld[s] % 8 ||
                in->ld[s] < in->width[s])
                return false;
            out->ptr[s] = in->ptr[s];
            out->idx[s] = in->idx[s];
            out->ld[s] = in->ld[s];
            out->c0[s] = col;
            col += in->width[s];
        } else {
            out->ptr[s] = nullptr;
            out->idx[s] = nullptr;
            out->ld[s] = 0;
            out->c0[s] = 1 << 30;
        }
    }
    out->nseg = in->nseg;
    out->trans = in->trans;
    return col == cover;
}

}  // namespace

extern "C" {

int sdem_sg_cells(int n, const double* posR, const sdem_sg_grid* g, int* cell, void* stream) {
    if (n < 0 || !g || g->cell <= 0.0 || g->dim[0] < 1 || g->dim[1] < 1 || g->dim[2] < 1 ||
        (long long)g->dim[0] * g->dim[1] * g->dim[2] >= (1ll << 31))
        return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    if (!posR || !cell) return SDEM_SG_E_ARG;
    k_cells<<<blocks(n, 256), 256, 0, st(stream)>>>(n, posR, *g, cell);
    return launched();
}

int sdem_sg_edge_count(int n, const double* posR, const sdem_sg_grid* g, const int* cell, const int* cell_start,
                       const int* sorted, int* degree, void* stream) {
    if (n < 0 || !g || g->cutoff > g->cell) return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    if (!posR || !cell || !cell_start || !sorted || !degree) return SDEM_SG_E_ARG;
    k_edges<false><<<blocks(n, 128), 128, 0, st(stream)>>>(n, posR, *g, cell, cell_start, sorted, degree, nullptr,
                                                           nullptr, nullptr, nullptr);
    return launched();
}

int sdem_sg_edge_fill(int n, const double* posR, const sdem_sg_grid* g, const int* cell, const int* cell_start,
                      const int* sorted, const int* row_off, int* dst, int* src, uint16_t* efeat, void* stream) {
    if (n < 0 || !g || g->cutoff > g->cell || g->scale <= 0.0) return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    if (!posR || !cell || !cell_start || !sorted || !row_off || !dst || !src || !efeat || !aligned16(efeat))
        return SDEM_SG_E_ARG;
    k_edges<true><<<blocks(n, 128), 128, 0, st(stream)>>>(n, posR, *g, cell, cell_start, sorted, nullptr, row_off,
                                                          dst, src, efeat);
    return launched();
}

namespace {
bool graph_args(int n, const double* posR, const sdem_sg_grid* g, const void* work, GridDiv* dv, float* margin) {
    if (n < 1 || !posR || !g || !work || g->cell <= 0.0 || g->scale <= 0.0 || g->cutoff > g->cell || g->cutoff <= 0.0 ||
        g->dim[0] < 1 || g->dim[1] < 1 || g->dim[2] < 1 ||
        (long long)g->dim[0] * g->dim[1] * g->dim[2] >= (1ll << 31) - 1 || (reinterpret_cast<uintptr_t>(work) & 255u) != 0)
        return false;
    dv->cell = fpi::divisor(g->cell);
    dv->scale = fpi::divisor(g->scale);
    // coordinates relative to a corner stay below 1.001 cells and differences
    // below 3: each of the ~8 roundings of a distance is below 3 cell 2^-24; the
    // margin is twice their sum
    *margin = (float)(24.0 * g->cell * ldexp(1.0, -23));
    return true;
}
}  // namespace

long long sdem_sg_graph_work(int n, const sdem_sg_grid* g) {
    if (n < 1 || !g || g->dim[0] < 1 || g->dim[1] < 1 || g->dim[2] < 1 ||
        (long long)g->dim[0] * g->dim[1] * g->dim[2] >= (1ll << 31) - 1)
        return 0;
    return (long long)graph_work(nullptr, n, (long long)g->dim[0] * g->dim[1] * g->dim[2]).bytes;
}

int sdem_sg_graph_count(int n, const double* posR, const sdem_sg_grid* g, void* work, int* row_off, void* stream) {
    GridDiv dv;
    float margin;
    if (!graph_args(n, posR, g, work, &dv, &margin) || !row_off || !aligned16(row_off)) return SDEM_SG_E_ARG;
    const long long ncell = (long long)g->dim[0] * g->dim[1] * g->dim[2];
    const GraphWork w = graph_work(work, n, ncell);
    const cudaStream_t q = st(stream);
    if (cudaMemsetAsync(work, 0, w.clear, q) != cudaSuccess) return SDEM_SG_E_CUDA;
    const unsigned b = blocks(n, GR_T);
    k_graph_bin<<<b, GR_T, 0, q>>>(n, posR, *g, dv, w);
    scan::scan_cells(w.cell_cnt, ncell, w.cell_start, w.cctl, w.cwords, w.status, q);
    k_graph_scatter<<<b, GR_T, 0, q>>>(n, w);
    k_graph_order<<<b, GR_T, 0, q>>>(n, posR, *g, w);
    k_graph_count<<<b, GR_T, 0, q>>>(n, *g, margin, w);
    scan::scan_cells(w.degree, n, row_off, w.rctl, w.rwords, w.status, q);
    return launched();
}

int sdem_sg_graph_fill(int n, const double* posR, const sdem_sg_grid* g, void* work, const int* row_off, int* dst,
                       int* src, uint16_t* efeat, void* stream) {
    GridDiv dv;
    float margin;
    if (!graph_args(n, posR, g, work, &dv, &margin) || !row_off || !dst || !src || !efeat || !aligned16(efeat))
        return SDEM_SG_E_ARG;
    const GraphWork w = graph_work(work, n, (long long)g->dim[0] * g->dim[1] * g->dim[2]);
    k_graph_fill<<<blocks(n, GF_S), GR_T, 0, st(stream)>>>(n, *g, dv, margin, w, row_off, dst, src, efeat);
    return launched();
}

int sdem_sg_node_features(int n, const double* posR, const double* vel, const double* omega, int nw,
                          const double* planes, double scale, double vscale, double dclip, uint16_t* nfeat,
                          void* stream) {
    if (n < 0 || nw < 0 || scale <= 0.0 || vscale <= 0.0 || dclip <= 0.0) return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    if (!posR || !vel || !omega || !nfeat || !aligned16(nfeat) || (nw > 0 && !planes)) return SDEM_SG_E_ARG;
    k_node_feat<<<blocks(n, 128), 128, 0, st(stream)>>>(n, posR, vel, omega, nw, planes, scale, vscale, dclip, nfeat);
    return launched();
}

int sdem_sg_gemm(int I, int J, int R, const sdem_sg_operand* a, const sdem_sg_operand* b,
                 const sdem_sg_epilogue* ep, int splits, float* partial, void* stream) {
    if (I < 0 || J < 0 || R < 0 || !ep || splits < 1) return SDEM_SG_E_ARG;
    if (I == 0 || J == 0) return SDEM_SG_OK;
    Operand A, B;
    if (!make_operand(a, a && a->trans ? I : R, &A) || !make_operand(b, b && b->trans ? J : R, &B))
        return SDEM_SG_E_ARG;
    if ((!A.trans || !B.trans) && R % 8) return SDEM_SG_E_ARG;
    if (ep->mask && ep->ld_mask < J) return SDEM_SG_E_ARG;
    if (ep->out && ep->ld_out < J) return SDEM_SG_E_ARG;
    if (ep->out_bf && ep->ld_out_bf < J) return SDEM_SG_E_ARG;
    if (ep->resid && ep->ld_resid < J) return SDEM_SG_E_ARG;
    if ((ep->res_out && ep->ld_res_out < J) || (ep->res_out_bf && ep->ld_res_out_bf < J)) return SDEM_SG_E_ARG;
    long long rchunk = R > 0 ? ((long long)R + splits - 1) / splits : BK;
    rchunk = (rchunk + BK - 1) / BK * BK;
    const int nsplit = R > 0 ? (int)((R + rchunk - 1) / rchunk) : 1;
    const dim3 grid(blocks(I, BM), blocks(J, BN), nsplit);
    if (grid.y > 65535 || grid.z > 65535) return SDEM_SG_E_ARG;
    const int jpad = (J + 15) / 16 * 16, kslices = (R + RW_K - 1) / RW_K;
    const size_t bbytes = (size_t)kslices * jpad * 128;
    if (nsplit == 1 && g_tc_enabled && !A.trans && R > 0 && jpad <= RW_J_MAX && bbytes <= RW_B_MAX &&
        (jpad <= 128 || kslices <= RW_STAGES / 2)) {
        // B fits in shared memory (with more than one block of columns a tile's
        // slices stay until the last block, so that two tiles must fit the ring)
        const size_t smem = bbytes + RW_STAGES * RW_SLICE;
        const bool wide = J % 32 == 0 && (!ep->out || (aligned32(ep->out) && ep->ld_out % 8 == 0)) &&
                          (!ep->out_bf || (aligned32(ep->out_bf) && ep->ld_out_bf % 16 == 0)) &&
                          (!ep->mask || (aligned32(ep->mask) && ep->ld_mask % 16 == 0)) &&
                          (!ep->resid || (aligned32(ep->resid) && ep->ld_resid % 8 == 0)) &&
                          (!ep->res_out || (aligned32(ep->res_out) && ep->ld_res_out % 8 == 0)) &&
                          (!ep->res_out_bf || (aligned32(ep->res_out_bf) && ep->ld_res_out_bf % 16 == 0));
        const int tiles = (I + RW_M - 1) / RW_M;
        const bool reads = wide && (ep->resid || ep->mask);
        const auto kernel = reads ? k_gemm_rows<true> : k_gemm_rows<false>;
        if (!set_smem((const void*)kernel, RW_B_MAX + RW_STAGES * RW_SLICE)) return SDEM_SG_E_CUDA;
        kernel<<<std::min(tiles, sm_count()), reads ? RW_T_READS : RW_T, smem, st(stream)>>>(I, J, R, A, B, *ep, wide ? 1 : 0);
        return launched();
    }
    if (nsplit == 1 && g_tc_enabled && !A.trans && !B.trans) {
        if (!set_smem((const void*)k_gemm_tc, TC_SMEM)) return SDEM_SG_E_CUDA;
        const dim3 tgrid(blocks(I, TC_M), blocks(J, TC_N));
        if (tgrid.y > 65535) return SDEM_SG_E_ARG;
        k_gemm_tc<<<tgrid, TC_T, TC_SMEM, st(stream)>>>(I, J, R, A, B, *ep);
        return launched();
    }
    const bool only_out = ep->out && !ep->bias && !ep->relu && !ep->mask && !ep->out_bf && !ep->resid;
    if (g_tc_enabled && A.trans && B.trans && R > 0 && only_out && (nsplit == 1 || partial)) {
        if (!set_smem((const void*)k_gemm_wgrad, WG_SMEM)) return SDEM_SG_E_CUDA;
        const dim3 wgrid(blocks(I, 128), blocks(J, 128), nsplit);
        k_gemm_wgrad<<<wgrid, WG_T, WG_SMEM, st(stream)>>>(I, J, R, A, B, ep->out, ep->ld_out, ep->accumulate, (int)rchunk,
                                                           nsplit > 1 ? partial : nullptr);
        if (nsplit == 1) return launched();
        if (cudaGetLastError() != cudaSuccess) return SDEM_SG_E_CUDA;
        k_split_reduce<<<blocks((long long)I * J, 32), 256, 0, st(stream)>>>(I, J, nsplit, partial, ep->out, ep->ld_out,
                                                                           ep->accumulate);
        return launched();
    }
    if (nsplit == 1) {
        k_gemm<<<grid, GT, 0, st(stream)>>>(I, J, R, A, B, *ep, (int)rchunk, nullptr);
        return launched();
    }
    if (!partial || !ep->out || ep->bias || ep->relu || ep->mask || ep->out_bf || ep->resid) return SDEM_SG_E_ARG;
    k_gemm<<<grid, GT, 0, st(stream)>>>(I, J, R, A, B, *ep, (int)rchunk, partial);
    if (cudaGetLastError() != cudaSuccess) return SDEM_SG_E_CUDA;
    k_split_reduce<<<blocks((long long)I * J, 32), 256, 0, st(stream)>>>(I, J, nsplit, partial, ep->out, ep->ld_out,
                                                                       ep->accumulate);
    return launched();
}

int sdem_sg_mlp(int M, int R, const sdem_sg_operand* a, const uint16_t* w1, const float* b1, const uint16_t* w2,
                const float* b2, int J, uint16_t* z, const float* resid, float* out, uint16_t* out_bf, int nagg,
                const int* row_off, const int* dst, uint16_t* agg_bf, void* stream) {
    if (M < 0 || R < 8 || R > 384 || R % 8 || (J != 16 && J != 128) || !w1 || !b1 || !w2 || !b2 || !aligned16(w1) ||
        !aligned16(w2) || nagg < 0)
        return SDEM_SG_E_ARG;
    if (M == 0) return SDEM_SG_OK;
    Operand A;
    if (!make_operand(a, R, &A) || A.trans) return SDEM_SG_E_ARG;
    if ((A.nseg > 1 && A.c0[1] % RW_K) || (A.nseg > 2 && A.c0[2] % RW_K)) return SDEM_SG_E_ARG;
    if ((z && !aligned32(z)) || (resid && (!aligned32(resid) || J != 128)) || (out && !aligned32(out)) ||
        (out_bf && !aligned32(out_bf)) || (!out && !out_bf && !agg_bf))
        return SDEM_SG_E_ARG;
    if (agg_bf && (J != 128 || !row_off || !dst || nagg < 1)) return SDEM_SG_E_ARG;
    MlpArgs g;
    g.M = M;
    g.R = R;
    g.J = J;
    g.w1 = w1;
    g.b1 = b1;
    g.w2 = w2;
    g.b2 = b2;
    g.z = z;
    g.resid = resid;
    g.out = out;
    g.out_bf = out_bf;
    g.nagg = nagg;
    g.row_off = row_off;
    g.dst = dst;
    g.agg = agg_bf;
    const int fixed = (R + RW_K - 1) / RW_K * 16384 + 2 * J * 128 + (agg_bf || out || out_bf ? ML_STRIP_BYTES : 0);
    g.stages = std::min((int)ML_MAX_STAGES, (ML_SMEM_MAX - fixed) / RW_SLICE);   // 5 at R = 384
    if (!set_smem((const void*)k_mlp, ML_SMEM_MAX)) return SDEM_SG_E_CUDA;
    k_mlp<<<std::min((M + 127) / 128, sm_count()), ML_T, fixed + g.stages * RW_SLICE, st(stream)>>>(A, g);
    return launched();
}

int sdem_sg_set_tensor_path(int use_tcgen05) {
    if (use_tcgen05 != 0 && use_tcgen05 != 1) return SDEM_SG_E_ARG;
    g_tc_enabled = use_tcgen05;
    return SDEM_SG_OK;
}

int sdem_sg_get_tensor_path(void) { return g_tc_enabled; }

int sdem_sg_tensor_timeouts(unsigned int* count) {
    if (!count) return SDEM_SG_E_ARG;
    return cudaMemcpyFromSymbol(count, g_tc_timeouts, sizeof(unsigned int)) == cudaSuccess ? SDEM_SG_OK
                                                                                         : SDEM_SG_E_CUDA;
}

int sdem_sg_segsum(int nrows, int J, const int* row_off, const int* perm, const float* x, int ldx, float* out,
                   int ld_out, int accumulate, uint16_t* out_bf, int ld_out_bf, void* stream) {
    if (nrows < 0 || J < 0 || ldx < J || (out && ld_out < J) || (out_bf && ld_out_bf < J)) return SDEM_SG_E_ARG;
    if (nrows == 0 || J == 0) return SDEM_SG_OK;
    if (!row_off || !x || (!out && !out_bf) || (accumulate && !out)) return SDEM_SG_E_ARG;
    k_segsum<<<blocks((long long)nrows * 32, 256), 256, 0, st(stream)>>>(nrows, J, row_off, perm, x, ldx, out, ld_out,
                                                                        accumulate, out_bf, ld_out_bf);
    return launched();
}

int sdem_sg_gather_add(int rows, int J, const int* idx, const float* x, int ldx, const float* y, int ldy, float* out,
                       int ld_out, uint16_t* out_bf, int ld_out_bf, void* stream) {
    if (rows < 0 || J < 0 || ldx < J || (y && ldy < J) || (out && ld_out < J) || (out_bf && ld_out_bf < J))
        return SDEM_SG_E_ARG;
    if (rows == 0 || J == 0) return SDEM_SG_OK;
    if (!x || (!out && !out_bf)) return SDEM_SG_E_ARG;
    if (J % 8 == 0 && ldx % 4 == 0 && aligned16(x) && (!y || (aligned16(y) && ldy % 4 == 0)) &&
        (!out || (aligned16(out) && ld_out % 4 == 0)) && (!out_bf || (aligned16(out_bf) && ld_out_bf % 8 == 0))) {
        k_gather_add8<<<blocks((long long)rows * (J / 8), 256), 256, 0, st(stream)>>>(rows, J / 8, idx, x, ldx, y, ldy, out,
                                                                                     ld_out, out_bf, ld_out_bf);
        return launched();
    }
    k_gather_add<<<blocks((long long)rows * J, 256), 256, 0, st(stream)>>>(rows, J, idx, x, ldx, y, ldy, out, ld_out,
                                                                          out_bf, ld_out_bf);
    return launched();
}

int sdem_sg_sphere_grad(int n, const int* row_off, const int* src_off, const int* src_perm, const float* x, int ldx,
                        const float* y, const float* d, float* out, uint16_t* out_bf, void* stream) {
    if (n < 0 || ldx < 128 || ldx % 4) return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    // (without edges there is no src_perm)
    if (!row_off || !src_off || !x || !y || !d || !out || !out_bf || !aligned16(x) || !aligned16(y) ||
        !aligned16(d) || !aligned16(out) || !aligned16(out_bf))
        return SDEM_SG_E_ARG;
    k_sphere_grad<<<blocks((long long)n * 32, 256), 256, 0, st(stream)>>>(n, row_off, src_off, src_perm, x, ldx, y, d, out,
                                                                         out_bf);
    return launched();
}

int sdem_sg_gather_add_sum(int rows, const int* idx, const float* x, int ldx, const float* y, uint16_t* out_bf, float* sum,
                           float* partial, void* stream) {
    if (rows < 0 || ldx < 128 || ldx % 4) return SDEM_SG_E_ARG;
    if (!sum || !partial || (rows > 0 && (!idx || !x || !y || !out_bf || !aligned16(x) || !aligned16(y) || !aligned16(out_bf))))
        return SDEM_SG_E_ARG;
    if (!set_smem((const void*)k_gather_add_sum, GS_SMEM)) return SDEM_SG_E_CUDA;
    k_gather_add_sum<<<dim3(kColsumBlocks, 128 / GS_COLS), GS_T, GS_SMEM, st(stream)>>>(rows, idx, x, ldx, y, out_bf, partial);
    if (cudaGetLastError() != cudaSuccess) return SDEM_SG_E_CUDA;
    k_split_reduce<<<blocks(128, 32), 256, 0, st(stream)>>>(1, 128, kColsumBlocks, partial, sum, 128, 1);
    return launched();
}

int sdem_sg_colsum_blocks(void) { return kColsumBlocks; }

int sdem_sg_colsum(int M, int J, const float* x, int ldx, float* out, int accumulate, float* partial, void* stream) {
    if (M < 0 || J < 0 || ldx < J) return SDEM_SG_E_ARG;
    if (J == 0) return SDEM_SG_OK;
    if (!out || !partial || (M > 0 && !x)) return SDEM_SG_E_ARG;
    if (J == 128 && ldx % 4 == 0 && aligned16(x)) {
        const int smem = CS_STAGES * CS_ROWS * CS_COLS * 4;
        if (!set_smem((const void*)k_colsum_part128, smem)) return SDEM_SG_E_CUDA;
        k_colsum_part128<<<dim3(kColsumBlocks, 128 / CS_COLS), 256, smem, st(stream)>>>(M, x, ldx, partial);
    } else {
        k_colsum_part<<<kColsumBlocks, 128, 0, st(stream)>>>(M, J, x, ldx, partial);
    }
    if (cudaGetLastError() != cudaSuccess) return SDEM_SG_E_CUDA;
    k_split_reduce<<<blocks(J, 32), 256, 0, st(stream)>>>(1, J, kColsumBlocks, partial, out, J, accumulate);
    return launched();
}

int sdem_sg_mse(int n, int K, const float* pred, int ldp, const float* target, float* rowerr, float* dpred,
                uint16_t* dpred_bf, void* stream) {
    if (n < 0 || K < 1 || ldp < K) return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    if (!pred || !target) return SDEM_SG_E_ARG;
    k_mse<<<blocks(n, 128), 128, 0, st(stream)>>>(n, K, pred, ldp, target, rowerr, dpred, dpred_bf);
    return launched();
}

int sdem_sg_adam(long long n, float* p, const float* g, float* m, float* v, uint16_t* p_bf, float lr, float beta1,
                 float beta2, float eps, float weight_decay, int step, void* stream) {
    if (n < 0 || step < 1) return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    if (!p || !g || !m || !v) return SDEM_SG_E_ARG;
    const float c1 = (float)(1.0 - pow((double)beta1, (double)step));
    const float c2 = (float)(1.0 - pow((double)beta2, (double)step));
    k_adam<<<blocks(n, 256), 256, 0, st(stream)>>>(n, p, g, m, v, p_bf, lr, beta1, beta2, eps, weight_decay, c1, c2);
    return launched();
}

int sdem_sg_to_bf16(long long n, const float* x, uint16_t* y, void* stream) {
    if (n < 0) return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    if (!x || !y) return SDEM_SG_E_ARG;
    k_to_bf16<<<blocks(n, 256), 256, 0, st(stream)>>>(n, x, y);
    return launched();
}

int sdem_sg_advance(int n, const float* pred, int ldp, double ascale, double gx, double gy, double gz, double h,
                    const sdem_sg_box* box, double* posR, double* vel, double* omega, void* stream) {
    if (n < 0 || ldp < 6 || !box) return SDEM_SG_E_ARG;
    if (n == 0) return SDEM_SG_OK;
    if (!pred || !posR || !vel || !omega) return SDEM_SG_E_ARG;
    k_advance<<<blocks(n, 128), 128, 0, st(stream)>>>(n, pred, ldp, ascale, gx, gy, gz, h, *box, posR, vel, omega);
    return launched();
}

}  // extern "C"
