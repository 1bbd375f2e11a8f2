// fastsolve.cu -- field_mode 2: FP64 iterative refinement whose inner solve
// applies the separable inverse of the symmetrised operator (fastsolve.cpp)
// as four dense FP32 products per pass.
//
// One refinement pass:
//   X = D^-1 (b - A x64) on the rectangle of unknowns (FP64 residual, FP32 out)
//   A1 = X V;  Y = (W^T A1) .* inv_eig;  A2 = Y V^T;  x64 += W A2
// and after the last pass phi_Pois and the final relative residual.  Each
// output element of a product is accumulated in k order from zero with
// separate multiply and add roundings (the file is built with --fmad=false),
// so a CPU loop reproduces it exactly, and no tiling changes it.
//
// The products are small (nx, ny of 33 to 513): what they cost is launches and
// the latency of fetching operands, not the 2 ny nx (nx + ny) flops (22 us of
// FP32 issue for both passes at 513x257, 0.3 us at 129x65).  So
//  * a CTA owns a strip of columns n.  Column n of Y needs column n of A1 only
//    and column n of E needs column n of A2 only, so the second product of each
//    pair follows in the same CTA with its operand in shared memory;
//  * every left operand is kept k-major (X and Y transposed, which is the node
//    order), so that it is copied as it lies and both operands are read along k
//    with constant strides;
//  * up to FS_CLUSTER_MAX unknowns a cluster runs the whole solve, all passes
//    and the final residual, with cluster barriers between the phases: the
//    strips of 16 CTAs keep up with a launch chain of the whole GPU there
//    (129x65 nodes: a step of 142 us with one launch per product, 119 us so);
//    above that each product is a launch of 32 x 32 tiles over the whole GPU, as
//    a strip's left operand would be read from L2 once per strip there (191x94
//    nodes, which the present cluster form does not take: a step of 254 us in
//    an earlier one, 232 in tiles; the eight products of a 513x257 solve 127 us in
//    strips over the whole GPU, 119 in tiles).  The line lies short of where the
//    two would meet: a step with 10 particles per cell takes, cluster and
//    tiles, 90 and 103 us at 8,127 unknowns, 95 and 108 at 9,730, and, past the
//    line, 99 and 110 at 10,400, 105 and 115 at 11,325, 117 and 121 at 12,000
//    (240x52 nodes), 116 and 121 at 13,203, 129 and 135 at 16,320, about the most
//    that the cluster form's other limits admit (fs_cluster_ctas).
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdint>

#include "devutil.cuh"
#include "kernels.cuh"
#include "prof.cuh"

namespace cg = cooperative_groups;

namespace hp {
namespace {

using namespace dv;

constexpr int FT = 512;    // threads per CTA
constexpr int FS_LDB = 16; // columns of a strip, at most: its row length in shared memory

__device__ __forceinline__ void copy16(float *smem, const float *gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// residual of the symmetrised system at unknown (i, j), times the row scale
__device__ __forceinline__ float scaled_residual(const DevCase &d, int i, int j) {
    const int node = (d.fs_i0 + i) * d.ngy + (d.fs_j0 + j), G = d.G, ngy = d.ngy;
    const float *st = d.st;
    const double *v = d.x64;
    double ax = 0.0;
    const float cw = st[node], cs = st[G + node], cc = st[2 * G + node], cn = st[3 * G + node], ce = st[4 * G + node];
    if (cw != 0.0f) ax += (double)cw * v[node - ngy];
    if (cs != 0.0f) ax += (double)cs * v[node - 1];
    ax += (double)cc * v[node];
    if (cn != 0.0f) ax += (double)cn * v[node + 1];
    if (ce != 0.0f) ax += (double)ce * v[node + ngy];
    const double r64 = d.b64[node] - ax;
    return (float)(r64 * (double)d.row_scale[node]);
}

// sum_k a[k][m] b[k][c] for the two columns of a thread, both operands in
// shared memory.  The row lengths are constants, so that a step of k is two
// loads with immediate offsets and four operations (with run-time lengths half
// of the instructions computed addresses).  One row and two columns per
// thread: a warp reads 128 bytes of a and one broadcast pair of b, and a
// strip of nine columns keeps ten warps busy at 129x65.
template <int LDA>
__device__ __forceinline__ void dot_columns(const float *a, const float *b, int K, float &c0, float &c1) {
    int k = 0;
    for (; k + 8 <= K; k += 8, a += 8 * LDA, b += 8 * FS_LDB) {
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const float q = a[u * LDA];
            const float2 p = *reinterpret_cast<const float2 *>(b + u * FS_LDB);
            c0 = c0 + q * p.x;
            c1 = c1 + q * p.y;
        }
    }
    for (; k < K; k++, a += LDA, b += FS_LDB) {
        const float2 p = *reinterpret_cast<const float2 *>(b);
        c0 = c0 + a[0] * p.x;
        c1 = c1 + a[0] * p.y;
    }
}

// epi(m, c, sum_k A[k][m] B[k][c], pre(m, c)) for m < M, c < ws, by the whole
// CTA: one row and columns c, c + 1 per thread (fs_cluster_ctas sees to it that
// the CTA has a thread for all), consecutive threads taking consecutive rows;
// pre is called before the sums, so that what it loads is there after them.
// A: rows of lda floats (32, 64, 96 or 128), B: rows of FS_LDB.
template <class Pre, class Epi>
__device__ __forceinline__ void product(const float *A, int lda, int M, int K, const float *B, int ws, Pre pre, Epi epi) {
    const int t = threadIdx.x;
    if (t < M * ((ws + 1) / 2)) {
        const int c = t / M * 2, m = t - c / 2 * M;
        const bool two = c + 1 < ws;
        const auto p0 = pre(m, c), p1 = pre(m, two ? c + 1 : c);
        float c0 = 0.0f, c1 = 0.0f;
        if (lda == 32) dot_columns<32>(A + m, B + c, K, c0, c1);
        else if (lda == 64) dot_columns<64>(A + m, B + c, K, c0, c1);
        else if (lda == 96) dot_columns<96>(A + m, B + c, K, c0, c1);
        else dot_columns<128>(A + m, B + c, K, c0, c1);
        epi(m, c, c0, p0);
        if (two) epi(m, c + 1, c1, p1);
    }
    __syncthreads(); // the epilogue's shared results
}

// a whole operand, rows x ld floats, into shared memory
__device__ __forceinline__ void load_operand(float *to, const float *from, int rows, int ld) {
    for (int u = threadIdx.x; u < rows * (ld >> 2); u += FT) copy16(to + 4 * u, from + 4 * u);
    copy_commit();
}

// columns n0 .. n0 + ws of a right operand into rows of FS_LDB floats
__device__ __forceinline__ void load_strip(float *to, const float *from, int ld, int K, int n0, int ws) {
    const int c = threadIdx.x % FS_LDB;
    if (c < ws)
        for (int k = threadIdx.x / FS_LDB; k < K; k += FT / FS_LDB) to[k * FS_LDB + c] = from[(size_t)k * ld + n0 + c];
}

// One chunk of FS_CHUNK nodes by 256 threads (tt): phi_Pois and the chunk's
// share of ||r||^2 and ||b||^2 (thread partials over nodes tt, tt + 256, ...,
// warp trees, then the eight warps in order by the caller's thread 0).  The
// four nodes' coefficients are loaded together, then all their values (a node
// outside the stencil stands for itself), then summed in order: node by
// node, each behind its own two loads, a chunk took 4.6 us.
__device__ __forceinline__ void final_chunk(const DevCase &d, int chunk, int tt, double &rr, double &bb) {
    constexpr int Q = FS_CHUNK / 256;
    const int G = d.G, ngy = d.ngy, n0 = chunk * FS_CHUNK + tt;
    const float *st = d.st;
    const double *v = d.x64;
    float c[Q][5];
    double x[Q][5], b[Q];
#pragma unroll
    for (int q = 0; q < Q; q++)
#pragma unroll
        for (int k = 0; k < 5; k++) c[q][k] = n0 + 256 * q < G ? st[(size_t)k * G + n0 + 256 * q] : 0.0f;
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int node = n0 + 256 * q;
        const bool on = node < G;
        const int off[5] = {-ngy, -1, 0, 1, ngy};
#pragma unroll
        for (int k = 0; k < 5; k++) x[q][k] = on ? v[node + (c[q][k] != 0.0f ? off[k] : 0)] : 0.0;
        b[q] = on ? d.b64[node] : 0.0;
    }
    rr = bb = 0.0;
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int node = n0 + 256 * q;
        if (node >= G) continue;
        d.phi_p[node] = c[q][2] == 0.0f ? 0.0f : (float)x[q][2];
        if (c[q][2] == 0.0f) continue;
        double ax = 0.0;
        if (c[q][0] != 0.0f) ax += (double)c[q][0] * x[q][0];
        if (c[q][1] != 0.0f) ax += (double)c[q][1] * x[q][1];
        ax += (double)c[q][2] * x[q][2];
        if (c[q][3] != 0.0f) ax += (double)c[q][3] * x[q][3];
        if (c[q][4] != 0.0f) ax += (double)c[q][4] * x[q][4];
        const double r = b[q] - ax;
        rr += r * r;
        bb += b[q] * b[q];
    }
    rr = warp_sum_d(rr);
    bb = warp_sum_d(bb);
}

// the chunks' sums in a fixed order, by one warp: the case's final residual
__device__ __forceinline__ void final_norm(const DevCase &d, int lane) {
    const int nch = (d.G + FS_CHUNK - 1) / FS_CHUNK;
    double a = 0.0, b = 0.0;
    for (int k = lane; k < nch; k += 32) {
        a += d.fs_res[2 + 2 * k];
        b += d.fs_res[3 + 2 * k];
    }
    a = warp_sum_d(a);
    b = warp_sum_d(b);
    if (lane == 0) {
        d.fs_res[0] = sqrt(a);
        d.fs_res[1] = sqrt(b);
        d.pcg_iters[0] = d.fs_passes;
        d.pcg_iters[1] = d.fs_passes;
        if (!(a == a) || isinf(a)) atomicOr(d.status, ST_NONFINITE);
        else if (b > 0.0 && sqrt(a) > 10.0 * d.pcg_rtol * sqrt(b)) atomicOr(d.status, ST_NOCONV);
    }
}

// ---------------------------------------------------------------- one cluster per case
__global__ void __launch_bounds__(FT, 1) k_gemm_solve(const DevCase *__restrict__ cases, const int *__restrict__ list,
                                                      int n, int passes) {
    enter_kernel();
    extern __shared__ __align__(16) float sm[];
    __shared__ double s_r[FT / 32], s_b[FT / 32];
    cg::cluster_group cl = cg::this_cluster();
    const int CS = (int)cl.num_blocks(), rank = (int)cl.block_rank(), li = (int)blockIdx.x / CS;
    if (li >= n) return;
    const DevCase &d = cases[list[li]];
    const int t = threadIdx.x, nx = d.fs_nx, ny = d.fs_ny, ldm = d.fs_ldm;
    const int wide = (nx + CS - 1) / CS, n0 = rank * wide, ws = max(0, min(nx, n0 + wide) - n0);
    float *const xy = sm, *const w = xy + nx * ldm, *const wt = w + ny * ldm, *const v = wt + ny * ldm,
                *const vt = v + nx * FS_LDB, *const mid = vt + nx * FS_LDB;
    // the constant operands, once for all passes
    load_operand(w, d.fs_W, ny, ldm);
    load_operand(wt, d.fs_Wt, ny, ldm);
    load_strip(v, d.fs_V, d.fs_ldv, nx, n0, ws);
    load_strip(vt, d.fs_Vt, d.fs_ldv, nx, n0, ws);
    for (int pass = 0; pass < passes; pass++) {
        for (int u = rank * FT + t; u < nx * ny; u += CS * FT) {
            const int i = u / ny, j = u - i * ny;
            d.fs_xt[(size_t)i * ldm + j] = scaled_residual(d, i, j);
        }
        cl.sync();
        for (int second = 0; second < 2; second++) {
            load_operand(xy, second ? d.fs_yt : d.fs_xt, nx, ldm);
            copy_wait<0>();
            __syncthreads();
            auto nothing = [](int, int) { return 0; };
            product(xy, ldm, ny, nx, second ? vt : v, ws, nothing,
                    [&](int m, int c, float q, int) { mid[m * FS_LDB + c] = q; });
            auto y_at = [&](int m, int c) { return (size_t)(n0 + c) * ldm + m; };
            auto x_at = [&](int m, int c) { return (size_t)(d.fs_i0 + n0 + c) * d.ngy + (d.fs_j0 + m); };
            if (!second)
                product(w, ldm, ny, ny, mid, ws, [&](int m, int c) { return d.fs_inv[y_at(m, c)]; },
                        [&](int m, int c, float q, float inv) { d.fs_yt[y_at(m, c)] = q * inv; });
            else
                product(wt, ldm, ny, ny, mid, ws, [&](int m, int c) { return d.x64[x_at(m, c)]; },
                        [&](int m, int c, float q, double x) { d.x64[x_at(m, c)] = x + (double)q; });
            cl.sync();
        }
    }
    const int nch = (d.G + FS_CHUNK - 1) / FS_CHUNK, half = t >> 8;
    for (int c0 = rank * (FT / 256); c0 < nch; c0 += CS * (FT / 256)) {
        const int chunk = c0 + half;
        double rr = 0.0, bb = 0.0;
        if (chunk < nch) final_chunk(d, chunk, t & 255, rr, bb);
        if ((t & 31) == 0) {
            s_r[t >> 5] = rr;
            s_b[t >> 5] = bb;
        }
        __syncthreads();
        if ((t & 255) == 0 && chunk < nch) {
            double a = 0.0, b = 0.0;
            for (int w = 0; w < 8; w++) { a += s_r[8 * half + w]; b += s_b[8 * half + w]; }
            d.fs_res[2 + 2 * chunk] = a;
            d.fs_res[3 + 2 * chunk] = b;
        }
        __syncthreads();
    }
    cl.sync();
    if (rank == 0 && t < 32) final_norm(d, t);
}

// ---------------------------------------------------------------- one launch per product
// These products and the residual before them are launched in stream order,
// without launch_next: a tile's CTA has about an SM to itself, and CTAs that
// are placed while the launch before still drains share SMs where others
// stay empty (513x257 nodes: a step of 1.376 ms with launch_next here, 1.312 so).
__global__ void __launch_bounds__(256) k_fs_resid(const DevCase *__restrict__ cases, const int *__restrict__ list,
                                                  const int *__restrict__ item_start, int n, int items) {
    const int t = (int)(blockIdx.x * (unsigned)blockDim.x + threadIdx.x);
    if (t >= items) return;
    const int li = find_case(item_start, n, t);
    const DevCase &d = cases[list[li]];
    const int u = t - item_start[li];
    const int i = u / d.fs_ny, j = u - i * d.fs_ny;
    d.fs_xt[(size_t)i * d.fs_ldm + j] = scaled_residual(d, i, j);
}

// Product S of a pass over the whole GPU: 32 x 32 output tiles, 256 threads of
// 2 x 2 outputs.  Both operands are k-major with the tile's edge contiguous,
// so a slice of 32 k is 32 rows of 128 bytes of each; GEMM_STAGES slices are
// in flight (with one slice read ahead into registers a k step took 57
// cycles at 513x257, the shared-memory reads and the arithmetic each ask for
// 16).  Lanes run along the edge that the result is stored along.
constexpr int GT = FS_TILE, GK = 32, GEMM_STAGES = 6, GEMM_THREADS = 256; // the host counts FS_TILE tiles
static_assert(GT == 32, "16 x 16 threads of 2 x 2 outputs, copies of 8 x 16 bytes per row");

template <int S>
__global__ void __launch_bounds__(GEMM_THREADS) k_gemm(const DevCase *__restrict__ cases,
                                                       const int *__restrict__ list,
                                                       const int *__restrict__ tile_start, int n) {
    extern __shared__ __align__(16) float sm[];
    const int li = find_case(tile_start, n, (int)blockIdx.x);
    const DevCase &d = cases[list[li]];
    const int nx = d.fs_nx, ny = d.fs_ny, lda = d.fs_ldm, ldb = d.fs_ldv;
    const int tiles_n = (nx + GT - 1) / GT, tile = (int)blockIdx.x - tile_start[li];
    const int m0 = tile / tiles_n * GT, n0 = tile % tiles_n * GT;
    const float *const A = S == 0 ? d.fs_xt : S == 1 ? d.fs_W : S == 2 ? d.fs_yt : d.fs_Wt;
    const float *const B = S == 0 ? d.fs_V : S == 2 ? d.fs_Vt : d.fs_mid;
    const int K = S == 0 || S == 2 ? nx : ny, slices = (K + GK - 1) / GK;
    const int t = threadIdx.x;
    constexpr bool ALONG_M = S == 1 || S == 3;
    const int tm = ALONG_M ? t & 15 : t >> 4, tn = ALONG_M ? t >> 4 : t & 15;
    // this thread's copies: units of four floats (t & 7) of row t >> 3 of each operand
    const int cu = 4 * (t & 7), cr = t >> 3;
    const bool ca = m0 + cu < lda, cb = n0 + cu < ldb;
    const float *const ga = A + (size_t)cr * lda + m0 + cu, *const gb = B + (size_t)cr * ldb + n0 + cu;
    auto copy = [&](int s) {
        if (s < slices && s * GK + cr < K) {
            float *to = sm + (s % GEMM_STAGES) * (2 * GK * GT) + cr * GT + cu;
            if (ca) copy16(to, ga + (size_t)s * GK * lda);
            if (cb) copy16(to + GK * GT, gb + (size_t)s * GK * ldb);
        }
        copy_commit();
    };
    float c00 = 0.0f, c01 = 0.0f, c10 = 0.0f, c11 = 0.0f; // c[m][n]
#pragma unroll
    for (int s = 0; s < GEMM_STAGES - 1; s++) copy(s);
    for (int s = 0; s < slices; s++) {
        copy_wait<GEMM_STAGES - 2>();
        __syncthreads(); // slice s is here, and every thread is done with the buffer refilled next
        copy(s + GEMM_STAGES - 1);
        const float *as = sm + (s % GEMM_STAGES) * (2 * GK * GT) + 2 * tm, *bs = as - 2 * tm + GK * GT + 2 * tn;
        auto mac = [&](int k) {
            const float2 a = *reinterpret_cast<const float2 *>(as + k * GT);
            const float2 b = *reinterpret_cast<const float2 *>(bs + k * GT);
            c00 = c00 + a.x * b.x;
            c01 = c01 + a.x * b.y;
            c10 = c10 + a.y * b.x;
            c11 = c11 + a.y * b.y;
        };
        const int rows = K - s * GK;
        if (rows >= GK) {
#pragma unroll
            for (int k = 0; k < GK; k++) mac(k);
        } else { // the last slice: exactly its terms, no padded ones
            for (int k = 0; k < rows; k++) mac(k);
        }
    }
    const float cv[2][2] = {{c00, c01}, {c10, c11}};
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const int m = m0 + 2 * tm + a, c = n0 + 2 * tn + b;
            if (m >= ny || c >= nx) continue;
            const size_t o = (size_t)c * lda + m;
            if (!ALONG_M) d.fs_mid[(size_t)m * ldb + c] = cv[a][b];
            else if (S == 1) d.fs_yt[o] = cv[a][b] * d.fs_inv[o];
            else d.x64[(size_t)(d.fs_i0 + c) * d.ngy + (d.fs_j0 + m)] += (double)cv[a][b];
        }
    copy_wait<0>();
}

// After the passes: FS_CHUNK nodes per CTA, CTA sums into fs_res, then one
// warp per case.
__global__ void __launch_bounds__(256) k_fs_final(const DevCase *__restrict__ cases, const int *__restrict__ list) {
    enter_kernel();
    const DevCase &d = cases[list[blockIdx.y]];
    if ((int)blockIdx.x * FS_CHUNK >= d.G) return;
    double rr, bb;
    final_chunk(d, (int)blockIdx.x, (int)threadIdx.x, rr, bb);
    __shared__ double s_r[8], s_b[8];
    if ((threadIdx.x & 31) == 0) {
        s_r[threadIdx.x >> 5] = rr;
        s_b[threadIdx.x >> 5] = bb;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < 8; w++) { a += s_r[w]; b += s_b[w]; }
        d.fs_res[2 + 2 * blockIdx.x] = a;
        d.fs_res[3 + 2 * blockIdx.x] = b;
    }
}

__global__ void __launch_bounds__(32) k_fs_norm(const DevCase *__restrict__ cases, const int *__restrict__ list) {
    enter_kernel();
    final_norm(cases[list[blockIdx.x]], (int)threadIdx.x);
}

inline unsigned nblocks(long long threads, int per) { return (unsigned)((threads + per - 1) / per); }

} // namespace

size_t fs_cluster_smem(int nx, int ny) {
    const size_t ldm = (size_t)((ny + 31) & ~31);
    return sizeof(float) * (nx * ldm + 2 * ny * ldm + 2 * (size_t)nx * FS_LDB + (size_t)ny * FS_LDB);
}

// 8 CTAs (a cluster any GPC can hold) where the outputs of an eighth of the
// columns take at most three quarters of a CTA, else 16; 0: not by a cluster
int fs_cluster_ctas(int nx, int ny) {
    if ((long long)nx * ny > FS_CLUSTER_MAX || ny > 128 || fs_cluster_smem(nx, ny) > FS_SMEM_MAX) return 0;
    for (int ctas = 8; ctas <= 16; ctas *= 2) {
        const int wide = (nx + ctas - 1) / ctas;
        if (wide <= FS_LDB && ny * ((wide + 1) / 2) <= (ctas == 8 ? 384 : FT)) return ctas;
    }
    return 0;
}

cudaError_t launch_fast_field(const DevCase *cases, const FastPlan &fp, cudaStream_t st) {
    cudaError_t e;
    for (const FastGroup &g : fp.groups) {
        if (g.n <= 0) continue;
        if ((e = allow_smem((const void *)k_gemm_solve, g.smem)) != cudaSuccess) return e;
        if ((e = cudaFuncSetAttribute(k_gemm_solve, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess)
            return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(g.n * g.ctas), 1, 1);
        cfg.blockDim = dim3(FT, 1, 1);
        cfg.dynamicSmemBytes = g.smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)g.ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; // as launch_next
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = prof::g_on ? 1 : 2;
        prof::mark(st, "k_gemm");
        if ((e = cudaLaunchKernelEx(&cfg, k_gemm_solve, cases, g.list, g.n, fp.passes)) != cudaSuccess) return e;
    }
    if (fp.n <= 0) return cudaSuccess;
    constexpr size_t smem = GEMM_STAGES * 2 * GK * GT * sizeof(float);
    auto gemm = [&](auto kernel) {
        cudaError_t g = allow_smem((const void *)kernel, smem);
        if (g != cudaSuccess) return g;
        prof::mark(st, "k_gemm");
        kernel<<<(unsigned)fp.tiles, GEMM_THREADS, smem, st>>>(cases, fp.list, fp.tile_start, fp.n);
        return cudaGetLastError();
    };
    for (int pass = 0; pass < fp.passes; pass++) {
        prof::mark(st, "k_fs_resid");
        k_fs_resid<<<nblocks(fp.items, 256), 256, 0, st>>>(cases, fp.list, fp.item_start, fp.n, fp.items);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = gemm(k_gemm<0>);
        if (e == cudaSuccess) e = gemm(k_gemm<1>);
        if (e == cudaSuccess) e = gemm(k_gemm<2>);
        if (e == cudaSuccess) e = gemm(k_gemm<3>);
        if (e != cudaSuccess) return e;
    }
    prof::mark(st, "k_fs_final");
    launch_next(k_fs_final, dim3((unsigned)fp.final_chunks, (unsigned)fp.n), 256, 0, st, cases, fp.list);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    prof::mark(st, "k_fs_norm");
    launch_next(k_fs_norm, (unsigned)fp.n, 32, 0, st, cases, fp.list);
    return cudaGetLastError();
}

} // namespace hp
