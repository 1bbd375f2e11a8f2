// fluid.cu -- the fluid species (Ar*, the O2 metastables and O atoms): the
// continuity solve and the averaging cycle that feeds it.
//
// Per step, after Deposit, in the reference's order (src/cuda_main.cu:84-91):
//   1. from the step after the first average on, the continuity solve
//      (Solve_Continuity_eqn, src/cuda_Fluid.cu:34-167): per species an
//      implicit sweep along every x line of plasma cells (a tridiagonal system
//      per line, Thomas algorithm) and the x-face fluxes, then the same along
//      the y lines;
//   2. the diagnostic cycle (Diagnostic_Basic, src/cuda_Diagnostic.cu:268-330):
//      N_ave steps sum the electron density, the next one averages it and the
//      collision tallies into rates and sources (Average_*_MCC_rate,
//      *_Update_Source, src/cuda_Diagnostic.cu:548-743); from that step on
//      the cell densities are copied to the nodes each step
//      (Sync_Fluid_GFCtoGFG_forDen, src/cuda_Fluid.cu:321-339), where the
//      collisions read them, and for Ar the electron collision probability of
//      each cell follows (src/cuda_mccAr.cu:57-58).
//
// The sweep is sequential along a line, so a warp owns a line: its lanes
// build the system's four diagonals in shared memory (from the Gummel
// coefficients, densities and fluxes, several loads per lane on the way at
// once), run the elimination and the back substitution, and write the
// densities and fluxes.  The chain of divisions and, on x lines, the strided
// loads bound it.  Measured on a B200, the x and the y lines of a 513x257
// case: 0.119 and 0.054 ms with one lane doing all three divisions of a cell,
// 0.070 and 0.030 ms so.  The float operations are those of the
// reference, each with the reference's operands, so the result is
// bit-identical to a sequential CPU sweep.  The diagnostic is one thread per
// node: a node's source, its density copy and its cell's probability read and
// write only that node and that cell.
#include <cstdint>

#include "devutil.cuh"
#include "hp_fluid.h"
#include "hp_math.h"
#include "kernels.cuh"
#include "prof.cuh"

namespace hp {
namespace {

using dv::find_case;
using dv::FULL;

__device__ __forceinline__ bool fluid_running(const DevCase &d) { return d.fluid_on && d.nfsp > 0; }

constexpr int FB = 4; // rows of 32 cells whose loads are issued together

// One warp per (case, species, line); DIR 0 an x line, 1 a y line.  Shared
// memory: 4 x L floats per warp (sub-, main and super-diagonal, right-hand
// side), the super-diagonal then holding gam and the right-hand side x.
template <int DIR>
__global__ void __launch_bounds__(128) k_fluid_sweep(const DevCase *__restrict__ cases,
                                                     const int *__restrict__ item_start, int ncases, int items,
                                                     int L) {
    extern __shared__ float sm[];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = (int)(blockIdx.x * (blockDim.x >> 5)) + wib;
    if (w >= items) return;
    const int ci = find_case(item_start, ncases, w);
    const DevCase &d = cases[ci];
    if (!fluid_running(d) || *d.tstep < (int64_t)d.n_ave + 2) return;
    const int nl = DIR ? d.nyl : d.nxl;
    const int n = w - item_start[ci];
    const int f = n / nl, k = n - f * nl;
    const int ngx = d.ngx, ngy = d.ngy, ncx = d.ncx, ncy = d.ncy, C = d.C;
    const int *Ln = (DIR ? d.fl_yl : d.fl_xl) + 3 * k;
    // x line: x1, x2, y; y line: x, y1, y2
    const int first = DIR ? Ln[1] : Ln[0], last = DIR ? Ln[2] : Ln[1], fixed = DIR ? Ln[0] : Ln[2];
    const int num = last - first + 1;
    const size_t fo = DIR ? (size_t)f * ncx * ngy : (size_t)f * ngx * ncy;
    const float *ga = (DIR ? d.gay : d.gax) + fo, *gb = (DIR ? d.gby : d.gbx) + fo;
    float *flux = (DIR ? d.ffly : d.fflx) + fo;
    const float *other = DIR ? d.fflx + (size_t)f * ngx * ncy : d.ffly + (size_t)f * ncx * ngy;
    float *den = d.fden + (size_t)f * C;
    const float *src = d.fsrc + (size_t)f * C;
    const float dtc = d.dtc, del_f = dtc / (DIR ? d.dy : d.dx), dother = DIR ? d.dx : d.dy;
    // faces and cells along the line, and the other direction's two faces of a cell
    auto face = [&](int q) { return DIR ? fixed * ngy + q : q * ncy + fixed; };
    auto cell = [&](int q) { return DIR ? fixed * ncy + q : q * ncy + fixed; };
    auto olo = [&](int q) { return DIR ? fixed * ncy + q : q * ngy + fixed; };
    auto ohi = [&](int q) { return DIR ? (fixed + 1) * ncy + q : q * ngy + fixed + 1; };
    float *A = sm + (size_t)wib * 4 * L, *B = A + L, *Cc = B + L, *D = Cc + L;
    // FB rows of 32 cells at a time: all of their loads are on the way together
    for (int i0 = lane; i0 < num; i0 += 32 * FB) {
        float a0[FB], a1[FB], b0[FB], b1[FB], n0[FB], s0[FB], oh[FB], ol[FB];
#pragma unroll
        for (int u = 0; u < FB; u++) {
            const int q = first + min(i0 + 32 * u, num - 1);
            a0[u] = ga[face(q)];
            a1[u] = ga[face(q + 1)];
            b0[u] = gb[face(q)];
            b1[u] = gb[face(q + 1)];
            n0[u] = den[cell(q)];
            s0[u] = src[cell(q)];
            oh[u] = other[ohi(q)];
            ol[u] = other[olo(q)];
        }
#pragma unroll
        for (int u = 0; u < FB; u++) {
            const int i = i0 + 32 * u;
            if (i < num) {
                A[i] = -a0[u] * del_f;
                B[i] = 1 + (a1[u] + b0[u]) * del_f;
                Cc[i] = -b1[u] * del_f;
                D[i] = n0[u] + s0[u] * dtc - (oh[u] - ol[u]) * dtc / dother;
            }
        }
    }
    __syncwarp();
    // tridiag, src/cuda_Fluid.cu:168-184.  Its chain is one division per cell
    // for the pivots (bet_j = B_j - A_j C_{j-1} / bet_{j-1}) and one for the
    // values (x_j = (D_j - A_j x_{j-1}) / bet_j).  Lane 0 takes the pivots and
    // the other lanes, two cells behind, the values: one division instruction
    // serves both, and a pivot crosses the lanes while the next is computed.
    // The divisions of gam = C / bet wait for no other cell and follow with a
    // cell per lane.
    const bool el = lane == 0;
    {
        // per lane: v is bet (lane 0) or x; row j reads a = A, y = C or D and
        // b = B at the lane's own cell, loaded one row ahead
        const float *PA = A - (el ? 0 : 2), *PY = el ? Cc - 1 : D - 2;
        float *W = el ? B : D - 2;
        float v = el ? B[0] : 0.f, pend = B[0], den, a = 0.f, y = 0.f, b = 0.f;
        auto load = [&](int j) {
            a = PA[j];
            y = PY[j];
            b = B[j];
        };
        auto row = [&](int j, bool el_runs, bool x_runs, bool more) {
            den = pend;
            pend = __shfl_sync(FULL, v, 0);
            const float t = a * (el ? y : v);
            const float nu = el ? t : j == 2 ? y : y - t, de = el ? v : den;
            const float bj = b;
            const bool run = el ? el_runs : x_runs;
            if (more && (el ? el_runs : true)) load(j + 1);
            const float q = (run ? nu : 0.f) / (run ? de : 1.f);
            v = run ? (el ? bj - q : q) : v;
            if (run && lane < 2) W[j] = v;
        };
        if (num > 1 && el) load(1);
        if (!el) load(2);
        if (num > 1) {
            row(1, true, false, false);
            if (el) load(2);
            for (int j = 2; j < num; j++) row(j, true, true, true);
            row(num, false, true, true);
        }
        if (num == 1) pend = B[0];
        row(num + 1, false, true, false);
    }
    __syncwarp();
    int ok = 1;
    for (int i = lane; i < num; i += 32) {
        const float bet = B[i];
        if (i > 0 && bet == 0) ok = 0;
        if (i < num - 1) Cc[i] = Cc[i] / bet;
    }
    ok = __all_sync(FULL, ok);
    __syncwarp();
    if (ok) {
        float x = D[num - 1];
        int j = num - 2;
        for (; j >= 7; j -= 8) {
            float dk[8], ck[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                dk[k] = D[j - k];
                ck[k] = Cc[j - k];
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                x = dk[k] - ck[k] * x;
                dk[k] = x;
            }
            __syncwarp();
            if (el) {
#pragma unroll
                for (int k = 0; k < 8; k++) D[j - k] = dk[k];
            }
        }
        for (; j >= 0; j--) {
            x = D[j] - Cc[j] * x;
            __syncwarp();
            if (el) D[j] = x;
        }
    }
    __syncwarp();
    if (!ok) return; // a vanishing pivot: the line keeps its state
    for (int i0 = lane; i0 < num; i0 += 32 * FB) {
        int pl[FB];
#pragma unroll
        for (int u = 0; u < FB; u++) pl[u] = d.plasma[cell(first + min(i0 + 32 * u, num - 1))];
#pragma unroll
        for (int u = 0; u < FB; u++) {
            const int i = i0 + 32 * u;
            if (i < num) {
                const float x = D[i];
                const float v = (pl[u] == 1 && x > 1e9f) ? x : 0.0f;
                den[cell(first + i)] = v;
                B[i] = v;
            }
        }
    }
    __syncwarp();
    // Calculate_Flux_x / _y (src/cuda_Fluid.cu:54-95)
    const float *fg = DIR ? d.fl_yfg : d.fl_xfg;
    for (int i0 = lane; i0 <= num; i0 += 32 * FB) {
        float fa[FB], fb[FB];
#pragma unroll
        for (int u = 0; u < FB; u++) {
            const int q = first + min(i0 + 32 * u, num);
            fa[u] = ga[face(q)];
            fb[u] = gb[face(q)];
        }
#pragma unroll
        for (int u = 0; u < FB; u++) {
            const int i = i0 + 32 * u;
            if (i > num) break;
            float v;
            if (i == 0) v = -fg[(size_t)f * nl + k] * fb[u] * B[0];
            else if (i == num) v = fg[(size_t)d.nfsp * nl + (size_t)f * nl + k] * fa[u] * B[num - 1];
            else v = fa[u] * B[i - 1] - fb[u] * B[i];
            flux[face(first + i)] = v;
        }
    }
}

// The diagnostic cycle of one node (see the file comment).
__global__ void __launch_bounds__(256) k_fluid_diag(const DevCase *__restrict__ cases,
                                                    const int *__restrict__ item_start, int ncases, int items) {
    const int t = (int)(blockIdx.x * (unsigned)blockDim.x + threadIdx.x);
    if (t >= items) return;
    const int ci = find_case(item_start, ncases, t);
    const DevCase &d = cases[ci];
    if (!fluid_running(d)) return;
    const int g = t - item_start[ci];
    const int N = d.n_ave;
    const int64_t per = (int64_t)N + 1, ts = *d.tstep;
    const int ph = (int)((ts - 1) % per);
    const int ngy = d.ngy, ncx = d.ncx, ncy = d.ncy, C = d.C, G = d.G, F = d.nfsp;
    const int i = g / ngy, j = g - i * ngy;
    const bool has_cell = i < ncx && j < ncy;
    const int cell = i * ncy + j;
    if (ph < N) {
        d.fl_sum[g] += d.den[g];
    } else {
        // Average_Particle_Density of the electrons, 0.25 x as the sources read it
        const float temp = d.denscale0 / (float)N;
        const float ave = temp * (float)(d.fl_sum[g] + d.den[g]);
        d.fl_sum[g] = 0.0;
        const float eden = (float)(0.25 * (double)ave);
        float R[96], S[5], nn[5];
        for (int ch = 0; ch < 96; ch++) R[ch] = 0.0f;
        if (has_cell) {
            const int st = d.mcc_stride;
            for (int ch = 0; ch < st && ch < d.tnrct; ch++) {
                const size_t q = (size_t)cell * st + ch;
                const unsigned now = d.mcc_count[q];
                R[ch] = d.rate_f[ch] * (float)(now - d.fl_base[q]);
                d.fl_base[q] = now;
            }
        }
        for (int f = 0; f < 5; f++) nn[f] = f < F ? d.fluid_den[(size_t)f * G + g] : 0.0f;
        const float bd1 = d.back_den1 ? d.back_den1[g] : 0.0f, bd2 = d.back_den2 ? d.back_den2[g] : 0.0f;
        hp_fluid_sources(d.gas, R, nn, bd1, bd2, eden, d.rr, S);
        if (has_cell)
            for (int f = 0; f < F; f++) d.fsrc[(size_t)f * C + cell] = S[f];
    }
    if (ts < per) return;
    // the node's density from its cell: (i, j) itself, or for the last row and
    // column of nodes the cell below-left; nodes (0, ncy) and (ncx, 0) have none
    int from = -1;
    if (has_cell) from = cell;
    else if (i == ncx && j >= 1) from = (ncx - 1) * ncy + (j - 1);
    else if (j == ncy && i >= 1) from = (i - 1) * ncy + (ncy - 1);
    if (from < 0) return;
    for (int f = 0; f < F; f++) d.fluid_den[(size_t)f * G + g] = d.fden[(size_t)f * C + from];
    if (d.gas == 0 && has_cell) {
        const float e = hp_expf(-1 * d.dt_mcc * d.sigv[1] * d.fluid_den[g]);
        d.prob[(size_t)C + cell] = d.prob[cell] + 1.0f - e;
    }
}

int blocks_for(int n, int per) { return (n + per - 1) / per; }

} // namespace

int fluid_sweep_warps(int L) {
    const size_t per_warp = (size_t)16 * (size_t)(L > 0 ? L : 1);
    int w = 4;
    while (w > 1 && per_warp * (size_t)w > FLUID_SMEM_MAX) w >>= 1;
    return per_warp > FLUID_SMEM_MAX ? 0 : w;
}

namespace {
cudaError_t launch_fluid_sweeps(const DevCase *cases, int ncases, const FluidPlan &fp, cudaStream_t st) {
    for (int dir = 0; dir < 2; dir++) {
        const int items = dir ? fp.n_y : fp.n_x, L = dir ? fp.len_y : fp.len_x;
        if (items <= 0) continue;
        const int w = fluid_sweep_warps(L);
        if (w == 0) return cudaErrorInvalidValue;
        const size_t smem = (size_t)w * 16 * (size_t)L;
        // The sweeps run beside the step's other kernels on a side stream.  An
        // SM changes its split between L1 and shared memory only when it is
        // empty, so blocks of a sweep under a small split keep the blocks of
        // the field's products and of Move, which need most of it as shared
        // memory, off their SMs (257x129 Ar/O2: a step of 0.689 ms, 0.622 so).
        const void *kern = dir == 0 ? (const void *)k_fluid_sweep<0> : (const void *)k_fluid_sweep<1>;
        cudaError_t ec = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (ec != cudaSuccess) return ec;
        if (dir == 0) {
            if (smem > 48 * 1024) cudaFuncSetAttribute(k_fluid_sweep<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            prof::mark(st, "k_fluid_sweep_x");
            k_fluid_sweep<0><<<blocks_for(items, w), 32 * w, smem, st>>>(cases, fp.xl_items, ncases, items, L);
        } else {
            if (smem > 48 * 1024) cudaFuncSetAttribute(k_fluid_sweep<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            prof::mark(st, "k_fluid_sweep_y");
            k_fluid_sweep<1><<<blocks_for(items, w), 32 * w, smem, st>>>(cases, fp.yl_items, ncases, items, L);
        }
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_fluid_diag(const DevCase *cases, const int *node_items, int ncases, int n_node_items,
                              const FluidPlan &fp, cudaStream_t st) {
    if (fp.n_x > 0 || fp.n_y > 0 || fp.any) {
        prof::mark(st, "k_fluid_diag");
        k_fluid_diag<<<blocks_for(n_node_items, 256), 256, 0, st>>>(cases, node_items, ncases, n_node_items);
        return cudaGetLastError();
    }
    return cudaSuccess;
}

bool forked(const FluidPlan &fp, const FluidFork &f) { return f.side && !prof::g_on && (fp.n_x > 0 || fp.n_y > 0); }
} // namespace

cudaError_t launch_fluid(const DevCase *cases, const int *node_items, int ncases, int n_node_items,
                         const FluidPlan &fp, cudaStream_t st) {
    cudaError_t e = launch_fluid_sweeps(cases, ncases, fp, st);
    if (e != cudaSuccess) return e;
    return launch_fluid_diag(cases, node_items, ncases, n_node_items, fp, st);
}

cudaError_t fluid_fork_create(FluidFork &f) {
    cudaError_t e = cudaStreamCreateWithFlags(&f.side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&f.fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&f.join, cudaEventDisableTiming);
    if (e != cudaSuccess) fluid_fork_destroy(f);
    return e;
}

void fluid_fork_destroy(FluidFork &f) {
    if (f.side) {
        cudaStreamSynchronize(f.side);
        cudaStreamDestroy(f.side);
    }
    if (f.fork) cudaEventDestroy(f.fork);
    if (f.join) cudaEventDestroy(f.join);
    f = FluidFork();
}

cudaError_t fluid_begin(const DevCase *cases, int ncases, const FluidPlan &fp, const FluidFork &f, cudaStream_t st) {
    if (!forked(fp, f)) return cudaSuccess;
    cudaError_t e = cudaEventRecord(f.fork, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(f.side, f.fork, 0);
    if (e == cudaSuccess) e = launch_fluid_sweeps(cases, ncases, fp, f.side);
    if (e == cudaSuccess) e = cudaEventRecord(f.join, f.side);
    return e;
}

cudaError_t fluid_end(const DevCase *cases, const int *node_items, int ncases, int n_node_items, const FluidPlan &fp,
                      const FluidFork &f, cudaStream_t st) {
    if (!forked(fp, f)) return launch_fluid(cases, node_items, ncases, n_node_items, fp, st);
    cudaError_t e = cudaStreamWaitEvent(st, f.join, 0);
    if (e != cudaSuccess) return e;
    return launch_fluid_diag(cases, node_items, ncases, n_node_items, fp, st);
}

// the event is recorded here as well: a begin that failed has not done so
cudaError_t fluid_join(const FluidPlan &fp, const FluidFork &f, cudaStream_t st) {
    if (!forked(fp, f)) return cudaSuccess;
    cudaError_t e = cudaEventRecord(f.join, f.side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, f.join, 0);
    return e;
}

} // namespace hp
