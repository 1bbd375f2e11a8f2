// pcg.cu -- the field modes 0 and 1 solve with the CG state on chip.
//
// The algorithm, the node partition and the order of every sum are k_pcg's
// (kernels.cu, from PCG_float, src/cuda_Field.cu:942-1072): CTA `rank` owns
// the nodes [rank*per, rank*per + per), thread t of it the nodes lo + t,
// lo + t + T, ..., and a dot product adds thread partials in a warp tree, the
// warps in order and the CTAs in rank order, in FP64.  So the iterates are
// those of k_pcg bit for bit; what differs is where they live.
//
// An iteration moves no byte that has to leave the SM except the sums and the
// residuals at the edges of the CTAs' node ranges; it is bound by the chain
// of its dependent phases.  k_pcg keeps x, r, p, Ap and the stencil in global
// memory (L2 latency in every phase) and funnels both sums through one thread
// and two block barriers.  Here a thread keeps its K nodes' x, r, p, Ap and
// stencil in registers and p also in shared memory (own nodes and the halo of
// ngy nodes on either side that the product reads), and
//  * a cluster's warps write their partial sums straight into every CTA's
//    shared memory; after the one cluster barrier each warp adds them up for
//    itself, in the order above, with no block barrier;
//  * the whole-GPU form (cases above one 16-CTA cluster) exchanges CTA sums
//    and edge residuals through global memory as 64-bit words that hold 32
//    bits of data and the number of the exchange, so a word that has arrived
//    says so itself: one round trip through L2 instead of a grid barrier and
//    the loads behind it, and no fence.  Every CTA writes its sum into the
//    inbox of every other one: 129 CTAs that poll one common list of sums
//    take 5.0 us per exchange (the polls queue up at the few L2 slices that
//    hold it), each at its own inbox 2.3 us, of which the 129 dependent FP64
//    additions that the order of the sum asks for are 0.6.
// Measured on a B200, us per iteration, k_pcg and this kernel: 129x65 nodes
// (4 CTAs) 12.2 and 2.8; 513x257 (129 CTAs, whole GPU) 13.0 and 6.9.
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

constexpr int MAXW = 16;      // warps per CTA
constexpr int MAXC = 16;      // CTAs of a cluster
constexpr int GRID_MAX = 512; // CTAs of the whole-GPU form
// A solve numbers its exchanges from past every number that the one before can
// have used.  After a wait that gave up the CTAs need not have stopped at the
// same number: one can have finished the exchange that another gave up on, and
// from its own last finished exchange a CTA sends at most three more before it
// leaves (in mode 1, the sum that gives up and the two of the next residual)
// and publishes its edges under at most the next number.  The stored number is
// CTA 0's last; words up to three past it may lie in the inboxes.
constexpr unsigned EXCHANGE_GAP = 8;

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long tagged(unsigned tag, unsigned data) {
    return ((unsigned long long)tag << 32) | data;
}
// the data of a word once it carries `tag`; false when it never did
__device__ __forceinline__ bool poll_word(const unsigned long long *p, unsigned tag, int polls, unsigned &data) {
    for (int k = 0; k < polls; k++) {
        const unsigned long long v = ld_word(p);
        if ((unsigned)(v >> 32) == tag) {
            data = (unsigned)v;
            return true;
        }
    }
    return false;
}
// a double as two such words, side by side (each says for itself that it is there)
__device__ __forceinline__ void st_double(unsigned long long *p, unsigned tag, double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(tagged(tag, (unsigned)u)),
                 "l"(tagged(tag, (unsigned)(u >> 32)))
                 : "memory");
}
__device__ __forceinline__ bool poll_double(const unsigned long long *p, unsigned tag, int polls, double &v) {
    for (int k = 0; k < polls; k++) {
        unsigned long long a, b;
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
        if ((unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag) {
            v = __longlong_as_double((long long)((b << 32) | (unsigned)a));
            return true;
        }
    }
    return false;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <bool GRID> struct Shared { // a cluster's exchanges
    double part[2][MAXC][MAXW + 1]; // warp partials of every CTA (two exchanges in turn)
};
template <> struct Shared<true> { // the whole GPU's
    double warp_part[MAXW];
    double cta[GRID_MAX];
    double own, bcast;
    int gave_up;
};

// K: nodes per thread.  Dynamic shared memory: p of the own nodes between its
// two halos (ngy + per + ngy floats), then (cluster) the own residuals at the edges,
// which the neighbours read.
template <bool GRID, int K>
__global__ void __launch_bounds__(512, 1) k_pcg_chip(const DevCase *__restrict__ cases, const int *__restrict__ list,
                                                  int nlist, int max_per, int max_ngy, int polls) {
    enter_kernel();
    extern __shared__ float dyn[];
    __shared__ Shared<GRID> sh;
    cg::cluster_group cl = cg::this_cluster();
    const int CS = GRID ? (int)gridDim.x : (int)cl.num_blocks();
    const int rank = GRID ? (int)blockIdx.x : (int)cl.block_rank();
    const int li = GRID ? 0 : (int)blockIdx.x / CS;
    if (li >= nlist) return;
    const DevCase &d = cases[list[li]];
    const int G = d.G, ngy = d.ngy;
    const int per = (G + CS - 1) / CS;
    const int lo = rank * per, hi = min(G, lo + per);
    const int T = blockDim.x, t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = T >> 5;
    float *const ps = dyn;                             // node n at n - lo + ngy
    float *const rs = dyn + max_per + 2 * max_ngy;     // node n at n - lo (cluster)
    const int mode = d.field_mode;
    const float *__restrict__ st = d.st;
    const float *__restrict__ ss = mode == 0 ? d.st : d.st_sym;

    // ---- exchanges
    int parity = 0;
    unsigned tag = GRID ? *d.pcg_seq + EXCHANGE_GAP : 0u; // pcg_seq: the last exchange of the solve before
    bool gave_up = false;
    if constexpr (GRID)
        if (t == 0) sh.gave_up = 0;
    // The sum of v over the case's CTAs, in two halves so that work that needs
    // no sum runs while it travels: sum_send, then sum_take.  fence (whole
    // GPU): also order the global writes before it, by any CTA, before the
    // reads after it.
    auto sum_send = [&](double v, bool fence = false) {
        v = warp_sum_d(v);
        if constexpr (GRID) {
            tag++;
            unsigned long long *in = d.pcg_slot + (size_t)(tag & 1u) * 2 * CS * CS; // [to][from]
            if (lane == 0) sh.warp_part[wid] = v;
            if (fence) __threadfence();
            __syncthreads();
            if (t == 0) {
                double a = 0.0;
                for (int k = 0; k < nw; k++) a += sh.warp_part[k];
                sh.own = a;
            }
            __syncthreads();
            if (fence) __threadfence();
            const double own = sh.own;
            for (int q = t; q < CS; q += T) st_double(in + 2 * ((size_t)q * CS + rank), tag, own);
        } else {
            if (lane < CS) *cl.map_shared_rank(&sh.part[parity][rank][wid], lane) = v;
            cluster_arrive();
        }
    };
    auto sum_take = [&](bool fence = false) -> double {
        if constexpr (GRID) {
            const unsigned long long *in = d.pcg_slot + (size_t)(tag & 1u) * 2 * CS * CS + 2 * (size_t)rank * CS;
            for (int q = t; q < CS; q += T)
                if (!poll_double(in + 2 * q, tag, polls, sh.cta[q])) sh.gave_up = 1;
            if (fence) __threadfence();
            __syncthreads();
            if (t == 0) { // 16 loads ahead of the chain of additions
                double a = 0.0;
                int q = 0;
                for (; q + 16 <= CS; q += 16) {
                    double c[16];
#pragma unroll
                    for (int k = 0; k < 16; k++) c[k] = sh.cta[q + k];
#pragma unroll
                    for (int k = 0; k < 16; k++) a += c[k];
                }
                for (; q < CS; q++) a += sh.cta[q];
                sh.bcast = a;
            }
            __syncthreads();
            if (fence) __threadfence();
            gave_up = sh.gave_up != 0;
            return sh.bcast;
        } else {
            cluster_wait();
            double a = 0.0;
            if (lane < CS) {
#pragma unroll
                for (int k = 0; k < MAXW; k++)
                    if (k < nw) a += sh.part[parity][lane][k];
            }
            parity ^= 1;
            double tot = 0.0;
            for (int r = 0; r < CS; r++) tot += __shfl_sync(FULL, a, r);
            return tot;
        }
    };
    auto sum = [&](double v, bool fence = false) -> double {
        sum_send(v, fence);
        return sum_take(fence);
    };

    // ---- the thread's nodes: stencil of the iterated system (0 off the
    // unknowns), the inverse of its diagonal
    float cw[K], cs[K], cc[K], cn[K], ce[K], iv[K];
    float x[K], r[K], p[K], ap[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int n = lo + t + k * T;
        cw[k] = cs[k] = cc[k] = cn[k] = ce[k] = iv[k] = 0.0f;
        x[k] = r[k] = p[k] = ap[k] = 0.0f;
        if (n < hi && ss[2 * G + n] != 0.0f) {
            cw[k] = ss[n];
            cs[k] = ss[G + n];
            cc[k] = ss[2 * G + n];
            cn[k] = ss[3 * G + n];
            ce[k] = ss[4 * G + n];
            iv[k] = 1 / cc[k];
        }
    }
    // ---- its halo nodes (at most two: ngy <= T): the inverse of the diagonal
    // and, whole GPU, the word that the owner's residual comes in.  They
    // belong to the CTAs next to this one: ngy <= T <= per where there are several.
    float hiv[2];
    const unsigned long long *hw[2];
    int hp_at[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int e = t + q * T;
        hiv[q] = 0.0f;
        hw[q] = nullptr;
        hp_at[q] = e < ngy ? e : per + e; // after the own nodes
        if (e < 2 * ngy) {
            const int h = e < ngy ? lo - ngy + e : lo + per + (e - ngy);
            if (h >= 0 && h < G) {
                const float c = ss[2 * G + h];
                if (c != 0.0f) {
                    hiv[q] = 1 / c;
                    if (GRID) hw[q] = d.pcg_edge + h;
                }
            }
            ps[hp_at[q]] = 0.0f;
        }
    }
    for (int k = t; k < per; k += T) ps[ngy + k] = 0.0f;
    // the own residuals the neighbours need, before the sum that follows
    auto publish = [&]() {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int q = t + k * T;
            if (cc[k] == 0.0f) continue;
            if (GRID) {
                if (q < ngy || q + ngy >= per) st_word(d.pcg_edge + lo + q, tagged(tag + 1, __float_as_uint(r[k])));
            } else {
                if (q < ngy || q + ngy >= per) rs[q] = r[k];
            }
        }
    };
    // residuals of the halo nodes (after that sum)
    auto halo_r = [&](int q) -> float {
        if constexpr (GRID) {
            unsigned u = 0;
            if (!poll_word(hw[q], tag, polls, u)) sh.gave_up = 1;
            return __uint_as_float(u);
        } else {
            const int e = t + q * T;
            return e < ngy ? *cl.map_shared_rank(rs + per - ngy + e, rank - 1)
                           : *cl.map_shared_rank(rs + e - ngy, rank + 1);
        }
    };
    // p_0 = D^-1 r_0, own nodes and halo
    auto first_dir = [&]() {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int q = t + k * T;
            p[k] = iv[k] * r[k];
            if (q < per) ps[ngy + q] = p[k];
        }
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (hiv[q] != 0.0f) ps[hp_at[q]] = hiv[q] * halo_r(q);
        __syncthreads();
    };
    // one CG iteration up to the new residual's r'z
    auto iterate = [&](double rz) -> double {
        double part = 0.0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int q = t + k * T;
            float out = 0.0f;
            if (q < per) {
                const float *c = ps + ngy + q;
                // CSR order W, S, C, N, E; a neighbour off the unknowns is skipped
                if (cw[k] != 0.0f) out += cw[k] * c[-ngy];
                if (cs[k] != 0.0f) out += cs[k] * c[-1];
                out += cc[k] * p[k];
                if (cn[k] != 0.0f) out += cn[k] * c[1];
                if (ce[k] != 0.0f) out += ce[k] * c[ngy];
            }
            ap[k] = out;
            if (cc[k] != 0.0f) part += (double)(p[k] * out);
        }
        const double pap = sum(part);
        const float alpha = (pap != 0.0) ? (mode == 0 ? (float)rz / (float)pap : (float)(rz / pap)) : 0.0f;
        part = 0.0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (cc[k] == 0.0f) continue;
            r[k] = -alpha * ap[k] + r[k];
            part += (double)(r[k] * (iv[k] * r[k]));
        }
        publish();
        sum_send(part);
#pragma unroll
        for (int k = 0; k < K; k++)
            if (cc[k] != 0.0f) x[k] = alpha * p[k] + x[k];
        return sum_take();
    };
    // p = beta p + D^-1 r, own nodes and halo
    auto next_dir = [&](float beta) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int q = t + k * T;
            if (cc[k] != 0.0f) {
                p[k] = beta * p[k] + iv[k] * r[k];
                ps[ngy + q] = p[k];
            }
        }
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (hiv[q] != 0.0f) ps[hp_at[q]] = beta * ps[hp_at[q]] + hiv[q] * halo_r(q);
        __syncthreads();
    };
    // no remote write into a CTA that has not started
    if (!GRID) cl.sync();

    const int maxit = d.pcg_max_iter;
    int iters = 0, outer = 0;
    bool bad = false;
    if (mode == 0) {
        const float *xg = d.pf_x;
        double part = 0.0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (cc[k] == 0.0f) continue;
            const int n = lo + t + k * T;
            const float ax = spmv_f(st, G, ngy, n, xg);
            const float rr = -1.0f * ax + (float)d.b64[n];
            x[k] = xg[n];
            r[k] = rr;
            part += (double)(rr * (iv[k] * rr));
        }
        publish();
        double rz = sum(part);
        // a non-finite right-hand side or warm start: the reference's loop
        // test (r'z > tol^2) is false for NaN and leaves x as it was
        if (!(rz == rz) || isinf(rz)) bad = true;
        first_dir();
        int iter = 1;
        while (rz > (double)d.pcg_tol2 && iter <= maxit && !gave_up) {
            const double rznew = iterate(rz);
            if (!(rznew == rznew) || isinf(rznew)) { bad = true; break; }
            const float beta = (rz != 0.0) ? (float)rznew / (float)rz : 0.0f;
            next_dir(beta);
            rz = rznew;
            iter++;
        }
        iters = iter;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int n = lo + t + k * T;
            if (n >= hi) continue;
            if (cc[k] != 0.0f) d.pf_x[n] = x[k];
            d.phi_p[n] = cc[k] != 0.0f ? x[k] : 0.0f;
        }
        if (iter > maxit && rank == 0 && t == 0) atomicOr(d.status, ST_NOCONV);
    } else {
        double *x64 = d.x64;
        const double *__restrict__ b64 = d.b64;
        double bb = 0.0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int n = lo + t + k * T;
            if (n < hi) bb += b64[n] * b64[n];
        }
        bb = sum(bb);
        const double target = d.pcg_rtol * d.pcg_rtol * bb;
        const double inner_rel2 = 1e-10; // inner solve: 1e-5 reduction of the preconditioned residual norm
        for (outer = 0; outer < 12; outer++) {
            double rr = 0.0, rz = 0.0;
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (cc[k] == 0.0f) continue;
                const int n = lo + t + k * T;
                const double r64 = b64[n] - spmv_d(st, G, ngy, n, x64);
                rr += r64 * r64;
                const float v = (float)(r64 * (double)d.row_scale[n]);
                r[k] = v;
                x[k] = 0.0f;
                rz += (double)(v * (iv[k] * v));
            }
            rr = sum(rr);
            publish();
            rz = sum(rz);
            if (gave_up) break;
            if (!(rr == rr) || isinf(rr)) { bad = true; break; }
            if (rr <= target || bb == 0.0) break;
            first_dir();
            const double rz0 = rz;
            int iter = 0;
            while (rz > inner_rel2 * rz0 && iter < maxit && !gave_up) {
                const double rznew = iterate(rz);
                if (!(rznew == rznew) || isinf(rznew)) { bad = true; break; }
                const float beta = (rz != 0.0) ? (float)(rznew / rz) : 0.0f;
                next_dir(beta);
                rz = rznew;
                iter++;
            }
            iters += iter;
            if (bad || gave_up) break;
#pragma unroll
            for (int k = 0; k < K; k++)
                if (cc[k] != 0.0f) x64[lo + t + k * T] += (double)x[k];
            if (GRID) sum(0.0, true);
            else cl.sync();
        }
        if (outer >= 12 && rank == 0 && t == 0) atomicOr(d.status, ST_NOCONV);
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int n = lo + t + k * T;
            if (n < hi) d.phi_p[n] = cc[k] != 0.0f ? (float)x64[n] : 0.0f;
        }
    }
    if (rank == 0 && t == 0) {
        d.pcg_iters[0] = iters;
        d.pcg_iters[1] = outer;
        if (bad) atomicOr(d.status, ST_NONFINITE);
        if (GRID) *d.pcg_seq = tag; // every CTA read it before its first exchange
    }
    if (GRID && gave_up && t == 0) atomicOr(d.status, ST_TIMEOUT);
    // no CTA may leave while another can still read its shared memory
    if (!GRID) cl.sync();
}

// The forms: 1, 2 and 4 nodes per thread; 5, which is what a grid of 2^a + 1
// by 2^b + 1 nodes comes to (65x33, 129x65 and 257x129 nodes: 1, 4 and 16 CTAs
// of 2,073 to 2,145 nodes at 512 threads, where 4 would miss by a few); and 8,
// the most that 128 registers hold at 512 threads (it spills 56 bytes, 88 on the
// whole GPU, the others up to 8).  A CTA of 6 or 7 nodes per thread runs the form
// for 8.  Forms of their own would take, us per iteration at 6 and 7 nodes: one
// CTA 4.1 and 5.9 against 6.2 and 6.7, a cluster of 16 5.7 and 7.5 against 7.9
// and 8.3 (k_pcg takes about 12), for 1.9 MB of code; they are not built.
struct Variant {
    int k;
    const void *cluster, *grid;
};
const Variant VARIANTS[] = {
    {1, (const void *)k_pcg_chip<false, 1>, (const void *)k_pcg_chip<true, 1>},
    {2, (const void *)k_pcg_chip<false, 2>, (const void *)k_pcg_chip<true, 2>},
    {4, (const void *)k_pcg_chip<false, 4>, (const void *)k_pcg_chip<true, 4>},
    {5, (const void *)k_pcg_chip<false, 5>, (const void *)k_pcg_chip<true, 5>},
    {8, (const void *)k_pcg_chip<false, 8>, (const void *)k_pcg_chip<true, 8>},
};

} // namespace

// The on-chip form takes a group whose CTAs own at most 8 nodes per thread
// (128 registers at 512 threads) and whose halo is at most two nodes per
// thread; a launch shape with fewer, wider CTAs than that (hp_tune) keeps
// k_pcg.  The halo rule holds for a group as a whole: a grid of more rows than
// threads per CTA (513x257 nodes with hp_tune.pcg_block 128 or 256) takes
// k_pcg, and with it its whole group (263x251 nodes: 18 us per iteration at 192
// threads, 24 at 128).
// Shared memory stays below 48 KB: 4 x (2 x 4096 + 2 x 512) bytes.
cudaError_t launch_pcg_chip(const DevCase *cases, const PcgGroup &pg, cudaStream_t st, bool &done, int polls) {
    done = false;
    const bool grid = pg.cluster > 16;
    // several CTAs own more than 1000 nodes each, so a halo reaches no further than the CTAs next to its own
    if (pg.max_ngy > pg.block) return cudaSuccess;
    const Variant *v = nullptr;
    for (const Variant &w : VARIANTS)
        if (!v && (long long)w.k * pg.block >= pg.max_per) v = &w;
    if (!v) return cudaSuccess;
    const void *fn = grid ? v->grid : v->cluster;
    const size_t smem = sizeof(float) * (size_t)(pg.max_per + 2 * pg.max_ngy + (grid ? 0 : pg.max_per));
    if (grid) { // every CTA has to be resident
        int dev = 0, sms = 0, per_sm = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, pg.block, smem);
        if (e != cudaSuccess) return e;
        if (pg.cluster > GRID_MAX || (long long)sms * per_sm < pg.cluster) return cudaSuccess;
    } else {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    for (int k = 0; k < (grid ? pg.n : 1); k++) { // the whole-GPU form: one case per launch
        const int *list = pg.list + k;
        int nlist = grid ? 1 : pg.n, per = pg.max_per, ngy = pg.max_ngy;
        void *args[] = {(void *)&cases, (void *)&list, (void *)&nlist, (void *)&per, (void *)&ngy, (void *)&polls};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(grid ? pg.cluster : pg.n * pg.cluster), 1, 1);
        cfg.blockDim = dim3((unsigned)pg.block, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        if (grid) {
            attr[0].id = cudaLaunchAttributeCooperative;
            attr[0].val.cooperative = 1;
        } else {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)pg.cluster;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
        }
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; // as launch_next
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = grid || prof::g_on ? 1 : 2;
        prof::mark(st, grid ? "k_pcg_grid" : "k_pcg");
        cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
        if (e != cudaSuccess) return e;
    }
    done = true;
    return cudaSuccess;
}

} // namespace hp
