// pcg_words.cu -- the whole-GPU solve of csrc/pcg.cu after a solve whose waits gave up.
//
// One case of 205 x 100 nodes (a 5-point operator, 20 CTAs) is solved twice, for two right-hand sides.  Then the same
// on fresh memory with a solve in between that may not poll at all: every wait of it gives up, it has to return and to
// set its status.  Then the words that a CTA ahead of the others can leave behind such a solve are put where it would
// have put them: sums and edge residuals under the next three exchange numbers.  The solve that follows must not take
// them for its own: same bits, same iterations.  Prints one line per field mode.
#include <cstdio>
#include <cstring>
#include <vector>

#include "pcg.cu"

using namespace hp;

constexpr int NX = 205, NY = 100, G = NX * NY, CTAS = 20, BLOCK = 512;

template <class T> T *device(const std::vector<T> &v) {
    T *p = nullptr;
    cudaMalloc(&p, v.size() * sizeof(T));
    cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
    return p;
}
template <class T> std::vector<T> host(const T *p, size_t n) {
    std::vector<T> v(n);
    cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost);
    return v;
}

struct Case {
    DevCase h;
    DevCase *d;
    int *list;
    double *b;
    int polls = 1 << 22;
    explicit Case(int mode) {
        std::memset(&h, 0, sizeof h);
        std::vector<float> st(5 * (size_t)G, 0.0f), one(G, 1.0f);
        auto unknown = [](int i, int j) { return i > 0 && j > 0 && i + 1 < NX && j + 1 < NY; };
        for (int i = 0; i < NX; i++)
            for (int j = 0; j < NY; j++) {
                if (!unknown(i, j)) continue;
                const int n = i * NY + j;
                st[0 * G + n] = unknown(i - 1, j) ? -1.0f : 0.0f;
                st[1 * G + n] = unknown(i, j - 1) ? -1.0f : 0.0f;
                st[2 * G + n] = 4.0f + 0.01f * (float)(n % 7);
                st[3 * G + n] = unknown(i, j + 1) ? -1.0f : 0.0f;
                st[4 * G + n] = unknown(i + 1, j) ? -1.0f : 0.0f;
            }
        h.G = G;
        h.ngx = NX;
        h.ngy = NY;
        h.field_mode = mode;
        h.st = h.st_sym = device(st);
        h.row_scale = device(one);
        h.pf_x = device(std::vector<float>(G, 0.0f));
        h.phi_p = device(std::vector<float>(G, 0.0f));
        h.x64 = device(std::vector<double>(G, 0.0));
        h.b64 = b = device(std::vector<double>(G, 0.0));
        h.pcg_max_iter = 2000;
        h.pcg_tol2 = 1e-8f;
        h.pcg_rtol = 1e-8;
        h.status = device(std::vector<uint32_t>(1, 0));
        h.pcg_iters = device(std::vector<int>(2, 0));
        h.pcg_slot = device(std::vector<unsigned long long>(4 * CTAS * CTAS, 0));
        h.pcg_edge = device(std::vector<unsigned long long>(G, 0));
        h.pcg_seq = device(std::vector<unsigned>(1, 0));
        d = device(std::vector<DevCase>(1, h));
        list = device(std::vector<int>(1, 0));
    }
    bool solve(int which) {
        std::vector<double> r(G, 0.0);
        for (int i = 1; i + 1 < NX; i++)
            for (int j = 1; j + 1 < NY; j++) r[i * NY + j] = (double)((i * 31 + j * 17 + which * 7) % 13) - 6.0;
        cudaMemcpy(b, r.data(), G * sizeof(double), cudaMemcpyHostToDevice);
        const PcgGroup pg{CTAS, BLOCK, list, 1, (G + CTAS - 1) / CTAS, NY};
        bool done = false;
        return launch_pcg_chip(d, pg, 0, done, polls) == cudaSuccess && done && cudaDeviceSynchronize() == cudaSuccess;
    }
};

int main() {
    for (int mode = 0; mode < 2; mode++) {
        Case a(mode), c(mode);
        bool ran = a.solve(1) && a.solve(2) && c.solve(1);
        c.polls = 0;
        ran = ran && c.solve(2);
        const uint32_t status = host(c.h.status, 1)[0];
        cudaMemset(c.h.status, 0, sizeof(uint32_t));
        const unsigned last = host(c.h.pcg_seq, 1)[0];
        auto slot = host(c.h.pcg_slot, 4 * CTAS * CTAS);
        auto edge = host(c.h.pcg_edge, G);
        for (unsigned tag = last + 1; tag <= last + 3; tag++) {
            unsigned long long *in = slot.data() + (size_t)(tag & 1u) * 2 * CTAS * CTAS;
            for (int q = 0; q < 2 * CTAS * CTAS; q++) in[q] = ((unsigned long long)tag << 32) | 0x40100000u;
        }
        for (int q = 0; q < G; q++) edge[q] = ((unsigned long long)(last + 1 + q % 3) << 32) | 0x3f800000u;
        cudaMemcpy(c.h.pcg_slot, slot.data(), slot.size() * 8, cudaMemcpyHostToDevice);
        cudaMemcpy(c.h.pcg_edge, edge.data(), edge.size() * 8, cudaMemcpyHostToDevice);
        c.polls = a.polls;
        ran = ran && c.solve(2);
        const auto x = host(a.h.phi_p, G), y = host(c.h.phi_p, G);
        const auto i = host(a.h.pcg_iters, 2), k = host(c.h.pcg_iters, 2);
        int nonzero = 0;
        for (float v : x) nonzero += v != 0.0f;
        std::printf("mode %d ran %d gave_up %d same %d iterations %d %d nonzero %d status %u %u\n", mode, (int)ran,
                    (int)((status & dv::ST_TIMEOUT) != 0), (int)(std::memcmp(x.data(), y.data(), G * 4) == 0), i[0], k[0],
                    (int)(nonzero == (NX - 2) * (NY - 2)), host(a.h.status, 1)[0], host(c.h.status, 1)[0]);
    }
}
