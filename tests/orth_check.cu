// The GMRES orthogonalisation kernel by itself, and its grid barrier with an
// arrival too few.
#include <algorithm>
#include <cstring>
#include <vector>

#include "../rhodst_b200/csrc/linalg.cuh"

using namespace rdst;

namespace {

template <typename VT>
int orth(long n, int m, int split, const double* W, double* out) {
    const long ldv = (n + 63) / 64 * 64;
    int nbv = red_blocks(n), sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
    if (split && nbv > sms) return -1;
    const int nb = split ? nbv : std::min(sms, (nbv + 1) / 2);
    VT* V = nullptr;
    double *w = nullptr, *part = nullptr;
    Scalars* sc = nullptr;
    cudaMalloc(&V, sizeof(VT) * ldv * (m + 1));
    cudaMalloc(&w, sizeof(double) * ldv);
    cudaMalloc(&part, sizeof(double) * (2 * m + 1) * nbv);
    cudaMalloc(&sc, sizeof(Scalars));
    cudaMemset(V, 0, sizeof(VT) * ldv * (m + 1));
    cudaMemset(w, 0, sizeof(double) * ldv);
    cudaMemset(sc, 0, sizeof(Scalars));
    unsigned wait_ms = 2000;
    for (int i = 0; i <= m; ++i) {
        // the FP64 basis is built in place, as the solver does it
        double* wi = sizeof(VT) == 8 ? reinterpret_cast<double*>(V + i * ldv) : w;
        cudaMemcpy(wi, W + i * n, sizeof(double) * n, cudaMemcpyHostToDevice);
        const VT* Vc = V;
        VT* vout = V + i * ldv;
        void* args[] = {&n, &i, &Vc, (void*)&ldv, &wi, &vout, &part, &sc, &m, &nbv, &wait_ms};
        auto* k = split ? k_orth_cgs2<VT, true> : k_orth_cgs2<VT, false>;
        cudaLaunchCooperativeKernel((const void*)k, dim3(nb), dim3(ORTH_TPB), args, 0, 0);
    }
    std::vector<VT> v(ldv * (m + 1));
    Scalars s;
    cudaMemcpy(v.data(), V, sizeof(VT) * v.size(), cudaMemcpyDeviceToHost);
    cudaMemcpy(&s, sc, sizeof(Scalars), cudaMemcpyDeviceToHost);
    for (int i = 0; i <= m; ++i)
        for (long k = 0; k < n; ++k) out[i * n + k] = v[i * ldv + k];
    int bad = s.flags != 0 || s.orth_bar != 0 || s.orth_out != 0 || s.gm_used != m;
    for (int i = 0; i <= m; ++i)            // the padding is still zero
        for (long k = n; k < ldv; ++k) bad |= v[i * ldv + k] != VT(0);
    cudaFree(V);
    cudaFree(w);
    cudaFree(part);
    cudaFree(sc);
    return cudaGetLastError() != cudaSuccess ? -2 : bad;
}

__global__ void k_lonely(Scalars* sc, unsigned wait_ms, int* passed) {
    if (grid_barrier(sc, 2, wait_ms) && threadIdx.x == 0) atomicAdd(passed, 1);
}

}  // namespace

// vectors W_0 .. W_m (n entries each) one after the other; out: the basis
extern "C" int orth_run(long n, int m, int fp32, int split, const double* W, double* out) {
    return fp32 ? orth<float>(n, m, split, W, out) : orth<double>(n, m, split, W, out);
}

// four blocks arrive once each at a barrier of eight: flags and, in out, blocks
// that passed, what is left of the solve, ms
extern "C" int lonely_run(unsigned wait_ms, double* out) {
    Scalars s;
    memset(&s, 0, sizeof(s));
    s.gm_active = s.gm_used = s.bi_active = 1;
    Scalars* sc = nullptr;
    int *d = nullptr, passed = 0;
    cudaMalloc(&sc, sizeof(Scalars));
    cudaMalloc(&d, sizeof(int));
    cudaMemcpy(sc, &s, sizeof(s), cudaMemcpyHostToDevice);
    cudaMemset(d, 0, sizeof(int));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0);
    k_lonely<<<4, 64>>>(sc, wait_ms, d);
    cudaEventRecord(e1);
    cudaMemcpy(&s, sc, sizeof(s), cudaMemcpyDeviceToHost);
    cudaMemcpy(&passed, d, sizeof(int), cudaMemcpyDeviceToHost);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    out[0] = passed;
    out[1] = s.gm_active + s.gm_used + s.bi_active + !s.converged;
    out[2] = ms;
    cudaFree(sc);
    cudaFree(d);
    return cudaGetLastError() != cudaSuccess ? -2 : s.flags;
}
