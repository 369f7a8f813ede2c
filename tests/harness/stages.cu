// Entry points for the tests: stages of a batch that the C ABI does not expose by themselves, on device buffers of the
// caller, linked against the built libgpt.so.
#include "gpt_common.cuh"
#include "gpt_internal.h"

#include <vector>

using namespace gpt;

namespace {

// a view of instances b0 .. b0 + B - 1 of a batch with the given knot offsets, per-instance activity and rho
struct View {
    BatchView bv = {};
    int *off = nullptr, *inst = nullptr;
    InstState *st = nullptr;
    cudaError_t err = cudaSuccess;
    View(int batch, const int *h_off, const unsigned char *h_active, float rho, int b0, int B)
    {
        std::vector<int> own(h_off[batch]);
        std::vector<InstState> s(batch);
        for (int b = 0; b < batch; ++b) {
            for (int k = h_off[b]; k < h_off[b + 1]; ++k) own[k] = b;
            s[b] = InstState{};
            s[b].rho = rho;
            s[b].active = h_active[b];
        }
        put(off, h_off, batch + 1);
        put(inst, own.data(), own.size());
        put(st, s.data(), batch);
        bv.B = B;
        bv.b0 = b0;
        bv.j0 = h_off[b0];
        bv.total_knots = h_off[b0 + B] - h_off[b0];
        bv.knot_off = off;
        bv.knot_inst = inst;
        bv.st = st;
    }
    template <class T> void put(T *&d, const T *h, size_t n)
    {
        if (err == cudaSuccess) err = cudaMalloc((void **)&d, n * sizeof(T));
        if (err == cudaSuccess) err = cudaMemcpy(d, h, n * sizeof(T), cudaMemcpyHostToDevice);
    }
    int done(cudaError_t e)
    {
        const cudaError_t w = cudaDeviceSynchronize();
        return (int)(err != cudaSuccess ? err : e != cudaSuccess ? e : w);
    }
    ~View()
    {
        cudaFree(off);
        cudaFree(inst);
        cudaFree(st);
    }
};

int sms()
{
    int d = 0, n = 0;
    cudaGetDevice(&d);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d);
    return n;
}

}  // namespace

// KKT formation of the SQP loop (C, g, c) with one knot per lane (lane 1) or by half-warps (0)
extern "C" int stage_kkt(int batch, const int *h_off, const unsigned char *h_active, int b0, int B, int lane, float dt,
                         int integrator, float qd_cost, float r_cost, int ref_terminal, const float *xu,
                         const float *goal, const float *xs, float *C, float *g, float *c)
{
    View v(batch, h_off, h_active, 1e-3f, b0, B);
    if (v.err != cudaSuccess) return (int)v.err;
    v.bv.kkt_lane = lane != 0;
    const ProblemParams P{dt, integrator, 1.f, qd_cost, r_cost, 10.f, ref_terminal};
    return v.done(launch_kkt(v.bv, P, xu, goal, xs, nullptr, C, g, c, sms(), 0, 16, KKT_G_NONE));
}

namespace {
__global__ void rcp_kernel(int n, int order, const double *x, double *r)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        r[i] = order == 3 ? rcp_cubic(x[i]) : rcp_newton(x[i]);
}
}  // namespace

// the kernels' FP64 reciprocals of each x: order 2 by two Newton-Raphson steps, 3 by one third-order step
extern "C" int stage_rcp(int n, int order, const double *x, double *r)
{
    rcp_kernel<<<256, 256>>>(n, order, x, r);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
