// Conjugate-gradient Poisson solve: the 'cg' and 'gmres' branches of the
// reference's Solver (src/Solvers.py:245-258, cupyx.scipy.sparse.linalg cg
// and gmres on the 5-point Laplacian with Dirichlet rows).  The system is
// symmetric, so conjugate gradients reach the solution GMRES would.
//
// lap(phi) = f on the free nodes, phi fixed on the Dirichlet nodes (the grid
// edges and the mask): with x = phi - phi_0 (zero on Dirichlet nodes), L x = r_0.
// Flexible preconditioned CG (Polak-Ribiere beta, which tolerates a
// preconditioner that is not exactly symmetric), preconditioned by one
// multigrid V-cycle from zero when a pic_mg is given.  Everything in FP64.
//
// The scalars (beta, alpha, the norms, the iteration count and the decision to
// stop) stay on the device: each kernel's last block to finish adds the block
// partials in a fixed order and derives what the next kernel needs, so an
// iteration is three launches besides the V-cycle's and one host round trip
// (three before; 385 x 257 to 1e-9: the call 855 -> 426 us).  With a
// preconditioner the host waits for the decision before it enqueues an iteration:
// one ahead of it is a V-cycle too many per solve, which costs what the waits of
// four iterations do at 65^2 and more on larger grids (513^2: 359 us ahead, 331
// waiting; from the converged potential 137 and 49).  Without one the host runs one
// iteration ahead, whose three kernels do nothing past the end.
#include <cmath>
#include <utility>
#include <vector>

#include "common.cuh"

namespace pic {

int mg_launch_graph(pic_mg* mg, double* phi, const double* f, double tol, int max_cycles, int min_cycles,
                    cudaStream_t st);
bool mg_is_rz(pic_mg* mg);

constexpr int kCgThreads = 256;

// The solve's scalars on the device.
struct CgState {
    double f2, r2;         // ||f||^2, ||r||^2
    double lim;            // tol^2 ||f||^2: converged below it
    double rz, alpha, beta;
    int it;                // iterations done
    int stop;              // converged, at the limit, or broken down
    unsigned done;         // blocks of the running kernel that have finished
};

struct CgImpl {
    int nx = 0, ny = 0;
    long G = 0;
    double cx = 0, cy = 0;
    uint8_t* free_ = nullptr;  // 1 = unknown
    pic_mg* mg = nullptr;
    double *r = nullptr, *r_prev = nullptr, *z = nullptr, *p = nullptr, *p2 = nullptr, *q = nullptr, *x = nullptr;
    double* part = nullptr;  // [2][blocks]
    CgState* state = nullptr;
    CgState* h_state = nullptr;  // page-locked: the state after each of the last two iterations
    cudaEvent_t ev[2] = {nullptr, nullptr};
    int blocks = 0;
    std::vector<void*> allocs;
};

__device__ __forceinline__ double lap_at(const double* __restrict__ v, long k, int nx, double cx, double cy) {
    const double c = v[k];
    return cx * ((v[k - 1] - c) + (v[k + 1] - c)) + cy * ((v[k - nx] - c) + (v[k + nx] - c));
}

// Sums a and b over the grid: true in thread 0 of the last block to finish,
// with the block partials added in a fixed order.
__device__ bool cg_sum(double& a, double& b, double* part, CgState* S) {
    __shared__ double ws[2][kCgThreads / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nb = gridDim.x;
    auto block = [&]() {
        a = warp_sum(a);
        b = warp_sum(b);
        __syncthreads();
        if (lane == 0) {
            ws[0][w] = a;
            ws[1][w] = b;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            a = b = 0.0;
            for (int k = 0; k < kCgThreads / 32; ++k) {
                a += ws[0][k];
                b += ws[1][k];
            }
        }
    };
    block();
    if (threadIdx.x == 0) {
        part[blockIdx.x] = a;
        part[nb + blockIdx.x] = b;
        __threadfence();
        last = atomicAdd(&S->done, 1u) == unsigned(nb - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    a = b = 0.0;
    const volatile double* P = part;
    for (int k = threadIdx.x; k < nb; k += kCgThreads) {
        a += P[k];
        b += P[nb + k];
    }
    block();
    if (threadIdx.x != 0) return false;
    S->done = 0u;
    return true;
}

__device__ __forceinline__ bool cg_stopped(const CgState* S) { return *reinterpret_cast<const volatile int*>(&S->stop); }

// r = f - lap(phi) on free nodes, 0 elsewhere; x = 0 (and z = 0); the norms
// and the first decision.
__global__ void __launch_bounds__(kCgThreads) k_cg_init(const double* __restrict__ phi, const double* __restrict__ f,
                                                        const uint8_t* __restrict__ fr, int nx, long G, double cx,
                                                        double cy, double* __restrict__ r, double* __restrict__ x,
                                                        double* __restrict__ z, double tol, double* __restrict__ part,
                                                        CgState* S) {
    double f2 = 0.0, r2 = 0.0;
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < G; k += long(gridDim.x) * blockDim.x) {
        double v = 0.0;
        if (fr[k]) {
            const double fv = f[k];
            v = fv - lap_at(phi, k, nx, cx, cy);
            f2 += fv * fv;
        }
        r[k] = v;
        x[k] = 0.0;
        if (z) z[k] = 0.0;
        r2 += v * v;
    }
    if (!cg_sum(f2, r2, part, S)) return;
    S->f2 = f2;
    S->r2 = r2;
    S->lim = tol * tol * (f2 > 0.0 ? f2 : 1.0);
    S->rz = 0.0;
    S->it = 0;
    S->stop = r2 < S->lim;
}

// Polak-Ribiere: beta = z.(r - r_prev) / (z_prev . r_prev), 0 in the first iteration.
__global__ void __launch_bounds__(kCgThreads) k_cg_beta(const double* __restrict__ r, const double* __restrict__ r_prev,
                                                        const double* __restrict__ z, const uint8_t* __restrict__ fr,
                                                        long G, double* __restrict__ part, CgState* S) {
    if (cg_stopped(S)) return;
    const int it = S->it;
    double rz = 0.0, rpz = 0.0;
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < G; k += long(gridDim.x) * blockDim.x) {
        if (!fr[k]) continue;
        const double v = z[k];
        rz += r[k] * v;
        if (it > 0) rpz += r_prev[k] * v;
    }
    if (!cg_sum(rz, rpz, part, S)) return;
    S->beta = it > 0 && S->rz != 0.0 ? (rz - rpz) / S->rz : 0.0;
    S->rz = rz;
}

// p2 = z + beta p on free nodes (0 elsewhere) and q = lap(p2), each node
// forming its neighbours' p2 itself, and alpha = r.z / p2.q.
__global__ void __launch_bounds__(kCgThreads) k_cg_apply(const double* __restrict__ z, const double* __restrict__ p,
                                                         const uint8_t* __restrict__ fr, int nx, long G, double cx,
                                                         double cy, double* __restrict__ p2, double* __restrict__ q,
                                                         double* __restrict__ part, CgState* S) {
    if (cg_stopped(S)) return;
    const double beta = S->beta;
    auto dir = [&](long k) { return !fr[k] ? 0.0 : beta != 0.0 ? z[k] + beta * p[k] : z[k]; };
    double pq = 0.0, none = 0.0;
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < G; k += long(gridDim.x) * blockDim.x) {
        double v = 0.0, l = 0.0;
        if (fr[k]) {
            v = dir(k);
            l = cx * ((dir(k - 1) - v) + (dir(k + 1) - v)) + cy * ((dir(k - nx) - v) + (dir(k + nx) - v));
            pq += v * l;
        }
        p2[k] = v;
        q[k] = l;
    }
    if (!cg_sum(pq, none, part, S)) return;
    if (pq == 0.0 || !isfinite(pq)) S->stop = 1;  // broken down
    else S->alpha = S->rz / pq;
}

// x += alpha p; r_prev = r; r -= alpha q; z = 0 (before the next V-cycle);
// ||r||^2 and the decision.
__global__ void __launch_bounds__(kCgThreads) k_cg_update(double* __restrict__ x, double* __restrict__ r,
                                                          double* __restrict__ r_prev, double* __restrict__ z,
                                                          const double* __restrict__ p, const double* __restrict__ q,
                                                          const uint8_t* __restrict__ fr, long G, int max_iter,
                                                          double* __restrict__ part, CgState* S) {
    if (cg_stopped(S)) return;
    const double alpha = S->alpha;
    double r2 = 0.0, none = 0.0;
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < G; k += long(gridDim.x) * blockDim.x) {
        const double old = r[k], v = old - alpha * q[k];
        x[k] += alpha * p[k];
        r_prev[k] = old;
        r[k] = v;
        if (z) z[k] = 0.0;
        if (fr[k]) r2 += v * v;
    }
    if (!cg_sum(r2, none, part, S)) return;
    const int it = S->it + 1;
    S->it = it;
    S->r2 = r2;
    S->stop = r2 < S->lim || it >= max_iter;
}

__global__ void k_cg_finish(double* __restrict__ phi, const double* __restrict__ x, const uint8_t* __restrict__ fr,
                            long G) {
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < G; k += long(gridDim.x) * blockDim.x)
        if (fr[k]) phi[k] += x[k];
}

int grid_blocks(long n, int threads);

static void cg_release(CgImpl& C) {
    for (void* a : C.allocs) cudaFree(a);
    C.allocs.clear();
    if (C.h_state) cudaFreeHost(C.h_state);
    C.h_state = nullptr;
    for (cudaEvent_t& e : C.ev) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
}

}  // namespace pic

struct pic_cg {
    pic::CgImpl c;
};

using namespace pic;

extern "C" {

int pic_cg_create(int nx, int ny, double dx, double dy, const uint8_t* h_dirichlet, pic_mg* precond, pic_cg** out) {
    clear_error();
    if (!out || !h_dirichlet || nx < 3 || ny < 3 || !(dx > 0) || !(dy > 0))
        return fail(PIC_ERR_BAD_ARG, "pic_cg_create: bad arguments");
    if (precond && mg_is_rz(precond))
        return fail(PIC_ERR_BAD_ARG, "pic_cg_create: the conjugate-gradient solve is Cartesian");
    pic_cg* h = new pic_cg;
    CgImpl& C = h->c;
    C.nx = nx;
    C.ny = ny;
    C.G = long(nx) * ny;
    C.cx = 1.0 / (dx * dx);
    C.cy = 1.0 / (dy * dy);
    C.mg = precond;
    C.blocks = 2 * num_sms();
    std::vector<uint8_t> fr(size_t(C.G));
    for (int j = 0; j < ny; ++j)
        for (int i = 0; i < nx; ++i) {
            const size_t k = size_t(j) * nx + i;
            fr[k] = (i > 0 && j > 0 && i < nx - 1 && j < ny - 1 && !h_dirichlet[k]) ? 1 : 0;
        }
    auto alloc = [&](void** p, size_t bytes) {
        if (cudaMalloc(p, bytes) != cudaSuccess) return false;
        C.allocs.push_back(*p);
        return cudaMemset(*p, 0, bytes) == cudaSuccess;
    };
    const size_t vb = sizeof(double) * size_t(C.G);
    bool ok = alloc(reinterpret_cast<void**>(&C.free_), size_t(C.G)) &&
              cudaMemcpy(C.free_, fr.data(), size_t(C.G), cudaMemcpyHostToDevice) == cudaSuccess;
    for (double** v : {&C.r, &C.r_prev, &C.z, &C.p, &C.p2, &C.q, &C.x})
        ok = ok && alloc(reinterpret_cast<void**>(v), vb);
    ok = ok && alloc(reinterpret_cast<void**>(&C.part), sizeof(double) * 2 * size_t(C.blocks)) &&
         alloc(reinterpret_cast<void**>(&C.state), sizeof(CgState)) &&
         cudaMallocHost(reinterpret_cast<void**>(&C.h_state), 2 * sizeof(CgState)) == cudaSuccess;
    for (cudaEvent_t& e : C.ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cg_release(C);
        delete h;
        return fail(PIC_ERR_CUDA, "pic_cg_create: out of device memory");
    }
    *out = h;
    return PIC_OK;
}

int pic_cg_destroy(pic_cg* h) {
    clear_error();
    if (!h) return PIC_OK;
    cudaDeviceSynchronize();
    cg_release(h->c);
    delete h;
    return PIC_OK;
}

int pic_cg_solve(pic_cg* h, double* d_phi, const double* d_f, double tol, int max_iter, pic_mg_info* info,
                 void* stream) {
    clear_error();
    if (!h || !d_phi || !d_f || !(tol > 0) || max_iter < 1) return fail(PIC_ERR_BAD_ARG, "pic_cg_solve: bad arguments");
    CgImpl& C = h->c;
    cudaStream_t st = as_stream(stream);
    const int B = C.blocks;
    double* z = C.mg ? C.z : nullptr;  // without a preconditioner z = r
    // a solve that ended early (an error return) may have left the block count of its last kernel
    PIC_CUDA(cudaMemsetAsync(C.state, 0, sizeof(CgState), st));
    k_cg_init<<<B, kCgThreads, 0, st>>>(d_phi, d_f, C.free_, C.nx, C.G, C.cx, C.cy, C.r, C.x, z, tol, C.part, C.state);
    PIC_LAUNCH_CHECK();
    // the state after the newest launches, on its way to the host, and whether it says stop
    int slot = 0;
    auto post = [&]() -> int {
        slot ^= 1;
        PIC_CUDA(cudaMemcpyAsync(C.h_state + slot, C.state, sizeof(CgState), cudaMemcpyDeviceToHost, st));
        PIC_CUDA(cudaEventRecord(C.ev[slot], st));
        return PIC_OK;
    };
    auto wait = [&](int s, bool& stop) -> int {
        PIC_CUDA(cudaEventSynchronize(C.ev[s]));
        stop = C.h_state[s].stop != 0;
        return PIC_OK;
    };
    PIC_TRY(post());
    for (int it = 0; it < max_iter; ++it) {
        bool stop = false;
        if (C.mg || it == 0) PIC_TRY(wait(slot, stop));
        if (stop) break;
        if (C.mg) PIC_TRY(mg_launch_graph(C.mg, C.z, C.r, 1e-300, 1, 1, st));
        const double* zz = C.mg ? C.z : C.r;
        k_cg_beta<<<B, kCgThreads, 0, st>>>(C.r, C.r_prev, zz, C.free_, C.G, C.part, C.state);
        k_cg_apply<<<B, kCgThreads, 0, st>>>(zz, C.p, C.free_, C.nx, C.G, C.cx, C.cy, C.p2, C.q, C.part, C.state);
        k_cg_update<<<B, kCgThreads, 0, st>>>(C.x, C.r, C.r_prev, z, C.p2, C.q, C.free_, C.G, max_iter, C.part,
                                              C.state);
        std::swap(C.p, C.p2);
        PIC_LAUNCH_CHECK();
        PIC_TRY(post());
        // without a preconditioner, the iteration before this one decides whether there is another
        if (!C.mg && it > 0) PIC_TRY(wait(slot ^ 1, stop));
        if (stop) break;
    }
    k_cg_finish<<<grid_blocks(C.G, kCgThreads), kCgThreads, 0, st>>>(d_phi, C.x, C.free_, C.G);
    PIC_LAUNCH_CHECK();
    PIC_TRY(post());
    PIC_CUDA(cudaStreamSynchronize(st));
    const CgState& S = C.h_state[slot];
    pic_mg_info loc{};
    const double ref = S.f2 > 0.0 ? S.f2 : 1.0;
    loc.cycles = S.it;
    loc.rhs_norm = std::sqrt(S.f2);
    loc.rel_res = std::sqrt(S.r2 / ref);
    loc.converged = S.r2 < tol * tol * ref ? 1 : 0;
    if (info) *info = loc;
    if (!loc.converged)
        return fail(PIC_ERR_NOT_CONVERGED, "pic_cg_solve: relative residual %.3e after %d iterations (tol %.1e)",
                    loc.rel_res, S.it, tol);
    return PIC_OK;
}

}  // extern "C"
