// Hand-written adjoint of the collisionless step: CIC deposit -> multigrid
// Poisson solve -> E = -grad(phi) -> kick -> drift with wall absorption, in
// FP64, with gradients of a final-density loss with respect to the potentials
// of electrode segments and to the amplitude of an initial-velocity
// perturbation.
//
// Forward model (the reference's order, src/simulation.py:622-660):
//   init:  rho_0 = D(x_0), phi_0 = P(rho_0; V), E_0 = G phi_0,
//          u_0 = v_0 + A dv - (k/2) I(x_0; E_0)
//   step n = 0 .. N-1:
//          x_{n+1} = x_n + c u_n          (absorbed when outside the grid)
//          rho_{n+1} = D(x_{n+1}), phi_{n+1} = P(rho_{n+1}; V), E_{n+1} = G phi_{n+1}
//          u_{n+1} = u_n + k I(x_{n+1}; E_{n+1})
//   loss:  L = mean over nodes of (n_s(x_N) - n_target)^2 for one species s
// D is the CIC deposit (src/Grid.py:96-154), P the Poisson solve with
// Dirichlet values V on the electrode segments (f = -rho/eps0 on free nodes),
// G the gradient stencil of src/Grid.py:167-194 (one-sided on the edges), I
// the bilinear gather (src/Particles.py:117-180), k = q dt/m, c = dt/dx.
//
// Adjoint, per step n from N-1 down to 0 (absorption is a fixed mask: a
// particle dead at a state takes no part in it):
//   kick:    lambda_u_n += lambda_u_{n+1};  lambda_x_{n+1} += k (dI/dx)^T lambda_u_{n+1}
//            lambda_E_{n+1} = k I^T lambda_u_{n+1}              (a CIC scatter)
//   field:   lambda_phi = G^T lambda_E;  solve A mu = lambda_phi on free nodes
//            (A is symmetric, so the adjoint solve is one more multigrid solve
//            with zero boundary values); dL/dV_seg += sum over the segment's
//            nodes of lambda_phi_B - sum of the free neighbours' couplings * mu
//   deposit: lambda_x_{n+1} += (q np2c/(dx dy)) (dW/dx)^T (-mu/eps0)
//   drift:   lambda_u_n += c lambda_x_{n+1};  lambda_x_n = lambda_x_{n+1}
// and for the init half-kick and the perturbation:
//   dL/dA = sum_p lambda_u_0 . dv_p, plus the field terms of the init kick.
// The forward pass keeps a checkpoint (positions, velocities, phi) every C
// steps; the backward pass recomputes each segment of C steps from its
// checkpoint, keeping the segment's positions and fields, then walks it back.
#include <climits>
#include <mutex>
#include <numeric>
#include <vector>

#include "sort_internal.cuh"

namespace pic {

int grid_blocks(long n, int threads);
int mg_create(int nx, int ny, double dx, double dy, const uint8_t* h_mask, const pic_mg_options* opts, pic_mg** out);
int mg_launch_cold(pic_mg* mg, double* phi, const double* f, double tol, int max_cycles, cudaStream_t st);
const int* mg_device_converged(pic_mg* mg);
int mg_info(pic_mg* mg, pic_mg_info* info);

struct AdSpecies {
    double kq[PIC_MAX_SPECIES];      // q dt / m
    double charge[PIC_MAX_SPECIES];  // q np2c / (dx dy): charge density of one particle at weight 1
    double dens[PIC_MAX_SPECIES];    // np2c / (dx dy): number density of one particle at weight 1
};

// Cell of a live particle (grid units, inside [0, n-1]) and its offsets;
// x = n-1 falls in the last cell with weight 1 on its far node.
struct AdCell {
    int i, j;
    double fx, fy;
};

__device__ __forceinline__ AdCell ad_cell(double x, double y, int nx, int ny) {
    AdCell c;
    c.i = max(0, min(int(floor(x)), nx - 2));
    c.j = max(0, min(int(floor(y)), ny - 2));
    c.fx = x - double(c.i);
    c.fy = y - double(c.j);
    return c;
}

// Gradient (per grid unit) of the bilinear interpolant of F at the particle.
__device__ __forceinline__ double2 ad_interp_grad(const double* __restrict__ F, const AdCell& c, int nx) {
    const long k = long(c.j) * nx + c.i;
    const double f00 = F[k], f10 = F[k + 1], f01 = F[k + nx], f11 = F[k + nx + 1];
    return make_double2((1.0 - c.fy) * (f10 - f00) + c.fy * (f11 - f01), (1.0 - c.fx) * (f01 - f00) + c.fx * (f11 - f10));
}

__device__ __forceinline__ bool alive(const int* __restrict__ death, int p, int state) { return death[p] > state; }

// ---- particle passes ---------------------------------------------------------------
//
// The particles are held in the cell order of their initial positions, species
// by species (AdjImpl::perm leads back to the caller's order), and a thread
// takes four consecutive slots with 32-byte accesses.
//   gather   E is stored per node as (Ex, Ey) here and at the east neighbour, 32
//            bytes: a particle reads two of them (of separate FP64 planes it reads
//            eight values in four sectors or more);
//   scatter  FP64 reductions run at the L2's rate of requests (about 145 per ns
//            whatever their order), so a thread adds up its particles while their
//            cell stays the same, the warp adds up lanes of one cell, and only the
//            sums go to the grid.  Ions stay in their cells for a whole run;
//            electrons leave theirs over some tens of steps.
// Per state, 1M electrons and 1M ions on 257^2 nodes: deposit, kick and drift,
// 129 us as three passes over planes, take one pass of 38 us; the adjoint of
// the kick and of the deposit and drift, 169 us as two passes, one of 65 us.

constexpr int kAdPer = 4;        // slots per thread
constexpr int kAdThreads = 128;

__device__ __forceinline__ void ld4(const double* __restrict__ p, double (&v)[4]) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}
__device__ __forceinline__ void st4(double* __restrict__ p, const double (&v)[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}

// (Ex, Ey) at a node and at its east neighbour.
struct alignas(32) AdQuad {
    double ex, ey, ex1, ey1;
};
__device__ __forceinline__ AdQuad ld_quad(const AdQuad* __restrict__ q) {
    AdQuad v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.ex), "=d"(v.ey), "=d"(v.ex1), "=d"(v.ey1) : "l"(q));
    return v;
}

// Sums of W values per corner of one cell: corners (i, j), (i+1, j), (i, j+1),
// (i+1, j+1) of the node k, each W consecutive doubles of the grid array.
template <int W>
struct AdSums {
    int k = -1;  // the cell's node, -1: none
    double v[4 * W];
    __device__ __forceinline__ void flush(double* __restrict__ F, int nx) {
        if (k < 0) return;
        double* a = F + long(k) * W;
        double* b = a + long(nx) * W;
#pragma unroll
        for (int q = 0; q < 2 * W; ++q) {
            atomicAdd(a + q, v[q]);
            atomicAdd(b + q, v[2 * W + q]);
        }
        k = -1;
    }
    // adds (value) * weights of a particle in cell c, flushing what another cell had
    __device__ __forceinline__ void add(const AdCell& c, const double (&val)[W], double* __restrict__ F, int nx) {
        const int n = c.j * nx + c.i;
        const double w[4] = {(1.0 - c.fx) * (1.0 - c.fy), c.fx * (1.0 - c.fy), (1.0 - c.fx) * c.fy, c.fx * c.fy};
        const bool fresh = n != k;
        if (fresh) flush(F, nx);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int d = 0; d < W; ++d) {
                const double t = w[q] * val[d];
                v[q * W + d] = fresh ? t : v[q * W + d] + t;
            }
        k = n;
    }
    // Adds the warp's lanes of one cell up (runs of consecutive lanes with the
    // same cell) where that leaves at most half of them to flush; every lane of
    // the warp takes part.
    __device__ __forceinline__ void merge(double* __restrict__ F, int nx) {
        const unsigned all = 0xffffffffu;
        const int lane = threadIdx.x & 31;
        const int before = __shfl_up_sync(all, k, 1);
        const unsigned heads = __ballot_sync(all, lane == 0 || before != k);
        if (__popc(heads) <= 16) {
            // lanes from this one to the end of its run
            const unsigned later = lane == 31 ? 0u : heads >> (lane + 1);
            const int run = later ? __ffs(later) : 32 - lane;
            if (k < 0) {
#pragma unroll
                for (int q = 0; q < 4 * W; ++q) v[q] = 0.0;
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
#pragma unroll
                for (int q = 0; q < 4 * W; ++q) {
                    const double t = __shfl_down_sync(all, v[q], o);
                    if (o < run) v[q] += t;
                }
            if (!((heads >> lane) & 1u)) k = -1;
        }
        flush(F, nx);
    }
};

// rho += charge (or number) density of the live particles; only species `only` if >= 0.
__global__ void __launch_bounds__(kAdThreads) k_ad_deposit(const double* __restrict__ x, const double* __restrict__ y,
                                                           const uint8_t* __restrict__ sp,
                                                           const int* __restrict__ death, int state, int n, int nx,
                                                           int ny, const __grid_constant__ AdSpecies S, int number,
                                                           int only, double* __restrict__ rho) {
    const int quads = (n + kAdPer - 1) / kAdPer, per = gridDim.x * blockDim.x;
    for (int q0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); q0 < quads; q0 += per) {
        const int q = q0 + (threadIdx.x & 31);
        AdSums<1> sum;
        if (q < quads) {
            double px[4], py[4];
            ld4(x + long(q) * kAdPer, px);
            ld4(y + long(q) * kAdPer, py);
#pragma unroll
            for (int r = 0; r < kAdPer; ++r) {
                const int p = q * kAdPer + r;
                if (p >= n || !alive(death, p, state)) continue;
                const int s = sp[p];
                if (only >= 0 && s != only) continue;
                const double v[1] = {number ? S.dens[s] : S.charge[s]};
                sum.add(ad_cell(px[r], py[r], nx, ny), v, rho, nx);
            }
        }
        sum.merge(rho, nx);
    }
}

// One particle pass of the forward model: u += factor k I(x; E) for particles
// alive at `state`, the state saved (cp), x += c u (a particle that leaves
// [0, n-1]^2 dies at state + 1, unless the absorption steps are frozen), and the
// charge of the survivors.  In and out may be the same arrays.
struct AdPass {
    const double *x, *y, *ux, *uy;
    double *xo, *yo, *uxo, *uyo;
    double* cp;     // the kicked state as four arrays of `stride` values, or null
    long stride;
    const uint8_t* sp;
    int* death;
    int state, n, nx, ny;
    const AdQuad* E;
    double factor, cx, cy;  // factor 0: no kick
    int drift, frozen;
    double* rho;  // null: no deposit
};

__global__ void __launch_bounds__(kAdThreads) k_ad_pass(const __grid_constant__ AdPass A,
                                                        const __grid_constant__ AdSpecies S) {
    const int quads = (A.n + kAdPer - 1) / kAdPer, per = gridDim.x * blockDim.x;
    for (int q0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); q0 < quads; q0 += per) {
        const int q = q0 + (threadIdx.x & 31);
        const long b = long(q) * kAdPer;
        AdSums<1> sum;
        if (q < quads) {
            double x[4], y[4], ux[4], uy[4];
            ld4(A.x + b, x);
            ld4(A.y + b, y);
            ld4(A.ux + b, ux);
            ld4(A.uy + b, uy);
            const int4 d4 = *reinterpret_cast<const int4*>(A.death + b);
            const uchar4 s4 = *reinterpret_cast<const uchar4*>(A.sp + b);
            const int dth[4] = {d4.x, d4.y, d4.z, d4.w};
            const int spc[4] = {s4.x, s4.y, s4.z, s4.w};
            if (A.factor != 0.0) {
#pragma unroll
                for (int r = 0; r < kAdPer; ++r) {
                    if (b + r >= A.n || dth[r] <= A.state) continue;
                    const AdCell c = ad_cell(x[r], y[r], A.nx, A.ny);
                    const AdQuad e = ld_quad(A.E + long(c.j) * A.nx + c.i), f = ld_quad(A.E + long(c.j + 1) * A.nx + c.i);
                    const double k = A.factor * S.kq[spc[r]];
                    const double w0 = (1.0 - c.fx) * (1.0 - c.fy), w1 = c.fx * (1.0 - c.fy), w2 = (1.0 - c.fx) * c.fy,
                                 w3 = c.fx * c.fy;
                    ux[r] += k * (w0 * e.ex + w1 * e.ex1 + w2 * f.ex + w3 * f.ex1);
                    uy[r] += k * (w0 * e.ey + w1 * e.ey1 + w2 * f.ey + w3 * f.ey1);
                }
            }
            if (A.cp) {
                st4(A.cp + b, x);
                st4(A.cp + A.stride + b, y);
                st4(A.cp + 2 * A.stride + b, ux);
                st4(A.cp + 3 * A.stride + b, uy);
            }
            if (A.drift) {
#pragma unroll
                for (int r = 0; r < kAdPer; ++r) {
                    if (b + r >= A.n || dth[r] <= A.state) continue;
                    x[r] += A.cx * ux[r];
                    y[r] += A.cy * uy[r];
                    bool live = dth[r] > A.state + 1;
                    if (!A.frozen) {
                        live = x[r] >= 0.0 && x[r] <= double(A.nx - 1) && y[r] >= 0.0 && y[r] <= double(A.ny - 1);
                        if (!live) A.death[b + r] = A.state + 1;
                        else live = dth[r] > A.state + 1;
                    }
                    if (A.rho && live) {
                        const double v[1] = {S.charge[spc[r]]};
                        sum.add(ad_cell(x[r], y[r], A.nx, A.ny), v, A.rho, A.nx);
                    }
                }
                st4(A.xo + b, x);
                st4(A.yo + b, y);
            }
            st4(A.uxo + b, ux);
            st4(A.uyo + b, uy);
        }
        if (A.rho) sum.merge(A.rho, A.nx);
    }
}

// f = -rho/eps0 on free nodes, 0 on Dirichlet nodes; clears rho for the next deposit.
__global__ void k_ad_rhs(double* __restrict__ rho, const uint8_t* __restrict__ mask, double neg_inv_eps0,
                         double* __restrict__ f, long G) {
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < G; k += long(gridDim.x) * blockDim.x) {
        f[k] = mask[k] ? 0.0 : rho[k] * neg_inv_eps0;
        rho[k] = 0.0;
    }
}

// Dirichlet values: V[segment] on electrode nodes, the fixed value elsewhere.
__global__ void k_ad_bc(double* __restrict__ phi, const uint8_t* __restrict__ mask, const int* __restrict__ seg,
                        const double* __restrict__ fixed, const double* __restrict__ V, long G) {
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < G; k += long(gridDim.x) * blockDim.x)
        if (mask[k]) phi[k] = seg[k] >= 0 ? V[seg[k]] : fixed[k];
}

// -grad(phi) at node (i, j) with the stencil of src/Grid.py:167-194.
__device__ __forceinline__ double2 ad_efield(const double* __restrict__ phi, int i, int j, int nx, int ny, double dx,
                                             double dy) {
    const long k = long(j) * nx + i;
    double ex, ey;
    if (i > 0 && i < nx - 1) ex = -(phi[k + 1] - phi[k - 1]) / (2.0 * dx);
    else if (i == 0) ex = -(phi[k + 1] - phi[k]) / dx;
    else ex = -(phi[k] - phi[k - 1]) / dx;
    if (j > 0 && j < ny - 1) ey = -(phi[k + nx] - phi[k - nx]) / (2.0 * dy);
    else if (j == 0) ey = -(phi[k + nx] - phi[k]) / dy;
    else ey = -(phi[k] - phi[k - nx]) / dy;
    return make_double2(ex, ey);
}

// E of every node and its east neighbour (the last column's own, never read);
// a solve that did not converge is counted.
__global__ void k_ad_efield(const double* __restrict__ phi, AdQuad* __restrict__ E, int nx, int ny, double dx,
                            double dy, const int* __restrict__ converged, int* __restrict__ failures) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (converged && i == 0 && j == 0 && !*converged) atomicAdd(failures, 1);
    if (i >= nx) return;
    const double2 a = ad_efield(phi, i, j, nx, ny, dx, dy), b = ad_efield(phi, min(i + 1, nx - 1), j, nx, ny, dx, dy);
    const double v[4] = {a.x, a.y, b.x, b.y};
    st4(reinterpret_cast<double*>(E + long(j) * nx + i), v);
}

// u = v0 + A dv
__global__ void k_ad_perturb(double* __restrict__ ux, double* __restrict__ uy, const double* __restrict__ vx0,
                             const double* __restrict__ vy0, const double* __restrict__ dvx,
                             const double* __restrict__ dvy, double A, int n) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        ux[p] = vx0[p] + A * dvx[p];
        uy[p] = vy0[p] + A * dvy[p];
    }
}

// The cell order of a species' initial positions (tile-major keys; clamped, so
// that any position has one).
__global__ void k_ad_keys(const double* __restrict__ x, const double* __restrict__ y, int n, int ncx, int ncy, int tile,
                          int tiles_x, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, int* __restrict__ n_dev) {
    if (blockIdx.x == 0 && threadIdx.x == 0) n_dev[0] = n_dev[1] = n;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const float gx = fminf(fmaxf(float(x[p]), 0.0f), float(ncx)), gy = fminf(fmaxf(float(y[p]), 0.0f), float(ncy));
        keys[p] = tile_key(gx, gy, ncx, ncy, tile, tiles_x, 0u);
        vals[p] = uint32_t(p);
    }
}

constexpr int kAdTile = 16;  // cells per side of the order's tiles

// The caller's slot of each slot of a species that starts at slot b.
__global__ void k_ad_slots(const uint32_t* __restrict__ perm, int n, uint32_t b, uint32_t* __restrict__ out) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) out[k] = b + perm[k];
}

// dst[k] = src[perm[k]] (0 without src).
__global__ void k_ad_gather(const double* __restrict__ src, const uint32_t* __restrict__ perm, int n,
                            double* __restrict__ dst) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        dst[k] = src ? src[perm[k]] : 0.0;
}

// The state in the caller's order, out[perm[k]] = state[k].
struct AdOut {
    const double* in[4];
    double* out[4];
    const int* death;
    int* death_out;
};
__global__ void k_ad_state(AdOut O, const uint32_t* __restrict__ perm, int n) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t p = perm[k];
#pragma unroll
        for (int q = 0; q < 4; ++q) O.out[q][p] = O.in[q][k];
        O.death_out[p] = O.death[k];
    }
}

// loss = sum (dens - target)^2 / G, and g = dL/d dens = 2 (dens - target) / G.
__global__ void k_ad_loss(const double* __restrict__ dens, const double* __restrict__ target, double* __restrict__ g,
                          long G, double* __restrict__ loss) {
    double s = 0.0;
    for (long k = blockIdx.x * long(blockDim.x) + threadIdx.x; k < G; k += long(gridDim.x) * blockDim.x) {
        const double d = dens[k] - target[k];
        g[k] = 2.0 * d / double(G);
        s += d * d / double(G);
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, s);
}

// ---- adjoint kernels --------------------------------------------------------------

// One particle pass of the backward model, either part optional:
//   dep   the deposit and drift adjoints at `sd`: lambda_x += charge (dW/dx)^T
//         (-mu/eps0) for particles alive at sd, then lambda_u += c lambda_x for
//         particles alive at sd - 1 (the drift into sd);
//   kick  the adjoint of u += factor k I(x; E) at `sk`: lambda_x += factor k
//         (dI/dx)^T lambda_u, and lambda_E += factor k I^T lambda_u (lE: per node
//         the x and y components).
struct AdBack {
    int n, nx, ny;
    const uint8_t* sp;
    const int* death;
    double *lx, *ly, *lux, *luy;
    int dep, sd;
    const double *xd, *yd, *mu;
    double neg_inv_eps0, cx, cy;
    int kick, sk;
    const double *xk, *yk;
    const AdQuad* E;
    double factor;
    double* lE;
};

__global__ void __launch_bounds__(kAdThreads) k_ad_back(const __grid_constant__ AdBack A,
                                                        const __grid_constant__ AdSpecies S) {
    const int quads = (A.n + kAdPer - 1) / kAdPer, per = gridDim.x * blockDim.x;
    for (int q0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); q0 < quads; q0 += per) {
        const int q = q0 + (threadIdx.x & 31);
        const long b = long(q) * kAdPer;
        AdSums<2> sum;
        if (q < quads) {
            double lx[4], ly[4], lux[4], luy[4], x[4], y[4];
            ld4(A.lx + b, lx);
            ld4(A.ly + b, ly);
            ld4(A.lux + b, lux);
            ld4(A.luy + b, luy);
            const int4 d4 = *reinterpret_cast<const int4*>(A.death + b);
            const uchar4 s4 = *reinterpret_cast<const uchar4*>(A.sp + b);
            const int dth[4] = {d4.x, d4.y, d4.z, d4.w};
            const int spc[4] = {s4.x, s4.y, s4.z, s4.w};
            if (A.dep) {
                ld4(A.xd + b, x);
                ld4(A.yd + b, y);
#pragma unroll
                for (int r = 0; r < kAdPer; ++r) {
                    if (b + r >= A.n || dth[r] <= A.sd - 1) continue;
                    if (dth[r] > A.sd) {
                        const double2 g = ad_interp_grad(A.mu, ad_cell(x[r], y[r], A.nx, A.ny), A.nx);
                        const double s = S.charge[spc[r]] * A.neg_inv_eps0;
                        lx[r] += s * g.x;
                        ly[r] += s * g.y;
                    }
                    lux[r] += A.cx * lx[r];
                    luy[r] += A.cy * ly[r];
                }
                st4(A.lux + b, lux);
                st4(A.luy + b, luy);
            }
            if (A.kick) {
                ld4(A.xk + b, x);
                ld4(A.yk + b, y);
#pragma unroll
                for (int r = 0; r < kAdPer; ++r) {
                    if (b + r >= A.n || dth[r] <= A.sk) continue;
                    const double k = A.factor * S.kq[spc[r]];
                    const double v[2] = {k * lux[r], k * luy[r]};
                    if (v[0] == 0.0 && v[1] == 0.0) continue;
                    const AdCell c = ad_cell(x[r], y[r], A.nx, A.ny);
                    const AdQuad e = ld_quad(A.E + long(c.j) * A.nx + c.i), f = ld_quad(A.E + long(c.j + 1) * A.nx + c.i);
                    const double gxx = (1.0 - c.fy) * (e.ex1 - e.ex) + c.fy * (f.ex1 - f.ex);
                    const double gxy = (1.0 - c.fx) * (f.ex - e.ex) + c.fx * (f.ex1 - e.ex1);
                    const double gyx = (1.0 - c.fy) * (e.ey1 - e.ey) + c.fy * (f.ey1 - f.ey);
                    const double gyy = (1.0 - c.fx) * (f.ey - e.ey) + c.fx * (f.ey1 - e.ey1);
                    lx[r] += v[0] * gxx + v[1] * gyx;
                    ly[r] += v[0] * gxy + v[1] * gyy;
                    sum.add(c, v, A.lE, A.nx);
                }
            }
            st4(A.lx + b, lx);
            st4(A.ly + b, ly);
        }
        if (A.kick) sum.merge(A.lE, A.nx);
    }
}

// lambda_phi = G^T lambda_E (transpose of k_ad_efield), and the right-hand
// side of the adjoint solve (lambda_phi on free nodes, 0 on Dirichlet nodes).
__global__ void k_ad_gradT(const double2* __restrict__ lE, const uint8_t* __restrict__ mask, double* __restrict__ lphi,
                           double* __restrict__ fa, int nx, int ny, double dx, double dy) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (i >= nx) return;
    const long k = long(j) * nx + i;
    const double hx = 0.5 / dx, hy = 0.5 / dy;
    double v = 0.0;
    if (i + 1 >= 1 && i + 1 <= nx - 2) v += hx * lE[k + 1].x;
    if (i - 1 >= 1 && i - 1 <= nx - 2) v -= hx * lE[k - 1].x;
    if (i == 0) v += lE[k].x / dx;
    if (i == 1) v -= lE[k - 1].x / dx;
    if (i == nx - 1) v -= lE[k].x / dx;
    if (i == nx - 2) v += lE[k + 1].x / dx;
    if (j + 1 >= 1 && j + 1 <= ny - 2) v += hy * lE[k + nx].y;
    if (j - 1 >= 1 && j - 1 <= ny - 2) v -= hy * lE[k - nx].y;
    if (j == 0) v += lE[k].y / dy;
    if (j == 1) v -= lE[k - nx].y / dy;
    if (j == ny - 1) v -= lE[k].y / dy;
    if (j == ny - 2) v += lE[k + nx].y / dy;
    lphi[k] = v;
    fa[k] = mask[k] ? 0.0 : v;
}

// After the adjoint solve: dL/dV[seg] += lambda_phi_B - sum over free
// neighbours of the coupling * mu, over the Dirichlet nodes B of each electrode
// segment; lambda_E cleared for the next scatter; a solve that did not converge
// counted.
__global__ void k_ad_dV(const double* __restrict__ lphi, const double* __restrict__ mu,
                        const uint8_t* __restrict__ mask, const int* __restrict__ seg, int nx, int ny, double cx,
                        double cy, double* __restrict__ dV, double2* __restrict__ lE,
                        const int* __restrict__ converged, int* __restrict__ failures) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (converged && i == 0 && j == 0 && !*converged) atomicAdd(failures, 1);
    if (i >= nx) return;
    const long k = long(j) * nx + i;
    lE[k] = make_double2(0.0, 0.0);
    if (!mask[k] || seg[k] < 0) return;
    double v = lphi[k];
    auto free_node = [&](int a, int b) {
        return a > 0 && b > 0 && a < nx - 1 && b < ny - 1 && !mask[long(b) * nx + a];
    };
    if (free_node(i - 1, j)) v -= cx * mu[k - 1];
    if (free_node(i + 1, j)) v -= cx * mu[k + 1];
    if (free_node(i, j - 1)) v -= cy * mu[k - nx];
    if (free_node(i, j + 1)) v -= cy * mu[k + nx];
    atomicAdd(dV + seg[k], v);
}

// lambda_x += dens (dW/dx)^T g for the loss species alive at the final state.
__global__ void k_ad_loss_adj(const double* __restrict__ x, const double* __restrict__ y,
                              const uint8_t* __restrict__ sp, const int* __restrict__ death, int state, int n, int nx,
                              int ny, const double* __restrict__ g, AdSpecies S, int only, double* __restrict__ lx,
                              double* __restrict__ ly) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        if (!alive(death, p, state) || sp[p] != only) continue;
        const double2 d = ad_interp_grad(g, ad_cell(x[p], y[p], nx, ny), nx);
        lx[p] += S.dens[sp[p]] * d.x;
        ly[p] += S.dens[sp[p]] * d.y;
    }
}

// dA = sum_p lambda_u . dv
__global__ void k_ad_dot(const double* __restrict__ lux, const double* __restrict__ luy,
                         const double* __restrict__ dvx, const double* __restrict__ dvy, int n,
                         double* __restrict__ out) {
    double s = 0.0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        s += lux[p] * dvx[p] + luy[p] * dvy[p];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// ---- host object ------------------------------------------------------------------

struct AdjImpl {
    pic_adj_desc d{};
    int n = 0;  // particles of all species
    long G = 0;
    int first[PIC_MAX_SPECIES + 1]{};
    AdSpecies S{};
    pic_mg* mg = nullptr;   // forward solves
    pic_mg* mga = nullptr;  // adjoint solves
    std::vector<void*> allocs;
    // particles, in the cell order of each species' initial positions; `perm`
    // holds the caller's slot of each.  Arrays are `stride` long (a multiple of
    // four slots).
    long stride = 0;
    uint32_t* perm = nullptr;
    double *x0 = nullptr, *y0 = nullptr, *vx0 = nullptr, *vy0 = nullptr, *dvx = nullptr, *dvy = nullptr;
    uint8_t* sp = nullptr;
    double *x = nullptr, *y = nullptr, *ux = nullptr, *uy = nullptr;    // the forward pass's state
    double *ru = nullptr, *rv = nullptr;                                // velocities of a recomputed segment
    int* death = nullptr;
    double* lam[4] = {};                                                // lambda_x, _y, _ux, _uy
    // the state after the last forward pass in the caller's order (pic_adj_state)
    double* out[4] = {};
    int* death_out = nullptr;
    // checkpoints: x, y, ux, uy per particle and phi, every C steps (states 0, C, 2C, ...)
    int ncp = 0;
    double* cp = nullptr;
    double* cp_phi = nullptr;
    // one segment of positions and fields (states a+1 .. a+C)
    double* seg_xy = nullptr;
    int* sort_cnt = nullptr;  // digit counts of the cell order's sort, their totals and the two counts
    // every species' sort works in the same scratch: on whatever streams and
    // threads species are set, one sort follows the other
    std::mutex sort_mutex;
    cudaEvent_t sorted = nullptr;
    AdQuad* seg_E = nullptr;
    // grids
    uint8_t* mask = nullptr;
    int* segid = nullptr;
    double *fixed = nullptr, *V = nullptr, *rho = nullptr, *f = nullptr, *phi = nullptr, *phi_out = nullptr;
    AdQuad* E = nullptr;
    double2* lE = nullptr;
    double *lphi = nullptr, *fa = nullptr, *mu = nullptr, *target = nullptr,
           *g = nullptr;
    double* red = nullptr;  // [0] loss, [1] dA, [2..] dV
    int* failures = nullptr;
    double A = 0.0;
    bool have_forward = false;
    bool frozen = false;  // reuse the absorption steps of the last forward pass
    double loss = 0.0;
};

template <class T>
static int adalloc(AdjImpl& J, T** p, size_t n) {
    PIC_CUDA(cudaMalloc(p, sizeof(T) * std::max<size_t>(n, 1)));
    J.allocs.push_back(*p);
    PIC_CUDA(cudaMemset(*p, 0, sizeof(T) * std::max<size_t>(n, 1)));
    return PIC_OK;
}

static void adj_free(AdjImpl& J) {
    if (J.mg) pic_mg_destroy(J.mg);
    if (J.mga) pic_mg_destroy(J.mga);
    J.mg = J.mga = nullptr;
    for (void* p : J.allocs) cudaFree(p);
    J.allocs.clear();
    if (J.sorted) cudaEventDestroy(J.sorted);
    J.sorted = nullptr;
}

static int adj_create(const pic_adj_desc* d, AdjImpl& J) {
    if (!d || d->nx < 3 || d->ny < 3 || !(d->dx > 0) || !(d->dy > 0) || !(d->dt > 0) || !(d->eps0 > 0) ||
        d->nspecies < 1 || d->nspecies > PIC_MAX_SPECIES || !d->h_dirichlet || !d->h_segment || d->nseg < 0 ||
        d->nseg > PIC_ADJ_MAX_SEGMENTS || d->steps < 1 || d->checkpoint_every < 1 || d->loss_species < 0 ||
        d->loss_species >= d->nspecies || !(d->tol >= 0) || d->max_cycles < 1)
        return fail(PIC_ERR_BAD_ARG, "pic_adj_create: bad descriptor");
    J.d = *d;
    J.G = long(d->nx) * d->ny;
    J.n = 0;
    for (int s = 0; s < d->nspecies; ++s) {
        const pic_adj_species& q = d->species[s];
        if (q.n < 0 || !(q.mass > 0) || !(q.np2c > 0)) return fail(PIC_ERR_BAD_ARG, "pic_adj_create: species %d", s);
        J.first[s] = J.n;
        J.n += q.n;
        J.S.kq[s] = q.charge * d->dt / q.mass;
        J.S.charge[s] = q.charge * q.np2c / (d->dx * d->dy);
        J.S.dens[s] = q.np2c / (d->dx * d->dy);
    }
    J.first[d->nspecies] = J.n;
    std::vector<uint8_t> mask(d->h_dirichlet, d->h_dirichlet + J.G);
    for (long k = 0; k < J.G; ++k) {
        const int i = int(k % d->nx), j = int(k / d->nx);
        mask[k] = (mask[k] || i == 0 || j == 0 || i == d->nx - 1 || j == d->ny - 1) ? 1 : 0;
        if (d->h_segment[k] >= d->nseg) return fail(PIC_ERR_BAD_ARG, "pic_adj_create: segment index out of range");
    }
    pic_mg_options o{};
    o.precision = PIC_MG_FP64;
    o.pre_sweeps = o.post_sweeps = 2;
    o.omega = 1.0;
    o.coarsest_max = 9;
    o.launch_mode = PIC_MG_GRAPH_LOOP;
    PIC_TRY(mg_create(d->nx, d->ny, d->dx, d->dy, mask.data(), &o, &J.mg));
    PIC_TRY(mg_create(d->nx, d->ny, d->dx, d->dy, mask.data(), &o, &J.mga));
    const size_t n = size_t(std::max(J.n, 1) + kAdPer - 1) / kAdPer * kAdPer, G = size_t(J.G);
    J.stride = long(n);
    for (double** p : {&J.x0, &J.y0, &J.vx0, &J.vy0, &J.dvx, &J.dvy, &J.x, &J.y, &J.ux, &J.uy, &J.ru, &J.rv, &J.lam[0],
                       &J.lam[1], &J.lam[2], &J.lam[3], &J.out[0], &J.out[1], &J.out[2], &J.out[3]})
        PIC_TRY(adalloc(J, p, n));
    PIC_TRY(adalloc(J, &J.perm, n));
    PIC_TRY(adalloc(J, &J.sp, n));
    PIC_TRY(adalloc(J, &J.death, n));
    PIC_TRY(adalloc(J, &J.death_out, n));
    J.ncp = (d->steps + d->checkpoint_every - 1) / d->checkpoint_every;  // states 0, C, ... < steps
    PIC_TRY(adalloc(J, &J.cp, size_t(J.ncp) * 4 * n));
    PIC_TRY(adalloc(J, &J.cp_phi, size_t(J.ncp) * G));
    const size_t C = size_t(std::min(d->checkpoint_every, d->steps));
    PIC_TRY(adalloc(J, &J.seg_xy, C * 2 * n));
    PIC_TRY(adalloc(J, &J.seg_E, C * G));
    PIC_CUDA(cudaEventCreateWithFlags(&J.sorted, cudaEventDisableTiming));
    PIC_TRY(adalloc(J, &J.sort_cnt, (size_t(num_sms() + 1) << kSortDigitMax) + 2));
    PIC_TRY(adalloc(J, &J.mask, G));
    PIC_CUDA(cudaMemcpy(J.mask, mask.data(), G, cudaMemcpyHostToDevice));
    PIC_TRY(adalloc(J, &J.segid, G));
    PIC_CUDA(cudaMemcpy(J.segid, d->h_segment, sizeof(int) * G, cudaMemcpyHostToDevice));
    PIC_TRY(adalloc(J, &J.fixed, G));
    if (d->h_phi_fixed) PIC_CUDA(cudaMemcpy(J.fixed, d->h_phi_fixed, sizeof(double) * G, cudaMemcpyHostToDevice));
    for (double** p : {&J.rho, &J.f, &J.phi, &J.phi_out, &J.lphi, &J.fa, &J.mu, &J.target, &J.g}) PIC_TRY(adalloc(J, p, G));
    PIC_TRY(adalloc(J, &J.E, G));
    PIC_TRY(adalloc(J, &J.lE, G));
    PIC_TRY(adalloc(J, &J.V, size_t(PIC_ADJ_MAX_SEGMENTS)));
    PIC_TRY(adalloc(J, &J.red, size_t(2 + PIC_ADJ_MAX_SEGMENTS)));
    PIC_TRY(adalloc(J, &J.failures, 1));
    // until a species' particles are set, its slots are the caller's
    std::vector<uint32_t> slots(n);
    std::iota(slots.begin(), slots.end(), 0u);
    PIC_CUDA(cudaMemcpy(J.perm, slots.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice));
    std::vector<uint8_t> spv(n, 0);
    for (int s = 0; s < d->nspecies; ++s)
        for (int p = J.first[s]; p < J.first[s + 1]; ++p) spv[p] = uint8_t(s);
    PIC_CUDA(cudaMemcpy(J.sp, spv.data(), n, cudaMemcpyHostToDevice));
    return PIC_OK;
}

static int grid2(const AdjImpl& J, dim3& g) {
    g = dim3(div_up(J.d.nx, 128), J.d.ny);
    return 128;
}

static int pass_blocks(const AdjImpl& J) {
    return std::max(1, std::min(div_up(div_up(J.n, kAdPer), kAdThreads), 16 * num_sms()));
}

// rho (deposited) -> phi -> E (phi holds the initial guess); clears rho.
static int field_of(AdjImpl& J, double* phi, AdQuad* E, cudaStream_t st) {
    k_ad_rhs<<<grid_blocks(J.G, 256), 256, 0, st>>>(J.rho, J.mask, -1.0 / J.d.eps0, J.f, J.G);
    PIC_LAUNCH_CHECK();
    PIC_TRY(mg_launch_cold(J.mg, phi, J.f, J.d.tol, J.d.max_cycles, st));
    dim3 g;
    const int t = grid2(J, g);
    k_ad_efield<<<g, t, 0, st>>>(phi, E, J.d.nx, J.d.ny, J.d.dx, J.d.dy,
                                 J.d.tol > 0 ? mg_device_converged(J.mg) : nullptr, J.failures);
    PIC_LAUNCH_CHECK();
    return PIC_OK;
}

static int deposit(AdjImpl& J, const double* x, const double* y, int state, int number, int only, cudaStream_t st) {
    k_ad_deposit<<<pass_blocks(J), kAdThreads, 0, st>>>(x, y, J.sp, J.death, state, J.n, J.d.nx, J.d.ny, J.S, number,
                                                        only, J.rho);
    PIC_LAUNCH_CHECK();
    return PIC_OK;
}

// The pass from `state` to state + 1 (k_ad_pass), in: x, y, ux, uy.
static AdPass pass_args(const AdjImpl& J, int state, const double* x, const double* y, const double* ux,
                        const double* uy, const AdQuad* E, double factor) {
    AdPass A{};
    A.x = x;
    A.y = y;
    A.ux = ux;
    A.uy = uy;
    A.stride = J.stride;
    A.sp = J.sp;
    A.death = J.death;
    A.state = state;
    A.n = J.n;
    A.nx = J.d.nx;
    A.ny = J.d.ny;
    A.E = E;
    A.factor = factor;
    A.cx = J.d.dt / J.d.dx;
    A.cy = J.d.dt / J.d.dy;
    A.drift = 1;
    A.frozen = J.frozen ? 1 : 0;
    A.rho = J.rho;
    return A;
}

// The error of a pass with so many unconverged solves: a timeout of one of their
// grid barriers (which is cleared with the report), else that they did not converge.
static int report(AdjImpl& J, int failures) {
    if (!failures && J.d.tol > 0) return PIC_OK;
    pic_mg_info info;
    PIC_TRY(mg_info(J.mg, &info));
    PIC_TRY(mg_info(J.mga, &info));
    if (failures) return fail(PIC_ERR_NOT_CONVERGED, "%d Poisson solves did not converge", failures);
    return PIC_OK;
}

static int adj_forward(AdjImpl& J, const double* h_V, double A, double* loss, cudaStream_t st) {
    const int pb = grid_blocks(J.n, 256), gb = grid_blocks(J.G, 256), ab = pass_blocks(J);
    const size_t G = size_t(J.G);
    if (J.d.nseg > 0) PIC_CUDA(cudaMemcpyAsync(J.V, h_V, sizeof(double) * J.d.nseg, cudaMemcpyHostToDevice, st));
    PIC_CUDA(cudaMemsetAsync(J.failures, 0, sizeof(int), st));
    PIC_CUDA(cudaMemsetAsync(J.red, 0, sizeof(double) * (2 + PIC_ADJ_MAX_SEGMENTS), st));
    if (!(J.frozen && J.have_forward))
        PIC_CUDA(cudaMemsetAsync(J.death, 0x7f, sizeof(int) * size_t(J.stride), st));  // alive at every state
    PIC_CUDA(cudaMemsetAsync(J.phi, 0, sizeof(double) * G, st));
    PIC_CUDA(cudaMemsetAsync(J.rho, 0, sizeof(double) * G, st));
    k_ad_bc<<<gb, 256, 0, st>>>(J.phi, J.mask, J.segid, J.fixed, J.V, J.G);
    k_ad_perturb<<<pb, 256, 0, st>>>(J.ux, J.uy, J.vx0, J.vy0, J.dvx, J.dvy, A, J.n);
    PIC_LAUNCH_CHECK();
    // init: E_0; the backward half kick is the first pass's
    PIC_TRY(deposit(J, J.x0, J.y0, 0, 0, -1, st));
    PIC_TRY(field_of(J, J.phi, J.E, st));
    const int C = J.d.checkpoint_every;
    for (int s = 0; s < J.d.steps; ++s) {
        // the kick at state s, its checkpoint, the drift to s + 1 and its deposit
        AdPass P = pass_args(J, s, s ? J.x : J.x0, s ? J.y : J.y0, J.ux, J.uy, J.E, s ? 1.0 : -0.5);
        P.xo = J.x;
        P.yo = J.y;
        P.uxo = J.ux;
        P.uyo = J.uy;
        if (s % C == 0) {
            P.cp = J.cp + size_t(s / C) * 4 * size_t(J.stride);
            PIC_CUDA(cudaMemcpyAsync(J.cp_phi + size_t(s / C) * G, J.phi, sizeof(double) * G, cudaMemcpyDeviceToDevice,
                                     st));
        }
        k_ad_pass<<<ab, kAdThreads, 0, st>>>(P, J.S);
        PIC_LAUNCH_CHECK();
        PIC_TRY(field_of(J, J.phi, J.E, st));
    }
    // the kick at the final state
    AdPass P = pass_args(J, J.d.steps, J.x, J.y, J.ux, J.uy, J.E, 1.0);
    P.uxo = J.ux;
    P.uyo = J.uy;
    P.drift = 0;
    P.rho = nullptr;
    k_ad_pass<<<ab, kAdThreads, 0, st>>>(P, J.S);
    PIC_LAUNCH_CHECK();
    // loss on the final density of the loss species
    PIC_TRY(deposit(J, J.x, J.y, J.d.steps, 1, J.d.loss_species, st));
    k_ad_loss<<<gb, 256, 0, st>>>(J.rho, J.target, J.g, J.G, J.red);
    PIC_CUDA(cudaMemsetAsync(J.rho, 0, sizeof(double) * G, st));
    PIC_CUDA(cudaMemcpyAsync(J.phi_out, J.phi, sizeof(double) * G, cudaMemcpyDeviceToDevice, st));
    AdOut O{{J.x, J.y, J.ux, J.uy}, {J.out[0], J.out[1], J.out[2], J.out[3]}, J.death, J.death_out};
    k_ad_state<<<pb, 256, 0, st>>>(O, J.perm, J.n);
    PIC_LAUNCH_CHECK();
    int failures = 0;
    PIC_CUDA(cudaMemcpyAsync(&J.loss, J.red, sizeof(double), cudaMemcpyDeviceToHost, st));
    PIC_CUDA(cudaMemcpyAsync(&failures, J.failures, sizeof(int), cudaMemcpyDeviceToHost, st));
    PIC_CUDA(cudaStreamSynchronize(st));
    J.A = A;
    J.have_forward = true;
    if (loss) *loss = J.loss;
    return report(J, failures);
}

// Field part of a kick adjoint already scattered into lambda_E: lambda_phi,
// the adjoint solve and the electrode-potential gradient; clears lambda_E.
static int field_adj(AdjImpl& J, cudaStream_t st) {
    dim3 g;
    const int t = grid2(J, g);
    k_ad_gradT<<<g, t, 0, st>>>(J.lE, J.mask, J.lphi, J.fa, J.d.nx, J.d.ny, J.d.dx, J.d.dy);
    PIC_LAUNCH_CHECK();
    PIC_TRY(mg_launch_cold(J.mga, J.mu, J.fa, J.d.tol, J.d.max_cycles, st));
    k_ad_dV<<<g, t, 0, st>>>(J.lphi, J.mu, J.mask, J.segid, J.d.nx, J.d.ny, 1.0 / (J.d.dx * J.d.dx),
                             1.0 / (J.d.dy * J.d.dy), J.red + 2, J.lE,
                             J.d.tol > 0 ? mg_device_converged(J.mga) : nullptr, J.failures);
    PIC_LAUNCH_CHECK();
    return PIC_OK;
}

// The backward particle pass (k_ad_back): the deposit and drift adjoints at
// state sd (positions xd, yd) unless xd is null, then the kick adjoint at
// state sk (positions xk, yk and field E) unless xk is null.
static int back(AdjImpl& J, int sd, const double* xd, const double* yd, int sk, const double* xk, const double* yk,
                const AdQuad* E, double factor, cudaStream_t st) {
    AdBack B{};
    B.n = J.n;
    B.nx = J.d.nx;
    B.ny = J.d.ny;
    B.sp = J.sp;
    B.death = J.death;
    B.lx = J.lam[0];
    B.ly = J.lam[1];
    B.lux = J.lam[2];
    B.luy = J.lam[3];
    B.dep = xd != nullptr;
    B.sd = sd;
    B.xd = xd;
    B.yd = yd;
    B.mu = J.mu;
    B.neg_inv_eps0 = -1.0 / J.d.eps0;
    B.cx = J.d.dt / J.d.dx;
    B.cy = J.d.dt / J.d.dy;
    B.kick = xk != nullptr;
    B.sk = sk;
    B.xk = xk;
    B.yk = yk;
    B.E = E;
    B.factor = factor;
    B.lE = reinterpret_cast<double*>(J.lE);
    k_ad_back<<<pass_blocks(J), kAdThreads, 0, st>>>(B, J.S);
    PIC_LAUNCH_CHECK();
    return PIC_OK;
}

static int adj_backward(AdjImpl& J, double* h_dV, double* h_dA, cudaStream_t st) {
    if (!J.have_forward) return fail(PIC_ERR_BAD_ARG, "pic_adj_backward: run pic_adj_forward first");
    const int pb = grid_blocks(J.n, 256), ab = pass_blocks(J);
    const size_t n = size_t(J.stride), G = size_t(J.G);
    const int N = J.d.steps, C = J.d.checkpoint_every;
    PIC_CUDA(cudaMemsetAsync(J.failures, 0, sizeof(int), st));
    PIC_CUDA(cudaMemsetAsync(J.red + 1, 0, sizeof(double) * (1 + PIC_ADJ_MAX_SEGMENTS), st));
    for (double* p : J.lam) PIC_CUDA(cudaMemsetAsync(p, 0, sizeof(double) * n, st));
    PIC_CUDA(cudaMemsetAsync(J.lE, 0, sizeof(double2) * G, st));
    PIC_CUDA(cudaMemsetAsync(J.mu, 0, sizeof(double) * G, st));
    // the loss gradient at the final state (positions are those the forward pass ended with)
    k_ad_loss_adj<<<pb, 256, 0, st>>>(J.x, J.y, J.sp, J.death, N, J.n, J.d.nx, J.d.ny, J.g, J.S, J.d.loss_species,
                                      J.lam[0], J.lam[1]);
    PIC_LAUNCH_CHECK();
    auto xs = [&](int k) { return J.seg_xy + size_t(k) * 2 * n; };  // positions of the segment's state a + 1 + k
    for (int c = J.ncp - 1; c >= 0; --c) {
        const int a = c * C, b = std::min(N, a + C);
        // recompute states a+1 .. b, keeping positions and fields; the checkpoint is kicked already
        const double* cp = J.cp + size_t(c) * 4 * n;
        PIC_CUDA(cudaMemcpyAsync(J.phi, J.cp_phi + size_t(c) * G, sizeof(double) * G, cudaMemcpyDeviceToDevice, st));
        for (int s = a; s < b; ++s) {
            const int k = s - a;
            AdPass P = k ? pass_args(J, s, xs(k - 1), xs(k - 1) + n, J.ru, J.rv, J.seg_E + size_t(k - 1) * G, 1.0)
                         : pass_args(J, s, cp, cp + n, cp + 2 * n, cp + 3 * n, nullptr, 0.0);
            P.xo = xs(k);
            P.yo = xs(k) + n;
            P.uxo = J.ru;
            P.uyo = J.rv;
            k_ad_pass<<<ab, kAdThreads, 0, st>>>(P, J.S);
            PIC_LAUNCH_CHECK();
            PIC_TRY(field_of(J, J.phi, J.seg_E + size_t(k) * G, st));
        }
        // walk the segment back: the kick adjoint at state s + 1, its field, then the deposit and drift into it,
        // which share a pass with the next kick adjoint
        PIC_TRY(back(J, 0, nullptr, nullptr, b, xs(b - 1 - a), xs(b - 1 - a) + n, J.seg_E + size_t(b - 1 - a) * G, 1.0, st));
        for (int s = b - 1; s >= a; --s) {
            const int k = s - a;  // state s + 1 is the segment's k-th
            PIC_TRY(field_adj(J, st));
            if (k > 0)
                PIC_TRY(back(J, s + 1, xs(k), xs(k) + n, s, xs(k - 1), xs(k - 1) + n, J.seg_E + size_t(k - 1) * G, 1.0,
                             st));
            else PIC_TRY(back(J, s + 1, xs(k), xs(k) + n, 0, nullptr, nullptr, nullptr, 0.0, st));
        }
    }
    // the init half kick at state 0 (positions x_0; its E_0 recomputed with the
    // forward's initial guess) and the perturbation amplitude
    PIC_CUDA(cudaMemcpyAsync(J.phi, J.cp_phi, sizeof(double) * G, cudaMemcpyDeviceToDevice, st));
    PIC_TRY(deposit(J, J.x0, J.y0, 0, 0, -1, st));
    PIC_TRY(field_of(J, J.phi, J.E, st));
    PIC_TRY(back(J, 0, nullptr, nullptr, 0, J.x0, J.y0, J.E, -0.5, st));
    PIC_TRY(field_adj(J, st));
    k_ad_dot<<<pb, 256, 0, st>>>(J.lam[2], J.lam[3], J.dvx, J.dvy, J.n, J.red + 1);
    PIC_LAUNCH_CHECK();
    double out[2 + PIC_ADJ_MAX_SEGMENTS];
    int failures = 0;
    PIC_CUDA(cudaMemcpyAsync(out, J.red, sizeof out, cudaMemcpyDeviceToHost, st));
    PIC_CUDA(cudaMemcpyAsync(&failures, J.failures, sizeof(int), cudaMemcpyDeviceToHost, st));
    PIC_CUDA(cudaStreamSynchronize(st));
    if (h_dA) *h_dA = out[1];
    if (h_dV)
        for (int q = 0; q < J.d.nseg; ++q) h_dV[q] = out[2 + q];
    return report(J, failures);
}

// The cell order of species s' new initial positions, and its arrays in it.
static int set_species(AdjImpl& J, int s, const double* const src[6], cudaStream_t st) {
    const int b = J.first[s], n = J.first[s + 1] - b;
    // the sort's scratch: keys and slots in the segment's position arrays (16
    // bytes per particle, used by the backward pass alone)
    std::lock_guard<std::mutex> lock(J.sort_mutex);
    // (in a capture the graph orders them: an event recorded outside cannot be waited on)
    cudaStreamCaptureStatus cs;
    PIC_CUDA(cudaStreamIsCapturing(st, &cs));
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    if (!capturing) PIC_CUDA(cudaStreamWaitEvent(st, J.sorted, 0));
    SortImpl R;
    PIC_TRY(sort_geometry(n, J.d.nx, J.d.ny, kAdTile, num_sms(), &R));
    uint32_t* scratch = reinterpret_cast<uint32_t*>(J.seg_xy);
    R.k0 = scratch;
    R.k1 = scratch + J.stride;
    R.v0 = scratch + 2 * J.stride;
    R.v1 = scratch + 3 * J.stride;
    R.cnt = J.sort_cnt;
    R.tot = R.cnt + (size_t(num_sms()) << kSortDigitMax);
    R.n_dev = R.tot + (size_t(1) << kSortDigitMax);
    k_ad_keys<<<grid_blocks(n, 256), 256, 0, st>>>(src[0], src[1], n, J.d.nx - 1, J.d.ny - 1, R.tile, R.tiles_x, R.k0,
                                                   R.v0, R.n_dev);
    const uint32_t* perm = nullptr;
    PIC_TRY(sort_passes(R, nullptr, nullptr, &perm, st));
    double* dst[6] = {J.x0, J.y0, J.vx0, J.vy0, J.dvx, J.dvy};
    for (int q = 0; q < 6; ++q) k_ad_gather<<<grid_blocks(n, 256), 256, 0, st>>>(src[q], perm, n, dst[q] + b);
    k_ad_slots<<<grid_blocks(n, 256), 256, 0, st>>>(perm, n, uint32_t(b), J.perm + b);
    PIC_LAUNCH_CHECK();
    if (!capturing) PIC_CUDA(cudaEventRecord(J.sorted, st));
    return PIC_OK;
}

}  // namespace pic

struct pic_adj {
    pic::AdjImpl j;
};

using namespace pic;

extern "C" {

int pic_adj_create(const pic_adj_desc* desc, pic_adj** out) {
    clear_error();
    if (!out) return fail(PIC_ERR_BAD_ARG, "pic_adj_create: out is NULL");
    pic_adj* a = new pic_adj;
    const int st = adj_create(desc, a->j);
    if (st != PIC_OK) {
        adj_free(a->j);
        delete a;
        return st;
    }
    *out = a;
    return PIC_OK;
}

int pic_adj_destroy(pic_adj* a) {
    clear_error();
    if (!a) return PIC_OK;
    cudaDeviceSynchronize();
    adj_free(a->j);
    delete a;
    return PIC_OK;
}

int pic_adj_set_particles(pic_adj* a, int s, const double* d_x, const double* d_y, const double* d_vx,
                          const double* d_vy, const double* d_dvx, const double* d_dvy, void* stream) {
    clear_error();
    if (!a || s < 0 || s >= a->j.d.nspecies || !d_x || !d_y || !d_vx || !d_vy)
        return fail(PIC_ERR_BAD_ARG, "pic_adj_set_particles: bad arguments");
    AdjImpl& J = a->j;
    cudaStream_t st = as_stream(stream);
    const int b = J.first[s], n = J.first[s + 1] - b;
    if (n == 0) return PIC_OK;
    const double* src[6] = {d_x, d_y, d_vx, d_vy, d_dvx, d_dvy};
    PIC_TRY(set_species(J, s, src, st));
    J.have_forward = false;
    return PIC_OK;
}

int pic_adj_set_target(pic_adj* a, const double* d_target, void* stream) {
    clear_error();
    if (!a || !d_target) return fail(PIC_ERR_BAD_ARG, "pic_adj_set_target: bad arguments");
    PIC_CUDA(cudaMemcpyAsync(a->j.target, d_target, sizeof(double) * a->j.G, cudaMemcpyDeviceToDevice,
                             as_stream(stream)));
    a->j.have_forward = false;
    return PIC_OK;
}

int pic_adj_forward(pic_adj* a, const double* h_V, double A, double* loss, void* stream) {
    clear_error();
    if (!a || (a->j.d.nseg > 0 && !h_V)) return fail(PIC_ERR_BAD_ARG, "pic_adj_forward: bad arguments");
    return adj_forward(a->j, h_V, A, loss, as_stream(stream));
}

int pic_adj_backward(pic_adj* a, double* h_dV, double* h_dA, void* stream) {
    clear_error();
    if (!a) return fail(PIC_ERR_BAD_ARG, "pic_adj_backward: bad arguments");
    return adj_backward(a->j, h_dV, h_dA, as_stream(stream));
}

int pic_adj_freeze_absorption(pic_adj* a, int on) {
    clear_error();
    if (!a) return fail(PIC_ERR_BAD_ARG, "pic_adj_freeze_absorption: bad arguments");
    if (on && !a->j.have_forward) return fail(PIC_ERR_BAD_ARG, "pic_adj_freeze_absorption: run a forward pass first");
    a->j.frozen = on != 0;
    return PIC_OK;
}

int pic_adj_state(pic_adj* a, double** x, double** y, double** ux, double** uy, int** death, double** phi) {
    clear_error();
    if (!a) return fail(PIC_ERR_BAD_ARG, "pic_adj_state: bad arguments");
    AdjImpl& J = a->j;
    if (x) *x = J.out[0];
    if (y) *y = J.out[1];
    if (ux) *ux = J.out[2];
    if (uy) *uy = J.out[3];
    if (death) *death = J.death_out;
    if (phi) *phi = J.phi_out;
    return PIC_OK;
}

}  // extern "C"
