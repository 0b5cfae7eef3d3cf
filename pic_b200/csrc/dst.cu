// Fast Poisson solve by discrete sine transforms, for grids whose Dirichlet
// nodes are exactly the four edges (the reference's poisson_fft_dirichlet,
// src/FFT.py:10-64, and poisson_solver_dirichlet_2d, :102-121).
//
// lap(phi) = f with the 5-point operator and phi given on the edges: the edge
// values move to the right-hand side of the interior nodes next to them
// (f - lap(phi_edges)), the interior is diagonalised by DST-I in x and y,
// divided by the operator's eigenvalues, and transformed back:
//
//   phi = (2/Mx)(2/My) Sx Sy [ (Sy Sx f') / lambda ],   Mx = nx - 1, My = ny - 1,
//   lambda(k, l) = -cx 4 sin^2(pi k / 2Mx) - cy 4 sin^2(pi l / 2My).
//
// A DST-I of length N = M - 1 is read off the FFT of the odd extension of
// length 2M, which is purely imaginary: FFT(y)_k = -2i X_k.  Two rows share
// one complex FFT (the first as the real part, the second as the imaginary
// part): Z_k = -2i A_k + 2 B_k, so A_k = -Im Z_k / 2 and B_k = Re Z_k / 2.
// M must be a power of two (grids of 2^q + 1 nodes, as the multigrid's).
//
// Three kernels, each block one complex FFT of 2M points (two in k_dst_cols):
//   k_dst_rows:  interior rows, forward along x, stored transposed, T[k][j];
//   k_dst_cols:  rows of T, forward along y, divide, inverse along y, in place;
//   k_dst_back:  columns of T, inverse along x, written to the interior of phi.
// What bounds them is the chain of passes in one block, so the FFT keeps eight
// points per thread in registers and makes radix-8 passes (Stockham order: no bit
// reversal; the first pass radix 2 or 4 where 2M is no power of eight), each one
// exchange through shared memory, padded by one element in eight so that neither
// its reads nor its writes conflict: four passes for 1024 points where radix 2
// makes ten, two barriers each.  Measured on 513^2 nodes: rows 12.1 -> 6.7 us,
// columns 19.3 -> 9.2 us, back 10.7 -> 5.9 us.
#include <cmath>
#include <vector>

#include "common.cuh"

namespace pic {

struct DstDev {
    int nx, ny;    // nodes
    int Nx, Ny;    // interior nodes per direction
    int Mx, My;    // Nx + 1, Ny + 1 (powers of two)
    int px, py;    // log2(2 Mx), log2(2 My)
    double cx, cy;
    const double2* twx;  // e^{-2 pi i m / (2 Mx)}, m < Mx
    const double2* twy;
    const double* lamx;  // 4 cx sin^2(pi k / 2Mx), k = 0..Mx
    const double* lamy;
    double* T;           // Nx * Ny, T[(k-1) * Ny + (j-1)]
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }  // -i a

// Forward transforms of 2, 4 and 8 points in place, natural order.
__device__ __forceinline__ void dft2(double2& a, double2& b) {
    const double2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}
__device__ __forceinline__ void dft4(double2& a, double2& b, double2& c, double2& d) {
    const double2 s0 = cadd(a, c), s1 = csub(a, c), s2 = cadd(b, d), s3 = mul_mi(csub(b, d));
    a = cadd(s0, s2);
    c = csub(s0, s2);
    b = cadd(s1, s3);
    d = csub(s1, s3);
}
__device__ __forceinline__ void dft8(double2 (&v)[8]) {
    const double h = 0.70710678118654752440;
    double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4(e0, e1, e2, e3);
    dft4(o0, o1, o2, o3);
    o1 = make_double2(h * (o1.x + o1.y), h * (o1.y - o1.x));   // e^{-i pi/4}
    o2 = mul_mi(o2);                                           // e^{-i pi/2}
    o3 = make_double2(h * (o3.y - o3.x), -h * (o3.x + o3.y));  // e^{-3 i pi/4}
    v[0] = cadd(e0, o0);
    v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1);
    v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2);
    v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3);
    v[7] = csub(e3, o3);
}

// Shared-memory index of point i: one element of padding in eight.
__device__ __forceinline__ int pad(int i) { return i + (i >> 3); }

// Threads of a block (eight points each; at least a warp) and its shared
// memory, 2^P padded points (the twiddles come from the L1: copied to shared
// memory first they cost more than they save).
template <int P>
struct DstShape {
    static constexpr int L = 1 << P, M = L / 2, T = L / 8, THREADS = T < 32 ? 32 : T;
    static constexpr int IT = (M + THREADS - 1) / THREADS;  // points of a row per thread
    static constexpr size_t smem = sizeof(double2) * size_t(L + L / 8);
};

// Fills s with (a_n, b_n), n = 1 .. M-1, every load of a thread issued before
// its first value is used, and meets the block at a barrier.
template <int P, class A>
__device__ __forceinline__ void load_pair(double2* s, const A& at) {
    using Z = DstShape<P>;
    double2 v[Z::IT];
#pragma unroll
    for (int u = 0; u < Z::IT; ++u) {
        const int n = threadIdx.x + u * Z::THREADS;
        v[u] = n > 0 && n < Z::M ? at(n) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int u = 0; u < Z::IT; ++u) {
        const int n = threadIdx.x + u * Z::THREADS;
        if (n > 0 && n < Z::M) s[pad(n)] = v[u];
    }
    __syncthreads();
}

// The DST-I of two real rows held as s[pad(n)] = (a_n, b_n), n = 1 .. M-1, by
// the FFT of their odd extension; out(k, A_k, B_k, r) for k = t + r T = 1 .. M-1
// on thread t.  tw[m] =
// e^{-2 pi i m / L}, m < M.  The caller has met the block at a barrier after
// filling s; s may be reused after a barrier.
template <int P, class Out>
__device__ __forceinline__ void dst_pair(double2* s, const double2* __restrict__ tw, Out out) {
    constexpr int L = 1 << P, M = L / 2, T = L / 8;
    constexpr int R0 = P % 3 == 0 ? 8 : P % 3 == 1 ? 2 : 4;  // radix of the first pass
    const int t = threadIdx.x;
    const bool on = t < T;
    double2 v[8];
    // first pass: no twiddles; butterfly g of the thread takes points
    // t + T g + r L / R0, r = 0 .. R0 - 1, of the odd extension
    constexpr int B = 8 / R0;
#pragma unroll
    for (int g = 0; g < B; ++g)
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int n = t + T * g + r * (L / R0);
            double2 z = make_double2(0.0, 0.0);
            if (on && (n & (M - 1))) {
                z = s[pad(n < M ? n : L - n)];
                if (n > M) z = make_double2(-z.x, -z.y);
            }
            v[g * R0 + r] = z;
        }
    if constexpr (R0 == 8) {
        dft8(v);
    } else if constexpr (R0 == 4) {
        dft4(v[0], v[1], v[2], v[3]);
        dft4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int g = 0; g < 4; ++g) dft2(v[2 * g], v[2 * g + 1]);
    }
    if constexpr (P > 3) {
        __syncthreads();
        if (on) {
#pragma unroll
            for (int g = 0; g < B; ++g)
#pragma unroll
                for (int r = 0; r < R0; ++r) s[pad((t + T * g) * R0 + r)] = v[g * R0 + r];
        }
        __syncthreads();
#pragma unroll
        for (int ns = R0; ns < L; ns *= 8) {
            const int q = t & (ns - 1);
            if (on) {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    v[r] = s[pad(t + r * T)];
                    if (r) {
                        const int m = r * q * (L / 8 / ns);
                        const double2 w = __ldg(tw + (m & (M - 1)));
                        v[r] = cmul(v[r], m & M ? make_double2(-w.x, -w.y) : w);
                    }
                }
                dft8(v);
            }
            if (ns * 8 < L) {
                __syncthreads();
                if (on) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) s[pad((t - q) * 8 + q + r * ns)] = v[r];
                }
                __syncthreads();
            }
        }
    }
    // Z_k = -2i A_k + 2 B_k, k = t + r T
    if (on) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (t + r * T) out(t + r * T, -0.5 * v[r].y, 0.5 * v[r].x, r);
    }
}

// Interior rows (j_a, j_b) = (1 + 2 blockIdx.x, 2 + 2 blockIdx.x): forward DST
// along x of f minus the edge terms, stored transposed in T.
template <int P>
__global__ void __launch_bounds__(DstShape<P>::THREADS) k_dst_rows(DstDev D, const double* __restrict__ phi,
                                                                   const double* __restrict__ f) {
    extern __shared__ __align__(16) unsigned char smem[];
    double2* s = reinterpret_cast<double2*>(smem);
    const int ja = 1 + 2 * int(blockIdx.x), jb = ja + 1;
    const int nx = D.nx;
    const double* fa = f + long(ja) * nx;
    const bool hb = jb <= D.Ny;
    load_pair<P>(s, [&](int n) { return make_double2(fa[n], hb ? fa[nx + n] : 0.0); });
    // f' = f - lap(phi on the edges), on the interior nodes next to an edge
    if (threadIdx.x == 0) {
        const double* pa = phi + long(ja) * nx;
        double2 l = s[pad(1)], r;
        l.x -= D.cx * pa[0];
        if (hb) l.y -= D.cx * pa[nx];
        s[pad(1)] = l;
        r = s[pad(D.Nx)];
        r.x -= D.cx * pa[nx - 1];
        if (hb) r.y -= D.cx * pa[2 * nx - 1];
        s[pad(D.Nx)] = r;
    }
    __syncthreads();
    if (ja == 1 || ja == D.Ny || jb == D.Ny) {
        for (int n = 1 + threadIdx.x; n < DstShape<P>::M; n += DstShape<P>::THREADS) {
            double2 v = s[pad(n)];
            if (ja == 1) v.x -= D.cy * phi[n];
            if (ja == D.Ny) v.x -= D.cy * phi[long(ja + 1) * nx + n];
            if (jb == D.Ny) v.y -= D.cy * phi[long(jb + 1) * nx + n];
            s[pad(n)] = v;
        }
        __syncthreads();
    }
    dst_pair<P>(s, D.twx, [&](int k, double a, double b, int) {
        double* t = D.T + long(k - 1) * D.Ny + (ja - 1);
        t[0] = a;
        if (hb) t[1] = b;
    });
}

// Rows (k_a, k_b) of T: forward DST along y, divide by the eigenvalues (and
// the normalisation 4 / (Mx My)), inverse DST along y, in place.
template <int P>
__global__ void __launch_bounds__(DstShape<P>::THREADS) k_dst_cols(DstDev D) {
    extern __shared__ __align__(16) unsigned char smem[];
    double2* s = reinterpret_cast<double2*>(smem);
    const int ka = 1 + 2 * int(blockIdx.x), kb = ka + 1;
    const bool hb = kb <= D.Nx;
    double* ra = D.T + long(ka - 1) * D.Ny;
    double* rb = D.T + long(kb - 1) * D.Ny;
    load_pair<P>(s, [&](int n) { return make_double2(ra[n - 1], hb ? rb[n - 1] : 0.0); });
    const double norm = 4.0 / (double(D.Mx) * double(D.My));
    const double la = D.lamx[ka], lb = hb ? D.lamx[kb] : 1.0;
    double2 u[4];
    dst_pair<P>(s, D.twy, [&](int l, double a, double b, int r) {
        const double ly = D.lamy[l];
        u[r] = make_double2(a * norm / -(la + ly), hb ? b * norm / -(lb + ly) : 0.0);
    });
    __syncthreads();
    if (threadIdx.x < DstShape<P>::T) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int l = threadIdx.x + r * DstShape<P>::T;
            if (l) s[pad(l)] = u[r];
        }
    }
    __syncthreads();
    dst_pair<P>(s, D.twy, [&](int l, double a, double b, int) {
        ra[l - 1] = a;
        if (hb) rb[l - 1] = b;
    });
}

// Interior rows (j_a, j_b): inverse DST along x of the columns of T, written
// to the interior of phi (the edges keep their values).
template <int P>
__global__ void __launch_bounds__(DstShape<P>::THREADS) k_dst_back(DstDev D, double* __restrict__ phi) {
    extern __shared__ __align__(16) unsigned char smem[];
    double2* s = reinterpret_cast<double2*>(smem);
    const int ja = 1 + 2 * int(blockIdx.x), jb = ja + 1;
    const bool hb = jb <= D.Ny;
    load_pair<P>(s, [&](int n) {
        const double* t = D.T + long(n - 1) * D.Ny + (ja - 1);
        return make_double2(t[0], hb ? t[1] : 0.0);
    });
    dst_pair<P>(s, D.twx, [&](int i, double a, double b, int) {
        phi[long(ja) * D.nx + i] = a;
        if (hb) phi[long(jb) * D.nx + i] = b;
    });
}

// ---- host plan ------------------------------------------------------------------------

struct DstPlan {
    DstDev d{};
    std::vector<void*> allocs;
};

// Calls F::run<P>() for P = p, the log of the FFT's length (3..12).
template <class F>
static int dst_dispatch(int p, const F& f) {
    switch (p) {
        case 3: return f.template run<3>();
        case 4: return f.template run<4>();
        case 5: return f.template run<5>();
        case 6: return f.template run<6>();
        case 7: return f.template run<7>();
        case 8: return f.template run<8>();
        case 9: return f.template run<9>();
        case 10: return f.template run<10>();
        case 11: return f.template run<11>();
        case 12: return f.template run<12>();
        default: return fail(PIC_ERR_BAD_ARG, "DST solver: FFT length 2^%d", p);
    }
}

struct DstLimits {
    template <int P>
    int run() const {
        for (const void* k : {reinterpret_cast<const void*>(k_dst_rows<P>), reinterpret_cast<const void*>(k_dst_cols<P>),
                              reinterpret_cast<const void*>(k_dst_back<P>)})
            PIC_TRY(raise_smem_limit(k, DstShape<P>::smem));
        return PIC_OK;
    }
};

struct DstX {  // the rows, or the way back
    const DstDev& D;
    double* phi;
    const double* f;  // null: the way back
    cudaStream_t st;
    template <int P>
    int run() const {
        const int g = (D.Ny + 1) / 2;
        if (f) k_dst_rows<P><<<g, DstShape<P>::THREADS, DstShape<P>::smem, st>>>(D, phi, f);
        else k_dst_back<P><<<g, DstShape<P>::THREADS, DstShape<P>::smem, st>>>(D, phi);
        return PIC_OK;
    }
};

struct DstY {
    const DstDev& D;
    cudaStream_t st;
    template <int P>
    int run() const {
        k_dst_cols<P><<<(D.Nx + 1) / 2, DstShape<P>::THREADS, DstShape<P>::smem, st>>>(D);
        return PIC_OK;
    }
};

static int log2_exact(int v) {
    int p = 0;
    while ((1 << p) < v) ++p;
    return (1 << p) == v ? p : -1;
}

void dst_destroy(DstPlan* P) {
    if (!P) return;
    for (void* a : P->allocs) cudaFree(a);
    delete P;
}

// nx - 1 and ny - 1 powers of two, 4..2048.
int dst_create(int nx, int ny, double dx, double dy, DstPlan** out) {
    const int qx = log2_exact(nx - 1), qy = log2_exact(ny - 1);
    if (qx < 2 || qy < 2 || qx > 11 || qy > 11)
        return fail(PIC_ERR_BAD_ARG, "DST solver: node counts must be 2^q + 1 with 2 <= q <= 11 (got %dx%d)", nx, ny);
    DstPlan* P = new DstPlan;
    DstDev& D = P->d;
    D.nx = nx;
    D.ny = ny;
    D.Mx = nx - 1;
    D.My = ny - 1;
    D.Nx = nx - 2;
    D.Ny = ny - 2;
    D.px = qx + 1;
    D.py = qy + 1;
    D.cx = 1.0 / (dx * dx);
    D.cy = 1.0 / (dy * dy);
    const double pi = 3.14159265358979323846;
    auto upload = [&](const void* h, size_t bytes, void** d) {
        if (cudaMalloc(d, bytes) != cudaSuccess) return false;
        P->allocs.push_back(*d);
        return cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
    };
    bool ok = true;
    for (int a = 0; a < 2 && ok; ++a) {
        const int M = a ? D.My : D.Mx;
        const double c = a ? D.cy : D.cx;
        std::vector<double2> tw(static_cast<size_t>(M));
        for (int m = 0; m < M; ++m) tw[m] = make_double2(std::cos(pi * m / M), -std::sin(pi * m / M));
        std::vector<double> lam(static_cast<size_t>(M) + 1);
        for (int k = 0; k <= M; ++k) {
            const double sn = std::sin(pi * k / (2.0 * M));
            lam[k] = 4.0 * c * sn * sn;
        }
        void *dt = nullptr, *dl = nullptr;
        ok = upload(tw.data(), tw.size() * sizeof(double2), &dt) && upload(lam.data(), lam.size() * sizeof(double), &dl);
        if (a) {
            D.twy = static_cast<const double2*>(dt);
            D.lamy = static_cast<const double*>(dl);
        } else {
            D.twx = static_cast<const double2*>(dt);
            D.lamx = static_cast<const double*>(dl);
        }
    }
    if (ok) {
        void* t = nullptr;
        ok = cudaMalloc(&t, sizeof(double) * size_t(D.Nx) * D.Ny) == cudaSuccess;
        if (ok) {
            P->allocs.push_back(t);
            D.T = static_cast<double*>(t);
        }
    }
    if (!ok) {
        dst_destroy(P);
        return fail(PIC_ERR_CUDA, "DST solver: out of device memory");
    }
    int rc = dst_dispatch(D.px, DstLimits{});
    if (rc == PIC_OK) rc = dst_dispatch(D.py, DstLimits{});
    if (rc != PIC_OK) {
        dst_destroy(P);
        return rc;
    }
    *out = P;
    return PIC_OK;
}

// phi: FP64 nx*ny with the edge values set (kept); f: FP64 right-hand side.
int dst_launch(DstPlan* P, double* phi, const double* f, cudaStream_t st) {
    const DstDev& D = P->d;
    PIC_TRY(dst_dispatch(D.px, DstX{D, phi, f, st}));
    PIC_TRY(dst_dispatch(D.py, DstY{D, st}));
    PIC_TRY(dst_dispatch(D.px, DstX{D, phi, nullptr, st}));
    PIC_LAUNCH_CHECK();
    return PIC_OK;
}

}  // namespace pic
