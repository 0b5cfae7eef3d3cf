// Host side of the null-collision MCC tables and the standalone MCC operator
// behind the drop-in MCC.null_collision_method (src/MCC.py:308-415).
#include <cmath>
#include <vector>

#include "mcc_host.cuh"

namespace pic {

int grid_blocks(long n, int threads);

int mcc_build(const pic_mcc_desc* d, int nspecies, const double* mass, double dt, MccHost* H) {
    constexpr double kQe = 1.6e-19;  // src/Consts.py:1
    constexpr double kKb = 1.380649e-23;
    if (!d || nspecies < 1 || nspecies > PIC_MAX_SPECIES || !mass || !(dt > 0))
        return fail(PIC_ERR_BAD_ARG, "mcc: bad arguments");
    if (d->ne < 2 || !d->h_energy || !(d->gas_density >= 0) || !(d->gas_mass > 0) || !(d->gas_temperature >= 0))
        return fail(PIC_ERR_BAD_ARG, "mcc: bad table or gas description");
    const int ne = d->ne;
    std::vector<float> energy(ne);
    for (int j = 0; j < ne; ++j) {
        energy[j] = float(d->h_energy[j]);
        if (!(energy[j] > 0) || (j && !(energy[j] > energy[j - 1])))
            return fail(PIC_ERR_BAD_ARG, "mcc: energies must be positive and increasing");
    }
    MccDev& M = H->dev;
    M = MccDev{};
    M.ne = ne;
    M.e_lo = energy[0];
    M.e_hi = energy[ne - 1];
    M.log_e0 = logf(energy[0]);
    M.inv_log_ratio = float(double(ne - 1) / std::log(double(energy[ne - 1]) / double(energy[0])));
    M.gas_density = float(d->gas_density);
    float* de = nullptr;
    PIC_CUDA(cudaMalloc(&de, sizeof(float) * ne));
    H->allocs.push_back(de);
    PIC_CUDA(cudaMemcpy(de, energy.data(), sizeof(float) * ne, cudaMemcpyHostToDevice));
    M.energy = de;
    for (int s = 0; s < nspecies; ++s) {
        const pic_mcc_species_desc& S = d->species[s];
        MccSpeciesDev& D = M.sp[s];
        D.nproc = S.nproc;
        H->nu_max[s] = 0.0;
        H->p_null[s] = 0.0;
        if (S.nproc <= 0) continue;
        if (S.nproc > PIC_MAX_PROCESSES) return fail(PIC_ERR_BAD_ARG, "mcc: species %d has too many processes", s);
        std::vector<float> sig(size_t(S.nproc) * ne);
        for (int k = 0; k < S.nproc; ++k) {
            if (!S.h_sigma[k]) return fail(PIC_ERR_BAD_ARG, "mcc: missing table %d of species %d", k, s);
            if (S.type[k] < PIC_ELASTIC || S.type[k] > PIC_CHARGE_EXCHANGE)
                return fail(PIC_ERR_BAD_ARG, "mcc: unknown process type %d", S.type[k]);
            D.type[k] = S.type[k];
            D.thr[k] = float(S.threshold[k]);
            for (int j = 0; j < ne; ++j) sig[size_t(k) * ne + j] = float(S.h_sigma[k][j]);
            if (S.type[k] == PIC_IONIZATION &&
                (S.born_electron_species < 0 || S.born_electron_species >= nspecies || S.born_ion_species < 0 ||
                 S.born_ion_species >= nspecies))
                return fail(PIC_ERR_BAD_ARG, "mcc: ionisation products of species %d out of range", s);
        }
        float* ds = nullptr;
        PIC_CUDA(cudaMalloc(&ds, sizeof(float) * sig.size()));
        H->allocs.push_back(ds);
        PIC_CUDA(cudaMemcpy(ds, sig.data(), sizeof(float) * sig.size(), cudaMemcpyHostToDevice));
        D.sigma = ds;
        D.half_m_over_q = float(0.5 * mass[s] / kQe);
        D.mass_ratio2 = float(2.0 * mass[s] / d->gas_mass);
        D.gas_vth = float(std::sqrt(kKb * d->gas_temperature / d->gas_mass));
        D.born_e = S.born_electron_species;
        D.born_i = S.born_ion_species;
        // nu' bounds n_g sigma_T(E) v(E) on every table interval (sigma is
        // linear in E there and v grows with E), from the float tables the
        // device interpolates.
        double numax = 0.0;
        for (int j = 0; j + 1 < ne; ++j) {
            double s0 = 0.0, s1 = 0.0;
            for (int k = 0; k < S.nproc; ++k) {
                s0 += sig[size_t(k) * ne + j];
                s1 += sig[size_t(k) * ne + j + 1];
            }
            const double v1 = std::sqrt(double(energy[j + 1]) / double(D.half_m_over_q));
            numax = std::max(numax, std::max(s0, s1) * v1);
        }
        numax *= double(d->gas_density) * (1.0 + 1e-5);
        D.nu_max = float(numax);
        if (D.nu_max > 0) {
            D.inv_log1m_p = -1.0 / (double(D.nu_max) * dt);
            H->p_null[s] = -std::expm1(-double(D.nu_max) * dt);
        } else {
            D.nproc = 0;
        }
        H->nu_max[s] = double(D.nu_max);
    }
    return PIC_OK;
}

void mcc_free(MccHost* H) {
    for (void* p : H->allocs) cudaFree(p);
    H->allocs.clear();
}

// The collision operator on its own.  What bounds it is the chain of one
// candidate (draws, the bin's table loads, Philox rounds, the scattering), so
// the block gives every thread a segment to draw and then every thread a
// candidate, however the candidates fall on the segments: `segs` segments of 256
// slots per block, the candidates numbered by a scan of the segments' counts.
// Counts are summed in shared memory first.  (One lane in sixteen drawing, the
// block then stepping over its slots: 20.5 us for 4M electrons; this way 8.5 us.)
// segs (mcc_segments): as many as a block has threads where few slots collide; in
// a dense gas only so many that a thread has kMccPerThread candidates on average,
// but never so few that the blocks (kMccResident to an SM) make a second wave, as
// drawing then leaves most of a block idle.  Measured, with 128 segments and by
// this rule: a candidate in two slots, 200k electrons 382 and 80 us, 1M 383 and 93,
// 16M 503 and 327; one in fifteen, 200k 77 and 33; one in 400, 4M 24 and 24.
constexpr int kMccBlockSegments = 128;  // most segments of a block, and its threads
constexpr int kMccPerThread = 2, kMccResident = 7;
constexpr int kMccWords = int(kMccSegment) / 32;

__global__ void __launch_bounds__(kMccBlockSegments) k_mcc_apply(const __grid_constant__ MccDev M, int s,
                                                                 const float* __restrict__ x,
                                                                 const float* __restrict__ y, float* __restrict__ vx,
                                                                 float* __restrict__ vy, float* __restrict__ vz, int n,
                                                                 uint32_t step, uint2 key, BirthDev B, int segs,
                                                                 unsigned long long* __restrict__ ctr) {
    __shared__ unsigned bits[kMccBlockSegments * (kMccWords + 1)];  // a segment's words, padded against bank conflicts
    __shared__ int first[kMccBlockSegments + 1];                    // the number of each segment's first candidate
    __shared__ int warp_tot[kMccBlockSegments / 32];
    __shared__ unsigned cnt[PIC_MAX_PROCESSES + 3];  // collisions, candidates, overflows, dropped births
    const MccSpeciesDev& S = M.sp[s];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const long g = long(blockIdx.x) * segs + t;
    unsigned* mine = bits + t * (kMccWords + 1);
#pragma unroll
    for (int q = 0; q < kMccWords; ++q) mine[q] = 0u;
    if (t < PIC_MAX_PROCESSES + 3) cnt[t] = 0u;
    const long b = g * long(kMccSegment);
    if (t < segs && b < n)
        mcc_mark_segment(S, uint32_t(s), g, n, int(b), int(min(long(n), b + long(kMccSegment))), step, key, mine);
    int c = 0;
#pragma unroll
    for (int q = 0; q < kMccWords; ++q) c += __popc(mine[q]);
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    int before = 0;
    for (int q = 0; q < w; ++q) before += warp_tot[q];
    first[t] = before + incl - c;
    if (t == kMccBlockSegments - 1) first[kMccBlockSegments] = before + incl;
    __syncthreads();
    const int total = first[kMccBlockSegments];
    for (int k = t; k < total; k += kMccBlockSegments) {
        int lo = 0, hi = segs - 1;  // the last segment whose first candidate is <= k
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first[mid] <= k) lo = mid;
            else hi = mid - 1;
        }
        // the (k - first)-th set bit of its words
        int r = k - first[lo], q = 0;
        const unsigned* words = bits + lo * (kMccWords + 1);
        while (r >= __popc(words[q])) r -= __popc(words[q++]);
        const int p = int((long(blockIdx.x) * segs + lo) * long(kMccSegment)) + 32 * q +
                      int(__fns(words[q], 0u, r + 1));
        const float px = x[p], py = y[p];
        if (!is_live(px)) continue;
        atomicAdd(&cnt[PIC_MAX_PROCESSES], 1u);
        float a = vx[p], d = vy[p], e = vz[p];
        const MccOutcome o = mcc_collide(M, S, uint32_t(s), uint32_t(p), step, key, a, d, e);
        if (o.overflow) atomicAdd(&cnt[PIC_MAX_PROCESSES + 1], 1u);
        if (o.proc < 0) continue;
        atomicAdd(&cnt[o.proc], 1u);
        vx[p] = a;
        vy[p] = d;
        vz[p] = e;
        if (o.born) {
            const bool ok_e = birth_push(B, S.born_e, px, py, o.be[0], o.be[1], o.be[2]);
            const bool ok_i = birth_push(B, S.born_i, px, py, o.bi[0], o.bi[1], o.bi[2]);
            if (!ok_e || !ok_i) atomicAdd(&cnt[PIC_MAX_PROCESSES + 2], 1u);
        }
    }
    __syncthreads();
    if (t < PIC_MAX_PROCESSES + 3 && cnt[t]) {
        const int at = t < PIC_MAX_PROCESSES        ? kCtrCollisions + s * PIC_MAX_PROCESSES + t
                       : t == PIC_MAX_PROCESSES     ? kCtrCandidates + s
                       : t == PIC_MAX_PROCESSES + 1 ? kCtrOverflow
                                                    : kCtrDropped;
        atomicAdd(ctr + at, (unsigned long long)cnt[t]);
    }
}

// Segments of a block of k_mcc_apply.
static int mcc_segments(int n, double p) {
    const double one_wave = double(n) / (double(kMccSegment) * kMccResident * num_sms());
    int segs = kMccBlockSegments;
    while (segs > 1 && segs / 2 >= one_wave &&
           segs * double(kMccSegment) * p > kMccPerThread * double(kMccBlockSegments))
        segs /= 2;
    return segs;
}

}  // namespace pic

struct pic_mcc {
    pic::MccHost h;
    int nspecies = 0;
};

using namespace pic;

extern "C" {

int pic_mcc_create(const pic_mcc_desc* desc, int nspecies, const double* species_mass, double dt, pic_mcc** out) {
    clear_error();
    if (!out) return fail(PIC_ERR_BAD_ARG, "pic_mcc_create: out is NULL");
    pic_mcc* m = new pic_mcc;
    m->nspecies = nspecies;
    const int st = mcc_build(desc, nspecies, species_mass, dt, &m->h);
    if (st != PIC_OK) {
        mcc_free(&m->h);
        delete m;
        return st;
    }
    *out = m;
    return PIC_OK;
}

int pic_mcc_destroy(pic_mcc* m) {
    clear_error();
    if (!m) return PIC_OK;
    mcc_free(&m->h);
    delete m;
    return PIC_OK;
}

int pic_mcc_query(pic_mcc* m, int s, double* nu_max, double* p_null, double* inv_log1m_p) {
    clear_error();
    if (!m || s < 0 || s >= m->nspecies) return fail(PIC_ERR_BAD_ARG, "pic_mcc_query: bad arguments");
    if (nu_max) *nu_max = double(m->h.dev.sp[s].nu_max);
    if (p_null) *p_null = m->h.p_null[s];
    if (inv_log1m_p) *inv_log1m_p = m->h.dev.sp[s].inv_log1m_p;
    return PIC_OK;
}

int pic_mcc_apply(pic_mcc* m, int s, const float* d_x, const float* d_y, float* d_vx, float* d_vy, float* d_vz, int n,
                  unsigned long long seed, unsigned int step, const pic_birth_buffer* births,
                  unsigned long long* d_counters, void* stream) {
    clear_error();
    if (!m || s < 0 || s >= m->nspecies || n < 0 || !d_counters || !births || !births->count ||
        (n > 0 && (!d_x || !d_y || !d_vx || !d_vy || !d_vz)))
        return fail(PIC_ERR_BAD_ARG, "pic_mcc_apply: bad arguments");
    if (n == 0 || m->h.dev.sp[s].nproc == 0) return PIC_OK;
    BirthDev B{births->x, births->y, births->vx, births->vy, births->vz, births->species, births->count,
               births->capacity};
    const uint2 key = make_uint2(uint32_t(seed), uint32_t(seed >> 32));
    const int segs = mcc_segments(n, m->h.p_null[s]);
    const int blocks = div_up(n, long(segs) * kMccSegment);
    k_mcc_apply<<<blocks, kMccBlockSegments, 0, as_stream(stream)>>>(m->h.dev, s, d_x, d_y, d_vx, d_vy, d_vz, n, step,
                                                                     key, B, segs, d_counters);
    PIC_LAUNCH_CHECK();
    return PIC_OK;
}

}  // extern "C"
