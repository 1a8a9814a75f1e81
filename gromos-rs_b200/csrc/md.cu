// md.cu -- MD steps around the force evaluation, device resident.
//
// One step is the sequence of gromos-md's md binary (md.rs:1144-1230) without
// thermostat: Forcefield::apply (the nonbonded path of this library) at r(t),
// leap-frog velocity v(t+dt/2) = v(t-dt/2) + F/m dt (leap_frog.rs:37-85),
// leap-frog position r(t+dt) = r(t) + v dt (leap_frog.rs:116-148) and SETTLE
// for every 3-site solvent molecule (constraints.rs:815-1010).  Positions,
// velocities and forces never leave the device between steps.
//
// Overflow recovery: list overflows (pairlist capacity, deferred water pairs)
// are detected after the fact from the device error flags.  The runner keeps
// a device snapshot of (positions, velocities) at the start of every block of
// pairlist periods (a period is the steps between two rebuilds), reads the
// flags at the end of the block, and on overflow grows the lists, restores
// the snapshot and runs the block again, so an overflow never leaks into the
// trajectory.
#include <cuda_runtime.h>

namespace gnb {

struct MdDev {
    double* vel;              // n_atoms*3
    const double* inv_mass;   // n_atoms
    const double* mass;       // n_atoms
    double dt, dt_i;
    int settle;               // SETTLE every solvent molecule
    double m_o, m_h, im_o, im_h, ra, rb, rc;  // canonical SETTLE triangle (constraints.rs:836-840)
    long long* ke;            // [5]: [0] kinetic energy of the velocities entering the step, [1] accumulator
                              // of the velocities leaving it (fixed point 2^24), [2] blocks finished,
                              // [3] excluded energies and [4] largest extent of the next step's records
    int* failures;            // [1] molecules SETTLE could not solve
    const double* t0;         // [1] Berendsen bath temperature (device memory: a replica exchange changes it
                              // without touching recorded graphs)
    double tau, dof;          // Berendsen bath (tau < 0: none)
    int prep_next;            // also write the next step's water records (SETTLE units, no rebuild next)
};

// Berendsen weak coupling (berendsen_thermostat.rs:74-98): lambda from the
// kinetic energy of the velocities entering this step.
__device__ __forceinline__ double berendsen_lambda(const MdDev& md) {
    if (md.tau < 0.0) return 1.0;
    const double kB = 0.00831446261815324;
    const double ekin = double(md.ke[0]) / kEnergyScale;
    const double t0 = *md.t0;
    double t = md.dof > 0.0 ? 2.0 * ekin / (md.dof * kB) : 0.0;
    if (t < 1e-10) t = t0;
    if (t < 1e-10) return 1.0;
    return md.tau == 0.0 ? sqrt(t0 / t) : sqrt(1.0 + md.dt / md.tau * (t0 / t - 1.0));
}

// Velocities scaled by `f` (temperature exchange), kinetic energy with them.
__global__ void k_scale_velocities(double* __restrict__ vel, int n3, double f, long long* ke) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) vel[i] *= f;
    if (blockIdx.x == 0 && threadIdx.x == 0) ke[0] = __double2ll_rn(double(ke[0]) * f * f);
}

struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 d3(double x, double y, double z) { return {x, y, z}; }
__device__ __forceinline__ D3 operator-(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3 operator+(D3 a, D3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3 operator*(D3 a, double s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ double dot3(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 cross3(D3 a, D3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// SETTLE for one molecule (Miyamoto & Kollman 1992, eqs. A3-A17): the frame
// is spanned by the old molecular plane and the new centre of mass; the
// three rotation sines are solved analytically.  Velocities receive the
// displacement / dt.  Returns false (molecule left unconstrained, as the
// reference does) when a sine leaves [-1, 1].
__device__ bool settle_molecule(const D3 old[3], D3 nw[3], D3 v[3], const MdDev& md) {
    D3 b0 = old[1] - old[0], c0 = old[2] - old[0];
    const double mt_i = 1.0 / (md.m_o + 2.0 * md.m_h);
    const D3 d0 = (nw[0] * md.m_o + nw[1] * md.m_h + nw[2] * md.m_h) * mt_i;
    D3 a1 = nw[0] - d0, b1 = nw[1] - d0, c1 = nw[2] - d0;
    D3 n0 = cross3(b0, c0);
    D3 n1 = cross3(a1, n0);
    D3 n2 = cross3(n0, n1);
    n0 = n0 * rsqrt(dot3(n0, n0));
    n1 = n1 * rsqrt(dot3(n1, n1));
    n2 = n2 * rsqrt(dot3(n2, n2));
    b0 = d3(dot3(n1, b0), dot3(n2, b0), dot3(n0, b0));
    c0 = d3(dot3(n1, c0), dot3(n2, c0), dot3(n0, c0));
    a1 = d3(dot3(n1, a1), dot3(n2, a1), dot3(n0, a1));
    b1 = d3(dot3(n1, b1), dot3(n2, b1), dot3(n0, b1));
    c1 = d3(dot3(n1, c1), dot3(n2, c1), dot3(n0, c1));
    const double sinphi = a1.z / md.ra;
    const double omp = 1.0 - sinphi * sinphi;
    if (omp < 0.0) return false;
    const double cosphi = sqrt(omp);
    const double sinpsi = (b1.z - c1.z) / (2.0 * md.rc * cosphi);
    const double omq = 1.0 - sinpsi * sinpsi;
    if (omq < 0.0) return false;
    const double cospsi = sqrt(omq);
    const double y_a2 = md.ra * cosphi, x_b2 = -md.rc * cospsi;
    const double y_b2 = -md.rb * cosphi - md.rc * sinpsi * sinphi;
    const double y_c2 = -md.rb * cosphi + md.rc * sinpsi * sinphi;
    const double alpha = x_b2 * (b0.x - c0.x) + b0.y * y_b2 + c0.y * y_c2;
    const double beta = x_b2 * (c0.y - b0.y) + b0.x * y_b2 + c0.x * y_c2;
    const double gamma = b0.x * b1.y - b1.x * b0.y + c0.x * c1.y - c1.x * c0.y;
    const double ab2 = alpha * alpha + beta * beta;
    const double disc = ab2 - gamma * gamma;
    if (disc < 0.0) return false;
    const double sintheta = (alpha * gamma - beta * sqrt(disc)) / ab2;
    const double omt = 1.0 - sintheta * sintheta;
    if (omt < 0.0) return false;
    const double costheta = sqrt(omt);
    const D3 r3[3] = {d3(-y_a2 * sintheta, y_a2 * costheta, a1.z),
                      d3(x_b2 * costheta - y_b2 * sintheta, x_b2 * sintheta + y_b2 * costheta, b1.z),
                      d3(-x_b2 * costheta - y_c2 * sintheta, -x_b2 * sintheta + y_c2 * costheta, c1.z)};
    // back to the lab frame: rows of the transposed basis
    const D3 m1 = d3(n1.x, n2.x, n0.x), m2 = d3(n1.y, n2.y, n0.y), m0 = d3(n1.z, n2.z, n0.z);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const D3 p = d3(dot3(r3[k], m1), dot3(r3[k], m2), dot3(r3[k], m0)) + d0;
        const D3 d = p - nw[k];
        nw[k] = p;
        v[k] = v[k] + d * md.dt_i;
    }
    return true;
}

// One thread per unit: a solute atom (leap-frog only) or a solvent molecule
// (leap-frog of its atoms, then SETTLE).
//
// FUSED (the fixed-point kernel): the step is also its evaluation's k_finalize.
// Each unit takes its forces from the fixed-point sums, writes the FP64
// forces, clears what it read and moves on with them; the last block to finish
// does the energies and the counters.  Separately the two kernels cost a launch
// and two latencies per step, which is most of them for a few thousand waters
// (1,000: 12.6 + 4.7 us, fused 12.4, ncu; 20 steps 1,328 -> 1,240 us).
// Without it (the plain kernel) the forces are those that k_finalize wrote.
//
// With prep_next the kernel also does the next evaluation's k_water_prep for
// each molecule from its new coordinates (same record, same cleared force
// sums, same excluded energies and extent; the slots are those of the current
// lists, so only when the next step keeps them): the next evaluation then
// skips k_water_prep.  Their energies and extent wait in ke[3] and ke[4] until
// the last block has read this step's accumulators.
struct MdUnit {
    long long ke;
    double e_excl;
    float m_ext;
};

// Forces of atom a: the fixed-point sums (cleared where nothing else clears
// them) or the finalized ones.  `sl` are the water's short and long slot sums
// of its first component, null for solute atoms.
template <bool FUSED>
__device__ __forceinline__ D3 md_force(const SysDev& s, double* __restrict__ f_out, int a, const long long* ws,
                                       const long long* wl, bool pa, bool twin) {
    if (!FUSED) return d3(f_out[3 * a], f_out[3 * a + 1], f_out[3 * a + 2]);
    long long f[3] = {0, 0, 0};
    if (pa) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            f[k] = s.f_short[3 * a + k];
            if (twin) f[k] += s.f_long[3 * a + k];
        }
    }
    if (ws) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            f[k] += ws[k];
            if (twin) f[k] += wl[k];
        }
    }
    const double inv = 1.0 / kForceScale;
    return d3(double(f[0]) * inv, double(f[1]) * inv, double(f[2]) * inv);
}

template <bool FUSED>
__device__ __forceinline__ void md_store(const SysDev& s, const MdDev& md, double* __restrict__ f_out, int a, D3 f, D3 x,
                                         D3 v, double mass, bool pa, long long& ke) {
    if (FUSED) {
        f_out[3 * a] = f.x;
        f_out[3 * a + 1] = f.y;
        f_out[3 * a + 2] = f.z;
        if (pa) s.f_short[3 * a] = s.f_short[3 * a + 1] = s.f_short[3 * a + 2] = 0;
    }
    s.pos[3 * a] = x.x;
    s.pos[3 * a + 1] = x.y;
    s.pos[3 * a + 2] = x.z;
    md.vel[3 * a] = v.x;
    md.vel[3 * a + 1] = v.y;
    md.vel[3 * a + 2] = v.z;
    ke += to_fixed_d(0.5 * mass * dot3(v, v), kEnergyScale);
}

// NA atoms from a0 (1: an atom, 3: a molecule that SETTLE constrains).
template <bool FUSED, int NA>
__device__ __forceinline__ void md_unit(const SysDev& s, const MdDev& md, int a0, double lambda, MdUnit& r) {
    double* __restrict__ f_out = s.f_out;
    const int nsa = s.n_solute_atoms, nscg = s.n_solute_cg;
    const bool twin = s.twin != 0, water = a0 >= nsa;
    // a water atom's per-atom sums hold something only when solute kernels,
    // excluded pairs or perturbation terms reach water atoms (as in k_finalize)
    const bool pa = !water || nscg > 0 || s.excl_atoms > nsa || s.n_pert > 0 || s.n_pp > 0;
    const bool rec = NA == 3 && md.prep_next;
    const int w = water ? (a0 - nsa) / 3 : 0;
    const int slot = water && (FUSED || rec) ? s.cg_slot[nscg + w] : -1;
    const long long *ws = nullptr, *wl = nullptr;
    if (FUSED && slot >= 0) {
        const size_t o = static_cast<size_t>(slot) * 9 + 3 * (a0 - nsa - 3 * w);
        ws = s.fs_short + o;
        wl = s.fs_long + o;
    }
    const bool excl = s.excl_atoms < s.n_atoms;
    double q3[3] = {0.0, 0.0, 0.0};
    D3 f[NA], old[NA], nw[NA], v[NA];
    double mass[NA];
#pragma unroll
    for (int k = 0; k < NA; ++k) {
        const int i = a0 + k;
        f[k] = md_force<FUSED>(s, f_out, i, ws ? ws + 3 * k : nullptr, wl ? wl + 3 * k : nullptr, pa, twin);
        if (rec && excl) q3[k] = s.charge[i];
        const double im = md.inv_mass[i];
        mass[k] = md.mass[i];
        v[k] = (d3(md.vel[3 * i], md.vel[3 * i + 1], md.vel[3 * i + 2]) + f[k] * im * md.dt) * lambda;
        old[k] = d3(s.pos[3 * i], s.pos[3 * i + 1], s.pos[3 * i + 2]);
        nw[k] = old[k] + v[k] * md.dt;
    }
    if constexpr (NA == 3) {
        if (!settle_molecule(old, nw, v, md)) atomicAdd(md.failures, 1);
        if (rec && slot >= 0) {
            const double p[9] = {nw[0].x, nw[0].y, nw[0].z, nw[1].x, nw[1].y, nw[1].z, nw[2].x, nw[2].y, nw[2].z};
            water_record(s, slot, p, q3, excl, r.e_excl, r.m_ext);
        }
    }
#pragma unroll
    for (int k = 0; k < NA; ++k) md_store<FUSED>(s, md, f_out, a0 + k, f[k], nw[k], v[k], mass[k], pa, r.ke);
}

// The end of a step kernel: the block's sums and, by the last block to finish,
// the step's energies and the counters.  Every thread of every block calls it.
template <bool FUSED>
__device__ __forceinline__ void md_step_end(const SysDev& s, const MdDev& md, const MdUnit& r) {
    // per-block sums: kinetic energy, the records' energies and extent
    __shared__ unsigned long long sh[2];
    __shared__ int mx, last;
    if (threadIdx.x == 0) {
        sh[0] = sh[1] = 0ull;
        mx = 0;
    }
    __syncthreads();
    const long long ke = warp_sum_ll(r.ke);
    if ((threadIdx.x & 31) == 0 && ke) atomicAdd(&sh[0], static_cast<unsigned long long>(ke));
    if (md.prep_next) {
        const long long ex = warp_sum_ll(to_fixed_d(r.e_excl, kEnergyScale));
        const int m = __reduce_max_sync(0xffffffffu, __float_as_int(r.m_ext));  // extents are >= 0: ordered as ints
        if ((threadIdx.x & 31) == 0) {
            if (ex) atomicAdd(&sh[1], static_cast<unsigned long long>(ex));
            if (m) atomicMax(&mx, m);
        }
    }
    __syncthreads();
    unsigned long long* acc = reinterpret_cast<unsigned long long*>(md.ke);
    if (threadIdx.x == 0) {
        if (sh[0]) atomicAdd(acc + 1, sh[0]);
        if (sh[1]) atomicAdd(acc + 3, sh[1]);
        if (mx) atomicMax(reinterpret_cast<int*>(acc + 4), mx);
        __threadfence();
        last = atomicAdd(acc + 2, 1ull) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // The last block to finish makes the accumulated kinetic energy the next
    // step's input (every block read ke[0] for its bath factor before adding),
    // and finalizes the step's energies.
    __threadfence();
    const int G = s.n_egroups, gs = s.solvent_group < 0 ? 0 : s.solvent_group;
    const int i_excl = G * G + gs * G + gs;
    const long long next_excl = md.prep_next ? static_cast<long long>(__ldcg(acc + 3)) : 0ll;
    if (FUSED) {
        for (int i = threadIdx.x; i < acc_size(G); i += blockDim.x) {
            double e = double(s.acc_short[i]) / kEnergyScale;
            if (s.twin) e += double(s.acc_long[i]) / kEnergyScale;
            s.e_out[i] = e;
            s.acc_short[i] = i == i_excl ? next_excl : 0ll;
        }
    } else if (threadIdx.x == 0 && next_excl) {
        s.acc_short[i_excl] += next_excl;
    }
    __syncthreads();  // next_excl read by every thread
    if (threadIdx.x == 0) {
        md.ke[0] = static_cast<long long>(__ldcg(acc + 1));
        const int m = __ldcg(reinterpret_cast<int*>(acc + 4));
        if (s.max_delta) *s.max_delta = md.prep_next ? __int_as_float(m) : 0.f;
        md.ke[1] = md.ke[2] = md.ke[3] = md.ke[4] = 0;
        if (FUSED)
            for (int k = 0; k < 6; ++k) s.n_deferred[k] = 0;
    }
}

template <bool FUSED>
__global__ void __launch_bounds__(128) k_md_step(const SysDev* __restrict__ sys, MdDev md) {
    pdl_wait();
    pdl_trigger();
    const SysDev& s = *sys;
    const int nsa = s.n_solute_atoms, n = s.n_atoms;
    const int n_units = md.settle ? nsa + (n - nsa) / 3 : n;
    const double lambda = berendsen_lambda(md);
    MdUnit r{0, 0.0, 0.f};
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n_units; u += gridDim.x * blockDim.x) {
        if (md.settle && u >= nsa)
            md_unit<FUSED, 3>(s, md, nsa + 3 * (u - nsa), lambda, r);
        else
            md_unit<FUSED, 1>(s, md, u, lambda, r);
    }
    md_step_end<FUSED>(s, md, r);
}

constexpr int kTile = 128;

// The fused step with SETTLE for a system that fills the chip (md_step_launch):
// a block takes kTile molecules, whose positions, velocities and force sums come
// in component by component, neighbouring threads on neighbouring addresses, and go
// through shared memory to the molecule's thread and back.  There a thread
// that reads its molecule's 72-byte rows itself touches a sector per lane with
// every load, and these set the time; a smaller system's time is the latency
// of one molecule, to which the tile only adds barriers.  All loads of a
// stage are issued before its first store, which they might alias.
__global__ void __launch_bounds__(kTile) k_md_step_tiled(const SysDev* __restrict__ sys, MdDev md) {
    pdl_wait();
    pdl_trigger();
    const SysDev& s = *sys;
    const int nsa = s.n_solute_atoms, nscg = s.n_solute_cg, n_mol = (s.n_atoms - nsa) / 3;
    const bool twin = s.twin != 0, excl = s.excl_atoms < s.n_atoms;
    const bool pa = nscg > 0 || s.excl_atoms > nsa || s.n_pert > 0 || s.n_pp > 0;  // as in md_unit
    const double lambda = berendsen_lambda(md);
    const double inv = 1.0 / kForceScale;
    MdUnit r{0, 0.0, 0.f};
    for (int u = blockIdx.x * kTile + threadIdx.x; u < nsa; u += gridDim.x * kTile)
        md_unit<true, 1>(s, md, u, lambda, r);
    __shared__ double sx[kTile * 9], sv[kTile * 9], sf[kTile * 9];
    __shared__ int sslot[kTile];
    double* f_out = s.f_out;
    double* pos = s.pos;
    double* vel = md.vel;
    const int t = threadIdx.x;
    for (int base = blockIdx.x * kTile; base < n_mol; base += gridDim.x * kTile) {
        const int cnt = min(kTile, n_mol - base);
        const int i0 = 3 * (nsa + 3 * base);  // the tile's first component
        if (t < cnt) sslot[t] = s.cg_slot[nscg + base + t];
        double x[9], v9[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int c = t + k * kTile;
            x[k] = c < 9 * cnt ? pos[i0 + c] : 0.0;
            v9[k] = c < 9 * cnt ? vel[i0 + c] : 0.0;
        }
        __syncthreads();
        long long f[9], g[9];
        size_t o[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int c = t + k * kTile, m = c / 9;
            const int slot = c < 9 * cnt ? sslot[m] : -1;
            o[k] = static_cast<size_t>(slot) * 9 + (c - 9 * m);
            f[k] = slot >= 0 ? s.fs_short[o[k]] : 0;
            g[k] = slot >= 0 && twin ? s.fs_long[o[k]] : 0;
            if (slot < 0) o[k] = ~size_t(0);
        }
        if (pa) {
            long long p[9], q[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const int c = t + k * kTile;
                p[k] = c < 9 * cnt ? s.f_short[i0 + c] : 0;
                q[k] = c < 9 * cnt && twin ? s.f_long[i0 + c] : 0;
            }
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const int c = t + k * kTile;
                f[k] += p[k] + q[k];
                if (c < 9 * cnt) s.f_short[i0 + c] = 0;
            }
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int c = t + k * kTile;
            if (c >= 9 * cnt) continue;
            const double fc = double(f[k] + g[k]) * inv;
            sx[c] = x[k];
            sv[c] = v9[k];
            sf[c] = fc;
            f_out[i0 + c] = fc;
            if (md.prep_next && o[k] != ~size_t(0)) s.fs_short[o[k]] = 0;  // for the records written below
        }
        __syncthreads();
        if (t < cnt) {
            D3 old[3], nw[3], v[3];
            const double im[3] = {md.im_o, md.im_h, md.im_h}, mass[3] = {md.m_o, md.m_h, md.m_h};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int c = 9 * t + 3 * k;
                v[k] = (d3(sv[c], sv[c + 1], sv[c + 2]) + d3(sf[c], sf[c + 1], sf[c + 2]) * im[k] * md.dt) * lambda;
                old[k] = d3(sx[c], sx[c + 1], sx[c + 2]);
                nw[k] = old[k] + v[k] * md.dt;
            }
            if (!settle_molecule(old, nw, v, md)) atomicAdd(md.failures, 1);
            const int slot = sslot[t];
            if (md.prep_next && slot >= 0) {
                double q3[3] = {0.0, 0.0, 0.0};
                if (excl)
#pragma unroll
                    for (int k = 0; k < 3; ++k) q3[k] = s.charge[nsa + 3 * (base + t) + k];
                const double p[9] = {nw[0].x, nw[0].y, nw[0].z, nw[1].x, nw[1].y, nw[1].z, nw[2].x, nw[2].y, nw[2].z};
                water_record<false>(s, slot, p, q3, excl, r.e_excl, r.m_ext);
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int c = 9 * t + 3 * k;
                sx[c] = nw[k].x;
                sx[c + 1] = nw[k].y;
                sx[c + 2] = nw[k].z;
                sv[c] = v[k].x;
                sv[c + 1] = v[k].y;
                sv[c + 2] = v[k].z;
                r.ke += to_fixed_d(0.5 * mass[k] * dot3(v[k], v[k]), kEnergyScale);
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int c = t + k * kTile;
            if (c >= 9 * cnt) continue;
            pos[i0 + c] = sx[c];
            vel[i0 + c] = sv[c];
        }
        __syncthreads();  // the next tile reuses the buffers
    }
    md_step_end<true>(s, md, r);
}

}  // namespace gnb

using namespace gnb;

gr_status NbSystem::md_init(const double* mass, const double* vel, const gr_md_params* p) {
    prepped_next = false;
    if (!uploaded) {
        set_error("gr_md_init before gr_system_upload");
        return GR_ERR_STATE;
    }
    if (!mass || !p) {
        set_error("gr_md_init: null mass or params");
        return GR_ERR_INVALID;
    }
    if (!(p->dt > 0.0)) {
        set_error("gr_md_init: dt must be positive");
        return GR_ERR_INVALID;
    }
    for (int i = 0; i < N; ++i)
        if (!(mass[i] > 0.0)) {
            set_error("gr_md_init: every mass must be positive");
            return GR_ERR_INVALID;
        }
    const bool settle = p->settle != 0 && N > NSA;
    if (settle) {
        if (aps != 3 || (N - NSA) % 3 != 0) {
            set_error("gr_md_init: SETTLE needs 3-site solvent molecules");
            return GR_ERR_UNSUPPORTED;
        }
        for (int i = NSA; i < N; i += 3)
            if (mass[i] != mass[NSA] || mass[i + 1] != mass[NSA + 1] || mass[i + 2] != mass[NSA + 1]) {
                set_error("gr_md_init: SETTLE needs one solvent with equal masses of sites 1 and 2");
                return GR_ERR_UNSUPPORTED;
            }
        if (!(p->dist_oh > 0.0) || !(p->dist_hh > 0.0) || !(p->dist_hh < 2.0 * p->dist_oh)) {
            set_error("gr_md_init: SETTLE lengths must satisfy 0 < dist_hh < 2 dist_oh");
            return GR_ERR_INVALID;
        }
    }
    std::vector<double> inv(N);
    for (int i = 0; i < N; ++i) inv[i] = 1.0 / mass[i];
    std::vector<double> v0(size_t(N) * 3, 0.0);
    if (vel) std::copy(vel, vel + size_t(N) * 3, v0.begin());
    gr_status st;
    if ((st = upload_array(&md_mass, mass, N)) || (st = upload_array(&md_inv_mass, inv.data(), N)) ||
        (st = upload_array(&md_vel, v0.data(), size_t(N) * 3)) || (st = alloc(&md_pos_snap, size_t(N) * 3)) ||
        (st = alloc(&md_vel_snap, size_t(N) * 3)) || (st = alloc(&md_ke, 5)) || (st = alloc(&md_ke_snap, 1)) ||
        (st = alloc(&md_psnap_pos, size_t(N) * 3)) || (st = alloc(&md_psnap_vel, size_t(N) * 3)) ||
        (st = alloc(&md_psnap_ke, 1)) || (st = alloc(&md_fail, 1)) || (st = alloc(&md_t0, 1)))
        return st;
    GR_CUDA(cudaMemcpy(md_t0, &p->temperature, sizeof(double), cudaMemcpyHostToDevice));
    {
        double ke0 = 0.0;
        for (int i = 0; i < N; ++i)
            ke0 += 0.5 * mass[i] * (v0[3 * i] * v0[3 * i] + v0[3 * i + 1] * v0[3 * i + 1] + v0[3 * i + 2] * v0[3 * i + 2]);
        const long long k[5] = {static_cast<long long>(std::llround(ke0 * kEnergyScale)), 0, 0, 0, 0};
        GR_CUDA(cudaMemcpy(md_ke, k, sizeof(k), cudaMemcpyHostToDevice));
    }
    GR_CUDA(cudaMemset(md_fail, 0, sizeof(int)));
    md_steps_total = 0;
    md_rollbacks = 0;
    md_step_idx = 0;
    md_psnap_valid = false;
    // an MD run starts a pairlist period with a build at its first step
    built = false;
    lr_computed = false;
    if (!md_err_host) GR_CUDA(pinned_alloc(&md_err_host, 8));
    if (!ev_md) GR_CUDA(cudaEventCreateWithFlags(&ev_md, cudaEventDisableTiming));
    mdp = *p;
    md_settle = settle;
    // degrees of freedom: 3N minus the solvent constraints (md.rs:1158-1172; NDFMIN 0)
    md_dof = 3.0 * N - (settle ? 3.0 * ((N - NSA) / 3) : 0.0);
    if (settle) {  // canonical triangle (constraints.rs:836-840)
        md_m_o = mass[NSA];
        md_m_h = mass[NSA + 1];
        const double half_mo_div_mh = 0.5 * md_m_o / md_m_h;
        md_rc = 0.5 * p->dist_hh;
        md_ra = std::sqrt(p->dist_oh * p->dist_oh - md_rc * md_rc) / (1.0 + half_mo_div_mh);
        md_rb = half_mo_div_mh * md_ra;
    }
    md_ready = true;
    return GR_OK;
}

// One MD step kernel: the finalization of the evaluation before it
// (eval(..., false)) and the step itself.
gr_status NbSystem::md_step_launch(cudaStream_t s, bool fuse_prep) {
    MdDev md;
    md.vel = md_vel;
    md.inv_mass = md_inv_mass;
    md.mass = md_mass;
    md.dt = mdp.dt;
    md.dt_i = 1.0 / mdp.dt;
    md.settle = md_settle ? 1 : 0;
    md.m_o = md_m_o;
    md.m_h = md_m_h;
    md.im_o = md_m_o > 0.0 ? 1.0 / md_m_o : 0.0;  // (SETTLE: every molecule has these masses)
    md.im_h = md_m_h > 0.0 ? 1.0 / md_m_h : 0.0;
    md.ra = md_ra;
    md.rb = md_rb;
    md.rc = md_rc;
    md.ke = md_ke;
    md.failures = md_fail;
    md.t0 = md_t0;
    md.tau = mdp.tau;
    md.dof = md_dof;
    // the next evaluation keeps this period's lists (no rebuild): its water
    // records come from this kernel
    md.prep_next = fuse_prep && md_settle && NCG > NSCG && h.wrec && !in_capture && built &&
                   steps_since_update < prm.nsnb;
    if (!in_capture) prepped_next = prep_in_acc = md.prep_next != 0;
    const int n_units = md_settle ? NSA + (N - NSA) / 3 : N;
    // a unit is one long FP64 chain: small blocks spread few units over more SMs
    const unsigned bt = n_units <= 128 * sm_count() ? 64 : 128;
    const unsigned grid = std::max(1u, std::min(unsigned((n_units + bt - 1) / bt), unsigned(sm_count() * 8)));
    if (prm.kernel == GR_KERNEL_FIXED) {
        if (md_settle && n_units > 128 * sm_count())
            GR_CUDA(launch(k_md_step_tiled, grid, kTile, 0, s, d_sys, md));
        else
            GR_CUDA(launch(k_md_step<true>, grid, bt, 0, s, d_sys, md));
        acc_clean = true;  // the step leaves the short-range accumulators zero
    } else {
        GR_CUDA(launch(k_md_step<false>, grid, bt, 0, s, d_sys, md));
    }
    return GR_OK;
}

gr_status NbSystem::md_stats(cudaStream_t s, gr_md_stats* out) {
    const int NA = acc_size(G);
    gr_status st = energy_buffer();
    if (st) return st;
    const double* e = e_dl_host;
    long long* ke_host = reinterpret_cast<long long*>(e_dl_host + NA);
    int* fails_host = reinterpret_cast<int*>(e_dl_host + NA + 1);
    GR_CUDA(cudaMemcpyAsync(ke_host, md_ke, sizeof(long long), cudaMemcpyDeviceToHost, s));
    GR_CUDA(cudaMemcpyAsync(fails_host, md_fail, sizeof(int), cudaMemcpyDeviceToHost, s));
    GR_CUDA(cudaMemcpyAsync(e_dl_host, h.e_out, size_t(NA) * sizeof(double), cudaMemcpyDeviceToHost, s));
    GR_CUDA(cudaStreamSynchronize(s));
    const long long ke = *ke_host;
    const int fails = *fails_host;
    double elj = 0.0, ecrf = 0.0;
    for (int g = 0; g < G * G; ++g) {
        elj += e[g];
        ecrf += e[G * G + g];
    }
    out->steps = md_steps_total;
    out->e_lj = elj;
    out->e_crf = ecrf;
    out->e_kin = double(ke) / kEnergyScale;
    out->settle_failures = fails;
    out->rollbacks = int(md_rollbacks);
    return GR_OK;
}

gr_status NbSystem::md_run(cudaStream_t s, int n_steps, gr_md_stats* out) {
    if (!md_ready) {
        set_error("gr_md_run before gr_md_init");
        return GR_ERR_STATE;
    }
    if (n_steps < 0) {
        set_error("gr_md_run: n_steps must be >= 0");
        return GR_ERR_INVALID;
    }
    const size_t bytes3 = size_t(N) * 3 * sizeof(double);
    // The error flags are sticky in device memory, so they are read once per
    // block of whole pairlist periods (one host synchronisation per block);
    // an overflow anywhere in the block rolls the whole block back.  Kernels
    // are launched one by one: the host runs ahead of the device, and the
    // recorded step graphs would add their per-step flag copy and timing
    // events (measured slower here).
    //
    // The rollback point of a block is its start when the block starts a
    // pairlist period.  A block that starts inside a period (the previous
    // call ended there) rolls back to that period's start, kept in md_psnap,
    // and replays the steps up to the block start: the lists are rebuilt at
    // the period's own first step, so the rebuild and long-range schedule is
    // that of a run without overflow, and (the sums being fixed point) the
    // replayed steps reproduce the block's starting state bit for bit.
    const int kblock = std::max(1, prm.nsnb) * 4;
    int done = 0, attempts = 0, rollbacks = 0;
    gr_status st;
    while (done < n_steps) {
        const int ssu0 = steps_since_update;
        const bool from_period = built && ssu0 < prm.nsnb && md_psnap_valid && md_step_idx - md_psnap_step == ssu0;
        GR_CUDA(cudaMemcpyAsync(md_pos_snap, from_period ? md_psnap_pos : h.pos, bytes3, cudaMemcpyDeviceToDevice, s));
        GR_CUDA(cudaMemcpyAsync(md_vel_snap, from_period ? md_psnap_vel : md_vel, bytes3, cudaMemcpyDeviceToDevice, s));
        GR_CUDA(cudaMemcpyAsync(md_ke_snap, from_period ? md_psnap_ke : md_ke, sizeof(long long),
                                cudaMemcpyDeviceToDevice, s));
        const long long idx0 = from_period ? md_psnap_step : md_step_idx;
        int replay = 0;  // steps re-run before the block's own steps (after a rollback)
        int k = 0;
        for (;;) {  // attempts at this block
            bool overflow = false;
            k = 0;
            for (int r = 0;;) {
                if (pending_check) {  // the flags of this period's rebuild
                    bool of = false;
                    if ((st = resolve_pending(&of))) return st;
                    if (of) {
                        overflow = true;
                        break;
                    }
                }
                if (!built || steps_since_update >= prm.nsnb) {  // this step starts a pairlist period
                    snapshot = MdSnapshot{md_psnap_pos, md_psnap_vel, md_psnap_ke, md_vel, md_ke};
                    md_psnap_step = md_step_idx;
                    md_psnap_valid = true;
                }
                if ((st = eval(s, 0, false, prm.kernel != GR_KERNEL_FIXED))) return st;
                if ((st = md_step_launch(s, true))) return st;
                ++md_step_idx;
                if (r < replay) {
                    ++r;
                    continue;
                }
                ++k;
                if (done + k >= n_steps || (steps_since_update >= prm.nsnb && k >= kblock)) break;
            }
            if (!overflow) {
                // everything of this block (builds and force kernels) has set its flags
                GR_CUDA(cudaMemcpyAsync(md_err_host, h.err, 4 * sizeof(int), cudaMemcpyDeviceToHost, s));
                GR_CUDA(cudaEventRecord(ev_md, s));
                GR_CUDA(cudaEventSynchronize(ev_md));
                const int* e = reinterpret_cast<const int*>(md_err_host);
                pending_check = false;  // a rebuild at the block's last step: its flags are in e[0] too
                several_images = e[1] != 0;
                if (e[0]) {
                    const int f = e[0];
                    GR_CUDA(cudaMemset(h.err, 0, 4 * sizeof(int)));
                    if (f & (ERR_CELL_TOO_DENSE | ERR_CG_TOO_LARGE)) {
                        set_error(f & ERR_CELL_TOO_DENSE ? "pairlist: a grid cell holds more than 2048 charge groups"
                                                         : "pairlist: solute charge group larger than 8 atoms");
                        return GR_ERR_UNSUPPORTED;
                    }
                    if (f & ERR_WLIST_OVERFLOW) wcap_want = std::max(wcap_want, wcap_alloc) * 2;
                    if (f & ERR_SLIST_OVERFLOW) scap_want = std::max(scap_want, scap_alloc) * 2;
                    if (f & ERR_PERT_OVERFLOW) pcap_want = std::max(pcap_want, pcap_alloc) * 2;
                    if (f & ERR_DEFER_OVERFLOW) {
                        defer_want = std::max(defer_want, h.defer_cap) * 4;
                        clus_alloc = 0;
                    }
                    overflow = true;
                }
            }
            if (!overflow) break;
            if (++attempts > 8) {
                set_error("md: list capacity could not be grown far enough");
                return GR_ERR_OVERFLOW;
            }
            GR_CUDA(cudaMemcpyAsync(h.pos, md_pos_snap, bytes3, cudaMemcpyDeviceToDevice, s));
            GR_CUDA(cudaMemcpyAsync(md_vel, md_vel_snap, bytes3, cudaMemcpyDeviceToDevice, s));
            GR_CUDA(cudaMemcpyAsync(md_ke, md_ke_snap, sizeof(long long), cudaMemcpyDeviceToDevice, s));
            prepped_next = false;
            md_step_idx = idx0;
            steps_since_update = prm.nsnb;
            built = false;  // the rollback point starts a period: rebuilt there with the grown lists
            lr_computed = false;
            replay = from_period ? ssu0 : 0;
            ++rollbacks;
        }
        attempts = 0;
        done += k;
    }
    md_steps_total += done;
    md_rollbacks += rollbacks;
    if (out) {
        if ((st = md_stats(s, out))) return st;
        out->steps = done;
        out->rollbacks = rollbacks;
    }
    return GR_OK;
}

extern "C" {

gr_status gr_md_init(gr_ctx* ctx, const double* mass, const double* vel, const gr_md_params* params) {
    CTX_GUARD(ctx);
    return ctx->sys.md_init(mass, vel, params);
}

gr_status gr_md_run(gr_ctx* ctx, int32_t n_steps, gr_md_stats* out) {
    CTX_GUARD(ctx);
    return ctx->sys.md_run(ctx->stream, n_steps, out);
}

gr_status gr_md_set_temperature(gr_ctx* ctx, double t0, int32_t rescale_velocities) {
    CTX_GUARD(ctx);
    NbSystem& S = ctx->sys;
    if (!S.md_ready) {
        set_error("gr_md_set_temperature before gr_md_init");
        return GR_ERR_STATE;
    }
    if (!(t0 > 0.0)) {
        set_error("gr_md_set_temperature: t0 must be positive");
        return GR_ERR_INVALID;
    }
    S.md_psnap_valid = false;  // a replay of earlier steps would see the new bath and unscaled velocities
    // the bath temperature lives in device memory (k_md_step reads it every
    // step): recorded step graphs stay valid, and the write is ordered after
    // the steps already enqueued on this context's stream
    GR_CUDA(cudaMemcpyAsync(S.md_t0, &t0, sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    if (rescale_velocities) {
        // Replica::rescale_velocities (replica.rs:355-371): scale to t0 from the
        // instantaneous temperature over 3N degrees of freedom
        long long ke = 0;
        GR_CUDA(cudaMemcpyAsync(&ke, S.md_ke, sizeof(ke), cudaMemcpyDeviceToHost, ctx->stream));
        GR_CUDA(cudaStreamSynchronize(ctx->stream));
        const double t_now = 2.0 * (double(ke) / gnb::kEnergyScale) / (3.0 * S.N * 0.00831446261815324);
        if (!(t_now > 0.0)) {
            S.mdp.temperature = t0;
            GR_CUDA(cudaStreamSynchronize(ctx->stream));
            return GR_OK;
        }
        const double f = std::sqrt(t0 / t_now);
        const int n3 = 3 * S.N;
        (++S.launches, gnb::k_scale_velocities<<<std::max(1, std::min((n3 + 255) / 256, 1024)), 256, 0, ctx->stream>>>(
            S.md_vel, n3, f, S.md_ke));
        GR_CUDA(cudaGetLastError());
    }
    S.mdp.temperature = t0;
    // complete before returning: a batch launches its members' steps on its own stream
    GR_CUDA(cudaStreamSynchronize(ctx->stream));
    return GR_OK;
}

gr_status gr_md_stats_get(gr_ctx* ctx, gr_md_stats* out) {
    CTX_GUARD(ctx);
    if (!ctx->sys.md_ready || !out) {
        set_error("gr_md_stats_get: MD not initialised or null out");
        return ctx->sys.md_ready ? GR_ERR_INVALID : GR_ERR_STATE;
    }
    return ctx->sys.md_stats(ctx->stream, out);
}

gr_status gr_md_download(gr_ctx* ctx, double* pos, double* vel) {
    CTX_GUARD(ctx);
    NbSystem& S = ctx->sys;
    if (!S.md_ready) {
        set_error("gr_md_download before gr_md_init");
        return GR_ERR_STATE;
    }
    const size_t bytes3 = size_t(S.N) * 3 * sizeof(double);
    cudaError_t e = cudaSuccess;
    if (pos) e = cudaMemcpyAsync(pos, S.h.pos, bytes3, cudaMemcpyDeviceToHost, ctx->stream);
    if (vel && e == cudaSuccess) e = cudaMemcpyAsync(vel, S.md_vel, bytes3, cudaMemcpyDeviceToHost, ctx->stream);
    // also after an error: no copy may still be under way into the caller's buffers
    const cudaError_t e2 = cudaStreamSynchronize(ctx->stream);
    GR_CUDA(e != cudaSuccess ? e : e2);
    return GR_OK;
}

}  // extern "C"
