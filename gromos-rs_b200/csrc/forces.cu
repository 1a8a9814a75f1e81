// forces.cu -- LJ + reaction-field force / energy / virial kernels.
//
// Pair physics: lj_crf_interaction (crates/gromos-forces/src/nonbonded/innerloops.rs:21-55)
//   inv_r2 = 1/r2, inv_r6 = inv_r2^3
//   e_lj  = (c12 inv_r6 - c6) inv_r6,  f_lj  = (12 c12 inv_r6 - 6 c6) inv_r6 inv_r2
//   e_crf = q (1/r - crf_2cut3i r2 - crf_cut),  f_crf = q (inv_r inv_r2 + crf_cut3i)
//   F_i += r f, F_j -= r f, virial[a][b] += r_a F_b;  r2 < 1e-10 -> no contribution.
//
// Image rules reproduced per list (forcefield.rs:417-727):
//   solvent short : one shift per CG pair from the first atoms (innerloops.rs:264-267)
//   solute short  : one shift per CG pair from the first atoms when the box is
//                   large (cg_grouped, innerloops.rs:118-124), else per atom
//   long lists    : per-atom nearest image (innerloops.rs:186)
// The FP32 kernels compute pair vectors from FP32 offsets relative to each
// CG's first atom plus an FP64 first-atom image; a pair whose FP32 vector is
// within 1e-4 nm of half a box edge is redone with the exact FP64 image, so
// the image choice is always the reference's.
//
// Kernels:
//   k_water_prep        per step: FP64 first-atom position + FP32 offsets, slot order;
//                       zeroes the slot force sums, pulls the short lists into L2
//   (water-water clusters: water.cu)
//   k_solute_force<..>  solute CG pairs (any CG size <= 8, LJ type table)
//   k_plain_force       baseline: thread per CG pair, absolute FP32, FP32 atomics
//   k_excluded_14       FP64 RF excluded / self terms (excluded.rs:25-112) and
//                       1-4 pairs (excluded.rs:131-206)
//   k_pert              FP64 soft-core pair correction (perturbed.rs:309-386) and the
//                       self / excluded / 1-4 / atom-pair corrections
//   k_finalize          fixed point -> FP64 outputs
#include <algorithm>

#include "nb_common.cuh"

namespace gnb {

constexpr float kF = 4294967296.0f;   // force fixed-point scale (2^32)
constexpr float kE = 16777216.0f;     // energy / virial fixed-point scale (2^24)

// ---------------------------------------------------------------------------
// The per-step record of one solvent molecule (coordinates p, charges q3 when
// the intra-molecular excluded pairs are done here): the slot's water record,
// its short-range force sums cleared, the line of the cluster's short list
// this member pulls into L2; returns the molecule's extent in m and adds its
// excluded-pair RF energies (-q_i q_j fpe crf_2cut3i r^2, rf_excluded_interactions,
// excluded.rs:81-96) to e_excl.  Used by k_water_prep and, for the next step,
// by the MD step kernel (the tiled one clears the force sums itself: CLEAR false).
template <bool CLEAR = true>
__device__ __forceinline__ void water_record(const SysDev& s, int slot, const double (&p)[9], const double (&q3)[3],
                                             bool excl, double& e_excl, float& m) {
    // descriptor fields first: the stores below go through pointers the
    // compiler cannot tell apart from the descriptor
    WaterRec* __restrict__ wrec = s.wrec;
    long long* fs_short = s.fs_short;  // the MD step kernel reads the slot's sums before they are cleared here
    const uint32_t* __restrict__ wl_s = s.wl_s;
    const int W = s.W, wcap = s.wcap;
    const bool rect = s.boundary == 1;
    const double bx = s.box[0], by = s.box[1], bz = s.box[2];
    const double ibx = s.inv_box[0], iby = s.inv_box[1], ibz = s.inv_box[2];
    const double fpe = s.fpe, crf2 = s.crf_2cut3i;
    WaterRec w;
    w.x0 = p[0];
    w.y0 = p[1];
    w.z0 = p[2];
    w.h1x = float(p[3] - p[0]);
    w.h1y = float(p[4] - p[1]);
    w.h1z = float(p[5] - p[2]);
    w.h2x = float(p[6] - p[0]);
    w.h2y = float(p[7] - p[1]);
    w.h2z = float(p[8] - p[2]);
    // extent of the molecule (per-atom images of the long list need it)
    m = fmaxf(m, fmaxf(fmaxf(fabsf(w.h1x), fabsf(w.h1y)), fmaxf(fabsf(w.h1z), fabsf(w.h2x))));
    m = fmaxf(m, fmaxf(fabsf(w.h2y), fabsf(w.h2z)));
    if (excl) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = a + 1; b < 3; ++b) {
                double rx = __dsub_rn(p[3 * a], p[3 * b]);
                double ry = __dsub_rn(p[3 * a + 1], p[3 * b + 1]);
                double rz = __dsub_rn(p[3 * a + 2], p[3 * b + 2]);
                if (rect) {
                    rx = image_exact(rx, bx, ibx);
                    ry = image_exact(ry, by, iby);
                    rz = image_exact(rz, bz, ibz);
                }
                e_excl += -q3[a] * q3[b] * fpe * crf2 * len2_exact(rx, ry, rz);
            }
    }
    wrec[slot] = w;
    // the slot's short-range force sums start at zero for this evaluation
    // (only slots that hold a water are ever added to or read)
    if (CLEAR) {
        long long* __restrict__ fz = fs_short + static_cast<size_t>(slot) * 9;
#pragma unroll
        for (int c = 0; c < 9; ++c) fz[c] = 0;
    }
    // the member k of a cluster pulls line k of the cluster's short list
    // into L2 for the force kernel (the list was written at the last rebuild)
    const int k = slot % W;
    if (32 * k < wcap) {
        const uint32_t* line = wl_s + static_cast<size_t>(slot / W) * wcap + 32 * k;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(line));
    }
}

// Block-level flush of water_record's outputs: one atomicMax of the extent
// and one energy add per block (the extents are >= 0, so their bit patterns
// order like the values).  Every thread of the block calls it.
__device__ __forceinline__ void water_record_flush(const SysDev& s, float m, double e_excl, bool excl) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const long long v = excl ? warp_sum_ll(to_fixed_d(e_excl, kEnergyScale)) : 0ll;
    __shared__ int mx;
    __shared__ unsigned long long sh;
    if (threadIdx.x == 0) {
        mx = 0;
        sh = 0ull;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        if (m > 0.f) atomicMax(&mx, __float_as_int(m));
        if (v) atomicAdd(&sh, static_cast<unsigned long long>(v));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int G = s.n_egroups, gs = s.solvent_group < 0 ? 0 : s.solvent_group;
        long long* acc = s.acc_short;
        if (mx) atomicMax(reinterpret_cast<int*>(s.max_delta), mx);
        if (sh) atomicAdd(reinterpret_cast<unsigned long long*>(acc + G * G + gs * G + gs), sh);
    }
}

__global__ void k_water_prep(const SysDev* __restrict__ sys) {
    pdl_wait();
    pdl_trigger();
    // One thread per solvent molecule in atom order (coalesced position
    // reads); the record goes to the molecule's slot.  Every load is issued
    // before the slot is tested: the coordinates do not depend on it.
    // Solvent molecules are 3-site (checked at upload).
    const SysDev& s = sys[blockIdx.y];
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    const int nsolv = s.n_cg - s.n_solute_cg;
    const int nsa = s.n_solute_atoms, nscg = s.n_solute_cg;
    const bool excl = s.excl_atoms < s.n_atoms;
    double e_excl = 0.0;
    float m = 0.f;
    if (w < nsolv) {
        const int slot = s.cg_slot[nscg + w];
        const int a0 = nsa + 3 * w;  // solvent CGs are whole 3-site molecules
        double p[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) p[q] = s.pos[3 * a0 + q];
        double q3[3] = {0.0, 0.0, 0.0};
        if (excl)
#pragma unroll
            for (int a = 0; a < 3; ++a) q3[a] = s.charge[a0 + a];
        if (slot >= 0) water_record(s, slot, p, q3, excl, e_excl, m);
    }
    water_record_flush(s, m, e_excl, excl);
}

// Per-block reduction of NV fixed-point accumulators into global memory.
template <int NV>
__device__ __forceinline__ void block_flush(long long (&acc)[NV], long long* __restrict__ dst,
                                            const int* __restrict__ idx) {
    __shared__ unsigned long long sh[NV];
    for (int v = threadIdx.x; v < NV; v += blockDim.x) sh[v] = 0ull;
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (acc[v]) atomicAdd(&sh[v], static_cast<unsigned long long>(acc[v]));
    __syncthreads();
    for (int v = threadIdx.x; v < NV; v += blockDim.x)
        if (sh[v]) atomicAdd(reinterpret_cast<unsigned long long*>(dst + idx[v]), sh[v]);
}

// ---------------------------------------------------------------------------
// Adds a warp's fixed-point (LJ, CRF) energies to the block's group sums, one
// value pair per lane under its group slot (-1: none).  Lanes of one slot, the
// common case, are summed by shuffles: 32 lanes adding to one 64-bit shared
// word retry one after the other.
__device__ __forceinline__ void warp_add_energies(unsigned long long* sh, int G, int sl, long long el, long long ec) {
    const int lead = __reduce_max_sync(0xffffffffu, sl);
    if (lead < 0) return;
    if (__all_sync(0xffffffffu, sl == lead || sl < 0)) {
        el = warp_sum_ll(el);
        ec = warp_sum_ll(ec);
        if ((threadIdx.x & 31) != 0) return;
        sl = lead;
    }
    if (el) atomicAdd(&sh[sl], static_cast<unsigned long long>(el));
    if (ec) atomicAdd(&sh[G * G + sl], static_cast<unsigned long long>(ec));
}

// Solute CG pairs (solute-solute, solute-solvent, intra-CG) of one range: the
// short entries fill a CG's list from the front, the long ones from the back.
// Work items are (solute CG, 64 or 32 of its entries), one warp per item and one
// lane per entry, so a CG's list is spread over many warps, each adding its
// share of the CG's forces with fixed-point reductions; sn_max bounds the
// items, so no warp walks the unused capacity of the lists.  Group energies
// and the virial are summed per lane in FP32 within one item and taken to
// fixed point at its end (energies also when the group slot changes), so the
// results do not depend on the grid or on which warp took which item.
//
// The kernel is bound by the latency of an item's dependent loads, not by its
// arithmetic, so an entry of the solvent (uniform solvent: every molecule has
// the first one's types and charges) needs one level of them after the list:
// the molecule's nine coordinates, at an address the index gives.
// MAXA bounds the atoms of the i groups (the largest solute CG: 1, up to 4, or
// up to 8): the per-atom force sums are registers and their loops unrolled code (168
// registers at 8, 128 at 1; eight replicas with single-atom groups gain 6%, an MD
// step of 3,000 waters with 200 ions 3%).  The molecule's
// charges come from the descriptor, the CG's LJ rows against the three
// solvent sites and its own atoms from shared memory, once per item.  The
// second round's molecule is loaded while the first one is computed.  200 ions in
// 3,000 waters: 32 us before, 25 now (ncu); replica exchange of eight systems of
// 1,500 waters and 200 ions 1.23x as fast.

// With a twin range the two lists are short and an item is one round of 32, else
// a system of few solute CGs has fewer items than the chip has warps.
__host__ __device__ constexpr int solute_chunk(bool twin) { return twin ? 32 : 64; }

template <int MAXA>
struct SoluteWarp {
    float4 at[MAXA];      // i atoms: offset from the CG's first atom, charge x fpe
    int2 tg[MAXA];        // LJ row (type x n_types), energy group
    float4 lj[MAXA * 3];  // c6, c12, 6 c6, 12 c12 against solvent site b at 3 a + b
};

template <bool LONG, int MAXA>
__global__ void __launch_bounds__(128) k_solute_force(const SysDev* __restrict__ sys) {
    pdl_wait();
    pdl_trigger();
    const SysDev& s = sys[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int G = s.n_egroups;
    long long* __restrict__ F = LONG ? s.f_long : s.f_short;
    extern __shared__ unsigned long long shg[];  // 2*G*G group energies (fixed)
    __shared__ SoluteWarp<MAXA> sw_all[4];
    SoluteWarp<MAXA>& sw = sw_all[threadIdx.x >> 5];
    for (int v = threadIdx.x; v < 2 * G * G; v += blockDim.x) shg[v] = 0ull;
    __syncthreads();
    const double* __restrict__ pos = s.pos;
    const int* __restrict__ cg_off = s.cg_off;
    const int* __restrict__ iac = s.iac;
    const double* __restrict__ charge = s.charge;
    const int* __restrict__ egroup = s.egroup;
    const int nsa = s.n_solute_atoms, nscg = s.n_solute_cg, scap = s.scap, n_types = s.n_types;
    const bool uniform = s.solvent_uniform != 0;
    const bool per_atom = LONG || !s.cg_grouped;
    const float crf2 = s.crf_2cut3i_f, crfc = s.crf_cut_f, crf3 = s.crf_cut3i_f;
    float v6[6] = {0, 0, 0, 0, 0, 0};
    __shared__ long long vfix[6][128];  // per lane, touched once per item
#pragma unroll
    for (int v = 0; v < 6; ++v) vfix[v][threadIdx.x] = 0;
    int cur_slot = -1;
    float e_lj = 0.f, e_cr = 0.f;
    auto to_slot = [&](int sl) {
        if (sl == cur_slot) return;
        if (cur_slot >= 0) {
            const long long fl = to_fixed_f(e_lj, kE), fc = to_fixed_f(e_cr, kE);
            if (fl) atomicAdd(&shg[cur_slot], static_cast<unsigned long long>(fl));
            if (fc) atomicAdd(&shg[G * G + cur_slot], static_cast<unsigned long long>(fc));
        }
        e_lj = e_cr = 0.f;
        cur_slot = sl;
    };
    const int chunk = solute_chunk(s.twin != 0);
    const int nitems = nscg * ((s.sn_max[LONG ? 1 : 0] + chunk - 1) / chunk);
    for (int it = blockIdx.x * wpb + (threadIdx.x >> 5); it < nitems; it += gridDim.x * wpb) {
        const int ci = it % nscg, e_beg = (it / nscg) * chunk;
        const int cnt = min(s.sn[2 * ci + (LONG ? 1 : 0)], e_beg + chunk);
        if (e_beg >= cnt) continue;  // warp-uniform
        // entry e of the CG's list of this range
        const size_t l0 = static_cast<size_t>(ci) * scap + (LONG ? scap - 1 : 0);
        auto place = [&](int e) { return LONG ? l0 - e : l0 + e; };
        int entry = e_beg + lane < cnt ? s.sl[place(e_beg + lane)] : -1;
        int entry_n = e_beg + 32 + lane < cnt ? s.sl[place(e_beg + 32 + lane)] : -1;  // (cnt ends the item)
        double p[9];
        auto load_solvent = [&](int entry_l) {
            if (entry_l >= 0 && (entry_l >> 1) >= nscg && uniform) {
                const double* __restrict__ pj = pos + 3 * static_cast<size_t>(nsa + 3 * ((entry_l >> 1) - nscg));
#pragma unroll
                for (int k = 0; k < 9; ++k) p[k] = pj[k];
            }
        };
        load_solvent(entry);
        const int i0 = cg_off[ci], ni = cg_off[ci + 1] - i0;
        double px = 0.0, py = 0.0, pz = 0.0;
        int ti = 0;
        if (lane < ni) {
            const int a = i0 + lane;
            px = pos[3 * a];
            py = pos[3 * a + 1];
            pz = pos[3 * a + 2];
            ti = iac[a] * n_types;
        }
        const double xi0 = __shfl_sync(0xffffffffu, px, 0), yi0 = __shfl_sync(0xffffffffu, py, 0);
        const double zi0 = __shfl_sync(0xffffffffu, pz, 0);
        __syncwarp();  // the previous item's reads are done
        if (lane < ni) {
            sw.at[lane] = make_float4(float(px - xi0), float(py - yi0), float(pz - zi0),
                                      float(charge[i0 + lane] * s.fpe));
            sw.tg[lane] = make_int2(ti, egroup[i0 + lane]);
        }
        if (uniform) {
            const int row = __shfl_sync(0xffffffffu, ti, lane / 3);
            if (lane < 3 * ni) {
                const float2 c = s.lj32[row + s.w_iac[lane % 3]];
                sw.lj[lane] = make_float4(c.x, c.y, 6.f * c.x, 12.f * c.y);
            }
        }
        __syncwarp();
        float fix[MAXA], fiy[MAXA], fiz[MAXA];
#pragma unroll
        for (int a = 0; a < MAXA; ++a) fix[a] = fiy[a] = fiz[a] = 0.f;
        // one atom pair: i atom a, j atom at its offset (djx, djy, djz) from its CG's
        // first atom, D the imaged vector between the first atoms; g the j force
        auto pair = [&](int a, int aj, float Dx, float Dy, float Dz, float djx, float djy, float djz, float4 c, float qj,
                        int gj, float& gx, float& gy, float& gz) {
            const float4 pi = sw.at[a];
            float x = (Dx + pi.x) - djx, y = (Dy + pi.y) - djy, z = (Dz + pi.z) - djz;
            if (per_atom && s.boundary) {
                const float m = 1e-4f;
                if (!(fabsf(x) < s.half_boxf[0] - m && fabsf(y) < s.half_boxf[1] - m && fabsf(z) < s.half_boxf[2] - m)) {
                    const int ai = i0 + a;
                    double dx, dy, dz;
                    nearest_image_exact(s, pos[3 * ai], pos[3 * ai + 1], pos[3 * ai + 2], pos[3 * aj], pos[3 * aj + 1],
                                        pos[3 * aj + 2], dx, dy, dz);
                    x = float(dx);
                    y = float(dy);
                    z = float(dz);
                }
            }
            const float r2 = fmaf(x, x, fmaf(y, y, z * z));
            if (r2 < 1e-10f) return;
            // one Newton step on the hardware reciprocal square root removes its
            // bias from the (cancelling) CRF energy sums of solute pairs
            float ri = rsqrtf(r2);
            ri = fmaf(0.5f * ri, fmaf(-r2 * ri, ri, 1.0f), ri);
            const float ri2 = ri * ri, ri6 = ri2 * ri2 * ri2;
            const float q = pi.w * qj;
            to_slot(group_slot(G, sw.tg[a].y, gj));
            e_lj += fmaf(c.y, ri6, -c.x) * ri6;
            e_cr += q * (fmaf(-crf2, r2, ri) - crfc);
            const float fs = fmaf(fmaf(c.w, ri6, -c.z), ri6 * ri2, q * fmaf(ri, ri2, crf3));
            const float fxx = x * fs, fyy = y * fs, fzz = z * fs;
            fix[a] += fxx;
            fiy[a] += fyy;
            fiz[a] += fzz;
            gx -= fxx;
            gy -= fyy;
            gz -= fzz;
            v6[0] = fmaf(x, fxx, v6[0]);
            v6[1] = fmaf(x, fyy, v6[1]);
            v6[2] = fmaf(x, fzz, v6[2]);
            v6[3] = fmaf(y, fyy, v6[3]);
            v6[4] = fmaf(y, fzz, v6[4]);
            v6[5] = fmaf(z, fzz, v6[5]);
        };
        for (int e0 = e_beg; e0 < cnt; e0 += 32) {
            const int cj = entry >> 1;
            const bool solvent = entry >= 0 && cj >= nscg && uniform;
            int j0 = 0;
            float Dx = 0.f, Dy = 0.f, Dz = 0.f, dj[9];
            if (solvent) {
                j0 = nsa + 3 * (cj - nscg);
                double dx, dy, dz;
                nearest_image_exact(s, xi0, yi0, zi0, p[0], p[1], p[2], dx, dy, dz);
                Dx = float(dx);
                Dy = float(dy);
                Dz = float(dz);
#pragma unroll
                for (int k = 0; k < 9; ++k) dj[k] = float(p[k] - p[k % 3]);
            }
            load_solvent(entry_n);
            if (solvent) {
                const int gj = s.solvent_group;
                long long* __restrict__ Fj = F + 3 * static_cast<size_t>(j0);
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    float gx = 0.f, gy = 0.f, gz = 0.f;
#pragma unroll
                    for (int a = 0; a < MAXA; ++a) {
                        if (a >= ni) break;
                        pair(a, j0 + b, Dx, Dy, Dz, dj[3 * b], dj[3 * b + 1], dj[3 * b + 2], sw.lj[3 * a + b], s.w_q[b],
                             gj, gx, gy, gz);
                    }
                    red_add(Fj + 3 * b, to_fixed_f(gx, kF));
                    red_add(Fj + 3 * b + 1, to_fixed_f(gy, kF));
                    red_add(Fj + 3 * b + 2, to_fixed_f(gz, kF));
                }
            } else if (entry >= 0) {
                const unsigned long long xm = s.sl_excl[place(e0 + lane)];
                j0 = cg_off[cj];
                const int nj = cg_off[cj + 1] - j0;
                double dx, dy, dz;
                nearest_image_exact(s, xi0, yi0, zi0, pos[3 * j0], pos[3 * j0 + 1], pos[3 * j0 + 2], dx, dy, dz);
                Dx = float(dx);
                Dy = float(dy);
                Dz = float(dz);
                for (int b = 0; b < nj; ++b) {
                    const int aj = j0 + b;
                    const float djx = float(pos[3 * aj] - pos[3 * j0]);
                    const float djy = float(pos[3 * aj + 1] - pos[3 * j0 + 1]);
                    const float djz = float(pos[3 * aj + 2] - pos[3 * j0 + 2]);
                    const int tj = iac[aj], gj = egroup[aj];
                    const float qj = float(charge[aj]);
                    float gx = 0.f, gy = 0.f, gz = 0.f;
#pragma unroll
                    for (int a = 0; a < MAXA; ++a) {
                        if (a >= ni) break;
                        if (xm & (1ull << (a * 8 + b))) continue;
                        const float2 c = s.lj32[sw.tg[a].x + tj];
                        pair(a, aj, Dx, Dy, Dz, djx, djy, djz, make_float4(c.x, c.y, 6.f * c.x, 12.f * c.y), qj, gj, gx,
                             gy, gz);
                    }
                    red_add(&F[3 * aj], to_fixed_f(gx, kF));
                    red_add(&F[3 * aj + 1], to_fixed_f(gy, kF));
                    red_add(&F[3 * aj + 2], to_fixed_f(gz, kF));
                }
            }
            entry = entry_n;
            entry_n = -1;
        }
        __syncwarp();
#pragma unroll
        for (int a = 0; a < MAXA; ++a) {
            if (a >= ni) break;
            const float vx = warp_sum(fix[a]), vy = warp_sum(fiy[a]), vz = warp_sum(fiz[a]);
            if (lane == a) {
                red_add(&F[3 * (i0 + a)], to_fixed_f(vx, kF));
                red_add(&F[3 * (i0 + a) + 1], to_fixed_f(vy, kF));
                red_add(&F[3 * (i0 + a) + 2], to_fixed_f(vz, kF));
            }
        }
        warp_add_energies(shg, G, cur_slot, to_fixed_f(e_lj, kE), to_fixed_f(e_cr, kE));
        e_lj = e_cr = 0.f;
        cur_slot = -1;
#pragma unroll
        for (int v = 0; v < 6; ++v) {
            vfix[v][threadIdx.x] += to_fixed_f(v6[v], kE);
            v6[v] = 0.f;
        }
    }
    long long* dst = LONG ? s.acc_long : s.acc_short;
    __syncthreads();
    for (int v = threadIdx.x; v < 2 * G * G; v += blockDim.x)
        if (shg[v]) atomicAdd(reinterpret_cast<unsigned long long*>(dst + v), shg[v]);
    long long vs[6];
#pragma unroll
    for (int v = 0; v < 6; ++v) vs[v] = warp_sum_ll(vfix[v][threadIdx.x]);
    long long acc[9] = {vs[0], vs[1], vs[2], vs[1], vs[3], vs[4], vs[2], vs[4], vs[5]};
    int idx[9];
#pragma unroll
    for (int v = 0; v < 9; ++v) idx[v] = 2 * G * G + v;
    block_flush<9>(acc, dst, idx);
}

// ---------------------------------------------------------------------------
// Baseline: one thread per CG pair, absolute FP32 coordinates, FP32 atomics.
__global__ void k_pos32(const SysDev* __restrict__ sys) {
    const SysDev& s = sys[blockIdx.y];
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= s.n_atoms) return;
    s.pos32[a] = make_float4(float(s.pos[3 * a]), float(s.pos[3 * a + 1]), float(s.pos[3 * a + 2]),
                             float(s.charge[a] * s.fpe));
}

__global__ void __launch_bounds__(256) k_plain_force(const SysDev* __restrict__ sys, int long_range) {
    const SysDev& s = sys[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const int n = s.n_cgp[long_range];
    float* __restrict__ F = long_range ? s.f32_long : s.f32;
    double* __restrict__ E = long_range ? s.e64_long : s.e64;
    float elj = 0.f, ecrf = 0.f, v6[6] = {0, 0, 0, 0, 0, 0};
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const int idx = long_range ? s.cgp_cap - 1 - p : p;
        const int ci = s.cgp[3 * idx], cj = s.cgp[3 * idx + 1];
        const unsigned long long xm = s.cgp_excl[idx];
        const int i0 = s.cg_off[ci], ni = s.cg_off[ci + 1] - i0;
        const int j0 = s.cg_off[cj], nj = s.cg_off[cj + 1] - j0;
        const bool solvent_pair = ci >= s.n_solute_cg;
        const bool shift = !long_range && (solvent_pair || s.cg_grouped);
        float sx = 0.f, sy = 0.f, sz = 0.f;
        if (shift && s.boundary) {
            float4 a = s.pos32[i0], b = s.pos32[j0];
            sx = s.boxf[0] * rintf((a.x - b.x) * s.inv_boxf[0]);
            sy = s.boxf[1] * rintf((a.y - b.y) * s.inv_boxf[1]);
            sz = s.boxf[2] * rintf((a.z - b.z) * s.inv_boxf[2]);
        }
        for (int a = 0; a < ni; ++a) {
            const float4 pi = s.pos32[i0 + a];
            const int ti = s.iac[i0 + a];
            float fxa = 0.f, fya = 0.f, fza = 0.f;
            for (int b = 0; b < nj; ++b) {
                if (xm & (1ull << (a * 8 + b))) continue;
                const float4 pj = s.pos32[j0 + b];
                float x = pi.x - pj.x, y = pi.y - pj.y, z = pi.z - pj.z;
                if (shift) {
                    x -= sx;
                    y -= sy;
                    z -= sz;
                } else if (s.boundary) {
                    x -= s.boxf[0] * rintf(x * s.inv_boxf[0]);
                    y -= s.boxf[1] * rintf(y * s.inv_boxf[1]);
                    z -= s.boxf[2] * rintf(z * s.inv_boxf[2]);
                }
                const float r2 = x * x + y * y + z * z;
                if (r2 < 1e-10f) continue;
                const float ri2 = 1.f / r2, ri6 = ri2 * ri2 * ri2, ri = sqrtf(ri2);
                const float2 lj = s.lj32[ti * s.n_types + s.iac[j0 + b]];
                const float q = pi.w * (pj.w / float(s.fpe));
                elj += (lj.y * ri6 - lj.x) * ri6;
                ecrf += q * (ri - s.crf_2cut3i_f * r2 - s.crf_cut_f);
                const float fs = (12.f * lj.y * ri6 - 6.f * lj.x) * ri6 * ri2 + q * (ri * ri2 + s.crf_cut3i_f);
                const float fxx = x * fs, fyy = y * fs, fzz = z * fs;
                fxa += fxx;
                fya += fyy;
                fza += fzz;
                atomicAdd(&F[3 * (j0 + b)], -fxx);
                atomicAdd(&F[3 * (j0 + b) + 1], -fyy);
                atomicAdd(&F[3 * (j0 + b) + 2], -fzz);
                v6[0] += x * fxx;
                v6[1] += x * fyy;
                v6[2] += x * fzz;
                v6[3] += y * fyy;
                v6[4] += y * fzz;
                v6[5] += z * fzz;
            }
            atomicAdd(&F[3 * (i0 + a)], fxa);
            atomicAdd(&F[3 * (i0 + a) + 1], fya);
            atomicAdd(&F[3 * (i0 + a) + 2], fza);
        }
    }
    float ev[8] = {elj, ecrf, v6[0], v6[1], v6[2], v6[3], v6[4], v6[5]};
    const int map[8] = {0, 1, 2, 3, 4, 6, 7, 10};  // lj, crf, xx, xy, xz, yy, yz, zz
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        double t = warp_sum_d(double(ev[v]));
        if (lane == 0 && t != 0.0) atomicAdd(&E[map[v]], t);
    }
}

// ---------------------------------------------------------------------------
// FP64 terms.  Shared-memory fixed-point accumulators per block, then global.
struct TermAcc {
    double* g;  // 2*G*G + 9 + 1 (FP64, per thread)
};

__device__ __forceinline__ void add_force_fixed(long long* F, int a, double fx, double fy, double fz) {
    red_add(&F[3 * a], to_fixed_d(fx, kForceScale));
    red_add(&F[3 * a + 1], to_fixed_d(fy, kForceScale));
    red_add(&F[3 * a + 2], to_fixed_d(fz, kForceScale));
}

__device__ __forceinline__ void shared_add(unsigned long long* sh, int idx, double v) {
    long long f = to_fixed_d(v, kEnergyScale);
    if (f) atomicAdd(&sh[idx], static_cast<unsigned long long>(f));
}

// rf_excluded_interactions (excluded.rs:25-112) + one_four_interaction_loop
// (excluded.rs:131-206, coulomb scaling 1).  One thread per term: the self
// term of a solute atom, an excluded pair, a 1-4 pair (i < j lists made once
// from the topology).  The terms are few and their cost is latency: a thread
// per atom that walked its exclusion list and added eleven values to shared
// 64-bit words that its whole block adds to took 28 us for 200 atoms in
// multi-atom CGs and 11 us for 200 ions (ncu).  Here a warp sums its values by
// shuffles, in FP64 and per group slot, and takes each sum to fixed point once:
// one shared add and one rounding per warp, 6.6 and 5.3 us.
__global__ void k_excluded_14(const SysDev* __restrict__ sys) {
    pdl_wait();
    pdl_trigger();
    const SysDev& s = sys[blockIdx.y];
    const int G = s.n_egroups;
    const int NA = acc_size(G);
    extern __shared__ unsigned long long sh[];
    for (int v = threadIdx.x; v < NA; v += blockDim.x) sh[v] = 0ull;
    __syncthreads();
    const int vb = 2 * G * G;
    const int nsa = s.n_solute_atoms, nex = s.n_ex_pairs, nterm = nsa + nex + s.n_14_pairs;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    int sl = -1;
    double el = 0.0, ec = 0.0;
    double v6[6] = {0, 0, 0, 0, 0, 0};  // xx, xy, xz, yy, yz, zz
    if (t < nsa) {
        const double qi = s.charge[t];
        const int gi = s.egroup[t];
        sl = group_slot(G, gi, gi);
        ec = -0.5 * qi * qi * s.fpe * s.crf_cut;
    } else if (t < nterm) {
        const int2 ij = s.term_pairs[t - nsa];
        const int i = ij.x, j = ij.y;
        const double qi = s.charge[i], qj = s.charge[j];
        const int gi = s.egroup[i], gj = s.egroup[j];
        double rx, ry, rz;
        nearest_image_exact(s, s.pos[3 * i], s.pos[3 * i + 1], s.pos[3 * i + 2], s.pos[3 * j], s.pos[3 * j + 1],
                            s.pos[3 * j + 2], rx, ry, rz);
        const double r2 = len2_exact(rx, ry, rz);
        const double q = qi * qj * s.fpe;
        double fs = 0.0;
        if (t < nsa + nex) {
            sl = group_slot(G, gi, gj);
            if (i < nsa) {
                ec = q * (-s.crf_2cut3i * r2 - s.crf_cut);
                fs = q * s.crf_cut3i;
            } else {
                ec = -qi * qj * s.fpe * s.crf_2cut3i * r2;
            }
        } else if (!(r2 < 1e-10)) {
            sl = group_slot(G, gi, gj);
            const double* lj = s.lj64 + 4 * (s.iac[i] * s.n_types + s.iac[j]);
            const double cs6 = lj[2], cs12 = lj[3];
            const double ir2 = 1.0 / r2, ir6 = ir2 * ir2 * ir2, ir = sqrt(ir2);
            el = (cs12 * ir6 - cs6) * ir6;
            ec = q * (ir - s.crf_2cut3i * r2 - s.crf_cut);
            fs = (12.0 * cs12 * ir6 - 6.0 * cs6) * ir6 * ir2 + q * (ir * ir2 + s.crf_cut3i);
        }
        if (fs != 0.0) {
            const double fx = rx * fs, fy = ry * fs, fz = rz * fs;
            add_force_fixed(s.f_short, i, fx, fy, fz);
            add_force_fixed(s.f_short, j, -fx, -fy, -fz);
            v6[0] = rx * fx;
            v6[1] = rx * fy;
            v6[2] = rx * fz;
            v6[3] = ry * fy;
            v6[4] = ry * fz;
            v6[5] = rz * fz;
        }
    }
    unsigned left = __ballot_sync(0xffffffffu, sl >= 0);
    while (left) {  // one round per group slot among the lanes
        const int lead = __shfl_sync(0xffffffffu, sl, __ffs(left) - 1);
        const bool mine = sl == lead;
        const double l = warp_sum_d(mine ? el : 0.0), c = warp_sum_d(mine ? ec : 0.0);
        if ((threadIdx.x & 31) == 0) {
            shared_add(sh, lead, l);
            shared_add(sh, G * G + lead, c);
        }
        left &= ~__ballot_sync(0xffffffffu, mine);
    }
    if (__any_sync(0xffffffffu, t >= nsa && t < nterm)) {
#pragma unroll
        for (int u = 0; u < 6; ++u) {
            const long long v = to_fixed_d(warp_sum_d(v6[u]), kEnergyScale);
            if ((threadIdx.x & 31) == 0 && v) {
                const int a = u < 3 ? 0 : u < 5 ? 1 : 2, b = u < 3 ? u : u < 5 ? u - 2 : 2;
                atomicAdd(&sh[vb + 3 * a + b], static_cast<unsigned long long>(v));
                if (a != b) atomicAdd(&sh[vb + 3 * b + a], static_cast<unsigned long long>(v));
            }
        }
    }
    __syncthreads();
    for (int v = threadIdx.x; v < NA; v += blockDim.x)
        if (sh[v]) atomicAdd(reinterpret_cast<unsigned long long*>(s.acc_short + v), sh[v]);
}

// perturbed_lj_crf_interaction (perturbed.rs:124-266), FP64.
__device__ void pert_interaction(const SysDev& s, double rx, double ry, double rz, double a_c6, double a_c12,
                                 double b_c6, double b_c12, double a_q, double b_q, double alj, double acrf,
                                 double out[5]) {
    const double* lp = s.lp;
    const double a_lj_n = lp[0], b_lj_n = lp[1], a_crf_n = lp[2], b_crf_n = lp[3];
    const double a_lj_n1 = lp[4], b_lj_n1 = lp[5], a_crf_n1 = lp[6], b_crf_n1 = lp[7];
    const double a_ljs = lp[8], b_ljs = lp[9], a_ljs2 = lp[10], b_ljs2 = lp[11];
    const double a_crfs = lp[12], b_crfs = lp[13], a_crfs2 = lp[14], b_crfs2 = lp[15];
    const double nexp = lp[16];
    const double r2 = len2_exact(rx, ry, rz);
    if (r2 < 1e-10) {
        for (int k = 0; k < 5; ++k) out[k] = 0.0;
        return;
    }
    const double r6 = r2 * r2 * r2, r4 = r2 * r2;
    const double a_c126 = fabs(a_c6) > 1e-10 ? a_c12 / a_c6 : 0.0;
    const double b_c126 = fabs(b_c6) > 1e-10 ? b_c12 / b_c6 : 0.0;
    // 1/sqrt and its powers from one rsqrt each: an FP64 division or square root is about
    // ten FP64 operations, and these are most of a pair's work
    const double a_dis = rsqrt(r2 + acrf * b_crfs2), a_d3is = a_dis * a_dis * a_dis;
    const double a_d6i = 1.0 / (r6 + alj * b_ljs2 * a_c126);
    const double b_dis = rsqrt(r2 + acrf * a_crfs2), b_d3is = b_dis * b_dis * b_dis;
    const double b_d6i = 1.0 / (r6 + alj * a_ljs2 * b_c126);
    const double cut2 = s.cutoff_sq;
    const double a_ci = rsqrt(cut2 + acrf * b_crfs2), b_ci = rsqrt(cut2 + acrf * a_crfs2);
    const double a_ci2 = a_ci * a_ci, b_ci2 = b_ci * b_ci;
    const double a_crf_2cut3i = s.crf_2cut3i * (a_ci2 * a_ci);
    const double b_crf_2cut3i = s.crf_2cut3i * (b_ci2 * b_ci);
    const double a_crf_cut3i = 2.0 * a_crf_2cut3i, b_crf_cut3i = 2.0 * b_crf_2cut3i;
    const double a_crf_pert = 3.0 * a_crf_2cut3i * a_ci2, b_crf_pert = 3.0 * b_crf_2cut3i * b_ci2;
    double force = (a_crf_n * a_q * (a_d3is + a_crf_cut3i) + b_crf_n * b_q * (b_d3is + b_crf_cut3i)) * s.fpe;
    force += -6.0 * (a_lj_n * a_c6 * a_d6i * a_d6i + b_lj_n * b_c6 * b_d6i * b_d6i) * r4;
    force += 12.0 * (a_lj_n * a_c12 * a_d6i * a_d6i * a_d6i + b_lj_n * b_c12 * b_d6i * b_d6i * b_d6i) * r4;
    const double a_e_lj = (a_c12 * a_d6i - a_c6) * a_d6i, b_e_lj = (b_c12 * b_d6i - b_c6) * b_d6i;
    const double a_e_crf = a_q * (a_dis - a_crf_2cut3i * r2 - s.crf_cut);
    const double b_e_crf = b_q * (b_dis - b_crf_2cut3i * r2 - s.crf_cut);
    out[0] = force;
    out[1] = a_lj_n * a_e_lj + b_lj_n * b_e_lj;
    out[2] = (a_crf_n * a_e_crf + b_crf_n * b_e_crf) * s.fpe;
    out[3] = -2.0 * alj *
                 (a_lj_n * b_ljs * a_c126 * a_d6i * a_d6i * (2.0 * a_c12 * a_d6i - a_c6) -
                  b_lj_n * a_ljs * b_c126 * b_d6i * b_d6i * (2.0 * b_c12 * b_d6i - b_c6)) +
             nexp * (b_lj_n1 * b_e_lj - a_lj_n1 * a_e_lj);
    out[4] = -(a_crf_n * a_q * b_crfs * (a_d3is - a_crf_pert * r2) -
               b_crf_n * b_q * a_crfs * (b_d3is - b_crf_pert * r2)) *
                 s.fpe * acrf +
             nexp * (b_crf_n1 * b_e_crf - a_crf_n1 * a_e_crf) * s.fpe;
}

struct PInfo {
    bool on;
    int a_iac, b_iac;
    double a_q, b_q, alj, acrf;
};

__device__ __forceinline__ PInfo pinfo(const SysDev& s, int a) {
    PInfo p{false, s.iac[a], s.iac[a], s.charge[a], s.charge[a], 0.0, 0.0};
    const int k = s.pert_idx[a];
    if (k >= 0) {
        p.on = true;
        p.a_iac = s.pert_iac[2 * k];
        p.b_iac = s.pert_iac[2 * k + 1];
        p.a_q = s.pert_q[2 * k];
        p.b_q = s.pert_q[2 * k + 1];
        p.alj = s.pert_alpha[2 * k];
        p.acrf = s.pert_alpha[2 * k + 1];
    }
    return p;
}

// perturbed_pairlist_correction (perturbed.rs:309-386) for the explicit list
// of (i perturbed, j) pairs of all lists, every step, per-atom image.
// One thread per pair: the pairs are some tens of thousands of FP64 chains, so
// runs of pairs per thread left most SMs without a block (35,000 pairs in runs of
// 16: 66 us, and 9.5 for the per-atom terms, launched over every atom; one launch of
// 18 us now, ncu).  Every pair's contribution goes to fixed point first
// and a warp's integers are summed by shuffles -- the i-force per distinct i
// (pairs are listed per solute charge group, so a warp has few) and the
// energies per group slot -- so the totals do not depend on the list's order,
// which the atomic appends of k_pert_pairs do not fix, and few same-address
// additions are issued.
__device__ __forceinline__ void pert_pairs(const SysDev& s, unsigned long long* sh, int block, int nblocks) {
    const int G = s.n_egroups, lane = threadIdx.x & 31;
    const int np = min(s.n_pert_pairs[0], s.pcap);
    for (int p0 = block * blockDim.x + threadIdx.x - lane; p0 < np; p0 += nblocks * blockDim.x) {  // warp-uniform
        const int p = p0 + lane;
        int i = -1, sl = -1;
        long long fx = 0, fy = 0, fz = 0, el = 0, ec = 0, dh = 0;
        if (p < np) {
            i = s.pert_pairs[3 * p];
            const int j = s.pert_pairs[3 * p + 1];
            const PInfo pi = pinfo(s, i), pj = pinfo(s, j);
            const double* lja = s.lj64 + 4 * (pi.a_iac * s.n_types + pj.a_iac);
            const double* ljb = s.lj64 + 4 * (pi.b_iac * s.n_types + pj.b_iac);
            const double a_q = pi.a_q * pj.a_q, b_q = pi.b_q * pj.b_q;
            const double alj = pj.on ? (pi.alj + pj.alj) * 0.5 : pi.alj;
            const double acrf = pj.on ? (pi.acrf + pj.acrf) * 0.5 : pi.acrf;
            double rx, ry, rz;
            nearest_image_exact(s, s.pos[3 * i], s.pos[3 * i + 1], s.pos[3 * i + 2], s.pos[3 * j], s.pos[3 * j + 1],
                                s.pos[3 * j + 2], rx, ry, rz);
            const double r2 = len2_exact(rx, ry, rz);
            double fa = 0, ela = 0, eca = 0;
            if (!(r2 < 1e-10)) {  // lj_crf_interaction, state A
                const double ir = rsqrt(r2), ir2 = ir * ir, ir6 = ir2 * ir2 * ir2;
                const double qa = a_q * s.fpe;
                ela = (lja[1] * ir6 - lja[0]) * ir6;
                eca = qa * (ir - s.crf_2cut3i * r2 - s.crf_cut);
                fa = (12.0 * lja[1] * ir6 - 6.0 * lja[0]) * ir6 * ir2 + qa * (ir * ir2 + s.crf_cut3i);
            }
            double o[5];
            pert_interaction(s, rx, ry, rz, lja[0], lja[1], ljb[0], ljb[1], a_q, b_q, alj, acrf, o);
            const double df = o[0] - fa;
            fx = to_fixed_d(rx * df, kForceScale);
            fy = to_fixed_d(ry * df, kForceScale);
            fz = to_fixed_d(rz * df, kForceScale);
            add_force_fixed(s.f_short, j, -rx * df, -ry * df, -rz * df);
            sl = group_slot(G, s.egroup[i], s.egroup[j]);
            el = to_fixed_d(o[1] - ela, kEnergyScale);
            ec = to_fixed_d(o[2] - eca, kEnergyScale);
            dh = to_fixed_d(o[3] + o[4], kEnergyScale);
        }
        unsigned left = __ballot_sync(0xffffffffu, i >= 0);
        while (left) {
            const int lead = __shfl_sync(0xffffffffu, i, __ffs(left) - 1);
            const bool mine = i == lead;
            const long long tx = warp_sum_ll(mine ? fx : 0), ty = warp_sum_ll(mine ? fy : 0);
            const long long tz = warp_sum_ll(mine ? fz : 0);
            if (lane == 0) {
                red_add(&s.f_short[3 * lead], tx);
                red_add(&s.f_short[3 * lead + 1], ty);
                red_add(&s.f_short[3 * lead + 2], tz);
            }
            left &= ~__ballot_sync(0xffffffffu, mine);
        }
        warp_add_energies(sh, G, sl, el, ec);
        dh = warp_sum_ll(dh);
        if (lane == 0 && dh) atomicAdd(&sh[acc_size(G) - 1], static_cast<unsigned long long>(dh));
    }
}

// Self / excluded / 1-4 / PERTATOMPAIR corrections (perturbed.rs:395-707).
// One thread per solute atom i (excluded and 1-4 pairs with j > i: only
// solute atoms are perturbed, so a pair with a perturbed atom starts at one);
// PERTATOMPAIR entries are handled by the threads i < n_pp.
__device__ __forceinline__ void pert_terms(const SysDev& s, unsigned long long* sh, int block) {
    const int G = s.n_egroups;
    const int NA = acc_size(G);
    const double* lp = s.lp;
    const double a_lj_n = lp[0], b_lj_n = lp[1], a_crf_n = lp[2], b_crf_n = lp[3];
    const double a_lj_n1 = lp[4], b_lj_n1 = lp[5], a_crf_n1 = lp[6], b_crf_n1 = lp[7];
    const double a_crfs = lp[12], b_crfs = lp[13], a_crfs2 = lp[14], b_crfs2 = lp[15];
    const double nexp = lp[16];
    const int i = block * blockDim.x + threadIdx.x;
    {  // perturbed_self_energy_correction
        int sl = -1;
        long long e = 0, dh = 0;
        if (i < s.n_solute_atoms && s.pert_idx[i] >= 0) {
            const PInfo pi = pinfo(s, i);
            const double qa2 = pi.a_q * pi.a_q, qb2 = pi.b_q * pi.b_q;
            const double e_rf = (-(a_crf_n * qa2) - b_crf_n * qb2 + qa2) * s.crf_cut * s.fpe;
            const double de_rf = nexp * (a_crf_n1 * qa2 - b_crf_n1 * qb2) * s.crf_cut * s.fpe;
            sl = group_slot(G, s.egroup[i], s.egroup[i]);
            e = to_fixed_d(0.5 * e_rf, kEnergyScale);
            dh = to_fixed_d(0.5 * de_rf, kEnergyScale);
        }
        warp_add_energies(sh, G, sl, 0, e);
        dh = warp_sum_ll(dh);
        if ((threadIdx.x & 31) == 0 && dh) atomicAdd(&sh[NA - 1], static_cast<unsigned long long>(dh));
    }
    if (i < s.n_solute_atoms || i < s.n_pp) {
        if (i < s.n_solute_atoms) {
            const PInfo pi = pinfo(s, i);
            const int gi = s.egroup[i];
            // perturbed_excluded_correction
            for (int k = s.excl_off[i]; k < s.excl_off[i + 1]; ++k) {
                const int j = s.excl[k];
                if (j <= i) continue;
                const PInfo pj = pinfo(s, j);
                if (!pi.on && !pj.on) continue;
                const double acrf = (pi.on && pj.on) ? (pi.acrf + pj.acrf) * 0.5 : (pi.on ? pi.acrf : pj.acrf);
                double rx, ry, rz;
                nearest_image_exact(s, s.pos[3 * i], s.pos[3 * i + 1], s.pos[3 * i + 2], s.pos[3 * j],
                                    s.pos[3 * j + 1], s.pos[3 * j + 2], rx, ry, rz);
                const double r2 = len2_exact(rx, ry, rz);
                const double a_q = pi.a_q * pj.a_q, b_q = pi.b_q * pj.b_q;
                const double cut2 = s.cutoff_sq;
                const double a_c2s = cut2 + acrf * b_crfs2, b_c2s = cut2 + acrf * a_crfs2;
                const double ra = cut2 / a_c2s, rb = cut2 / b_c2s;
                const double a_crf_2cut3i = s.crf_2cut3i * sqrt(ra * (ra * ra));
                const double b_crf_2cut3i = s.crf_2cut3i * sqrt(rb * (rb * rb));
                const double a_crf_pert = 3.0 * a_crf_2cut3i / a_c2s, b_crf_pert = 3.0 * b_crf_2cut3i / b_c2s;
                const double a_e_crf = a_q * (-a_crf_2cut3i * r2 - s.crf_cut);
                const double b_e_crf = b_q * (-b_crf_2cut3i * r2 - s.crf_cut);
                const double e_p = (a_crf_n * a_e_crf + b_crf_n * b_e_crf) * s.fpe;
                const double f_p = (a_crf_n * a_q * 2.0 * a_crf_2cut3i + b_crf_n * b_q * 2.0 * b_crf_2cut3i) * s.fpe;
                const double e_a = a_q * s.fpe * (-s.crf_2cut3i * r2 - s.crf_cut);
                const double f_a = a_q * s.fpe * s.crf_cut3i;
                const double de = ((a_crf_n * a_q * b_crfs * a_crf_pert - b_crf_n * b_q * a_crfs * b_crf_pert) * r2 * acrf +
                                   nexp * (b_crf_n1 * b_e_crf - a_crf_n1 * a_e_crf)) *
                                  s.fpe;
                const double df = f_p - f_a;
                add_force_fixed(s.f_short, i, rx * df, ry * df, rz * df);
                add_force_fixed(s.f_short, j, -rx * df, -ry * df, -rz * df);
                shared_add(sh, G * G + group_slot(G, gi, s.egroup[j]), e_p - e_a);
                shared_add(sh, NA - 1, de);
            }
        for (int k = s.o14_off[i]; k < s.o14_off[i + 1]; ++k) {  // perturbed_one_four_correction
            const int j = s.o14[k];
            if (j <= i) continue;
            const PInfo pj = pinfo(s, j);
            if (!pi.on && !pj.on) continue;
            double rx, ry, rz;
            nearest_image_exact(s, s.pos[3 * i], s.pos[3 * i + 1], s.pos[3 * i + 2], s.pos[3 * j], s.pos[3 * j + 1],
                                s.pos[3 * j + 2], rx, ry, rz);
            const double r2 = len2_exact(rx, ry, rz);
            if (r2 < 1e-10) continue;
            const double* lja = s.lj64 + 4 * (pi.a_iac * s.n_types + pj.a_iac);
            const double* ljb = s.lj64 + 4 * (pi.b_iac * s.n_types + pj.b_iac);
            const double a_q = pi.a_q * pj.a_q, b_q = pi.b_q * pj.b_q;
            const double alj = (pi.on && pj.on) ? (pi.alj + pj.alj) * 0.5 : (pi.on ? pi.alj : pj.alj);
            const double acrf = (pi.on && pj.on) ? (pi.acrf + pj.acrf) * 0.5 : (pi.on ? pi.acrf : pj.acrf);
            const double ir2 = 1.0 / r2, ir6 = ir2 * ir2 * ir2, ir = sqrt(ir2);
            const double e_lj_a = (lja[3] * ir6 - lja[2]) * ir6;
            const double f_lj_a = (12.0 * lja[3] * ir6 - 6.0 * lja[2]) * ir6 * ir2;
            const double e_crf_a = a_q * s.fpe * (ir - s.crf_2cut3i * r2 - s.crf_cut);
            const double f_crf_a = a_q * s.fpe * (ir * ir2 + s.crf_cut3i);
            double o[5];
            pert_interaction(s, rx, ry, rz, lja[2], lja[3], ljb[2], ljb[3], a_q, b_q, alj, acrf, o);
            const double df = o[0] - (f_lj_a + f_crf_a);
            add_force_fixed(s.f_short, i, rx * df, ry * df, rz * df);
            add_force_fixed(s.f_short, j, -rx * df, -ry * df, -rz * df);
            const int sl = group_slot(G, gi, s.egroup[j]);
            shared_add(sh, sl, o[1] - e_lj_a);
            shared_add(sh, G * G + sl, o[2] - e_crf_a);
            shared_add(sh, NA - 1, o[3] + o[4]);
        }
        }
        if (i < s.n_pp) {  // perturbed_atom_pair_correction
            const int a = s.pp[4 * i], b = s.pp[4 * i + 1], at = s.pp[4 * i + 2], bt = s.pp[4 * i + 3];
            bool in14 = false;
            for (int k = s.o14_off[a]; k < s.o14_off[a + 1]; ++k) in14 |= s.o14[k] == b;
            for (int k = s.o14_off[b]; k < s.o14_off[b + 1]; ++k) in14 |= s.o14[k] == a;
            double rx, ry, rz;
            nearest_image_exact(s, s.pos[3 * a], s.pos[3 * a + 1], s.pos[3 * a + 2], s.pos[3 * b], s.pos[3 * b + 1],
                                s.pos[3 * b + 2], rx, ry, rz);
            const double r2 = len2_exact(rx, ry, rz);
            if (in14 && !(r2 < 1e-10)) {
                const double ir2 = 1.0 / r2, ir6 = ir2 * ir2 * ir2, ir = sqrt(ir2);
                const double* lj = s.lj64 + 4 * (s.iac[a] * s.n_types + s.iac[b]);
                const double e_lj_reg = (lj[3] * ir6 - lj[2]) * ir6;
                const double f_lj_reg = (12.0 * lj[3] * ir6 - 6.0 * lj[2]) * ir6 * ir2;
                const double q = s.charge[a] * s.charge[b] * s.fpe;
                const double e_crf_reg = q * (ir - s.crf_2cut3i * r2 - s.crf_cut);
                const double f_crf_reg = q * (ir * ir2 + s.crf_cut3i);
                double e_lj_a, f_lj_a, e_lj_b = 0.0, f_lj_b = 0.0;
                const int ca = at == 0 ? 0 : 2;
                e_lj_a = (lj[ca + 1] * ir6 - lj[ca]) * ir6;
                f_lj_a = (12.0 * lj[ca + 1] * ir6 - 6.0 * lj[ca]) * ir6 * ir2;
                if (bt >= 0) {
                    const int cb = bt == 0 ? 0 : 2;
                    e_lj_b = (lj[cb + 1] * ir6 - lj[cb]) * ir6;
                    f_lj_b = (12.0 * lj[cb + 1] * ir6 - 6.0 * lj[cb]) * ir6 * ir2;
                }
                const double e_crf_b = bt >= 0 ? e_crf_reg : 0.0, f_crf_b = bt >= 0 ? f_crf_reg : 0.0;
                const double e_lj_p = a_lj_n * e_lj_a + b_lj_n * e_lj_b;
                const double f_lj_p = a_lj_n * f_lj_a + b_lj_n * f_lj_b;
                const double f_crf_p = a_crf_n * f_crf_reg + b_crf_n * f_crf_b;
                const double de_lj = nexp * (b_lj_n1 * e_lj_b - a_lj_n1 * e_lj_a);
                const double de_crf = nexp * (b_crf_n1 * e_crf_b - a_crf_n1 * e_crf_reg);
                const double df = (f_lj_p - f_lj_reg) + (f_crf_p - f_crf_reg);
                add_force_fixed(s.f_short, a, rx * df, ry * df, rz * df);
                add_force_fixed(s.f_short, b, -rx * df, -ry * df, -rz * df);
                // forcefield.rs:907-933 adds only the LJ energy change of this pass
                shared_add(sh, group_slot(G, s.egroup[a], s.egroup[b]), e_lj_p - e_lj_reg);
                shared_add(sh, NA - 1, de_lj + de_crf);
            }
        }
    }
}

// All perturbation corrections in one launch: the first term_blocks blocks
// take the per-atom terms, the others the listed pairs.
__global__ void __launch_bounds__(128) k_pert(const SysDev* __restrict__ sys, int term_blocks) {
    pdl_wait();
    pdl_trigger();
    const SysDev& s = sys[blockIdx.y];
    const int NA = acc_size(s.n_egroups);
    extern __shared__ unsigned long long sh[];
    for (int v = threadIdx.x; v < NA; v += blockDim.x) sh[v] = 0ull;
    __syncthreads();
    if (int(blockIdx.x) < term_blocks)
        pert_terms(s, sh, blockIdx.x);
    else
        pert_pairs(s, sh, blockIdx.x - term_blocks, gridDim.x - term_blocks);
    __syncthreads();
    for (int v = threadIdx.x; v < NA; v += blockDim.x)
        if (sh[v]) atomicAdd(reinterpret_cast<unsigned long long*>(s.acc_short + v), sh[v]);
}

// Fixed point -> FP64 results.  plain != 0 adds the FP32 baseline buffers.
__global__ void k_finalize(const SysDev* __restrict__ sys, int plain) {
    pdl_wait();
    pdl_trigger();
    // One thread per force component; a water atom's component also gathers
    // its cluster slot's sum (solvent CG w = atoms nsa + 3w .. nsa + 3w + 2).
    // The descriptor's fields are read into registers first and every load is
    // issued before the first store: a store through a pointer taken from the
    // descriptor would otherwise force the later field reads to wait for it.
    const SysDev& s = sys[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n3 = 3 * s.n_atoms, nsa = s.n_solute_atoms, nscg = s.n_solute_cg;
    const int twin = s.twin, NA = acc_size(s.n_egroups);
    long long* __restrict__ f_short = s.f_short;
    const long long* __restrict__ f_long = s.f_long;
    const long long* __restrict__ fs_short = s.fs_short;
    const long long* __restrict__ fs_long = s.fs_long;
    const int* __restrict__ cg_slot = s.cg_slot;
    const float* __restrict__ f32 = s.f32;
    const float* __restrict__ f32_long = s.f32_long;
    double* __restrict__ f_out = s.f_out;
    long long* __restrict__ acc_short = s.acc_short;
    const long long* __restrict__ acc_long = s.acc_long;
    double* __restrict__ e_out = s.e_out;
    float* max_delta = s.max_delta;
    int* n_deferred = s.n_deferred;
    const bool water = s.wrec != nullptr && !plain;
    // a water atom's per-atom accumulators hold something only when solute
    // kernels, excluded pairs or perturbation terms reach water atoms
    const bool water_pa = plain || nscg > 0 || s.excl_atoms > nsa || s.n_pert > 0 || s.n_pp > 0;
    const double inv = 1.0 / kForceScale;
    // Every per-atom short-range accumulator is read by exactly one thread
    // here, which also clears it for the next evaluation (the per-slot water
    // sums are cleared by one contiguous memset; the long-range cache persists).
    if (i < n3) {
        const int a = i / 3;
        const bool pa = a < nsa || water_pa;
        long long fx = pa ? f_short[i] : 0ll;
        if (twin && pa) fx += f_long[i];
        if (a >= nsa && water) {
            const int w = (a - nsa) / 3;
            const int slot = cg_slot[nscg + w];
            const int k = i - 3 * (nsa + 3 * w);
            if (slot >= 0) {  // (no slot: the build failed on this molecule's cell and reported it)
                fx += fs_short[slot * 9 + k];
                if (twin) fx += fs_long[slot * 9 + k];
            }
        }
        double v = double(fx) * inv;
        if (plain) {
            v += double(f32[i]);
            if (twin) v += double(f32_long[i]);
        }
        f_out[i] = v;
        if (pa) f_short[i] = 0;
    }
    if (i < NA) {
        double v = double(acc_short[i]) / kEnergyScale;
        if (twin) v += double(acc_long[i]) / kEnergyScale;
        e_out[i] = v;
        acc_short[i] = 0;
    }
    if (i == 0) {
        if (max_delta) *max_delta = 0.f;
        if (n_deferred)
            for (int k = 0; k < 6; ++k) n_deferred[k] = 0;
    }
}

__global__ void k_finalize_plain_energies(const SysDev* __restrict__ sys) {
    const SysDev& s = sys[blockIdx.y];
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int G = s.n_egroups;
    const int gs = s.solvent_group < 0 ? 0 : s.solvent_group;
    const int sl = group_slot(G, gs, gs);
    double lj = s.e64[0] + (s.twin ? s.e64_long[0] : 0.0);
    double crf = s.e64[1] + (s.twin ? s.e64_long[1] : 0.0);
    s.e_out[sl] += lj;
    s.e_out[G * G + sl] += crf;
    const int vb = 2 * G * G;
    const int map[9] = {2, 3, 4, 3, 6, 7, 4, 7, 10};
    for (int v = 0; v < 9; ++v) s.e_out[vb + v] += s.e64[map[v]] + (s.twin ? s.e64_long[map[v]] : 0.0);
}

// Explicit instantiations used by the host runtime.
template __global__ void k_solute_force<false, 8>(const SysDev*);
template __global__ void k_solute_force<true, 8>(const SysDev*);
template __global__ void k_solute_force<false, 4>(const SysDev*);
template __global__ void k_solute_force<true, 4>(const SysDev*);
template __global__ void k_solute_force<false, 1>(const SysDev*);
template __global__ void k_solute_force<true, 1>(const SysDev*);

}  // namespace gnb

namespace gnb {
// lj_crf_innerloop over an explicit atom-pair list (innerloops.rs:169-210),
// the body behind the reference's C-ABI stub (ffi.rs:55-103).  One thread
// per pair, per-atom nearest image; q_i q_j scaled by fpe.
//
// The kernel is bound by its atomic additions, so it issues few.  A warp takes
// kPairIters x 32 consecutive pairs; pair lists are written i by i, so its
// lanes mostly share i: the i-force is summed in registers and by shuffles
// and added once per run of pairs (any other order is correct too: rounds of
// mixed i add group by group, or lane by lane when there are many).  The three
// components of a j-force are one 8-byte and one 4-byte reduction, whichever
// way round the address allows.  Energies and the virial go to FP64 per warp
// chunk and once per block to memory, where eleven FP64 atomics per warp went to
// one cache line.  6.3 M pairs of 30,000 atoms: 613 us with one addition per pair
// and component, 83 now (ncu).  The arithmetic hides behind the reductions:
// IEEE division and square root, which round once where a reciprocal square
// root would give r^-6 2.3 times the rounding, cost nothing.
constexpr int kPairIters = 8;

__device__ __forceinline__ void red_add3(float* p, float x, float y, float z) {
    const bool odd = (reinterpret_cast<uintptr_t>(p) & 4u) != 0;  // 4 bytes off an 8-byte boundary
    float* two = p + (odd ? 1 : 0);
    float* one = p + (odd ? 0 : 2);
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(two), "f"(odd ? y : x), "f"(odd ? z : y) : "memory");
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(one), "f"(odd ? x : z) : "memory");
}

__global__ void __launch_bounds__(256) k_innerloop_pairs(
    const float* __restrict__ pos, const float* __restrict__ q, const uint32_t* __restrict__ iac,
    const uint32_t* __restrict__ pairs, uint32_t n_pairs, const float2* __restrict__ lj, uint32_t n_types, float bx,
    float by, float bz, int rect, float crf_cut, float crf_2cut3i, float crf_cut3i, float fpe, float* __restrict__ F,
    double* __restrict__ E) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const bool al8 = (reinterpret_cast<uintptr_t>(pairs) & 7u) == 0;
    const float ibx = 1.f / bx, iby = 1.f / by, ibz = 1.f / bz;
    const float hx = 0.5f * bx, hy = 0.5f * by, hz = 0.5f * bz;
    double sums[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // lj, crf, xx, xy, xz, yy, yz, zz
    const size_t nwarps = size_t(gridDim.x) * (blockDim.x >> 5);
    const size_t step = size_t(kPairIters) * 32;
    for (size_t c = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; c * step < n_pairs; c += nwarps) {
        float e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        float fx = 0.f, fy = 0.f, fz = 0.f;  // this run's share of the force on atom cur
        uint32_t cur = 0xffffffffu;
        auto flush = [&]() {  // warp-uniform
            if (cur == 0xffffffffu) return;
            const float sx = warp_sum(fx), sy = warp_sum(fy), sz = warp_sum(fz);
            if (lane == 0) red_add3(F + 3 * size_t(cur), sx, sy, sz);
            fx = fy = fz = 0.f;
        };
#pragma unroll 2
        for (int it = 0; it < kPairIters; ++it) {
            const size_t p = c * step + size_t(it) * 32 + lane;
            const bool valid = p < n_pairs;
            uint2 ij = make_uint2(0xffffffffu, 0u);
            if (valid) ij = al8 ? reinterpret_cast<const uint2*>(pairs)[p] : make_uint2(pairs[2 * p], pairs[2 * p + 1]);
            float gx = 0.f, gy = 0.f, gz = 0.f;
            if (valid) {
                const size_t i3 = 3 * size_t(ij.x), j3 = 3 * size_t(ij.y);
                float x = pos[i3] - pos[j3], y = pos[i3 + 1] - pos[j3 + 1], z = pos[i3 + 2] - pos[j3 + 2];
                const float2 k = lj[iac[ij.x] * n_types + iac[ij.y]];
                const float qq = q[ij.x] * q[ij.y] * fpe;
                if (rect) {
                    // the product with the rounded reciprocal may fall on the other side of a
                    // tie: the remainder shows it, and the quotients decide (by division
                    // for every pair a call takes 3% longer)
                    const float dx = fmaf(-rintf(x * ibx), bx, x), dy = fmaf(-rintf(y * iby), by, y);
                    const float dz = fmaf(-rintf(z * ibz), bz, z);
                    if (fabsf(dx) >= hx || fabsf(dy) >= hy || fabsf(dz) >= hz) {
                        x -= bx * rintf(x / bx);
                        y -= by * rintf(y / by);
                        z -= bz * rintf(z / bz);
                    } else {
                        x = dx;
                        y = dy;
                        z = dz;
                    }
                }
                const float r2 = x * x + y * y + z * z;
                if (!(r2 < 1e-10f)) {
                    const float ri2 = 1.f / r2, ri6 = ri2 * ri2 * ri2, ri = sqrtf(ri2);
                    e[0] += (k.y * ri6 - k.x) * ri6;
                    e[1] += qq * (ri - crf_2cut3i * r2 - crf_cut);
                    const float fs = (12.f * k.y * ri6 - 6.f * k.x) * ri6 * ri2 + qq * (ri * ri2 + crf_cut3i);
                    gx = x * fs;
                    gy = y * fs;
                    gz = z * fs;
                    e[2] = fmaf(x, gx, e[2]);
                    e[3] = fmaf(x, gy, e[3]);
                    e[4] = fmaf(x, gz, e[4]);
                    e[5] = fmaf(y, gy, e[5]);
                    e[6] = fmaf(y, gz, e[6]);
                    e[7] = fmaf(z, gz, e[7]);
                    red_add3(F + j3, -gx, -gy, -gz);
                }
            }
            const uint32_t lead = __shfl_sync(full, ij.x, 0);  // lane 0 is valid whenever any lane is
            if (__all_sync(full, !valid || ij.x == lead)) {
                if (lead != cur) {
                    flush();
                    cur = lead;
                }
                fx += gx;
                fy += gy;
                fz += gz;
                continue;
            }
            flush();
            cur = 0xffffffffu;
            unsigned left = __ballot_sync(full, valid);
            for (int g = 0; left && g < 4; ++g) {  // the first few i's by sums over their lanes
                const uint32_t i = __shfl_sync(full, ij.x, __ffs(left) - 1);
                const bool mine = valid && ij.x == i;
                const float sx = warp_sum(mine ? gx : 0.f), sy = warp_sum(mine ? gy : 0.f);
                const float sz = warp_sum(mine ? gz : 0.f);
                if (lane == 0) red_add3(F + 3 * size_t(i), sx, sy, sz);
                left &= ~__ballot_sync(full, mine);
            }
            if ((left >> lane) & 1u) red_add3(F + 3 * size_t(ij.x), gx, gy, gz);
        }
        flush();
#pragma unroll
        for (int k = 0; k < 8; ++k) sums[k] += double(e[k]);
    }
    __shared__ double sh[8][8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const double t = warp_sum_d(sums[k]);
        if (lane == 0) sh[threadIdx.x >> 5][k] = t;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        double t = 0.0;
        for (int w = 0; w < int(blockDim.x >> 5); ++w) t += sh[w][threadIdx.x];
        const int k = threadIdx.x;
        const int at = k < 5 ? k : k == 5 ? 6 : k == 6 ? 7 : 10;           // E: lj, crf, then the 3 x 3 virial
        const int mirror = k == 3 ? 5 : k == 4 ? 8 : k == 6 ? 9 : -1;
        if (t != 0.0) {
            atomicAdd(&E[at], t);
            if (mirror >= 0) atomicAdd(&E[mirror], t);
        }
    }
}

// Blocks for n_pairs: every warp a chunk, at most four blocks per SM (more only
// add block sums).
inline unsigned innerloop_grid(uint32_t n_pairs) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
        sms = 148;
    const size_t per_block = size_t(kPairIters) * 256;
    return unsigned(std::min<size_t>((size_t(n_pairs) + per_block - 1) / per_block, size_t(sms) * 4));
}
}  // namespace gnb

namespace gnb {
// FP32 FMA-pipe rate microbenchmark: eight independent FFMA chains per
// thread; every FFMA counts as one operation (the convention of the force
// kernel's 37 operations per pair).
__global__ void k_ffma_peak(float* out, int iters, float a, float b) {
    float x0 = threadIdx.x * 1e-7f, x1 = x0 + 1e-6f, x2 = x0 + 2e-6f, x3 = x0 + 3e-6f;
    float x4 = x0 + 4e-6f, x5 = x0 + 5e-6f, x6 = x0 + 6e-6f, x7 = x0 + 7e-6f;
    for (int k = 0; k < iters; ++k) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            x0 = fmaf(x0, a, b);
            x1 = fmaf(x1, a, b);
            x2 = fmaf(x2, a, b);
            x3 = fmaf(x3, a, b);
            x4 = fmaf(x4, a, b);
            x5 = fmaf(x5, a, b);
            x6 = fmaf(x6, a, b);
            x7 = fmaf(x7, a, b);
        }
    }
    float s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
    if (s == 1234.5678f) out[0] = s;  // keeps the chains live
}
}  // namespace gnb
