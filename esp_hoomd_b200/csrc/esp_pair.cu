// a8: the short-range pair term (EvaluatorPairPSWF over a neighbour list,
// src/EvaluatorPairPSWF.h:274-295 with the HOOMD PotentialPair loop).
#include "esp_common.cuh"
#include "esp_kernels.h"
#include "esp_pair.cuh"

namespace espb {

// ============================================================================
// a8: short-range pair term over a HOOMD-layout neighbour list
// (neighbours of i: nlist[head[i] + k], k < n_neigh[i], local indices).
// TPP lanes cooperate on one particle; per pair
//   pair_eng = qiqj/(4 pi) (1/r - Q(u)/r_c),  u = r^2/r_c^2
//   force_divr = qiqj/(4 pi) (1/r^3 + 2 Q'(u)/r_c^3)
// (the split form of EvaluatorPairPSWF::evalForceAndEnergy).
// ============================================================================

// Rows in 16-byte segments of four entries, one segment per lane and step; the
// next segment is loaded one step ahead of the gathers that use this one.
template <int TPP, bool WRAP, typename Eval>
__device__ __forceinline__ void pair_row(Eval& ev, const uint4* __restrict__ row, uint32_t n4, uint32_t sub,
                                         const float4& pi, const float4* __restrict__ pos) {
    uint4 jn = sub < n4 ? __ldg(&row[sub]) : make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t k4 = sub; k4 < n4; k4 += TPP) {
        const uint4 jj = jn;
        if (k4 + TPP < n4) jn = __ldg(&row[k4 + TPP]);
        const float4 p0 = __ldg(&pos[(int)jj.x]);
        const float4 p1 = __ldg(&pos[(int)jj.y]);
        const float4 p2 = __ldg(&pos[(int)jj.z]);
        const float4 p3 = __ldg(&pos[(int)jj.w]);
        ev.template pair<WRAP>(pi, p0);
        ev.template pair<WRAP>(pi, p1);
        ev.template pair<WRAP>(pi, p2);
        ev.template pair<WRAP>(pi, p3);
    }
}

// EN: pair energies (per particle and per system); without them the split
// polynomial Q itself is not needed, only Q', and the kernel (40 registers)
// keeps 6 CTAs per SM resident so that more position gathers are in flight.
template <int TPP, int NQ, bool VIR, bool EN>
__global__ void __launch_bounds__(256, EN ? 5 : 6)
    k_pair(const int2* __restrict__ chunks, const SysDev* __restrict__ sys, const ParamSet* __restrict__ psets,
           const float4* __restrict__ posq, const uint32_t* __restrict__ head, const uint32_t* __restrict__ nn,
           const uint32_t* __restrict__ nlist, float4* __restrict__ force, double* __restrict__ acc, int accumulate,
           const PairCoef pc, float* __restrict__ vpp, int vpitch, const uint32_t* __restrict__ outidx) {
    __shared__ double red[32 * 7];
    const int2 ch = chunks[blockIdx.x];
    const SysDev S = sys[ch.x];
    const ParamSet& ps = psets[S.pset];
    PairEval<NQ, VIR, EN> ev{pc};
    ev.rc2 = ps.rcut2;
    ev.irc = ps.inv_rcut;
    ev.irc2 = ps.inv_rcut * ps.inv_rcut;
    ev.tirc3 = ps.two_inv_rcut3;
    ev.Lx = S.Lx;
    ev.Ly = S.Ly;
    ev.Lz = S.Lz;
    ev.iLx = S.inv_Lx;
    ev.iLy = S.inv_Ly;
    ev.iLz = S.inv_Lz;
    const int i = ch.y + threadIdx.x / TPP;
    const int sub = threadIdx.x % TPP;
    const bool valid = i < S.p_off + S.N;
    // particles at least r_c from every face (positions are wrapped into
    // the box) see every in-cutoff neighbour in the same image; a warp whose
    // particles all are skips the minimum-image wrap (out-of-cutoff pairs
    // are masked whatever their displacement)
    bool inner = true;
    if (valid) {
        const float4 p = posq[i];
        const float rc = ps.rcut;
        inner = p.x >= rc && p.x <= S.Lx - rc && p.y >= rc && p.y <= S.Ly - rc && p.z >= rc && p.z <= S.Lz - rc;
    }
    const bool interior = __all_sync(0xffffffffu, inner);
    if (valid) {
        const float4 pi = posq[i];
        const uint32_t n = nn[i], h = head[i];
        const float4* pos = posq + S.p_off;
        const uint32_t* row = nlist + h;
        uint32_t k0 = 0;
        if ((h & 3u) == 0u) {
            const uint4* row4 = reinterpret_cast<const uint4*>(row);
            const uint32_t n4 = n >> 2;
            if (interior) pair_row<TPP, false>(ev, row4, n4, sub, pi, pos);
            else pair_row<TPP, true>(ev, row4, n4, sub, pi, pos);
            k0 = n4 << 2;
        }
        for (uint32_t k = k0 + sub; k < n; k += TPP) ev.pair(pi, __ldg(&pos[(int)__ldg(&row[k])]));
    }
    float fx = ev.fx, fy = ev.fy, fz = ev.fz, en = ev.en;
#pragma unroll
    for (int o = TPP / 2; o > 0; o >>= 1) {
        fx += __shfl_xor_sync(0xffffffffu, fx, o);
        fy += __shfl_xor_sync(0xffffffffu, fy, o);
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
        en += __shfl_xor_sync(0xffffffffu, en, o);
    }
    // rows by slot (the library's pair list): results go to the particle of the slot
    const int oi = (outidx && valid) ? (int)outidx[i] : i;
    if (valid && sub == 0) {
        float4 f = accumulate ? force[oi] : make_float4(0.f, 0.f, 0.f, 0.f);
        f.x += fx;
        f.y += fy;
        f.z += fz;
        f.w += 0.5f * en;
        force[oi] = f;
    }
    if (VIR && vpp) {
        // this particle's half of its pairs' virial (HOOMD's per-particle virial)
        float v[6] = {ev.vxx, ev.vxy, ev.vxz, ev.vyy, ev.vyz, ev.vzz};
#pragma unroll
        for (int o = TPP / 2; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 6; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if (valid && sub == 0)
#pragma unroll
            for (int k = 0; k < 6; ++k) vpp[(size_t)k * vpitch + oi] += 0.5f * v[k];
    }
    if (VIR) {
        double e[7] = {sub == 0 ? 0.5 * (double)en : 0.0, 0.5 * (double)ev.vxx, 0.5 * (double)ev.vxy,
                       0.5 * (double)ev.vxz, 0.5 * (double)ev.vyy, 0.5 * (double)ev.vyz, 0.5 * (double)ev.vzz};
        block_sum_f64<7>(e, red);
        if (threadIdx.x == 0) {
            atomicAdd(&acc[ch.x * ACC_STRIDE + ACC_E], e[0]);
#pragma unroll
            for (int k = 0; k < 6; ++k) atomicAdd(&acc[ch.x * ACC_STRIDE + ACC_WP + k], e[1 + k]);
        }
    } else if (EN) {
        double e[1] = {sub == 0 ? 0.5 * (double)en : 0.0};
        block_sum_f64<1>(e, red);
        if (threadIdx.x == 0) atomicAdd(&acc[ch.x * ACC_STRIDE + ACC_E], e[0]);
    }
}

template <int TPP, bool VIR, bool EN>
static cudaError_t launch_pair_t(const LaunchArgs& a, cudaStream_t st) {
    // the library's pair list: rows by slot over the slot-ordered positions
    const PairList* pl = a.plist;
    const float4* posq = pl ? pl->spos : a.posq;
    const uint32_t* head = pl ? pl->head : a.nl_head;
    const uint32_t* nn = pl ? pl->nn : (a.nn_limited ? a.nn_limited : a.nl_n);
    const uint32_t* nl = pl ? pl->nl : a.nl_list;
    const uint32_t* outidx = pl ? pl->slot2idx : nullptr;
#define ESPB_PAIR(NQ)                                                                                          \
    k_pair<TPP, NQ, VIR, EN><<<a.n_pchunks, 256, 0, st>>>(a.pchunks, a.sys, a.psets, posq, head, nn, nl, a.force, \
                                                          a.acc, a.accumulate, a.pc, a.virial_pp, a.vpp_pitch,    \
                                                          outidx)
    if (a.nq <= 8) { ESPB_PAIR(8); }
    else if (a.nq <= 10) { ESPB_PAIR(10); }
    else if (a.nq <= 11) { ESPB_PAIR(11); }
    else if (a.nq <= 12) { ESPB_PAIR(12); }
    else if (a.nq <= 13) { ESPB_PAIR(13); }
    else if (a.nq <= 14) { ESPB_PAIR(14); }
    else if (a.nq <= 16) { ESPB_PAIR(16); }
    else if (a.nq <= 20) { ESPB_PAIR(20); }
    else if (a.nq <= 24) { ESPB_PAIR(24); }
    else { ESPB_PAIR(32); }
#undef ESPB_PAIR
    return cudaGetLastError();
}

cudaError_t launch_pair(const LaunchArgs& a, cudaStream_t st) {
    if (a.n_pchunks == 0) return cudaSuccess;
    if (a.want_virial) {
        switch (a.tpp) {
            case 4: return launch_pair_t<4, true, true>(a, st);
            case 8: return launch_pair_t<8, true, true>(a, st);
            case 16: return launch_pair_t<16, true, true>(a, st);
            case 32: return launch_pair_t<32, true, true>(a, st);
            default: return cudaErrorInvalidValue;
        }
    }
    if (a.want_energy) {
        switch (a.tpp) {
            case 4: return launch_pair_t<4, false, true>(a, st);
            case 8: return launch_pair_t<8, false, true>(a, st);
            case 16: return launch_pair_t<16, false, true>(a, st);
            case 32: return launch_pair_t<32, false, true>(a, st);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (a.tpp) {
        case 4: return launch_pair_t<4, false, false>(a, st);
        case 8: return launch_pair_t<8, false, false>(a, st);
        case 16: return launch_pair_t<16, false, false>(a, st);
        case 32: return launch_pair_t<32, false, false>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace espb
