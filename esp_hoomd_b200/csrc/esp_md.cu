// MD harness kernels: cell-list neighbour list and velocity-Verlet halves.
// These stand in for the HOOMD-blue pieces the reference relies on
// (NeighborList and the integrator; not vendored in the reference) so the
// ESP path can run standalone.
#include <algorithm>

#include "esp_cells.cuh"
#include "esp_common.cuh"
#include "esp_kernels.h"
#include "esp_md.h"

namespace espb {

// Cell of each particle.
__global__ void k_cell_bin(const int2* __restrict__ chunks, const SysDev* __restrict__ sys,
                           const CellDev* __restrict__ cells, const float4* __restrict__ pos,
                           uint32_t* __restrict__ ckey, uint32_t* __restrict__ ccount, float4* __restrict__ wpos) {
    const int2 ch = chunks[blockIdx.x];
    const SysDev& S = sys[ch.x];
    const CellDev& C = cells[ch.x];
    const int i = ch.y + threadIdx.x;
    const bool valid = i < S.p_off + S.N;
    const float4 p = valid ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    float x = p.x - S.Lx * floorf(p.x * S.inv_Lx);
    float y = p.y - S.Ly * floorf(p.y * S.inv_Ly);
    float z = p.z - S.Lz * floorf(p.z * S.inv_Lz);
    if (x >= S.Lx) x -= S.Lx;
    if (y >= S.Ly) y -= S.Ly;
    if (z >= S.Lz) z -= S.Lz;
    int cx = min((int)(x * C.inv_wx), C.ncx - 1), cy = min((int)(y * C.inv_wy), C.ncy - 1),
        cz = min((int)(z * C.inv_wz), C.ncz - 1);
    cx = max(cx, 0);
    cy = max(cy, 0);
    cz = max(cz, 0);
    const uint32_t k = valid ? (uint32_t)(C.c_off + (cz * C.ncy + cy) * C.ncx + cx) : 0xffffffffu;
    // one atomic per distinct cell of the warp
    const unsigned grp = __match_any_sync(0xffffffffu, k);
    if (!valid) return;
    if ((threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&ccount[k], (uint32_t)__popc(grp));
    ckey[i] = k;
    wpos[i] = make_float4(x, y, z, __int_as_float(i));
}

// Deterministic order inside each cell (ascending particle index) and the
// cell-sorted positions. One thread per unsorted slot ranks its particle
// among its cell's (about 5 at density 1 and rlist 3.4): the cell's indices
// are neighbours in perm_u, so the loop reads the L1.
__global__ void __launch_bounds__(256)
    k_cell_sort(int total, const uint32_t* __restrict__ ckey, const uint32_t* __restrict__ start,
                const uint32_t* __restrict__ perm_u, const float4* __restrict__ wpos, float4* __restrict__ cpos,
                uint32_t* __restrict__ slot2idx, uint32_t* __restrict__ idx2slot) {
    const int t = blockIdx.x * 256 + threadIdx.x;
    if (t >= total) return;
    const uint32_t v = perm_u[t];
    const uint32_t c = ckey[v];
    const float4 p = wpos[v];
    const uint32_t b = start[c], e = start[c + 1];
    uint32_t r = b;
    for (uint32_t j = b; j < e; ++j) r += perm_u[j] < v ? 1u : 0u;
    cpos[r] = p;
    if (slot2idx) slot2idx[r] = v;
    if (idx2slot) idx2slot[v] = r;
}

// One CTA per cell, one thread per particle of the cell (passes of
// NL_THREADS). The particles of the 27 surrounding cells are staged in
// shared memory, in the fixed (dz, dy, dx) order and ascending slot inside
// each cell (in windows of NL_STAGE when there are more), so every row is
// deterministic; each thread scans them with broadcast shared loads (one
// wavefront serves the whole warp). With at least 3 cells on every axis each
// surrounding cell is a distinct periodic image and its particles are staged
// already shifted by that image, so the test needs no wrap; smaller cell
// grids take the minimum-image test.
constexpr int NL_THREADS = 64;
constexpr int NL_STAGE = 1024;

// Appends the staged candidates within rlist of pi, other than `self`, to
// row (staged values are already local indices or slots); threads without a
// particle carry a NaN position, which tests false against everything. Hits
// past cap are counted, and stored over the row's last entry (so an
// overflowing row still holds only neighbours; the build reports it).
// One candidate's test and append, as straight-line predicated code (no
// branch per candidate): stores w at p when r2 < rlist2 and w != self, and
// returns 1 then (0 otherwise).
__device__ __forceinline__ uint32_t append_if(float r2, float rlist2, int w, int self, uint32_t* p) {
    uint32_t inc;
    asm volatile(
        "{\n\t.reg .pred q, r;\n\tsetp.lt.f32 q, %1, %2;\n\tsetp.ne.s32 r, %3, %4;\n\tand.pred q, q, r;\n\t"
        "@q st.global.u32 [%5], %3;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(inc)
        : "f"(r2), "f"(rlist2), "r"(w), "r"(self), "l"(p)
        : "memory");
    return inc;
}

template <bool MINIMG>
__device__ __forceinline__ uint32_t nl_scan(const float4* __restrict__ cand, int n, float4 pi, int self,
                                            const SysDev& S, float rlist2, uint32_t cap, uint32_t* __restrict__ row,
                                            uint32_t cnt) {
    const uint32_t cap1 = cap - 1u;
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
        const float4 pj = cand[k];
        float ddx = pi.x - pj.x, ddy = pi.y - pj.y, ddz = pi.z - pj.z;
        if (MINIMG) {
            ddx -= S.Lx * rintf(ddx * S.inv_Lx);
            ddy -= S.Ly * rintf(ddy * S.inv_Ly);
            ddz -= S.Lz * rintf(ddz * S.inv_Lz);
        }
        cnt += append_if(ddx * ddx + ddy * ddy + ddz * ddz, rlist2, __float_as_int(pj.w), self, row + min(cnt, cap1));
    }
    return cnt;
}

// SORTED = false: HOOMD-layout rows -- the row of particle i at nl_off +
// local i * cap, entries local particle indices, head/nn indexed by
// particle. SORTED = true: the library's pair list -- the same layout indexed
// by the cell-sorted slot (row of slot s at nl_off + local s * cap, head and
// nn by slot), entries local slots. Rows longer than cap keep their first cap
// entries and set the overflow flag; overflow[1] receives the longest row and
// overflow[2] the row capacity. nn holds the counts up to nn_max.
template <bool SORTED>
__global__ void __launch_bounds__(NL_THREADS) k_nlist_cta(const int* __restrict__ cell_sys, const SysDev* __restrict__ sys,
                                                          const CellDev* __restrict__ cells,
                                                      const uint32_t* __restrict__ cstart,
                                                      const float4* __restrict__ cpos, float rlist2, int cap,
                                                      uint32_t* __restrict__ head, uint32_t* __restrict__ nn,
                                                      uint32_t* __restrict__ nl, int* __restrict__ overflow,
                                                      uint32_t nn_max) {
    __shared__ float4 cand[NL_STAGE];
    __shared__ CellNbhd nb;
    const uint32_t cidx = blockIdx.x;
    const uint32_t c0 = cstart[cidx], c1 = cstart[cidx + 1];
    if (c0 == c1) return;
    const int si = cell_sys[cidx];
    const SysDev& S = sys[si];
    const CellDev& C = cells[si];
    const int tid = threadIdx.x;
    if (tid < 32) cell_nbhd_warp((int)cidx - C.c_off, C, S, cstart, nb);
    __syncthreads();
    const bool minimg = nb.minimg != 0;
    const uint32_t total = nb.off[27];
    // staged value: the candidate's local particle index (HOOMD rows; the
    // cell-sorted positions carry the index) or its local slot (pair list)
    auto stage = [&](uint32_t base) {
        const uint32_t top = min(total, base + (uint32_t)NL_STAGE);
        for (int s = 0; s < 27; ++s) {
            const uint32_t lo = max(nb.off[s], base), hi = min(nb.off[s + 1], top);
            for (uint32_t g = lo + tid; g < hi; g += NL_THREADS) {
                const uint32_t slot = nb.src[s] + (g - nb.off[s]);
                float4 p = cpos[slot];
                p.x += nb.shift[s][0];
                p.y += nb.shift[s][1];
                p.z += nb.shift[s][2];
                // local values: the pair list's slot, or the particle index
                p.w = __int_as_float((SORTED ? (int)slot : __float_as_int(p.w)) - S.p_off);
                cand[g - base] = p;
            }
        }
    };
    const bool one_stage = total <= (uint32_t)NL_STAGE;
    if (one_stage) {
        stage(0);
        __syncthreads();
    }
    for (uint32_t p0 = c0; p0 < c1; p0 += NL_THREADS) {
        const uint32_t slot = p0 + tid;
        const bool active = slot < c1;
        const float4 pi = active ? cpos[slot] : make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, __int_as_float(-1));
        const int idx = __float_as_int(pi.w);
        const int self = (SORTED ? (int)slot : idx) - S.p_off;
        const uint32_t key = SORTED ? slot : (uint32_t)idx;  // owner of the row
        const long long hrow = C.nl_off + (long long)((int)key - S.p_off) * cap;
        uint32_t* row = nl + (active ? hrow : 0);
        uint32_t cnt = 0;
        for (uint32_t base = 0; base < total; base += NL_STAGE) {
            if (!one_stage) {
                __syncthreads();
                stage(base);
                __syncthreads();
            }
            const int n = (int)min((uint32_t)NL_STAGE, total - base);
            cnt = minimg ? nl_scan<true>(cand, n, pi, self, S, rlist2, (uint32_t)cap, row, cnt)
                         : nl_scan<false>(cand, n, pi, self, S, rlist2, (uint32_t)cap, row, cnt);
        }
        if (active) {
            head[key] = (uint32_t)hrow;
            nn[key] = min(cnt, nn_max);
            if (cnt > (uint32_t)cap) {
                atomicOr(overflow, 1);
                atomicMax(overflow + 1, (int)cnt);
                overflow[2] = cap;
            }
        }
    }
}

// Neighbour rows. One warp per cell; the cell's particles are taken eight at
// a time, their positions held by every lane, and the surrounding cells'
// particles stream past, one candidate per lane: a (dz, dy) row of up to five
// cells is contiguous in the cell-sorted order (two pieces at a periodic
// face), the rows' candidates are numbered consecutively so that every segment
// of 32 is full, and the next segment's positions are in flight. A ballot and
// a population count place each hit in its row, so a row's entries are written
// in order, neighbouring lanes side by side. Rows list the (dz, dy, dx) cells
// in that order and ascending slots inside each: they are deterministic. With
// at least 5 cells on every axis a surrounding cell is one periodic image and
// its particles are shifted by it; smaller grids visit every cell of the axis
// and take the minimum image per pair.
// Bound by issue slots (72% active; 72 registers for 7 CTAs per SM, 96 and
// fewer CTAs: 20% slower). Cells of half the list radius leave 15.6 rlist^3 of
// volume to test instead of the CTA kernel's 27, and the work falls into more
// and shorter warps (nlist_half_cells has both kernels' times). Packed FP32 pairs in
// the distance test saved no instruction (register moves) and measured 5%
// slower.
constexpr int NL_WARPS = 4;
constexpr int NL_GROUP = 8;  // particles of the cell tested per pass
constexpr int NL_MAXEX = 8;  // excluded partners per particle kept in shared memory

struct NlGroup {
    float px[NL_GROUP], py[NL_GROUP], pz[NL_GROUP];
    uint32_t pos[NL_GROUP];   // next entry of the row - 1
    uint32_t end[NL_GROUP];   // end of the row's capacity
    uint32_t hits[NL_GROUP];  // hits before exclusions (EX only)
};

// Tests candidate c (one per lane) against the group and appends value v to
// the rows of the particles within range. SELF: c may be one of the group
// (slot = c's slot, g0 = the group's first slot). EX: excluded partners'
// slots in exs, nex per particle.
template <bool MINIMG, bool SELF, bool EX>
__device__ __forceinline__ void nl_test(NlGroup& g, int ng, float4 c, uint32_t slot, uint32_t v, uint32_t g0,
                                        const SysDev& S, float rlist2, uint32_t lemask, uint32_t* __restrict__ nl,
                                        const uint32_t (*exs)[NL_MAXEX], const uint32_t* nex) {
#pragma unroll
    for (int i = 0; i < NL_GROUP; ++i) {
        if (i >= ng) break;
        float dx = g.px[i] - c.x, dy = g.py[i] - c.y, dz = g.pz[i] - c.z;
        if (MINIMG) {
            dx -= S.Lx * rintf(dx * S.inv_Lx);
            dy -= S.Ly * rintf(dy * S.inv_Ly);
            dz -= S.Lz * rintf(dz * S.inv_Lz);
        }
        const float d2 = dx * dx + dy * dy + dz * dz;
        bool in = d2 < rlist2;
        if (SELF) in = in && slot != g0 + i;
        if (EX) {
            g.hits[i] += (uint32_t)__popc(__ballot_sync(0xffffffffu, in));
            for (uint32_t x = 0; x < nex[i]; ++x) in = in && slot != exs[i][x];
        }
        const uint32_t inc = (uint32_t)__popc(__ballot_sync(0xffffffffu, in) & lemask);  // hits up to this lane
        const uint32_t e = g.pos[i] + inc;
        if (in && e < g.end[i]) nl[e] = v;
        g.pos[i] += __shfl_sync(0xffffffffu, inc, 31);
    }
}

// SORTED = false: HOOMD-layout rows -- the row of particle i at nl_off +
// local i * cap, entries local particle indices, head/nn indexed by
// particle. SORTED = true: the library's pair list -- the same layout indexed
// by the cell-sorted slot (row of slot s at nl_off + local s * cap, head and
// nn by slot), entries local slots. Rows longer than cap keep their first cap
// entries, the overflow flag is set, overflow[1] receives the longest row and
// overflow[2] the row capacity. nn holds the counts up to nn_max: the true ones
// in a caller's HOOMD rows, whose readers then take no more than overflow[2]
// entries, the kept ones in the pair list and in a server's rows. EX: the excluded partners are left out of the
// rows (a row whose hits exceed cap before that counts as overflowing).
template <bool SORTED, bool EX>
__global__ void __launch_bounds__(32 * NL_WARPS, EX ? 4 : 7)
    k_nlist(const int* __restrict__ cell_sys, int n_cells, const SysDev* __restrict__ sys,
            const CellDev* __restrict__ cells, const uint32_t* __restrict__ cstart, const float4* __restrict__ cpos,
            float rlist2, uint32_t cap, uint32_t* __restrict__ head, uint32_t* __restrict__ nn,
            uint32_t* __restrict__ nl, int* __restrict__ overflow, const uint32_t* __restrict__ ex_n,
            const uint32_t* __restrict__ ex_list, int ex_pitch, const uint32_t* __restrict__ idx2slot,
            uint32_t nn_max) {
    __shared__ uint4 srow[NL_WARPS][25];     // (dz, dy) row: its two pieces' slots (see below), first candidate
    __shared__ float2 sshift[NL_WARPS][25];  // its periodic image along y and z
    __shared__ uint32_t soff[NL_WARPS][28];  // first candidate of each row, then the total
    __shared__ uint32_t sex[NL_WARPS][EX ? NL_GROUP : 1][NL_MAXEX], snex[NL_WARPS][NL_GROUP];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cidx = blockIdx.x * NL_WARPS + warp;
    if (cidx >= (uint32_t)n_cells) return;
    const uint32_t c0 = cstart[cidx], c1 = cstart[cidx + 1];
    if (c0 + blockIdx.y * NL_GROUP >= c1) return;
    const int si = cell_sys[cidx];
    const SysDev& S = sys[si];
    const CellDev& C = cells[si];
    const int p_off = S.p_off;
    const uint32_t lemask = 0xffffffffu >> (31 - lane);
    const int ncx = C.ncx, ncy = C.ncy, ncz = C.ncz;
    const int lc = (int)cidx - C.c_off;
    const int cx = lc % ncx, cy = (lc / ncx) % ncy, cz = lc / (ncx * ncy);
    const bool minimg = ncx < 5 || ncy < 5 || ncz < 5;
    const int nry = min(ncy, 5), nrows = nry * min(ncz, 5);
    const int rself = (ncy >= 5 ? 2 : cy) + nry * (ncz >= 5 ? 2 : cz);  // the cell's own row
    // five cells from cx - 2; at a face the part beyond it is the second piece
    // (its last cells' piece first at the low face)
    const bool wlo = ncx >= 5 && cx < 2, whi = ncx >= 5 && cx + 2 >= ncx;
    uint32_t len = 0;
    uint4 t = make_uint4(0u, 0u, 0u, 0u);
    if (lane < nrows) {
        int yy = lane % nry, zz = lane / nry;
        float shy = 0.f, shz = 0.f;
        if (ncy >= 5) {
            yy += cy - 2;
            if (yy < 0) { yy += ncy; shy = -S.Ly; } else if (yy >= ncy) { yy -= ncy; shy = S.Ly; }
        }
        if (ncz >= 5) {
            zz += cz - 2;
            if (zz < 0) { zz += ncz; shz = -S.Lz; } else if (zz >= ncz) { zz -= ncz; shz = S.Lz; }
        }
        const uint32_t* rowc = cstart + C.c_off + (zz * ncy + yy) * ncx;
        const int xa = wlo ? cx - 2 + ncx : (ncx >= 5 ? cx - 2 : 0);
        const int xb = wlo || whi || ncx < 5 ? ncx : cx + 3;
        t.x = rowc[xa];
        t.y = rowc[xb] - t.x;
        len = t.y;
        if (wlo || whi) {
            t.z = rowc[0];
            len += rowc[wlo ? cx + 3 : cx + 3 - ncx] - t.z;
        }
        sshift[warp][lane] = minimg ? make_float2(0.f, 0.f) : make_float2(shy, shz);
    }
    // the rows' candidates numbered consecutively; candidate g of row r is the
    // slot (g < y ? x : z) + g of its srow entry (slot offsets less the row's
    // first candidate)
    uint32_t inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    if (lane < nrows) {
        const uint32_t o = inc - len;
        soff[warp][lane + 1] = inc;
        srow[warp][lane] = make_uint4(t.x - o, t.y + o, t.z - t.y - o, 0u);
        if (lane == 0) soff[warp][0] = 0u;
    }
    __syncwarp();
    const uint32_t self0 = soff[warp][rself], self1 = soff[warp][rself + 1];
    const float shx1 = wlo && !minimg ? -S.Lx : 0.f, shx2 = whi && !minimg ? S.Lx : 0.f;
    // several CTAs share a row of cells (grid y) when the cells hold more than a group
    for (uint32_t g0 = c0 + blockIdx.y * NL_GROUP; g0 < c1; g0 += gridDim.y * NL_GROUP) {
        const int ng = (int)min(c1 - g0, (uint32_t)NL_GROUP);
        NlGroup g;
        uint32_t mykey = 0, myrow = 0;  // lane k < ng: owner and first entry of the k-th row
#pragma unroll
        for (int i = 0; i < NL_GROUP; i += 2) {
            // past the group's last particle: the cell's last one again, which
            // nl_test leaves out (i >= ng)
            const float4 a = cpos[min(g0 + i, c1 - 1)], b = cpos[min(g0 + i + 1, c1 - 1)];
            g.px[i] = a.x, g.py[i] = a.y, g.pz[i] = a.z;
            g.px[i + 1] = b.x, g.py[i + 1] = b.y, g.pz[i + 1] = b.z;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t key = SORTED ? g0 + i + h : (uint32_t)__float_as_int(h ? b.w : a.w);
                const uint32_t row = (uint32_t)(C.nl_off + (long long)((int)key - p_off) * (long long)cap);
                g.pos[i + h] = row - 1u;
                g.end[i + h] = row + cap;
                g.hits[i + h] = 0u;
                if (lane == i + h) {
                    mykey = key;
                    myrow = row;
                }
            }
            if (EX) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (lane == i + h && lane < ng) {
                        const uint32_t idx = (uint32_t)__float_as_int(h ? b.w : a.w);
                        const uint32_t ne = min(ex_n[idx], (uint32_t)ex_pitch);
                        uint32_t m = 0;
                        for (uint32_t x = 0; x < ne && m < NL_MAXEX; ++x) {
                            const uint32_t jl = ex_list[(size_t)idx * ex_pitch + x];
                            if (jl < (uint32_t)S.N) sex[warp][lane][m++] = idx2slot[p_off + (int)jl];
                        }
                        snex[warp][lane] = m;
                    }
            }
        }
        if (EX) {
            if (lane >= ng && lane < NL_GROUP) snex[warp][lane] = 0u;
            __syncwarp();
        }
        // segments of 32 candidates, the next one's positions in flight
        int r = 0;  // row of this lane's candidate
        float4 cn = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t slot_n = 0;
        auto fetch = [&](uint32_t c) {  // candidate c of this lane (a NaN position past the last)
            cn = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
            if (c < total) {
                while (c >= soff[warp][r + 1]) ++r;
                const uint4 w = srow[warp][r];
                const float2 sh = sshift[warp][r];
                const bool second = c >= w.y;
                slot_n = (second ? w.z : w.x) + c;
                cn = cpos[slot_n];
                cn.x += second ? shx2 : shx1;
                cn.y += sh.x;
                cn.z += sh.y;
            }
        };
        fetch(lane);
        for (uint32_t b0 = 0; b0 < total; b0 += 32) {
            const float4 c = cn;
            const uint32_t slot = slot_n, v = (SORTED ? slot : (uint32_t)__float_as_int(c.w)) - (uint32_t)p_off;
            if (b0 + 32 < total) fetch(b0 + 32 + lane);
            if (minimg) nl_test<true, true, EX>(g, ng, c, slot, v, g0, S, rlist2, lemask, nl, sex[warp], snex[warp]);
            else if (b0 < self1 && b0 + 32 > self0)
                nl_test<false, true, EX>(g, ng, c, slot, v, g0, S, rlist2, lemask, nl, sex[warp], snex[warp]);
            else nl_test<false, false, EX>(g, ng, c, slot, v, g0, S, rlist2, lemask, nl, sex[warp], snex[warp]);
        }
        uint32_t cnt = 0, hits = 0;
#pragma unroll
        for (int i = 0; i < NL_GROUP; ++i)
            if (lane == i) {
                cnt = g.pos[i] + 1u - myrow;
                hits = EX ? g.hits[i] : cnt;
            }
        if (lane < ng) {
            head[mykey] = myrow;
            nn[mykey] = min(cnt, nn_max);
            if (hits > cap) {
                atomicOr(overflow, 1);
                atomicMax(overflow + 1, (int)hits);
                overflow[2] = (int)cap;
            }
        }
        __syncwarp();
    }
}

// Leaves the excluded partners out of the rows of particles with more than
// `done` exclusions: one thread per row, in place, the kept entries in their
// order; the count drops by the entries removed from the stored part.
template <bool SORTED>
__global__ void k_nlist_exclude(const int2* __restrict__ chunks, const SysDev* __restrict__ sys,
                                const uint32_t* __restrict__ head, uint32_t* __restrict__ nn,
                                uint32_t* __restrict__ nl, int cap, const uint32_t* __restrict__ ex_n,
                                const uint32_t* __restrict__ ex_list, int ex_pitch,
                                const uint32_t* __restrict__ slot2idx, const uint32_t* __restrict__ idx2slot, int done) {
    const int2 ch = chunks[blockIdx.x];
    const SysDev& S = sys[ch.x];
    const int key = ch.y + threadIdx.x;  // the row: a slot (pair list) or a particle
    if (key >= S.p_off + S.N) return;
    const int i = SORTED ? (int)slot2idx[key] : key;
    const int ne = min((int)ex_n[i], ex_pitch);
    if (ne <= done) return;
    uint32_t* row = nl + head[key];
    const uint32_t cnt = nn[key];
    const uint32_t n = min(cnt, (uint32_t)cap);
    uint32_t w = 0;
    for (uint32_t r = 0; r < n; ++r) {
        const uint32_t v = row[r];
        bool drop = false;
        for (int k = 0; k < ne; ++k) {
            const uint32_t jl = ex_list[(size_t)i * ex_pitch + k];
            if (jl < (uint32_t)S.N) drop |= v == (SORTED ? idx2slot[S.p_off + (int)jl] - (uint32_t)S.p_off : jl);
        }
        if (!drop) row[w++] = v;
    }
    nn[key] = cnt - (n - w);
}

// skip (may be NULL): per system, the local particle range [x, y) of rigid
// molecules, which the constraint kernels integrate instead
__global__ void k_nve1(const int2* __restrict__ chunks, const SysDev* __restrict__ sys, float4* __restrict__ pos,
                       float4* __restrict__ vel, const float4* __restrict__ force, float dt,
                       const int2* __restrict__ skip) {
    const int2 ch = chunks[blockIdx.x];
    const SysDev& S = sys[ch.x];
    const int i = ch.y + threadIdx.x;
    if (i >= S.p_off + S.N) return;
    if (skip) {
        const int2 r = skip[ch.x];
        if (i - S.p_off >= r.x && i - S.p_off < r.y) return;
    }
    float4 v = vel[i];
    const float4 f = force[i];
    const float h = 0.5f * dt / v.w;
    v.x += h * f.x;
    v.y += h * f.y;
    v.z += h * f.z;
    float4 p = pos[i];
    p.x += dt * v.x;
    p.y += dt * v.y;
    p.z += dt * v.z;
    p.x -= S.Lx * floorf(p.x * S.inv_Lx);
    p.y -= S.Ly * floorf(p.y * S.inv_Ly);
    p.z -= S.Lz * floorf(p.z * S.inv_Lz);
    if (p.x >= S.Lx) p.x -= S.Lx;
    if (p.y >= S.Ly) p.y -= S.Ly;
    if (p.z >= S.Lz) p.z -= S.Lz;
    pos[i] = p;
    vel[i] = v;
}

__global__ void k_nve2(const int2* __restrict__ chunks, const SysDev* __restrict__ sys, float4* __restrict__ vel,
                       const float4* __restrict__ force, float dt) {
    const int2 ch = chunks[blockIdx.x];
    const SysDev& S = sys[ch.x];
    const int i = ch.y + threadIdx.x;
    if (i >= S.p_off + S.N) return;
    float4 v = vel[i];
    const float4 f = force[i];
    const float h = 0.5f * dt / v.w;
    v.x += h * f.x;
    v.y += h * f.y;
    v.z += h * f.z;
    vel[i] = v;
}

// Lennard-Jones core repulsion of the MD harness (the C1 workload's
// LJ eps, sigma, r_cut), over the same full neighbour list: adds forces and
// half the pair energy per particle to force, the system total to energy[s].
// TPP lanes share one particle's row (consecutive lanes read consecutive
// entries) and a 256-particle chunk is spread over TPP CTAs; the kernel is a
// chain of dependent gathers, so its time is the entries per lane. One lane
// per particle left 164 of them in series on 4 CTAs (N = 1,000, FP64: 102 us
// per launch); 32 lanes leave 6 on 125 CTAs (5.8 us).
template <typename T4, typename T, int TPP>
__global__ void __launch_bounds__(256)
    k_lj(const int2* __restrict__ chunks, const SysDev* __restrict__ sys, const T4* __restrict__ pos,
         const uint32_t* __restrict__ head, const uint32_t* __restrict__ nn, const uint32_t* __restrict__ nl,
         const uint32_t* __restrict__ row_limit, T eps, T sig2, T rc2, T4* __restrict__ force,
         double* __restrict__ energy) {
    __shared__ double red[32];
    const int2 ch = chunks[blockIdx.x / TPP];
    const SysDev& S = sys[ch.x];
    const int i = ch.y + (blockIdx.x % TPP) * (256 / TPP) + threadIdx.x / TPP, sub = threadIdx.x % TPP;
    const T Lx = (T)S.Lxd, Ly = (T)S.Lyd, Lz = (T)S.Lzd;
    const T iLx = (T)1 / Lx, iLy = (T)1 / Ly, iLz = (T)1 / Lz;
    const bool valid = i < S.p_off + S.N;
    const int po = S.p_off;
    T fx = 0, fy = 0, fz = 0, en = 0;
    if (valid) {
        const T4 pi = pos[i];
        const uint32_t h = head[i], n = row_entries(nn[i], row_limit);
        uint32_t jn = sub < n ? nl[h + sub] : 0u;
        for (uint32_t k = sub; k < n; k += TPP) {
            const T4 pj = pos[po + (int)jn];
            if (k + TPP < n) jn = nl[h + k + TPP];  // loaded one step ahead of its gather
            T dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            // minimum image by the reciprocal box length; it differs from a
            // division only for pairs at |d| = L/2, beyond every listed cutoff
            dx -= Lx * rint(dx * iLx);
            dy -= Ly * rint(dy * iLy);
            dz -= Lz * rint(dz * iLz);
            const T r2 = dx * dx + dy * dy + dz * dz;
            if (r2 < rc2 && r2 > 0) {
                const T i2 = (T)1 / r2, s2 = sig2 * i2, s6 = s2 * s2 * s2;
                const T fdr = (T)24 * eps * ((T)2 * s6 * s6 - s6) * i2;
                en += (T)4 * eps * (s6 * s6 - s6);
                fx += fdr * dx;
                fy += fdr * dy;
                fz += fdr * dz;
            }
        }
    }
#pragma unroll
    for (int o = TPP / 2; o > 0; o >>= 1) {
        fx += __shfl_xor_sync(0xffffffffu, fx, o);
        fy += __shfl_xor_sync(0xffffffffu, fy, o);
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
        en += __shfl_xor_sync(0xffffffffu, en, o);
    }
    double e1[1] = {0.0};
    if (valid && sub == 0) {
        T4 f = force[i];
        f.x += fx;
        f.y += fy;
        f.z += fz;
        f.w += (T)0.5 * en;
        force[i] = f;
        e1[0] = 0.5 * (double)en;
    }
    block_sum_f64<1>(e1, red);
    if (threadIdx.x == 0 && energy) atomicAdd(&energy[ch.x], e1[0]);
}

__global__ void k64_nve1(const int2* __restrict__ chunks, const SysDev* __restrict__ sys, double4* __restrict__ pos,
                         double4* __restrict__ vel, const double4* __restrict__ force, double dt,
                         const int2* __restrict__ skip) {
    const int2 ch = chunks[blockIdx.x];
    const SysDev& S = sys[ch.x];
    const int i = ch.y + threadIdx.x;
    if (i >= S.p_off + S.N) return;
    if (skip) {
        const int2 r = skip[ch.x];
        if (i - S.p_off >= r.x && i - S.p_off < r.y) return;
    }
    double4 v = vel[i];
    const double4 f = force[i];
    const double h = 0.5 * dt / v.w;
    v.x += h * f.x;
    v.y += h * f.y;
    v.z += h * f.z;
    double4 p = pos[i];
    const double L[3] = {S.Lxd, S.Lyd, S.Lzd};
    double x[3] = {p.x + dt * v.x, p.y + dt * v.y, p.z + dt * v.z};
    for (int a = 0; a < 3; ++a) {
        x[a] -= L[a] * floor(x[a] / L[a]);
        if (x[a] >= L[a]) x[a] -= L[a];
        if (x[a] < 0.0) x[a] += L[a];
    }
    pos[i] = make_double4(x[0], x[1], x[2], p.w);
    vel[i] = v;
}

__global__ void k64_nve2(const int2* __restrict__ chunks, const SysDev* __restrict__ sys, double4* __restrict__ vel,
                         const double4* __restrict__ force, double dt) {
    const int2 ch = chunks[blockIdx.x];
    const SysDev& S = sys[ch.x];
    const int i = ch.y + threadIdx.x;
    if (i >= S.p_off + S.N) return;
    double4 v = vel[i];
    const double4 f = force[i];
    const double h = 0.5 * dt / v.w;
    v.x += h * f.x;
    v.y += h * f.y;
    v.z += h * f.z;
    vel[i] = v;
}

constexpr int LJ_WARP_CHUNKS = 37;  // 148 SMs x 64 warps / 256 particles

template <typename T4, typename T>
static void lj_launch(const int2* chunks, int n_chunks, const SysDev* sys, const void* pos, const uint32_t* head,
                      const uint32_t* nn, const uint32_t* nl, const uint32_t* row_limit, double eps, double sigma,
                      double rcut, void* force, double* energy, cudaStream_t st) {
    const T e = (T)eps, s2 = (T)(sigma * sigma), r2 = (T)(rcut * rcut);
    // a warp per particle while that does not oversubscribe the GPU (148 SMs
    // x 64 warps, 256-particle chunks), else 8 lanes: fewer idle lanes in the
    // last pass over a row and cheaper reductions
    if (n_chunks <= LJ_WARP_CHUNKS)
        k_lj<T4, T, 32><<<n_chunks * 32, 256, 0, st>>>(chunks, sys, (const T4*)pos, head, nn, nl, row_limit, e, s2, r2,
                                                       (T4*)force, energy);
    else
        k_lj<T4, T, 8><<<n_chunks * 8, 256, 0, st>>>(chunks, sys, (const T4*)pos, head, nn, nl, row_limit, e, s2, r2,
                                                     (T4*)force, energy);
}

cudaError_t launch_lj(const int2* chunks, int n_chunks, const SysDev* sys, const void* pos, const uint32_t* head,
                      const uint32_t* nn, const uint32_t* nl, const uint32_t* row_limit, double eps, double sigma,
                      double rcut, void* force, double* energy, bool f64, cudaStream_t st) {
    if (n_chunks == 0) return cudaSuccess;
    if (f64)
        lj_launch<double4, double>(chunks, n_chunks, sys, pos, head, nn, nl, row_limit, eps, sigma, rcut, force, energy,
                                   st);
    else
        lj_launch<float4, float>(chunks, n_chunks, sys, pos, head, nn, nl, row_limit, eps, sigma, rcut, force, energy,
                                 st);
    return cudaGetLastError();
}

cudaError_t launch_nve64(int half, const int2* chunks, int n_chunks, const SysDev* sys, double4* pos, double4* vel,
                         const double4* force, double dt, cudaStream_t st, const int2* skip) {
    if (n_chunks == 0) return cudaSuccess;
    if (half == 1) k64_nve1<<<n_chunks, 256, 0, st>>>(chunks, sys, pos, vel, force, dt, skip);
    else k64_nve2<<<n_chunks, 256, 0, st>>>(chunks, sys, vel, force, dt);
    return cudaGetLastError();
}

cudaError_t launch_nlist(const NlistArgs& a, cudaStream_t st) {
    if (a.n_chunks == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(a.overflow, 0, NLIST_STATE * sizeof(int), st);
    if (e != cudaSuccess) return e;
    k_cell_bin<<<a.n_chunks, 256, 0, st>>>(a.chunks, a.sys, a.cells, a.pos, a.ckey, a.ccount, a.wpos);
    if ((e = launch_scan(a.ccount, a.cstart, a.n_cells, a.scan_ws, st)) != cudaSuccess) return e;
    if ((e = launch_scatter(a.chunks, a.n_chunks, a.sys, a.ckey, a.cstart, a.ccount, a.perm_u, st)) != cudaSuccess)
        return e;
    k_cell_sort<<<(a.total + 255) / 256, 256, 0, st>>>(a.total, a.ckey, a.cstart, a.perm_u, a.wpos, a.cpos, a.slot2idx,
                                                       a.idx2slot);
    const uint32_t nn_max = a.clamp_counts ? (uint32_t)a.cap : 0xffffffffu;
    if (a.half) {
        // one warp per group of NL_GROUP particles in a cell of the mean occupancy
        const dim3 grid((a.n_cells + NL_WARPS - 1) / NL_WARPS,
                        std::min(8, 1 + (int)(a.total / ((long long)NL_GROUP * a.n_cells))));
        const auto rows = a.sorted ? (a.ex_n ? k_nlist<true, true> : k_nlist<true, false>)
                                   : (a.ex_n ? k_nlist<false, true> : k_nlist<false, false>);
        rows<<<grid, 32 * NL_WARPS, 0, st>>>(a.cell_sys, a.n_cells, a.sys, a.cells, a.cstart, a.cpos, a.rlist2,
                                             (uint32_t)a.cap, a.head, a.nn, a.nl, a.overflow, a.ex_n, a.ex_list,
                                             a.ex_pitch, a.idx2slot, nn_max);
    } else {
        const auto rows = a.sorted ? k_nlist_cta<true> : k_nlist_cta<false>;
        rows<<<a.n_cells, NL_THREADS, 0, st>>>(a.cell_sys, a.sys, a.cells, a.cstart, a.cpos, a.rlist2, a.cap, a.head,
                                               a.nn, a.nl, a.overflow, nn_max);
    }
    const int done = a.half ? NL_MAXEX : 0;  // exclusions per particle left out already
    if (a.ex_n && a.ex_pitch > done) {
        const auto rest = a.sorted ? k_nlist_exclude<true> : k_nlist_exclude<false>;
        rest<<<a.n_chunks, 256, 0, st>>>(a.chunks, a.sys, a.head, a.nn, a.nl, a.cap, a.ex_n, a.ex_list, a.ex_pitch,
                                         a.slot2idx, a.idx2slot, done);
    }
    return cudaGetLastError();
}

cudaError_t launch_nve1(const int2* chunks, int n_chunks, const SysDev* sys, float4* pos, float4* vel,
                        const float4* force, float dt, cudaStream_t st, const int2* skip) {
    if (n_chunks == 0) return cudaSuccess;
    k_nve1<<<n_chunks, 256, 0, st>>>(chunks, sys, pos, vel, force, dt, skip);
    return cudaGetLastError();
}

cudaError_t launch_nve2(const int2* chunks, int n_chunks, const SysDev* sys, float4* vel, const float4* force,
                        float dt, cudaStream_t st) {
    if (n_chunks == 0) return cudaSuccess;
    k_nve2<<<n_chunks, 256, 0, st>>>(chunks, sys, vel, force, dt);
    return cudaGetLastError();
}

}  // namespace espb
