// Shared device-side definitions for the ESP kernels (sm_100a).
//
// Every kernel is batched: it reads a per-system descriptor (SysDev) and a
// work-item list, so the plain one-system path is the same code launched on
// a batch of one. Mesh layout is x-fastest, cell = (z*ny + y)*nx + x, as in
// the reference (src/ESPForceComputeGPU.cu:267).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace espb {

constexpr int MAX_P = 12;      // ESP_MAX_ORDER (src/ESPForceCompute.h:63)
constexpr int MAX_D = 15;      // window polynomial degree limit
constexpr int MAX_QC = 32;     // split polynomial coefficients
constexpr int ACC_STRIDE = 24; // doubles of per-system accumulators
constexpr int FFT_MAX_N = 256; // longest 1D transform (2/3/5-smooth)
// Columns per CTA in the y/z passes: 8 (25 KB of shared memory at 200 points, 5
// CTAs per SM by registers) where 16 let 4 of them wait out their stages (mesh
// 200^3: z pass 77.5 -> 63.0 us, y passes 38.1 -> 33.7). The x passes keep 8
// row pairs: with 4 they took 47.7 / 52.9 us instead of 36.3 / 48.2.
constexpr int FFT_B_YZ = 8;
constexpr int FFT_B_X = 8;     // row pairs per CTA in the x passes
constexpr int FFT_SB_X = 9;    // padded line stride of the x passes (bank-conflict free)
constexpr float INV_4PI_F = 0.0795774715459476678f;
constexpr double INV_4PI_D = 0.079577471545947673;  // ESP_INV_4PI, src/ESPForceCompute.cc:36

// Accumulator slots (double[ACC_STRIDE] per system).
enum AccSlot {
    ACC_QSUM = 0,   // sum q
    ACC_Q2SUM = 1,  // sum q^2
    ACC_E = 2,      // sum of per-particle energies (mesh + self + pair)
    ACC_EK = 3,     // k-space energy (diagnostic, with the virial; equals the mesh energy)
    ACC_WK = 4,     // k-space virial xx,xy,xz,yy,yz,zz (4..9)
    ACC_WP = 10,    // pair virial (10..15)
    ACC_WX = 16,    // exclusion-correction virial (16..21)
};

struct SysDev {
    int N;             // particles
    int p_off;         // first particle in the concatenated arrays
    int nx, ny, nz, nxh;
    long long m_off;   // real-mesh element offset
    long long s_off;   // half-spectrum element offset (float2)
    long long g_off;   // influence-table element offset (float2)
    int ntx, nty, ntz, t_off;  // tile grid and first tile
    float Lx, Ly, Lz;
    float inv_Lx, inv_Ly, inv_Lz;
    double gxd, gyd, gzd;  // n / L in FP64
    double Lxd, Lyd, Lzd;  // box lengths in FP64 (FP64 mode)
    double V;
    int pset;          // parameter-set index
    int twx, twy, twz; // twiddle-table offsets per axis
    uint32_t radx, rady, radz;  // packed radix plans (4 bits per stage)
    // potential mesh with a periodic halo: nxp x nyp x nzp (x fastest) at
    // element offset mp_off, point (x, y, z) holding phi(x mod nx, y mod ny,
    // z mod nz), so every tile's extended region is one box without wrap
    long long mp_off;
    int nxp, nyp, nzp;
};

// Padded extent of the halo potential mesh along an axis of n points with
// tiles of edge T and support P: every tile's extended region [t T, t T +
// T + P - 1) lies inside; x rows are rounded up to whole 16-byte groups.
__host__ __device__ inline int halo_extent(int n, int T, int P, bool x_axis) {
    const int e = ((n + T - 1) / T) * T + P - 1;
    return x_axis ? (e + 3) & ~3 : e;
}

struct ParamSet {
    float wcoef[MAX_P * (MAX_D + 1)];  // window polynomial [a][j] in t
    float qv[MAX_QC];    // Q(v) = sum qv[j] v^j, v = 2u - 1, u = r^2/r_c^2
    float dqv[MAX_QC];   // dQ/du as a series in v
    int nq;              // number of Q coefficients (dQ has nq-1)
    float rcut, rcut2, inv_rcut, two_inv_rcut3;
    double self_coef;    // per-particle self energy = self_coef * q^2
    double bg_coef;      // E_bg = bg_coef * Q^2 / V
    double rcut_d;       // r_c in FP64 (FP64 mode)
};

// ----------------------------------------------------------------------------
// small helpers
// ----------------------------------------------------------------------------
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {  // a * conj(b)
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// Kahan-compensated update of (sum, comp) in shared memory; rounding is
// pinned with the _rn intrinsics so the compiler cannot re-associate.
__device__ __forceinline__ void kahan_add(float* sum, float* comp, float v) {
    const float s = *sum;
    const float y = __fsub_rn(v, *comp);
    const float t = __fadd_rn(s, y);
    *comp = __fsub_rn(__fsub_rn(t, s), y);
    *sum = t;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide FP64 sum of K values; result valid in thread 0.
template <int K>
__device__ __forceinline__ void block_sum_f64(double (&v)[K], double* red /* smem [32*K] */) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = warp_sum(v[k]);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) red[wid * K + k] = v[k];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double x = lane < nw ? red[lane * K + k] : 0.0;
            v[k] = warp_sum(x);
        }
    }
}

// Window weights: every segment is evaluated at the same local t.
__device__ __forceinline__ float horner_w(const float* c, int D, float t) {
    float v = c[D];
    for (int j = D - 1; j >= 0; --j) v = fmaf(v, t, c[j]);
    return v;
}
__device__ __forceinline__ float horner_dw(const float* c, int D, float t) {
    float v = D * c[D];
    for (int j = D - 1; j >= 1; --j) v = fmaf(v, t, j * c[j]);
    return v;
}

// Default window degree of the FP32 path for support P (what the planner
// picks when the degree is not set; the staging kernels unroll this case
// fully): P for P >= 8 (fit error 4.7e-9 at P = 8, below the FP32
// evaluation's rounding), 9 below that. The FP64 mode uses max(P + 2, 9).
__host__ __device__ constexpr int default_window_degree(int P) { return P >= 8 ? P : 9; }
template <int P>
constexpr int default_window_degree() {
    return default_window_degree(P);
}

// One window segment held in registers by the thread that evaluates it
// (degree DD at compile time, or a runtime degree through shared memory).
template <int DD>
struct SegPoly {
    float c[DD + 1];  // w(t)  = sum_j c[j] t^j
    float d[DD];      // w'(t) = sum_j d[j] t^j, d[j] = (j+1) c[j+1]
    __device__ __forceinline__ void load(const float* wc_seg) {
#pragma unroll
        for (int j = 0; j <= DD; ++j) c[j] = wc_seg[j];
#pragma unroll
        for (int j = 0; j < DD; ++j) d[j] = (float)(j + 1) * c[j + 1];
    }
    __device__ __forceinline__ float w(float t) const {
        float v = c[DD];
#pragma unroll
        for (int j = DD - 1; j >= 0; --j) v = fmaf(v, t, c[j]);
        return v;
    }
    __device__ __forceinline__ float dw(float t) const {
        float v = d[DD - 1];
#pragma unroll
        for (int j = DD - 2; j >= 0; --j) v = fmaf(v, t, d[j]);
        return v;
    }
};

// Launch FN<P> for a stencil order known at run time (2..ESP_MAX_ORDER).
#define ESPB_DISPATCH_P(FN, P_, ...)                 \
    switch (P_) {                                    \
        case 2: return FN<2>(__VA_ARGS__);           \
        case 3: return FN<3>(__VA_ARGS__);           \
        case 4: return FN<4>(__VA_ARGS__);           \
        case 5: return FN<5>(__VA_ARGS__);           \
        case 6: return FN<6>(__VA_ARGS__);           \
        case 7: return FN<7>(__VA_ARGS__);           \
        case 8: return FN<8>(__VA_ARGS__);           \
        case 9: return FN<9>(__VA_ARGS__);           \
        case 10: return FN<10>(__VA_ARGS__);         \
        case 11: return FN<11>(__VA_ARGS__);         \
        case 12: return FN<12>(__VA_ARGS__);         \
        default: return cudaErrorInvalidValue;       \
    }

// Buckets of the per-tile sorts: y origins inside a tile (the tile edge is at most 64), or ranges of
// particle indices.
constexpr int SORT_BUCKETS = 64;

// starts of the buckets from their counts (first warp); cnt becomes the fill
// cursor, a bucket's end once it is filled
__device__ __forceinline__ void bucket_starts(uint32_t* cnt, uint32_t* beg) {
    if (threadIdx.x >= 32) return;
    const int l = threadIdx.x;
    const uint32_t a = cnt[2 * l], b = cnt[2 * l + 1];
    uint32_t x = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (l >= o) x += y;
    }
    beg[2 * l] = x - a - b;
    beg[2 * l + 1] = x - b;
    cnt[2 * l] = x - a - b;
    cnt[2 * l + 1] = x - b;
}

// First mesh point of the stencil of a particle at grid coordinate g, from
// u = g - P/2: floor(u) + 1, in [-P + 1, n + 1]. g lies in [0, n) unless the
// position is not finite or too large to be wrapped; then some point of that
// range is returned, so that every index stays inside the mesh, and the stencil
// coordinate carries the non-finite value on into the forces.
__device__ __forceinline__ int stencil_origin(double u, int P, int n) {
    return min(max(__double2int_rd(u), -P), n) + 1;
}

// Entries of a neighbour row that may be read: n, or the row capacity when the
// limit is set (the library built the rows and one of them overflowed, so that
// n may be a count its row does not hold).
__device__ __forceinline__ uint32_t row_entries(uint32_t n, uint32_t limit) { return limit ? min(n, limit) : n; }
__device__ __forceinline__ uint32_t row_entries(uint32_t n, const uint32_t* __restrict__ limit) {
    return limit ? row_entries(n, *limit) : n;
}

// shift that puts index offsets up to `range` into 2^LOG buckets, in order
template <int LOG = 6>
__device__ __forceinline__ int index_bucket_shift(uint32_t range) {
    return max(0, 32 - LOG - __clz((int)range));
}
static_assert(1 << 6 == SORT_BUCKETS);

// Index order of a tile that the shared memory of the tile sorts does not hold
// (perm_u[s0, s0 + n) in any order): LARGE_BUCKETS ranges of indices counted in
// shared memory (cnt, beg: LARGE_BUCKETS words each; lo, hi: one word), the
// indices laid out range by range in perm, each ranked inside its range, and
// the records gathered. Called by the whole CTA. Ranking such a tile against
// all of itself is n^2 reads of memory, which beside the pair term waited for
// its place in the L1 as well (98,304 water charges, support 6, FP64: r_c 1.2
// nm, tiles of 4,700, 5,097 -> 728 us per evaluation; r_c 1.0, 2,700, 914 ->
// 498; 32,768 ions, r_c 6, 6,008 -> 495).
constexpr int LARGE_LOG = 10, LARGE_BUCKETS = 1 << LARGE_LOG;
template <typename T4>
__device__ void sort_large_tile(uint32_t s0, uint32_t n, uint32_t* perm_u, uint32_t* perm,
                                const T4* __restrict__ trec, const uint32_t* __restrict__ rel,
                                T4* __restrict__ srec, uint32_t* __restrict__ srel, uint32_t* cnt, uint32_t* beg,
                                uint32_t* lo, uint32_t* hi) {
    for (uint32_t i = threadIdx.x; i < LARGE_BUCKETS; i += blockDim.x) cnt[i] = 0u;
    if (threadIdx.x == 0) {
        *lo = 0xffffffffu;
        *hi = 0u;
    }
    __syncthreads();
    uint32_t a = 0xffffffffu, b = 0u;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t v = perm_u[s0 + i];
        a = min(a, v);
        b = max(b, v);
    }
    a = __reduce_min_sync(0xffffffffu, a);
    b = __reduce_max_sync(0xffffffffu, b);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(lo, a);
        atomicMax(hi, b);
    }
    __syncthreads();
    const uint32_t v0 = *lo;
    const int sh = index_bucket_shift<LARGE_LOG>(*hi - v0);
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&cnt[(perm_u[s0 + i] - v0) >> sh], 1u);
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t carry = 0;
        for (int k = threadIdx.x; k < LARGE_BUCKETS; k += 32) {
            const uint32_t c = cnt[k];
            uint32_t x = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if ((int)threadIdx.x >= o) x += y;
            }
            beg[k] = cnt[k] = carry + x - c;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t v = perm_u[s0 + i];
        perm[s0 + atomicAdd(&cnt[(v - v0) >> sh], 1u)] = v;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t v = perm[s0 + i], bk = (v - v0) >> sh, b0 = beg[bk], b1 = cnt[bk];
        const T4 rec = trec[v];
        const uint32_t rl = rel[v];
        uint32_t r = b0;
        for (uint32_t j = b0; j < b1; ++j) r += perm[s0 + j] < v ? 1u : 0u;
        perm_u[s0 + r] = v;
        srec[s0 + r] = rec;
        srel[s0 + r] = rl;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) perm[s0 + i] = perm_u[s0 + i];
}

}  // namespace espb
