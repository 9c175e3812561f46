// zsc_init.cu -- initial condition kernels.
//
// bubble_phi_kernel   : src/init.c:39-59 (phi from the bubble list, on the GPU)
// equilibrium_*kernel : src/init_f.cu:42-79 and src/init_g.cu:46-93
#include "lattice.cuh"

namespace lbm {
namespace {

constexpr float kW0 = 0.33333333333333333333f;  // src/constants.h:52-54
constexpr float kW1 = 0.05555555555555555556f;
constexpr float kW2 = 0.02777777777777777778f;
constexpr float kInv6 = 0.16666666666666666667f;

// phi on nx * ny * (nz + 2) nodes: plane kk is the reference's plane
// k = kk + kk0 (the two ghost planes included; kk0 = z0 for a z-slab starting
// at plane z0 of a larger box, as a rank of the reference sets its own planes
// from the bubble list), x and y 0-based.  For each bubble in file
// order, nodes with R <= Rc + width take phiStar * tanh(2 (Rc - R) / width),
// the others keep -phiStar; the last bubble that covers a node wins.  The
// distance and the comparison use round-to-nearest float operations without
// contraction, so the covered set is the one the reference's host code gets.
__global__ void bubble_phi_kernel(Box b, const float *__restrict__ bubbles, int nbubbles, float phiStar,
                                  float width, int kk0, float *__restrict__ phig)
{
    const long long total = b.nxy * (long long)(b.nz + 2);
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % b.nx);
        const int j = (int)((t / b.nx) % b.ny);
        const int kk = (int)(t / b.nxy);
        float v = -phiStar;
        for (int m = 0; m < nbubbles; m++) {
            const float xc = __ldg(bubbles + 4 * m + 0), yc = __ldg(bubbles + 4 * m + 1);
            const float zc = __ldg(bubbles + 4 * m + 2), rc = __ldg(bubbles + 4 * m + 3);
            const float dx = __fsub_rn((float)i, xc);
            const float dy = __fsub_rn((float)j, yc);
            const float dz = __fsub_rn((float)(kk + kk0), zc);
            const float s = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
            const float R = __fsqrt_rn(s);
            if (R <= __fadd_rn(rc, width)) v = phiStar * tanhf(__fdiv_rn(2.f * __fsub_rn(rc, R), width));
        }
        phig[t] = v;
    }
}

// The same phi, per tile of 32 x 8 x 4 nodes of the ghosted grid: the block
// first lists, in file order, the bubbles that can reach the tile (the
// distance from the centre to the tile's box, in double, against
// Rc + width + 0.01, which no rounding of the float test can exceed), then
// makes the float test of bubble_phi_kernel for those only, so the node set
// and the last covering bubble are the same.  A tile reached by more than
// kTileBubbles bubbles tests them all.
constexpr int BTX = 32, BTY = 8, BTZ = 4, kTileBubbles = 1024;

__global__ void __launch_bounds__(BTX * BTY) bubble_phi_tiled_kernel(Box b, const float *__restrict__ bubbles,
                                                                     int nbubbles, float phiStar, float width,
                                                                     int kk0, float *__restrict__ phig)
{
    __shared__ int list[kTileBubbles];
    __shared__ int warp_off[BTY];
    __shared__ int count, overflow;
    const int lane = threadIdx.x, warp = threadIdx.y;
    const int x0 = blockIdx.x * BTX, y0 = blockIdx.y * BTY, k0 = blockIdx.z * BTZ;
    const int k1 = min(k0 + BTZ, b.nz + 2) - 1;
    if (lane == 0 && warp == 0) {
        count = 0;
        overflow = 0;
    }
    __syncthreads();
    for (int base = 0; base < nbubbles; base += BTX * BTY) {
        const int m = base + warp * BTX + lane;
        bool hit = false;
        if (m < nbubbles) {
            const double xc = bubbles[4 * m + 0], yc = bubbles[4 * m + 1], zc = bubbles[4 * m + 2];
            const double reach = (double)bubbles[4 * m + 3] + (double)width + 0.01;
            const double dx = fmax(fmax((double)x0 - xc, xc - (double)(x0 + BTX - 1)), 0.0);
            const double dy = fmax(fmax((double)y0 - yc, yc - (double)(y0 + BTY - 1)), 0.0);
            const double dz = fmax(fmax((double)(k0 + kk0) - zc, zc - (double)(k1 + kk0)), 0.0);
            hit = dx * dx + dy * dy + dz * dz <= reach * reach;
        }
        const unsigned ballot = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) warp_off[warp] = __popc(ballot);
        __syncthreads();
        if (lane == 0 && warp == 0) {   // exclusive prefix over the warps, in bubble order
            int run = count;
            for (int w = 0; w < BTY; w++) {
                const int c = warp_off[w];
                warp_off[w] = run;
                run += c;
            }
            count = run;
        }
        __syncthreads();
        if (hit) {
            const int pos = warp_off[warp] + __popc(ballot & ((1u << lane) - 1u));
            if (pos < kTileBubbles) list[pos] = m;
            else overflow = 1;
        }
        __syncthreads();
    }
    const bool every = overflow != 0;
    const int nlist = every ? nbubbles : min(count, kTileBubbles);
    const int i = x0 + lane, j = y0 + warp;
    for (int kk = k0; kk <= k1; kk++) {
        float v = -phiStar;
        for (int q = 0; q < nlist; q++) {
            const int m = every ? q : list[q];
            const float xc = __ldg(bubbles + 4 * m + 0), yc = __ldg(bubbles + 4 * m + 1);
            const float zc = __ldg(bubbles + 4 * m + 2), rc = __ldg(bubbles + 4 * m + 3);
            const float dx = __fsub_rn((float)i, xc);
            const float dy = __fsub_rn((float)j, yc);
            const float dz = __fsub_rn((float)(kk + kk0), zc);
            const float s = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
            const float R = __fsqrt_rn(s);
            if (R <= __fadd_rn(rc, width)) v = phiStar * tanhf(__fdiv_rn(2.f * __fsub_rn(rc, R), width));
        }
        phig[(size_t)kk * (size_t)b.nxy + (size_t)j * (size_t)b.nx + (size_t)i] = v;
    }
}

// At-rest equilibrium of a node from phi and rho: f_0, the common value of
// f_1..f_6, and g_0, of g_1..g_6 and of g_7..g_18.  z neighbours outside
// [0, nz) come from ghost_lo / ghost_hi (nx*ny each) when given, else by
// periodic wrap.  The last product of each g is kept from contracting with
// what its reader subtracts, so every kernel below sees the same FP32 values.
struct EqConst {
    float alpha4, kappa, phiStarSq, Gamma;
};
struct Eq {
    float f0, f1, g0, g1, g2;
};
__device__ __forceinline__ Eq equilibrium_at(const Box &b, const EqConst &c, const float *__restrict__ phi,
                                             const float *__restrict__ rho, const float *__restrict__ ghost_lo,
                                             const float *__restrict__ ghost_hi, int i, int j, int k)
{
    const int ie = i == b.nx - 1 ? 0 : i + 1, iw = i == 0 ? b.nx - 1 : i - 1;
    const int rn = (j == b.ny - 1 ? 0 : j + 1) * b.nx, rs = (j == 0 ? b.ny - 1 : j - 1) * b.nx, rc = j * b.nx;
    const float *const pc = phi + (size_t)k * b.nxy;
    const float *const pt = k == b.nz - 1 ? (ghost_hi ? ghost_hi : phi) : pc + b.nxy;
    const float *const pb = k == 0 ? (ghost_lo ? ghost_lo : phi + (size_t)(b.nz - 1) * b.nxy) : pc - b.nxy;
    const float phin = pc[rc + i];
    const float lap = (pc[rn + ie] + pc[rs + iw] + pc[rs + ie] + pc[rn + iw] + pt[rc + ie] + pb[rc + iw] + pb[rc + ie]
                       + pt[rc + iw] + pt[rn + i] + pb[rs + i] + pb[rn + i] + pt[rs + i]
                       + 2.f * (pc[rc + ie] + pc[rc + iw] + pc[rn + i] + pc[rs + i] + pt[rc + i] + pb[rc + i]
                                - 12.f * phin)) * kInv6;
    const float mu = c.alpha4 * phin * (phin * phin - c.phiStarSq) - c.kappa * lap;
    const float rhon = rho[(size_t)k * b.nxy + rc + i];
    Eq e;
    e.f0 = phin - 3.f * c.Gamma * mu;
    e.f1 = 0.5f * c.Gamma * mu;
    e.g0 = __fmul_rn(kW0, rhon - 6.f * phin * mu);
    e.g1 = __fmul_rn(kW1, 3.f * phin * mu + rhon);
    e.g2 = __fmul_rn(kW2, 3.f * phin * mu + rhon);
    return e;
}

// A block: a 32 x 8 tile (16-bit: 16 words of the pair layout, i.e. 32 nodes, x
// 8 rows) of EQZ planes.  The stores bound these kernels (104 or 54 bytes a
// node against 8 read): 256^3 FP32 297 us, 6.3 TB/s; FP16 171 us (6.1 TB/s) and
// 107 for the maxima (325, 210 and 129 on a grid of three dimensions).  The equilibrium into an FP32 scratch copy, the maxima of
// that and its conversion took 700, 289 and 498.
constexpr int EQZ = 4;

// The block's tile and first plane.  The grid has one dimension: a box's y or z
// may need more blocks than the 65535 of a grid's second and third.
struct EqTile {
    int bx, by, z0;
};
__device__ __forceinline__ EqTile eq_tile(const Box &b)
{
    const unsigned ntx = (unsigned)b.nx / 32u, nty = (unsigned)b.ny / 8u, t = blockIdx.x;
    return EqTile{(int)(t % ntx), (int)(t / ntx % nty), (int)(t / (ntx * nty)) * EQZ};
}

// FP32 storage: the streamed natural layout is the equilibrium itself.
__global__ void __launch_bounds__(256) equilibrium_kernel(Box b, EqConst c, const float *__restrict__ phi,
                                                          const float *__restrict__ rho,
                                                          const float *__restrict__ ghost_lo,
                                                          const float *__restrict__ ghost_hi, float *__restrict__ f0,
                                                          float *__restrict__ fq, float *__restrict__ g)
{
    const EqTile tile = eq_tile(b);
    const int i = tile.bx * 32 + threadIdx.x, j = tile.by * 8 + threadIdx.y;
#pragma unroll 1
    for (int k = tile.z0, k_end = min(b.nz, k + EQZ); k < k_end; k++) {
        const Eq e = equilibrium_at(b, c, phi, rho, ghost_lo, ghost_hi, i, j, k);
        const size_t t = (size_t)k * b.nxy + j * b.nx + i;
        f0[t] = e.f0;
#pragma unroll
        for (int q = 0; q < kQf - 1; q++) fq[q * b.n + t] = e.f1;
        g[t] = e.g0;
#pragma unroll
        for (int q = 1; q < kQg; q++) g[q * b.n + t] = q < 7 ? e.g1 : e.g2;
    }
}

// 16-bit storage: the two nodes of one pair-layout word, mapped and stored as
// one word per field (the values a quantize_kernel of the FP32 equilibrium
// would store, without that scratch copy).
template <typename ST>
__global__ void __launch_bounds__(128) equilibrium_store_kernel(Box b, EqConst c, Quant q,
                                                                const float *__restrict__ phi,
                                                                const float *__restrict__ rho,
                                                                const float *__restrict__ ghost_lo,
                                                                const float *__restrict__ ghost_hi,
                                                                float *__restrict__ f0, ST *__restrict__ fq,
                                                                ST *__restrict__ g)
{
    using T2 = typename Fmt<ST>::T2;
    const EqTile tile = eq_tile(b);
    const int w = tile.bx * 16 + threadIdx.x, j = tile.by * 8 + threadIdx.y;
#pragma unroll 1
    for (int k = tile.z0, k_end = min(b.nz, k + EQZ); k < k_end; k++) {
        const Eq a = equilibrium_at(b, c, phi, rho, ghost_lo, ghost_hi, w, j, k);
        const Eq d = equilibrium_at(b, c, phi, rho, ghost_lo, ghost_hi, w + b.nx / 2, j, k);
        const size_t t = (size_t)k * b.nxy + j * b.nx + 2 * w;   // the word's first element
        *reinterpret_cast<float2 *>(f0 + t) = make_float2(a.f0, d.f0);
        const T2 f1 = Fmt<ST>::store2(make_float2(__fmul_rn(a.f1, q.f_scale), __fmul_rn(d.f1, q.f_scale)));
#pragma unroll
        for (int m = 0; m < kQf - 1; m++) *reinterpret_cast<T2 *>(fq + m * b.n + t) = f1;
        auto map = [&](float va, float vb, int m) {
            return Fmt<ST>::store2(make_float2((va - q.g_shift[m]) * q.g_scale, (vb - q.g_shift[m]) * q.g_scale));
        };
        const T2 g0 = map(a.g0, d.g0, 0), g1 = map(a.g1, d.g1, 1), g2 = map(a.g2, d.g2, 7);
        *reinterpret_cast<T2 *>(g + t) = g0;
#pragma unroll
        for (int m = 1; m < kQg; m++) *reinterpret_cast<T2 *>(g + m * b.n + t) = m < 7 ? g1 : g2;
    }
}

// out_bits[0..4] = bits of max |f_0|, |f_1..6|, |g_0 - s_0|, |g_1..6 - s_1|,
// |g_7..18 - s_2| over the equilibrium (non-negative floats order like their
// bits), from which the 16-bit storage map is chosen.
__global__ void __launch_bounds__(256) equilibrium_maxabs_kernel(Box b, EqConst c, float s0, float s1, float s2,
                                                                 const float *__restrict__ phi,
                                                                 const float *__restrict__ rho,
                                                                 const float *__restrict__ ghost_lo,
                                                                 const float *__restrict__ ghost_hi,
                                                                 unsigned *__restrict__ out_bits)
{
    __shared__ unsigned red[8][5];
    const EqTile tile = eq_tile(b);
    const int i = tile.bx * 32 + threadIdx.x, j = tile.by * 8 + threadIdx.y;
    float m[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int k = tile.z0, k_end = min(b.nz, k + EQZ); k < k_end; k++) {
        const Eq e = equilibrium_at(b, c, phi, rho, ghost_lo, ghost_hi, i, j, k);
        m[0] = fmaxf(m[0], fabsf(e.f0));
        m[1] = fmaxf(m[1], fabsf(e.f1));
        m[2] = fmaxf(m[2], fabsf(e.g0 - s0));
        m[3] = fmaxf(m[3], fabsf(e.g1 - s1));
        m[4] = fmaxf(m[4], fabsf(e.g2 - s2));
    }
#pragma unroll
    for (int v = 0; v < 5; v++) {
        const unsigned r = __reduce_max_sync(0xffffffffu, __float_as_uint(m[v]));
        if (threadIdx.x == 0) red[threadIdx.y][v] = r;
    }
    __syncthreads();
    if (threadIdx.y == 0 && threadIdx.x < 5) {
        unsigned r = red[0][threadIdx.x];
        for (int w = 1; w < 8; w++) r = max(r, red[w][threadIdx.x]);
        // most blocks do not raise the maximum: look before the atomic
        if (r > *reinterpret_cast<volatile unsigned *>(out_bits + threadIdx.x)) atomicMax(out_bits + threadIdx.x, r);
    }
}

__global__ void fill_kernel(float *p, long long n, float v)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        p[t] = v;
}

unsigned grid_for(long long n)
{
    long long blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    return (unsigned)(blocks < 1 ? 1 : blocks);
}

}  // namespace

cudaError_t launch_bubble_phi(const Box &b, const float *bubbles_dev, int nbubbles, float phiStar, float width,
                              int z0, float *phi_ghosted, cudaStream_t s)
{
    if (b.nx % BTX == 0 && b.ny % BTY == 0) {
        const dim3 grid((unsigned)(b.nx / BTX), (unsigned)(b.ny / BTY), (unsigned)((b.nz + 2 + BTZ - 1) / BTZ));
        bubble_phi_tiled_kernel<<<grid, dim3(BTX, BTY), 0, s>>>(b, bubbles_dev, nbubbles, phiStar, width, z0,
                                                                 phi_ghosted);
    } else {
        bubble_phi_kernel<<<grid_for(b.nxy * (b.nz + 2)), 256, 0, s>>>(b, bubbles_dev, nbubbles, phiStar, width,
                                                                        z0, phi_ghosted);
    }
    return cudaGetLastError();
}

namespace {
EqConst eq_const(const lbm_derived &d, float Gamma) { return EqConst{d.alpha4, d.kappa, d.phiStarSq, Gamma}; }
unsigned eq_grid(const Box &b)
{
    return (unsigned)(b.nx / 32) * (unsigned)(b.ny / 8) * (unsigned)((b.nz + EQZ - 1) / EQZ);
}
}  // namespace

cudaError_t launch_equilibrium(const Box &b, const lbm_derived &d, float Gamma, const Quant &q, int storage,
                               const float *phi, const float *rho, const float *ghost_lo, const float *ghost_hi,
                               float *f0, void *fq, void *g, cudaStream_t s)
{
    if (b.nx % 32 != 0 || b.ny % 8 != 0) return cudaErrorInvalidValue;
    const EqConst c = eq_const(d, Gamma);
    const dim3 pair(16, 8);
    switch (storage) {
    case LBM_STORAGE_FP32:
        equilibrium_kernel<<<eq_grid(b), dim3(32, 8), 0, s>>>(b, c, phi, rho, ghost_lo, ghost_hi, f0,
                                                             static_cast<float *>(fq), static_cast<float *>(g));
        break;
    case LBM_STORAGE_FP16:
        equilibrium_store_kernel<__half><<<eq_grid(b), pair, 0, s>>>(b, c, q, phi, rho, ghost_lo, ghost_hi, f0,
                                                                     static_cast<__half *>(fq),
                                                                     static_cast<__half *>(g));
        break;
    case LBM_STORAGE_BF16:
        equilibrium_store_kernel<__nv_bfloat16><<<eq_grid(b), pair, 0, s>>>(
            b, c, q, phi, rho, ghost_lo, ghost_hi, f0, static_cast<__nv_bfloat16 *>(fq),
            static_cast<__nv_bfloat16 *>(g));
        break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_equilibrium_maxabs(const Box &b, const lbm_derived &d, float Gamma, const float *g_shift,
                                      const float *phi, const float *rho, const float *ghost_lo,
                                      const float *ghost_hi, unsigned *out_bits, cudaStream_t s)
{
    if (b.nx % 32 != 0 || b.ny % 8 != 0) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(out_bits, 0, 5 * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    equilibrium_maxabs_kernel<<<eq_grid(b), dim3(32, 8), 0, s>>>(b, eq_const(d, Gamma), g_shift[0], g_shift[1],
                                                                 g_shift[7], phi, rho, ghost_lo, ghost_hi, out_bits);
    return cudaGetLastError();
}

cudaError_t launch_fill(float *p, long long n, float v, cudaStream_t s)
{
    fill_kernel<<<grid_for(n), 256, 0, s>>>(p, n, v);
    return cudaGetLastError();
}

}  // namespace lbm
