// zsc_adjoint.cu -- discrete adjoint of the fused ZSC step (no counterpart in
// the reference).
//
// The forward step maps the streamed state s^n = (f^n, g^n) to s^{n+1}:
//   moments phi = sum f, rho = sum g, u = sum c g / rho;
//   lap, grad: 19-point stencils of phi (src/collision_f.cu:61-94);
//   mu = alpha4 phi (phi^2 - phiStar^2) - kappa lap;  F = mu grad (+ grav on phi > 0);
//   u* = u + F / (2 rho);  P = collision_f, Q = collision_g (src/collision_*.cu);
//   f'_i(x) = eta P_i(x - c_i) + (1 - eta) P_i(x);  g'_i(x) = Q_i(x - c_i).
// Its transpose, applied to lambda^{n+1} = dJ/ds^{n+1}:
//   stream:   lP_i(x) = eta lf'_i(x + c_i) + (1 - eta) lf'_i(x);  lQ_i(x) = lg'_i(x + c_i)
//   collision (local): direct terms (1 - 1/tau) lP, lQ plus the adjoints of
//             phi, mu, rho, u*, F, UF, 3 phi mu; dJ/dgrav += lambda_Fz H(phi > 0)
//   stencil:  lambda_phi += L[lambda_lap] - sum_k D_k[lambda_grad_k]
//             (the Laplacian stencil is symmetric, the gradient antisymmetric)
//   moments:  lf_i += lambda_phi;  lg_i += lambda_rho + c_i . lambda_m
// All seven lf hold the same part: with a = 1 - 1/tauPhi, lf_i = q_i + L where
// q_i = a lP_i of the step before and L = lambda_phi + the stencil part.  So
// lambda is kept as L (one field), lg (19) and, only when tauPhi is not 1, the
// seven q_i.
//
// The forward state is read where the step kernel keeps it (a checkpoint slot
// or the context's buffers): f_0 FP32, f_1..f_6 post-collision (the eta-blend
// is redone on read), g in the AA layout, 16-bit formats mapped back to FP32.
// The collision's Jacobian needs g only through rho and the momentum, and f
// only through phi, so only phi is materialised (the stencil needs it at the
// neighbours).  Per step (bytes per node, FP32 / 16-bit state, tauPhi = 1):
//   adjoint_phi_kernel     s^n -> phi                                 32 / 20
//   adjoint_march_kernel   lambda^{n+1}, s^n, phi -> lg^n, lambda_phi
//                          and (lambda_lap, mu lambda_F)              256 / 218
//   adjoint_stencil_kernel these four, lambda_phi -> L^n              24
// All per-node arithmetic is FP32; the objective sums and dJ/dgrav are FP64.
// The kernels work on 32 x 8 column tiles, each block marching z planes.
// 32-bit node indices (n * 19 < 2^32 is checked at init).
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "lattice.cuh"

namespace lbm {
namespace {

constexpr int TXA = 32, TYA = 8, NTA = TXA * TYA;
#ifndef ZSC_ADJ_PLANES
#define ZSC_ADJ_PLANES 4
#endif
constexpr int kPlanes = ZSC_ADJ_PLANES;
constexpr int kStencilBlocks = 8;   // resident blocks of the stencil kernel per SM
constexpr float kInv6 = 0.16666666666666666667f;
constexpr float kInv12 = 0.08333333333333333333f;
constexpr float kW0 = 0.33333333333333333333f, kW1 = 0.05555555555555555556f, kW2 = 0.02777777777777777778f;

// Node indices of the 3 x 3 x 3 neighbourhood of (x, y, z), periodic.
struct Nb {
    unsigned X[3], Y[3], Z[3];
    __device__ __forceinline__ unsigned at(int dx, int dy, int dz) const { return X[dx + 1] + Y[dy + 1] + Z[dz + 1]; }
};

__device__ __forceinline__ Nb neighbourhood(const Box &b, int x, int y, int z)
{
    Nb r;
    const unsigned nx = (unsigned)b.nx, nxy = (unsigned)b.nxy;
    r.X[0] = x == 0 ? nx - 1 : x - 1;
    r.X[1] = x;
    r.X[2] = x == b.nx - 1 ? 0 : x + 1;
    r.Y[0] = (y == 0 ? b.ny - 1 : y - 1) * nx;
    r.Y[1] = y * nx;
    r.Y[2] = (y == b.ny - 1 ? 0 : y + 1) * nx;
    r.Z[0] = (z == 0 ? b.nz - 1 : z - 1) * nxy;
    r.Z[1] = z * nxy;
    r.Z[2] = (z == b.nz - 1 ? 0 : z + 1) * nxy;
    return r;
}

// The same neighbourhood as element indices of the state's fields (FP32:
// the node indices; 16-bit storage: the pair layout, see storage_index).
template <typename ST>
__device__ __forceinline__ Nb state_neighbourhood(const Box &b, int x, int y, int z)
{
    Nb r = neighbourhood(b, x, y, z);
    if constexpr (sizeof(ST) == 2) {
        const unsigned h = (unsigned)b.nx >> 1;
#pragma unroll
        for (int k = 0; k < 3; k++) r.X[k] = r.X[k] < h ? 2u * r.X[k] : 2u * (r.X[k] - h) + 1u;
    }
    return r;
}

__device__ __forceinline__ unsigned node_index_of(const Box &b, int x, int y, int z)
{
    return (unsigned)x + (unsigned)b.nx * ((unsigned)y + (unsigned)b.ny * (unsigned)z);
}

// index of the node at sign * c_i from the centre of p
__device__ __forceinline__ unsigned dir_at(const Nb &p, int i, int sign)
{
    return p.at(sign * kCx(i), sign * kCy(i), sign * kCz(i));
}

// 19-point Laplacian and gradient of field v at the centre of p
// (src/collision_f.cu:61-94), the stencil points taken in D3Q19 order.
__device__ __forceinline__ void stencil19(const float *__restrict__ v, const Nb &p, float &lap, float &gx, float &gy,
                                          float &gz)
{
    float s[kQg];
#pragma unroll
    for (int i = 0; i < kQg; i++) s[i] = __ldg(v + dir_at(p, i, 1));
    lap = (s[7] + s[8] + s[9] + s[10] + s[11] + s[12] + s[13] + s[14] + s[15] + s[16] + s[17] + s[18]
           + 2.f * (s[1] + s[2] + s[3] + s[4] + s[5] + s[6] - 12.f * s[0])) * kInv6;
    gx = (2.f * (s[1] - s[2]) + s[7] - s[8] + s[9] - s[10] + s[11] - s[12] + s[13] - s[14]) * kInv12;
    gy = (2.f * (s[3] - s[4]) + s[7] - s[8] + s[10] - s[9] + s[15] - s[16] + s[17] - s[18]) * kInv12;
    gz = (2.f * (s[5] - s[6]) + s[11] - s[12] + s[14] - s[13] + s[15] - s[16] + s[18] - s[17]) * kInv12;
}

// What the 19-point stencils of a node take from one plane of phi (row pitch
// PITCH), at the node p points to: the Laplacian sums to mid of the node's own
// plane plus a of the planes above and below, and the gradient likewise.
struct PlaneSums {
    float c, a, fx, fy;    // centre; e + w + n + s + 2 c; e - w; n - s
    float mid, gx, gy;     // corners + 2 (e + w + n + s) - 24 c; own-plane parts of the x and y gradient
};
template <int PITCH>
__device__ __forceinline__ PlaneSums plane_sums(const float *p)
{
    const float e = p[1], w = p[-1], n = p[PITCH], s = p[-PITCH];
    const float en = p[PITCH + 1], ws = p[-PITCH - 1], es = p[-PITCH + 1], wn = p[PITCH - 1];
    PlaneSums r;
    r.c = p[0];
    const float f4 = (e + w) + (n + s), d1 = en - ws, d2 = es - wn;
    r.fx = e - w;
    r.fy = n - s;
    r.a = f4 + 2.f * r.c;
    r.mid = 2.f * (f4 - 12.f * r.c) + ((en + ws) + (es + wn));
    r.gx = 2.f * r.fx + (d1 + d2);
    r.gy = 2.f * r.fy + (d1 - d2);
    return r;
}

// Per-field base pointers of a state (kernel parameters: a field's address is
// one multiply-add on the node index).
struct GFields {
    const void *f[kQg];       // g, AA layout
};
struct FQFields {
    const void *f[kQf - 1];   // f_1 .. f_6
};

// Streamed g_i at the centre of p, FP32.
template <typename ST, bool ODD>
__device__ __forceinline__ float g_streamed(const GFields &g, const Quant &q, const Nb &p, int i)
{
    const ST v = ODD ? static_cast<const ST *>(g.f[kOpp(i)])[dir_at(p, i, -1)]
                     : static_cast<const ST *>(g.f[i])[p.at(0, 0, 0)];
    if constexpr (Fmt<ST>::kMapped)
        return Fmt<ST>::load(v) * q.g_inv + q.g_shift[i];
    else
        return Fmt<ST>::load(v);
}

// rho and momentum of the streamed g at the centre of p.
template <typename ST, bool ODD>
__device__ __forceinline__ void g_moments(const GFields &g, const Quant &q, const Nb &p, float &rho, float m[3])
{
    rho = 0.f;
    m[0] = m[1] = m[2] = 0.f;
#pragma unroll
    for (int i = 0; i < kQg; i++) {
        const float gi = g_streamed<ST, ODD>(g, q, p, i);
        rho += gi;
        if (kCx(i)) m[0] += kCx(i) * gi;
        if (kCy(i)) m[1] += kCy(i) * gi;
        if (kCz(i)) m[2] += kCz(i) * gi;
    }
}

__device__ __forceinline__ double block_sum(double v, double *red)
{
    const int tid = threadIdx.y * TXA + threadIdx.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (tid == 0)
        for (int w = 0; w < NTA / 32; w++) r += red[w];
    __syncthreads();
    return r;
}

__device__ __forceinline__ unsigned block_id() { return blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z); }

// The light phase's weight sum of one block of a phi kernel (NT threads, linear
// thread number tid) into *out.
template <int NT>
__device__ __forceinline__ void weight_sum(double v, int tid, double *out)
{
    __shared__ double red[NT / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    if (tid == 0) {
        double r = 0.0;
        for (int w = 0; w < NT / 32; w++) r += red[w];
        *out = r;
    }
}

// phi = sum of the streamed f of a native state (FP32 storage).  With SUM also
// the per-block sums of w = (phiStar - phi) / (2 phiStar), the objective's
// weight, which an adjoint step of the averaging window needs.
template <bool SUM>
__global__ void __launch_bounds__(NTA) adjoint_phi_kernel(Box b, float eta, const float *__restrict__ f0,
                                                          const FQFields fq, int f_streamed, float *__restrict__ phi,
                                                          float phiStar, double *__restrict__ partials)
{
    const float eta2 = 1.f - eta, half_inv = 0.5f / phiStar;
    double B = 0.0;
    const int x = blockIdx.x * TXA + threadIdx.x, y = blockIdx.y * TYA + threadIdx.y;
    for (int z = blockIdx.z * kPlanes, z_end = min(b.nz, z + kPlanes); z < z_end; z++) {
        const Nb p = neighbourhood(b, x, y, z);
        const unsigned t = p.at(0, 0, 0);
        float s = f0[t];
#pragma unroll
        for (int i = 1; i < kQf; i++) {
            const float *a = static_cast<const float *>(fq.f[i - 1]);
            const float here = a[t];
            s += f_streamed ? here : eta * a[dir_at(p, i, -1)] + eta2 * here;
        }
        phi[t] = s;
        if (SUM) B += (double)((phiStar - s) * half_inv);
    }
    if (SUM) weight_sum<NTA>(B, threadIdx.y * TXA + threadIdx.x, partials + block_id());
}

// The same for 16-bit storage: a thread sums the two nodes of one pair-layout
// word, so that every load is a whole word: 60 us at 256^3 (with two-byte loads
// 87; the 20 bytes a node take 49 at the copy bandwidth).  Bound by the latency
// of its loads at 85 % of the warps.
template <typename ST, bool SUM>
__global__ void __launch_bounds__(TXA / 2 * TYA) adjoint_phi_pair_kernel(Box b, float eta, float inv,
                                                                         const float *__restrict__ f0,
                                                                         const FQFields fq, int f_streamed,
                                                                         float *__restrict__ phi, float phiStar,
                                                                         double *__restrict__ partials)
{
    using T2 = typename Fmt<ST>::T2;
    const float eta2 = 1.f - eta, half_inv = 0.5f / phiStar;
    double B = 0.0;
    const int h = b.nx / 2, w = blockIdx.x * (TXA / 2) + threadIdx.x, y = blockIdx.y * TYA + threadIdx.y;
    // the words at x - 1 and x + 1; past the x seam a word's nodes are swapped
    const int wl = w == 0 ? h - 1 : w - 1, wr = w == h - 1 ? 0 : w + 1;
    const unsigned sel_l = w == 0 ? kSwap : kKeep, sel_r = w == h - 1 ? kSwap : kKeep;
    const int yl = y == 0 ? b.ny - 1 : y - 1, yr = y == b.ny - 1 ? 0 : y + 1;
    for (int z = blockIdx.z * kPlanes, z_end = min(b.nz, z + kPlanes); z < z_end; z++) {
        const int zl = z == 0 ? b.nz - 1 : z - 1, zr = z == b.nz - 1 ? 0 : z + 1;
        auto word = [&](int ww, int yy, int zz) { return (unsigned)ww + (unsigned)h * ((unsigned)yy + (unsigned)b.ny * (unsigned)zz); };
        const unsigned t = word(w, y, z);
        // where the streamed f_i comes from: x - c_i
        const unsigned up[kQf - 1] = {word(wl, y, z), word(wr, y, z), word(w, yl, z),
                                      word(w, yr, z), word(w, y, zl), word(w, y, zr)};
        float2 s = reinterpret_cast<const float2 *>(f0)[t];
#pragma unroll
        for (int i = 0; i < kQf - 1; i++) {
            const T2 *a = static_cast<const T2 *>(fq.f[i]);
            const float2 c = Fmt<ST>::load2(a[t]);
            const float hx = c.x * inv, hy = c.y * inv;
            if (f_streamed) {
                s.x += hx;
                s.y += hy;
            } else {
                const float2 v = Fmt<ST>::load2(Fmt<ST>::perm2(a[up[i]], i == 0 ? sel_l : i == 1 ? sel_r : kKeep));
                s.x += eta * (v.x * inv) + eta2 * hx;
                s.y += eta * (v.y * inv) + eta2 * hy;
            }
        }
        const unsigned r = (unsigned)b.nx * ((unsigned)y + (unsigned)b.ny * (unsigned)z) + (unsigned)w;
        phi[r] = s.x;
        phi[r + (unsigned)h] = s.y;
        if (SUM) B += (double)((phiStar - s.x) * half_inv) + (double)((phiStar - s.y) * half_inv);
    }
    if (SUM) weight_sum<TXA / 2 * TYA>(B, threadIdx.y * (TXA / 2) + threadIdx.x, partials + block_id());
}

// Objective sums of one state: A = sum w q, B = sum w, with
// w = (phiStar - phi) / (2 phiStar) and q = u_z (objective 0) or the reference
// plane index z + 1 (objective 1); per-block partials.
template <typename ST, bool ODD>
__global__ void __launch_bounds__(NTA) objective_kernel(Box b, int objective, float phiStar, Quant q,
                                                        const GFields g, const float *__restrict__ phi,
                                                        double *__restrict__ partials)
{
    __shared__ double red[NTA / 32];
    const float half_inv = 0.5f / phiStar;
    double A = 0.0, B = 0.0;
    const int x = blockIdx.x * TXA + threadIdx.x, y = blockIdx.y * TYA + threadIdx.y;
    for (int z = blockIdx.z * kPlanes, z_end = min(b.nz, z + kPlanes); z < z_end; z++) {
        const float w = (phiStar - phi[node_index_of(b, x, y, z)]) * half_inv;
        float qv;
        if (objective == 0) {
            float rho, m[3];
            g_moments<ST, ODD>(g, q, state_neighbourhood<ST>(b, x, y, z), rho, m);
            qv = m[2] / rho;
        } else {
            qv = (float)(z + 1);
        }
        A += (double)(w * qv);
        B += (double)w;
    }
    A = block_sum(A, red);
    B = block_sum(B, red);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        partials[2 * block_id()] = A;
        partials[2 * block_id() + 1] = B;
    }
}

// ab[0..1] = sums of the partials, ab[2] = A / B, ab[3] = scale / B;
// acc[0] (J) += scale * A / B.
__global__ void __launch_bounds__(NTA) objective_fold_kernel(const double *__restrict__ partials, int nparts,
                                                             double scale, double *__restrict__ ab,
                                                             double *__restrict__ acc)
{
    __shared__ double red[NTA / 32];
    double A = 0.0, B = 0.0;
    for (int p = threadIdx.y * TXA + threadIdx.x; p < nparts; p += NTA) {
        A += partials[2 * p];
        B += partials[2 * p + 1];
    }
    A = block_sum(A, red);
    B = block_sum(B, red);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        ab[0] = A;
        ab[1] = B;
        ab[2] = A / B;
        ab[3] = scale / B;
        acc[0] += scale * A / B;
    }
}

// ab[1] = B = sum of the phi kernel's weight sums, ab[3] = scale / B.
// One block, bound by the latency of its reads: 4 us at 128^3 (cold), on the
// side stream.
__global__ void __launch_bounds__(NTA) weight_fold_kernel(const double *__restrict__ partials, int nparts, double scale,
                                                          double *__restrict__ ab)
{
    __shared__ double red[NTA / 32];
    double B = 0.0;
    for (int p = threadIdx.y * TXA + threadIdx.x; p < nparts; p += NTA) B += partials[p];
    B = block_sum(B, red);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        ab[1] = B;
        ab[3] = scale / B;
    }
}

// ab[0] = A = sum of the march kernel's sums of w u_z, ab[2] = A / B; acc[0] (J)
// += scale A / B.  One block, 7 us at 128^3 (cold); with the two it takes the
// place of a pass over the state's g (42 us).
__global__ void __launch_bounds__(1024) velocity_fold_kernel(const double *__restrict__ parts, int nparts, double scale,
                                                             double *__restrict__ ab, double *__restrict__ acc)
{
    __shared__ double red[32];
    const int tid = threadIdx.x;
    double A = 0.0;
#pragma unroll 4
    for (int p = tid; p < nparts; p += 1024) A += parts[p];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) A += __shfl_down_sync(0xffffffffu, A, o);
    if ((tid & 31) == 0) red[tid >> 5] = A;
    __syncthreads();
    if (tid < 32) {
        A = red[tid];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) A += __shfl_down_sync(0xffffffffu, A, o);
        if (tid == 0) {
            ab[0] = A;
            ab[2] = A / ab[1];
            acc[0] += scale * A / ab[1];
        }
    }
}

// Per-launch coefficients of the objective's derivative: J += scale A / B
// gives dJ/dw = scale (q - A/B) / B and dJ/dq = scale w / B, with
// dw/dphi = -1 / (2 phiStar).
struct SourceCoef {
    float ratio;    // A / B
    float s_over_b; // scale / B
    float half_inv; // 1 / (2 phiStar)
};

__device__ __forceinline__ SourceCoef source_coef(const double *ab, float phiStar)
{
    SourceCoef k;
    k.ratio = (float)ab[2];
    k.s_over_b = (float)ab[3];
    k.half_inv = 0.5f / phiStar;
    return k;
}

// d(scale * A / B)/d(state) at a node of plane z (FP32 per node).
__device__ __forceinline__ void objective_source(int z, int objective, const SourceCoef &k, float phiStar, float ph,
                                                 float rho, float mz, float &dphi, float &drho, float &dmz)
{
    const float w = (phiStar - ph) * k.half_inv;
    if (objective == 0) {
        const float inv = 1.0f / rho;
        const float uz = mz * inv;
        dphi = -k.half_inv * k.s_over_b * (uz - k.ratio);
        const float duz = k.s_over_b * w;
        dmz = duz * inv;
        drho = -duz * uz * inv;
    } else {
        dphi = -k.half_inv * k.s_over_b * ((float)(z + 1) - k.ratio);
        drho = 0.f;
        dmz = 0.f;
    }
}

// lambda^T: only the objective source of the final state.
template <typename ST, bool ODD>
__global__ void __launch_bounds__(NTA) source_init_kernel(Box b, int objective, double scale,
                                                          const double *__restrict__ ab, float phiStar, Quant q,
                                                          const GFields g, const float *__restrict__ phi,
                                                          float *__restrict__ lq, float *__restrict__ lg,
                                                          float *__restrict__ L)
{
    const unsigned n = (unsigned)b.n;
    const SourceCoef k = source_coef(ab, phiStar);
    const int x = blockIdx.x * TXA + threadIdx.x, y = blockIdx.y * TYA + threadIdx.y;
    for (int z = blockIdx.z * kPlanes, z_end = min(b.nz, z + kPlanes); z < z_end; z++) {
        const unsigned t = node_index_of(b, x, y, z);
        float rho, m[3];
        g_moments<ST, ODD>(g, q, state_neighbourhood<ST>(b, x, y, z), rho, m);
        float dphi, drho, dmz;
        objective_source(z, objective, k, phiStar, phi[t], rho, m[2], dphi, drho, dmz);
        L[t] = dphi;
        if (lq)
            for (int i = 0; i < kQf; i++) lq[i * n + t] = 0.f;
#pragma unroll
        for (int i = 0; i < kQg; i++) lg[i * n + t] = drho + kCz(i) * dmz;
    }
}

struct AdjIn {
    // per-field base pointers (kernel parameters: a field's address is one
    // multiply-add on the node index, with no i * n on the load's path)
    const void *g_f[kQg];                  // the state's g fields
    const float *lg_f[kQg];                // lambda_g^{n+1}
    float *lg_o[kQg];                      // lambda_g^n
    const float *lq_f[kQf];                // q^{n+1} and q^n (tauPhi != 1 only)
    float *lq_o[kQf];
    const float *phi;                      // phi of s^n
    const float *L;                        // L^{n+1}
    float *lphi;                           // lambda_phi^n (L^n without its stencil part)
    float *lsrc[4];                        // lambda_lap, mu lambda_F at every node
    double *dgrav;                         // per warp of each block, accumulated over steps
    double *wuz;                           // per warp: sum of w u_z of s^n (when add_source)
    const double *ab;                      // objective sums of s^n: ab[3] = scale / B (when add_source)
    int add_source;                        // s^n is in the averaging window of the u_z objective
};

__device__ __forceinline__ int wrap_to(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

// 16-byte global -> shared copy, cached in L2 only; completes asynchronously.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const unsigned sm = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sm), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_prior()   // all but this thread's last N groups
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

template <int I>
struct Dir {
    static constexpr int value = I;
};
// f(Dir<i>) for i = I, I + D, I + 2D, ... < 19
template <int I, int D, typename F>
__device__ __forceinline__ void for_dirs(F &&f)
{
    if constexpr (I < kQg) {
        f(Dir<I>{});
        for_dirs<I + D, D>(f);
    }
}
// the same from the run-time first direction q < D (uniform per warp)
template <int D, int Q = 0, typename F>
__device__ __forceinline__ void for_dirs_of(int q, F &&f)
{
    if constexpr (Q < D) {
        if (q == Q) for_dirs<Q, D>(f);
        else for_dirs_of<D, Q + 1>(q, f);
    }
}

// Shared-memory geometry of the march kernel.  A tile is 32 nodes x 8 rows.
// For an FP32 state the 32 nodes are consecutive; for a 16-bit state, kept in
// the pair layout, they are the two nodes of 16 consecutive words (x = w and
// x = w + nx/2: lanes 0..15 and 16..31), so that every staged byte of g is used.
// The FP32 fields are then staged as two segments of 16 nodes, a segment's rows
// kSeg floats apart with kSeg = 16 mod 32, which keeps the two half-warps in
// different banks.
template <typename ST>
struct Geo {
    static constexpr bool kPair = sizeof(ST) == 2;
    static constexpr int SEGS = kPair ? 2 : 1;
    static constexpr int W = TXA / SEGS;                // nodes of a segment
    static constexpr int LP = W + 4;                    // lambda_g row: a chunk for the x-shifted nodes
    static constexpr int LSEG = kQg * TYA * LP + (kPair ? 16 : 0);   // floats between segments
    static constexpr int LSTAGE = SEGS * LSEG;          // floats per plane
    static constexpr int GP = kPair ? 2 * (W + 4) : LP; // g row, elements
    static constexpr int GSTAGE = kQg * TYA * GP;       // elements per plane
    static constexpr int HP = W + 8;                    // phi / L row with its halo
    static constexpr int HROWS = TYA + 2;
    static constexpr int HSEG = HROWS * HP;             // (16-bit: 240 = 16 mod 32)
    static constexpr int HPLANE = SEGS * HSEG;
    static constexpr int HCHUNKS = HPLANE / 4;          // 16-byte chunks of a phi / L plane
    static constexpr int L_OFF = 0;                     // bytes: [2][LSTAGE] floats
    static constexpr int G_OFF = L_OFF + 2 * LSTAGE * 4;
    static constexpr int PHI_OFF = G_OFF + 2 * GSTAGE * (int)sizeof(ST);   // [3][HPLANE] floats
    static constexpr int LF_OFF = PHI_OFF + 3 * HPLANE * 4;                // [3][HPLANE] floats
    static constexpr int SMEM = LF_OFF + 3 * HPLANE * 4;
    static constexpr int GCH = kPair ? 4 : 8;           // chunks of an unshifted g row
    static constexpr int GD = NTA / (TYA * GCH);        // directions the block stages at a time
    static_assert(HCHUNKS <= NTA / 2, "one chunk of phi and of L per thread at most");
    static_assert(G_OFF % 16 == 0 && PHI_OFF % 16 == 0 && LF_OFF % 16 == 0 && HPLANE % 4 == 0, "16-byte stages");
};

// The local part of one adjoint step (see the file comment).
//
// A block owns a 32 x 8 tile of columns and marches tz planes.  Everything a
// node reads comes from shared memory, staged one plane ahead with 16-byte
// cp.async copies (periodic in x and y by their addresses): the 19 lambda_g
// rows the node's directions point to (x + c_i), the 19 g rows of the state
// (own slots, or in the odd AA layout the reversed slots of x - c_i), and phi
// and L on the tile plus one node; phi of the plane above is reduced to the
// sums its stencils need (PlaneSums) once and carried down the march.
//
// 256 bytes a node with an FP32 state, 218 with a 16-bit one: 632 and 538 us at
// 256^3 at the copy bandwidth.  It takes 651 and 652 (DRAM bounds the first,
// the instructions and the shared-memory pipe of two blocks of 128 registers
// the second); read straight from global memory, with all seven lambda_f kept,
// the step took 1055 and 1066.  128^3 FP32 86 us (126 before), 64^3 16 (22).
// Two blocks, not more: the state's and lambda's two stages of rows take 83 to
// 95 KB, and one plane ahead hides the latency of a plane.
template <typename ST, bool ODD, bool LQ>
__global__ void __launch_bounds__(NTA, 2)
adjoint_march_kernel(Box b, StepConst c, float phiStar, Quant q, const __grid_constant__ AdjIn a, int tz)
{
    using Gm = Geo<ST>;
    constexpr bool PAIR = Gm::kPair;
    constexpr int W = Gm::W;
    extern __shared__ __align__(128) unsigned char smem[];
    float *const SL = reinterpret_cast<float *>(smem + Gm::L_OFF);
    ST *const SG = reinterpret_cast<ST *>(smem + Gm::G_OFF);
    float *const SP = reinterpret_cast<float *>(smem + Gm::PHI_OFF);
    float *const SF = reinterpret_cast<float *>(smem + Gm::LF_OFF);

    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TXA + tx;
    const int half = b.nx / Gm::SEGS;             // x distance of the segments
    const int ntx = b.nx / TXA, nty = b.ny / TYA;
    const int bx = blockIdx.x % ntx, by = (blockIdx.x / ntx) % nty, bz = blockIdx.x / (ntx * nty);
    const int w0 = bx * W, y0 = by * TYA;         // first node of segment 0
    const int z0 = bz * tz, nzc = min(tz, b.nz - z0);
    const int seg = PAIR ? tx >> 4 : 0, k = tx & (W - 1);
    const int x = w0 + seg * half + k, y = y0 + ty;
    const unsigned nxy = (unsigned)b.nxy;

    // ---- staging roles, fixed per thread ----
    // lambda_g: row s_r, chunk s_k (of segment s_seg) of every 4th direction from s_q
    const int s_q = tid >> 6, s_r = (tid >> 3) & 7, s_c = tid & 7;
    const int s_seg = PAIR ? s_c >> 2 : 0, s_k = PAIR ? s_c & 3 : s_c;
    const int s_x = w0 + s_seg * half + 4 * s_k;                       // first node of the chunk
    const int s_xl = wrap_to(w0 + s_seg * half - 4, b.nx), s_xr = wrap_to(w0 + s_seg * half + W, b.nx);
    const int s_row0 = b.nx * (y0 + s_r), s_rowp = b.nx * wrap_to(y0 + s_r + 1, b.ny),
              s_rowm = b.nx * wrap_to(y0 + s_r - 1, b.ny);
    // g: the same for FP32; 16-bit rows are 4 chunks of 8 elements, every 8th direction
    const int g_q = PAIR ? tid >> 5 : s_q, g_r = PAIR ? (tid >> 2) & 7 : s_r, g_k = PAIR ? tid & 3 : s_k;
    constexpr int GE = PAIR ? 8 : 4;              // elements per chunk
    const int g_x = (PAIR ? 2 * w0 : w0) + GE * g_k;
    const int g_xl = wrap_to((PAIR ? 2 * w0 : w0) - GE, b.nx), g_xr = wrap_to((PAIR ? 2 : 1) * (w0 + W), b.nx);
    const int g_row0 = b.nx * (y0 + g_r), g_rowp = b.nx * wrap_to(y0 + g_r + 1, b.ny),
              g_rowm = b.nx * wrap_to(y0 + g_r - 1, b.ny);
    // phi (threads 0..127) and L (threads 128..255): one chunk of the tile and its halo
    const int h_t = tid & (NTA / 2 - 1);
    const bool h_issuer = h_t < Gm::HCHUNKS;
    int h_xy = 0;
    {
        constexpr int RC = Gm::HP / 4;            // chunks per row
        const int sg = h_t / (Gm::HROWS * RC), rr = (h_t / RC) % Gm::HROWS, kk = h_t % RC;
        if (h_issuer)
            h_xy = wrap_to(w0 + sg * half - 4 + 4 * kk, b.nx) + b.nx * wrap_to(y0 - 1 + rr, b.ny);
    }
    auto issue_h = [&](int z) {                   // plane z >= z0 - 1 into ring slot (z - z0 + 1) % 3
        if (!h_issuer) return;
        const int slot = (int)((unsigned)(z - z0 + 1) % 3u);
        const unsigned t = (unsigned)wrap_to(z, b.nz) * nxy + (unsigned)h_xy;
        cp_async16((tid < NTA / 2 ? SP : SF) + slot * Gm::HPLANE + 4 * h_t, (tid < NTA / 2 ? a.phi : a.L) + t);
    };
    auto issue = [&](int z, int stage) {          // lambda_g and g rows of plane z
        const unsigned zc = (unsigned)z * nxy, zp = (unsigned)wrap_to(z + 1, b.nz) * nxy,
                       zm = (unsigned)wrap_to(z - 1, b.nz) * nxy;
        float *dl = SL + stage * Gm::LSTAGE + s_seg * Gm::LSEG + s_r * Gm::LP;
        for_dirs_of<4>(s_q, [&](auto d) {
            constexpr int i = decltype(d)::value;
            constexpr int sx = kCx(i), sy = kCy(i), sz = kCz(i);
            const float *src = a.lg_f[i] + ((sz > 0 ? zp : sz < 0 ? zm : zc) +
                                            (unsigned)(sy > 0 ? s_rowp : sy < 0 ? s_rowm : s_row0));
            float *dst = dl + i * TYA * Gm::LP;
            cp_async16(dst + (sx < 0 ? 4 : 0) + 4 * s_k, src + s_x);
            if (sx != 0 && s_k == 0) cp_async16(dst + (sx < 0 ? 0 : W), src + (sx < 0 ? s_xl : s_xr));
        });
        ST *dg = SG + stage * Gm::GSTAGE + g_r * Gm::GP;
        for_dirs_of<Gm::GD>(g_q, [&](auto d) {
            constexpr int i = decltype(d)::value;
            constexpr int sx = ODD ? -kCx(i) : 0, sy = ODD ? -kCy(i) : 0, sz = ODD ? -kCz(i) : 0;
            const ST *src = static_cast<const ST *>(a.g_f[ODD ? kOpp(i) : i]) +
                            ((sz > 0 ? zp : sz < 0 ? zm : zc) +
                             (unsigned)(sy > 0 ? g_rowp : sy < 0 ? g_rowm : g_row0));
            ST *dst = dg + i * TYA * Gm::GP;
            cp_async16(dst + (sx < 0 ? GE : 0) + GE * g_k, src + g_x);
            if (sx != 0 && g_k == 0)
                cp_async16(dst + (sx < 0 ? 0 : GE * Gm::GCH), src + (sx < 0 ? g_xl : g_xr));
        });
    };

    // where the node finds its values: column of a row staged with x shift sx
    constexpr auto col = [](int sx) { return sx > 0 ? 1 : sx < 0 ? 3 : 0; };
    const float *const rl = SL + seg * Gm::LSEG + ty * Gm::LP + k;
    const ST *const rg = SG + ty * Gm::GP + (PAIR ? 2 * k : k);
    // 16-bit g: the half of the word; past the x seam (word nx/2 - 1 -> 0 and
    // back) a word's halves are the other way round
    const int hf = PAIR ? seg : 0;
    const int hf_r = PAIR && k == W - 1 && w0 + W == half ? 1 - seg : hf;
    const int hf_l = PAIR && k == 0 && w0 == 0 ? 1 - seg : hf;
    const int hc = seg * Gm::HSEG + (ty + 1) * Gm::HP + k + 4;   // the node in a phi / L plane
    auto hslot = [&](int z) { return (int)((unsigned)(z - z0 + 1) % 3u) * Gm::HPLANE + hc; };

    issue_h(z0 - 1);
    issue_h(z0);
    issue_h(z0 + 1);
    issue(z0, 0);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    const PlaneSums below = plane_sums<Gm::HP>(SP + hslot(z0 - 1));
    float a_b = below.a, fx_b = below.fx, fy_b = below.fy;
    PlaneSums cur = plane_sums<Gm::HP>(SP + hslot(z0));
    float L_m = SF[hslot(z0 - 1)], L_c = SF[hslot(z0)];
    double dg = 0.0, wuz = 0.0;

    for (int j = 0; j < nzc; ++j) {
        const int z = z0 + j, st = j & 1;
        cp_async_wait_all();
        __syncthreads();   // plane z has landed; the stages of plane z - 1 are free
        if (j + 1 < nzc) {
            issue(z + 1, 1 - st);
            issue_h(z + 2);
        }
        cp_async_commit();
        const unsigned t = (unsigned)z * nxy + (unsigned)y * (unsigned)b.nx + (unsigned)x;

        const PlaneSums top = plane_sums<Gm::HP>(SP + hslot(z + 1));
        const float ph = cur.c;
        const float lap = ((cur.mid + top.a) + a_b) * kInv6;
        const float gr[3] = {(cur.gx + (top.fx + fx_b)) * kInv12, (cur.gy + (top.fy + fy_b)) * kInv12,
                             (top.a - a_b) * kInv12};
        a_b = cur.a;
        fx_b = cur.fx;
        fy_b = cur.fy;
        cur = top;

        // moments of the streamed g, summed in direction order (as g_moments)
        float rh = 0.f, m[3] = {0.f, 0.f, 0.f};
        {
            const ST *gs = rg + st * Gm::GSTAGE;
#pragma unroll
            for (int i = 0; i < kQg; i++) {
                const int sx = ODD ? -kCx(i) : 0;
                const int cc = PAIR ? 2 * (sx > 0 ? 1 : sx < 0 ? 3 : 0) + (sx > 0 ? hf_r : sx < 0 ? hf_l : hf) : col(sx);
                float gi = Fmt<ST>::load(gs[i * TYA * Gm::GP + cc]);
                if constexpr (Fmt<ST>::kMapped) gi = gi * q.g_inv + q.g_shift[i];
                rh += gi;
                if (kCx(i)) m[0] += kCx(i) * gi;
                if (kCy(i)) m[1] += kCy(i) * gi;
                if (kCz(i)) m[2] += kCz(i) * gi;
            }
        }
        const float inv = 1.0f / rh;
        const float u[3] = {m[0] * inv, m[1] * inv, m[2] * inv};
        const float mu = c.alpha4 * ph * (ph * ph - c.phiStarSq) - c.kappa * lap;
        float F[3] = {mu * gr[0], mu * gr[1], mu * gr[2]};
        const bool heavy = ph > 0.f;
        if (heavy) F[2] += c.grav;
        const float us[3] = {u[0] + 0.5f * F[0] * inv, u[1] + 0.5f * F[1] * inv, u[2] + 0.5f * F[2] * inv};
        const float v[3] = {3.f * us[0], 3.f * us[1], 3.f * us[2]};
        const float vsq6 = (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) * kInv6;
        const float Cf = c.invTauPhi * c.invEta2 * ph;

        // stream adjoint
        float lP[kQf], lQ[kQg];
        {
            const float *Lp = SF + hslot(z);
            const float L_p = SF[hslot(z + 1)];
            const float up[kQf] = {L_c, Lp[1], Lp[-1], Lp[Gm::HP], Lp[-Gm::HP], L_p, L_m};
            lP[0] = L_c;
#pragma unroll
            for (int i = 1; i < kQf; i++) lP[i] = c.eta * up[i] + c.eta2 * L_c;
            if constexpr (LQ) {   // lf_i = q_i + L
                const Nb p = neighbourhood(b, x, y, z);
                lP[0] += __ldg(a.lq_f[0] + t);
#pragma unroll
                for (int i = 1; i < kQf; i++)
                    lP[i] += c.eta * __ldg(a.lq_f[i] + dir_at(p, i, 1)) + c.eta2 * __ldg(a.lq_f[i] + t);
            }
            L_m = L_c;
            L_c = L_p;
            const float *ls = rl + st * Gm::LSTAGE;
#pragma unroll
            for (int i = 0; i < kQg; i++) lQ[i] = ls[i * TYA * Gm::LP + col(kCx(i))];
        }

        // D3Q7 collision
        float lphi = 0.f, lmu = 0.f, lus[3] = {0.f, 0.f, 0.f}, lF[3] = {0.f, 0.f, 0.f}, lrho = 0.f;
        {
            const float lAf = -6.f * lP[0] + lP[1] + lP[2] + lP[3] + lP[4] + lP[5] + lP[6];
            float lCf = 0.f;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float d = lP[1 + 2 * k] - lP[2 + 2 * k];
                lCf += us[k] * d;
                lus[k] += Cf * d;
            }
            lphi += c.invTauPhi * lP[0] + c.invTauPhi * c.invEta2 * lCf;
            lmu += 0.5f * c.Gamma * c.invTauPhi * lAf;
        }
        // D3Q19 collision with forcing
        float ls, lvsq6, lUF, lv[3];
        {
            // A weight class's constants are taken out of its sums, and the sums
            // over lambda_Q that several terms share are formed once: the kernel
            // runs at half the issue rate, and with every term written out it
            // took 825 instructions a node and plane in place of 737 (192^3 FP16
            // state 306 -> 290 us, FP32 297 -> 287).
            const float K1r = c.K1 * rh, K2r = c.K2 * rh;
            const float G1[3] = {c.KC1 * F[0], c.KC1 * F[1], c.KC1 * F[2]};
            const float G2[3] = {c.KC2 * F[0], c.KC2 * F[1], c.KC2 * F[2]};
            float ltemp1 = 0.f, lrho1 = 0.f, lF1[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float S = lQ[1 + 2 * k] + lQ[2 + 2 * k], A = lQ[1 + 2 * k] - lQ[2 + 2 * k];
                const float SA = S + A, vS = v[k] * S;
                ltemp1 += S;
                lrho1 += v[k] * (0.5f * vS + A);
                lv[k] = K1r * (vS + A) + G1[k] * SA;
                lF1[k] = v[k] * SA;
            }
            // pairs (7,8) x+y, (9,10) x-y, (11,12) x+z, (13,14) x-z, (15,16) y+z, (17,18) y-z
            constexpr int PA[6] = {0, 0, 0, 0, 1, 1}, PB[6] = {1, 1, 2, 2, 2, 2};
            constexpr float SG[6] = {1.f, -1.f, 1.f, -1.f, 1.f, -1.f};
            float ltemp2 = 0.f, lrho2 = 0.f, lF2[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int pp = 0; pp < 6; pp++) {
                const int ia = PA[pp], ib = PB[pp];
                const float sg = SG[pp];
                const float w = v[ia] + sg * v[ib], Gs = G2[ia] + sg * G2[ib];
                const float S = lQ[7 + 2 * pp] + lQ[8 + 2 * pp], A = lQ[7 + 2 * pp] - lQ[8 + 2 * pp];
                const float wS = w * S, B = wS + A;
                ltemp2 += S;
                lrho2 += w * (0.5f * wS + A);
                const float lw = K2r * B + Gs * S;
                lv[ia] += lw;
                lv[ib] += sg * lw;
                lF2[ia] += B;
                lF2[ib] += sg * B;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) lF[k] = c.KC1 * lF1[k] + c.KC2 * lF2[k];
            const float T0 = c.K0 * lQ[0], T = c.K2 * ltemp2 + (c.K1 * ltemp1 + T0);
            ls = T - 3.f * T0;
            lUF = -(c.KC2 * ltemp2 + (c.KC1 * ltemp1 + c.KC0 * lQ[0]));
            lvsq6 = -rh * T * (1.f / 3.f);
            lrho += (1.f - vsq6) * T + (c.K1 * lrho1 + c.K2 * lrho2);
        }
#pragma unroll
        for (int k = 0; k < 3; k++) {
            lv[k] += lvsq6 * v[k];
            lus[k] += lUF * F[k] + 3.f * lv[k];
            lF[k] += lUF * us[k];
        }
        const float ls3 = 3.f * ls;
        lphi += mu * ls3;
        lmu += ph * ls3;
        float lm[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            lm[k] = lus[k] * inv;
            lF[k] += 0.5f * lm[k];
            lrho -= lm[k] * us[k];   // us = u + F / (2 rho)
        }
#pragma unroll
        for (int k = 0; k < 3; k++) lmu += gr[k] * lF[k];
        if (heavy) dg += lF[2];
        lphi += c.alpha4 * (3.f * ph * ph - c.phiStarSq) * lmu;
        a.lsrc[0][t] = -c.kappa * lmu;
#pragma unroll
        for (int k = 0; k < 3; k++) a.lsrc[1 + k][t] = mu * lF[k];
        if (a.add_source) {
            // the objective's source but for its part of A / B, which is the
            // same at every node and which the stencil kernel adds when A is
            // known (objective_source with ratio 0)
            const float half_inv = 0.5f / phiStar, s_over_b = (float)a.ab[3];
            const float w = (phiStar - ph) * half_inv, uz = m[2] * inv, duz = s_over_b * w;
            wuz += (double)(w * (m[2] / rh));
            lphi += -half_inv * s_over_b * uz;
            lrho += -duz * uz * inv;
            lm[2] += duz * inv;
        }
        a.lphi[t] = lphi;
        if constexpr (LQ) {
#pragma unroll
            for (int i = 0; i < kQf; i++) a.lq_o[i][t] = c.invTauPhiOne * lP[i];
        }
#pragma unroll
        for (int i = 0; i < kQg; i++) {
            float o = c.invTauRhoOne * lQ[i] + lrho;
            if (kCx(i)) o += kCx(i) * lm[0];
            if (kCy(i)) o += kCy(i) * lm[1];
            if (kCz(i)) o += kCz(i) * lm[2];
            a.lg_o[i][t] = o;
        }
    }
    // per-warp sums into the warp's own slot, in a fixed order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dg += __shfl_down_sync(0xffffffffu, dg, o);
    if (tx == 0) a.dgrav[blockIdx.x * (NTA / 32) + ty] += dg;
    if (a.add_source) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wuz += __shfl_down_sync(0xffffffffu, wuz, o);
        if (tx == 0) a.wuz[blockIdx.x * (NTA / 32) + ty] = wuz;
    }
}

// L = lambda_phi + Lap[lambda_lap] - sum_k D_k[lambda_grad_k]: the transposed
// stencils, added to lambda_phi in place.  Laplacian weights: 2/6 on faces, 1/6
// on edges, -4 at the centre; gradient component k: c_ik times 2/12 on faces,
// 1/12 on edges.
//
// A block marches tz planes of a 32 x 8 tile.  The four source fields of a
// plane (the tile plus one node) are staged two planes ahead with 16-byte
// cp.async copies.  Regrouped by plane, a node takes three numbers from each:
// what it adds to the node in it, to the node above and to the node below,
// which two registers carry down the march.  A thread has two rows of the
// tile, which share the rows between them: 20 shared-memory reads a node and
// plane (31 with one row, 49 without the regrouping), and eight blocks of 128
// threads stay on an SM.  24 bytes a node, 59 us at 256^3 at the copy
// bandwidth; 84 us (one row a thread and lambda_phi read where it is used
// 104, the kernel before with no staging 152), 128^3 16 us (20, 24): bound by
// the latency of its shared-memory reads and barriers beside DRAM at 70 %.
struct StencilGeo {
    static constexpr int P = TXA + 8, ROWS = TYA + 2;      // staged row and rows (floats)
    static constexpr int FIELD = P * ROWS, PLANE = 4 * FIELD;
    static constexpr int CHUNKS = PLANE / 4;               // 16-byte chunks of a plane
    static constexpr int NT = NTA / 2;                     // threads of a block, two rows each
    static constexpr int PER = (CHUNKS + NT - 1) / NT;     // per thread
    static constexpr int STAGES = 4;
};

__global__ void __launch_bounds__(StencilGeo::NT, kStencilBlocks)
adjoint_stencil_kernel(Box b, const float *__restrict__ lsrc, float *__restrict__ lphi, int tz,
                       const double *__restrict__ ab, float phiStar)
{
    // the objective's source common to all nodes (see the march kernel)
    const float common = ab ? 0.5f / phiStar * (float)ab[3] * (float)ab[2] : 0.f;
    using G = StencilGeo;
    __shared__ __align__(16) float sm[G::STAGES][G::PLANE];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TXA + tx;
    const int ntx = b.nx / TXA, nty = b.ny / TYA;
    const int bx = blockIdx.x % ntx, by = (blockIdx.x / ntx) % nty, bz = blockIdx.x / (ntx * nty);
    const int x0 = bx * TXA, y0 = by * TYA, z0 = bz * tz, nzc = min(tz, b.nz - z0);
    const unsigned nxy = (unsigned)b.nxy;
    const unsigned n = (unsigned)b.n;
    // the chunks this thread stages: in-plane offset (periodic) and field
    unsigned off[G::PER];
#pragma unroll
    for (int q = 0; q < G::PER; q++) {
        const int e = tid + q * G::NT, f = e / (G::FIELD / 4), r = e % (G::FIELD / 4);
        const int row = r / (G::P / 4), kk = r % (G::P / 4);
        off[q] = (unsigned)f * n + (unsigned)(b.nx * wrap_to(y0 - 1 + row, b.ny) + wrap_to(x0 - 4 + 4 * kk, b.nx));
    }
    auto issue = [&](int z, int stage) {
        const unsigned zo = (unsigned)wrap_to(z, b.nz) * nxy;
#pragma unroll
        for (int q = 0; q < G::PER; q++) {
            const int e = tid + q * G::NT;
            if (e < G::CHUNKS) cp_async16(&sm[stage][4 * e], lsrc + zo + off[q]);
        }
    };
    // contributions of plane values at this thread's nodes (rows 2 ty and
    // 2 ty + 1 of the tile): to their own plane, to the plane below it (it is
    // the plane above that one) and to the plane above
    const int cell = (2 * ty + 1) * G::P + tx + 4;
    struct Part {
        float own[2], below[2], above[2];
    };
    auto part = [&](int stage) -> Part {
        constexpr int N = G::P;
        const float *l = sm[stage] + cell - N, *gx = l + G::FIELD, *gy = gx + G::FIELD, *gz = gy + G::FIELD;
        // rows -1 .. 2 about row 2 ty: sums over x - 1, x + 1 and differences
        float lc[4], ls[4], xd[4], yc[4], yd[4], ys[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            lc[r] = l[r * N];
            ls[r] = l[r * N + 1] + l[r * N - 1];
            xd[r] = gx[r * N + 1] - gx[r * N - 1];
            yc[r] = gy[r * N];
            ys[r] = gy[r * N + 1] + gy[r * N - 1];
        }
        Part p;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int c = k + 1;
            const float lf = ls[c] + (lc[c + 1] + lc[c - 1]), le = ls[c + 1] + ls[c - 1];
            const float sx = xd[c], sy = yc[c + 1] - yc[c - 1];
            const float dx = xd[c + 1] + xd[c - 1], dy = ys[c + 1] - ys[c - 1];
            const float *g = gz + c * N;
            const float sz = ((g[1] + g[-1]) + (g[N] + g[-N])) + 2.f * g[0];
            p.own[k] = (le + 2.f * (lf - 12.f * lc[c])) * kInv6 - (2.f * (sx + sy) + (dx + dy)) * kInv12;
            const float side = (lf + 2.f * lc[c]) * kInv6 - (sx + sy) * kInv12;
            p.below[k] = side - sz * kInv12;   // c_z = +1 of the node below
            p.above[k] = side + sz * kInv12;
        }
        return p;
    };
    // plane z0 - 1 + m is staged in stage m % STAGES, two planes ahead of its use
    auto at = [&](int m) { return (int)((unsigned)m % (unsigned)G::STAGES); };
#pragma unroll
    for (int m = 0; m < 3; m++) {
        issue(z0 - 1 + m, at(m));
        cp_async_commit();
    }
    unsigned t = (unsigned)z0 * nxy + (unsigned)((y0 + 2 * ty) * b.nx + x0 + tx);
    const unsigned row = (unsigned)b.nx;
    float next[2] = {lphi[t], lphi[t + row]};
    cp_async_wait_prior<2>();
    __syncthreads();
    Part cur = part(at(0));
    float from_below[2] = {cur.above[0], cur.above[1]};   // what plane z0 - 1 adds to plane z0
    cp_async_wait_prior<1>();
    __syncthreads();
    cur = part(at(1));
    for (int j = 0; j < nzc; ++j, t += nxy) {
        const float base[2] = {next[0], next[1]};
        // plane z + 2 takes the stage of plane z - 2, read before the last barrier
        if (j + 1 < nzc) {
            issue(z0 + j + 2, at(j + 3));
            next[0] = lphi[t + nxy];
            next[1] = lphi[t + nxy + row];
        }
        cp_async_commit();
        cp_async_wait_prior<1>();
        __syncthreads();   // plane z + 1 has landed
        const Part top = part(at(j + 2));
#pragma unroll
        for (int k = 0; k < 2; k++) {
            lphi[t + (unsigned)k * row] = (base[k] + common) + ((cur.own[k] + top.below[k]) + from_below[k]);
            from_below[k] = cur.above[k];
        }
        cur = top;
    }
}

// acc[1] (dJ/dgrav) = sum of the per-warp sums.
__global__ void __launch_bounds__(NTA) dgrav_fold_kernel(const double *__restrict__ parts, int nparts,
                                                         double *__restrict__ acc)
{
    __shared__ double red[NTA / 32];
    double s = 0.0;
    for (int p = threadIdx.y * TXA + threadIdx.x; p < nparts; p += NTA) s += parts[p];
    s = block_sum(s, red);
    if (threadIdx.x == 0 && threadIdx.y == 0) acc[1] = s;
}

// dJ/dphi0 through the initial equilibrium (src/init_f.cu:57-78,
// src/init_g.cu:69-91), local part; llap receives lambda of the Laplacian.
// The 19 lambda_g are loaded before anything waits for phi: 256^3 450 -> 275 us
// (92 bytes a node, 227 us at the copy bandwidth), 128^3 65 -> 38, 64^3 17 -> 8.5.
__global__ void __launch_bounds__(NTA) init_adjoint_kernel(Box b, float alpha4, float kappa, float phiStarSq,
                                                           float Gamma, const float *__restrict__ phi0,
                                                           const float *__restrict__ lq,
                                                           const float *__restrict__ L,
                                                           const float *__restrict__ lg, float *__restrict__ lphi0,
                                                           float *__restrict__ llap)
{
    const unsigned n = (unsigned)b.n;
    const int x = blockIdx.x * TXA + threadIdx.x, y = blockIdx.y * TYA + threadIdx.y;
    for (int z = blockIdx.z * kPlanes, z_end = min(b.nz, z + kPlanes); z < z_end; z++) {
        const Nb p = neighbourhood(b, x, y, z);
        const unsigned t = p.at(0, 0, 0);
        float l[kQg];
#pragma unroll
        for (int i = 0; i < kQg; i++) l[i] = __ldg(lg + (i * n + t));
        const float add = L[t];   // lf_i = q_i + L
        float lap, gx, gy, gz;
        stencil19(phi0, p, lap, gx, gy, gz);
        const float ph = phi0[t];
        const float mu = alpha4 * ph * (ph * ph - phiStarSq) - kappa * lap;
        const float l0 = lq ? lq[t] + add : add;
        float lfs = 6.f * add, lga = 0.f, lgd = 0.f;
        if (lq)
            for (int i = 1; i < kQf; i++) lfs += lq[i * n + t];
#pragma unroll
        for (int i = 1; i < 7; i++) lga += l[i];
#pragma unroll
        for (int i = 7; i < kQg; i++) lgd += l[i];
        const float lg0 = l[0];
        const float lmu = -3.f * Gamma * l0 + 0.5f * Gamma * lfs - 6.f * kW0 * ph * lg0 + 3.f * kW1 * ph * lga
                          + 3.f * kW2 * ph * lgd;
        float lphi = l0 - 6.f * kW0 * mu * lg0 + 3.f * kW1 * mu * lga + 3.f * kW2 * mu * lgd;
        lphi += alpha4 * (3.f * ph * ph - phiStarSq) * lmu;
        llap[t] = -kappa * lmu;
        lphi0[t] = lphi;
    }
}

__global__ void __launch_bounds__(NTA) init_adjoint_stencil_kernel(Box b, const float *__restrict__ llap,
                                                                   float *__restrict__ lphi0)
{
    const int x = blockIdx.x * TXA + threadIdx.x, y = blockIdx.y * TYA + threadIdx.y;
    for (int z = blockIdx.z * kPlanes, z_end = min(b.nz, z + kPlanes); z < z_end; z++) {
        const Nb p = neighbourhood(b, x, y, z);
        float l1, d0, d1, d2;
        stencil19(llap, p, l1, d0, d1, d2);
        lphi0[p.at(0, 0, 0)] += l1;
    }
}

dim3 adjoint_grid(const Box &b)
{
    return dim3((unsigned)(b.nx / TXA), (unsigned)(b.ny / TYA), (unsigned)((b.nz + kPlanes - 1) / kPlanes));
}

// The march kernel's planes per block and its blocks.  Constants of the cost
// (march_depth), fitted to depths 1 to 32 on seven boxes and checked on 21
// others: a block's prologue is about one plane, two blocks on an SM take 1.3
// times as long as one, and a last round pays for its second block on an SM
// almost in full.  Against an earlier fit that took that block for a third of
// its time: 128^3 FP32 state 87 -> 85 us, FP16 92 -> 88.5, 128 x 64 x 128 51
// -> 47.6, the 42 cases 0.8 % on average, the worst 3 % slower.
struct March {
    int tz, blocks;
};
March march_of(const Box &b)
{
    constexpr MarchCost cost = {32, 1.2, {0.0, 1.0, 1.3}, {0.4, 1.1, 1.8}};
    const int tiles = (b.nx / TXA) * (b.ny / TYA);
    const int tz = march_depth(tiles, b.nz, sm_count(), 2, cost).tz;
    return March{tz, tiles * ((b.nz + tz - 1) / tz)};
}
// The stencil kernel's: a prologue of two planes, kStencilBlocks blocks on an
// SM.  Depths from 2 to 32 measured on seven boxes: the choice is within 5 % of
// the best (64^3 2 planes 5.7 us, best 3 planes 5.5; 128^3 16.1, best; 256^3
// 20 to 24 planes 84, 16 85, 32 86.5, 8 91.5).
March stencil_march(const Box &b)
{
    constexpr MarchCost cost = {24, 2.0, {0.0, 1.0, 1.05, 1.15, 1.3, 1.45, 1.65, 1.85, 2.1}, {0.88, 0.88, 0.93, 1.02, 1.15, 1.28, 1.46, 1.64, 1.85}};
    const int tiles = (b.nx / TXA) * (b.ny / TYA);
    const int tz = march_depth(tiles, b.nz, sm_count(), kStencilBlocks, cost).tz;
    return March{tz, tiles * ((b.nz + tz - 1) / tz)};
}

size_t blocks_of(const dim3 &g) { return (size_t)g.x * g.y * g.z; }

const dim3 kBlock(TXA, TYA);

// fn(ST{}, std::integral_constant<bool, ODD>{}) for the state's storage type and g layout.
template <typename Fn>
cudaError_t dispatch(const NativeState &st, Fn &&fn)
{
    auto with = [&](auto tag) { return st.g_odd ? fn(tag, std::true_type{}) : fn(tag, std::false_type{}); };
    switch (st.storage) {
    case LBM_STORAGE_FP32: return with(float{});
    case LBM_STORAGE_FP16: return with(__half{});
    case LBM_STORAGE_BF16: return with(__nv_bfloat16{});
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// per-field pointers of a native state
GFields g_fields(const Box &b, const NativeState &st)
{
    GFields r;
    const size_t stride = (size_t)b.n * storage_bytes(st.storage);
    for (int i = 0; i < kQg; i++) r.f[i] = static_cast<const unsigned char *>(st.g) + (size_t)i * stride;
    return r;
}
FQFields fq_fields(const Box &b, const NativeState &st)
{
    FQFields r;
    const size_t stride = (size_t)b.n * storage_bytes(st.storage);
    for (int i = 0; i < kQf - 1; i++) r.f[i] = static_cast<const unsigned char *>(st.fq) + (size_t)i * stride;
    return r;
}

size_t adjoint_dgrav_parts(const Box &b) { return (size_t)march_of(b).blocks * (NTA / 32); }

size_t adjoint_blocks(const Box &b) { return blocks_of(adjoint_grid(b)); }

cudaError_t launch_adjoint_phi(const Box &b, float eta, const Quant &q, const NativeState &st, float *phi,
                               cudaStream_t s, float phiStar, double scale, double *partials, double *ab)
{
    const int streamed = st.f_streamed ? 1 : 0;
    const dim3 grid = adjoint_grid(b), pair(TXA / 2, TYA);
    const FQFields fq = fq_fields(b, st);
    auto go = [&](auto sum) {
        constexpr bool SUM = decltype(sum)::value;
        switch (st.storage) {
        case LBM_STORAGE_FP32:
            adjoint_phi_kernel<SUM><<<grid, kBlock, 0, s>>>(b, eta, st.f0, fq, streamed, phi, phiStar, partials);
            break;
        case LBM_STORAGE_FP16:
            adjoint_phi_pair_kernel<__half, SUM><<<grid, pair, 0, s>>>(b, eta, q.f_inv, st.f0, fq, streamed, phi,
                                                                       phiStar, partials);
            break;
        case LBM_STORAGE_BF16:
            adjoint_phi_pair_kernel<__nv_bfloat16, SUM><<<grid, pair, 0, s>>>(b, eta, q.f_inv, st.f0, fq, streamed,
                                                                              phi, phiStar, partials);
            break;
        default: return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    };
    if (!ab) return go(std::false_type{});
    const cudaError_t e = go(std::true_type{});
    if (e != cudaSuccess) return e;
    weight_fold_kernel<<<1, kBlock, 0, s>>>(partials, (int)blocks_of(grid), scale, ab);
    return cudaGetLastError();
}

cudaError_t launch_objective(const Box &b, int objective, float phiStar, double scale, const Quant &q,
                             const NativeState &st, const float *phi, double *partials, double *ab, double *acc,
                             cudaStream_t s)
{
    cudaError_t e = dispatch(st, [&](auto tag, auto odd) {
        using ST = decltype(tag);
        objective_kernel<ST, decltype(odd)::value><<<adjoint_grid(b), kBlock, 0, s>>>(
            b, objective, phiStar, q, g_fields(b, st), phi, partials);
        return cudaGetLastError();
    });
    if (e != cudaSuccess) return e;
    objective_fold_kernel<<<1, kBlock, 0, s>>>(partials, (int)blocks_of(adjoint_grid(b)), scale, ab, acc);
    return cudaGetLastError();
}

cudaError_t launch_source_init(const Box &b, int objective, double scale, const double *ab, float phiStar,
                               const Quant &q, const NativeState &st, const float *phi, float *lq, float *lg,
                               float *L, cudaStream_t s)
{
    return dispatch(st, [&](auto tag, auto odd) {
        using ST = decltype(tag);
        source_init_kernel<ST, decltype(odd)::value><<<adjoint_grid(b), kBlock, 0, s>>>(
            b, objective, scale, ab, phiStar, q, g_fields(b, st), phi, lq, lg, L);
        return cudaGetLastError();
    });
}

cudaError_t launch_adjoint_step(const Box &b, const StepConst &c, float phiStar, const Quant &q,
                                const NativeState &st, const AdjointBuffers &a, bool add_source, double scale,
                                cudaStream_t s)
{
    AdjIn in;
    std::memset(&in, 0, sizeof(in));
    in.phi = a.phi;
    in.L = a.L_in;
    in.lphi = a.L_out;
    const size_t n = (size_t)b.n, esz = storage_bytes(st.storage);
    for (int i = 0; i < kQg; i++) {
        in.g_f[i] = static_cast<const unsigned char *>(st.g) + (size_t)i * n * esz;
        in.lg_f[i] = a.lg_in + (size_t)i * n;
        in.lg_o[i] = a.lg_out + (size_t)i * n;
    }
    for (int i = 0; i < kQf && a.lq_in; i++) {
        in.lq_f[i] = a.lq_in + (size_t)i * n;
        in.lq_o[i] = a.lq_out + (size_t)i * n;
    }
    for (int k = 0; k < 4; k++) in.lsrc[k] = a.lsrc + (size_t)k * n;
    in.dgrav = a.dgrav;
    in.wuz = a.wuz;
    in.ab = a.ab;
    in.add_source = add_source ? 1 : 0;
    const March march = march_of(b);
    cudaError_t e = dispatch(st, [&](auto tag, auto odd) {
        using ST = decltype(tag);
        auto go = [&](auto kernel) {
            // per launch: the attribute belongs to the device's function, and this is not a hot path of the host
            cudaError_t ea = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo<ST>::SMEM);
            if (ea != cudaSuccess) return ea;
            kernel<<<(unsigned)march.blocks, kBlock, Geo<ST>::SMEM, s>>>(b, c, phiStar, q, in, march.tz);
            return cudaGetLastError();
        };
        return a.lq_in ? go(adjoint_march_kernel<ST, decltype(odd)::value, true>)
                       : go(adjoint_march_kernel<ST, decltype(odd)::value, false>);
    });
    if (e != cudaSuccess) return e;
    if (add_source) {
        velocity_fold_kernel<<<1, 1024, 0, s>>>(a.wuz, march.blocks * (NTA / 32), scale, a.ab, a.acc);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    const March sten = stencil_march(b);
    adjoint_stencil_kernel<<<(unsigned)sten.blocks, dim3(TXA, TYA / 2), 0, s>>>(b, a.lsrc, a.L_out, sten.tz,
                                                                         add_source ? a.ab : nullptr, phiStar);
    return cudaGetLastError();
}

cudaError_t launch_dgrav_fold(const Box &b, const double *dgrav, double *acc, cudaStream_t s)
{
    dgrav_fold_kernel<<<1, kBlock, 0, s>>>(dgrav, (int)adjoint_dgrav_parts(b), acc);
    return cudaGetLastError();
}

cudaError_t launch_init_adjoint(const Box &b, const lbm_derived &d, float Gamma, const float *phi0, const float *lq,
                                const float *L, const float *lg, float *lphi0, float *llap, cudaStream_t s)
{
    init_adjoint_kernel<<<adjoint_grid(b), kBlock, 0, s>>>(b, d.alpha4, d.kappa, d.phiStarSq, Gamma, phi0, lq, L,
                                                           lg, lphi0, llap);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    init_adjoint_stencil_kernel<<<adjoint_grid(b), kBlock, 0, s>>>(b, llap, lphi0);
    return cudaGetLastError();
}

}  // namespace lbm
