// zsc_stats.cu -- statistics of the phi, rho, u arrays in FP64.
//
// Replaces the host loops of src/stats.c:39-58 and the pressure part of
// src/logsave.c:63-150.  One pass over the five arrays: per-thread
// compensated float sums (a float pair hi + lo updated with Knuth's two-sum,
// products split exactly with an FMA), which hold ~48 bits like an FP64 sum
// at FP32 throughput (GB300's FP64 rate is a small fraction of its FP32 rate);
// the sums of a warp in three floats, FP64 across warps and blocks, all in a
// fixed order (deterministic for a given box).
//
// Partial / result layout (doubles):
//   0 max |u|^2 (compat)    1 #phi>=0 (compat)   2..4 sum u over phi>=0 (compat)
//   5 sum p over phi>=0     6 sum p over phi<0 (compat)
//   7 sum phi   8 sum rho   9..11 sum rho u   12 #phi>=0   13 max |u|^2
//   14 #non-finite nodes    15 unused
// "compat" skips the planes x = 0, nx-1 and y = 0, ny-1 like the reference.
#include <algorithm>

#include "lbm_internal.h"

namespace lbm {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int SX = 32;                       // columns of a warp, two rows a thread
constexpr int kBlocksPerSm = 2;              // resident blocks the launch bounds ask for (128 registers)
constexpr int kMaxBlocks = 152 * kBlocksPerSm;
constexpr float kInv6 = 0.16666666666666666667f;
constexpr float kInv12 = 0.08333333333333333333f;

constexpr float kCsSq = 0.33333333333333333333f;   // src/constants.h:48

struct StatsConst {
    float alpha, kappa, phiStarSq;
};

__device__ __forceinline__ bool is_max(int v) { return v == 0 || v == 13; }

// row index of (y, z)
__device__ __forceinline__ int kk_row(int y, int z, int ny) { return y + ny * z; }

// Compensated float accumulator: the sum is hi + lo.  The _rn intrinsics keep
// the compiler from contracting the two-sum's operations into FMAs, which
// would break the exact error terms.
struct Sum2 {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float x)
    {
        const float s = __fadd_rn(hi, x);
        const float bp = __fsub_rn(s, hi);
        lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(x, bp)));
        hi = s;
    }
    // a * b exactly (the product's rounding error from an FMA)
    __device__ __forceinline__ void add_product(float a, float b)
    {
        const float p = __fmul_rn(a, b);
        add(p);
        lo = __fadd_rn(lo, fmaf(a, b, -p));
    }
};

// s + e = a + b exactly (Knuth's two-sum)
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = __fadd_rn(a, b);
    const float bp = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

// A sum in three floats, for the sums of the threads' pairs.
struct Sum3 {
    float hi, lo, rest;
    __device__ __forceinline__ void add(const Sum3 &o)
    {
        float e1, e2, e3;
        two_sum(hi, o.hi, hi, e1);
        two_sum(lo, o.lo, lo, e2);
        two_sum(lo, e1, lo, e3);
        rest = __fadd_rn(__fadd_rn(rest, o.rest), __fadd_rn(e2, e3));
    }
    __device__ __forceinline__ Sum3 shuffled(int offset) const   // the value of the lane `offset` away
    {
        return Sum3{__shfl_xor_sync(0xffffffffu, hi, offset), __shfl_xor_sync(0xffffffffu, lo, offset),
                    __shfl_xor_sync(0xffffffffu, rest, offset)};
    }
    __device__ __forceinline__ double value() const { return (double)hi + ((double)lo + (double)rest); }
};

// What a node needs of one plane of phi for the 19-point Laplacian, the
// gradient and its own value: with f4 = e + w + n + s and e4 the four diagonal
// neighbours of the plane, the Laplacian sums to
//   (e4 + 2 f4 - 24 c) of its own plane + (f4 + 2 c) of the planes above and below,
// and the gradient components likewise (src/logsave.c:94-127 regrouped by
// plane): marching in z reads 9 values per node instead of 19.
struct Plane {
    float c, a, fx, fy;       // centre; f4 + 2 c; e - w; n - s
    float mid, gx, gy;        // e4 + 2 f4 - 24 c; own-plane parts of the x and y gradient
};

// One block: eight warps, a 32 x 2 WY tile of columns (WY = 8, fewer in a box
// of fewer rows, whose other warps take the next runs of planes); item `it` is
// one tile and 8 / WY runs of kz planes, one of which every thread marches at
// its two columns (rows y and y + 1, which share 6 of the 18 values of phi they
// need).  Plane z + 2 of phi and plane z + 1 of the other fields are loaded
// while plane z is computed.
// |u|^2 and the pressure are evaluated in float as the reference does
// (src/stats.c:45, src/logsave.c:94-137); sums are compensated, counts exact.
// phi_lo / phi_hi: the phi planes just below and above a z-slab (NULL for a
// periodic box, whose z neighbours wrap).  The pressure is summed over the
// reference's region only, so x and y need no wrap.
//
// Bound by instruction issue: the 20 bytes a node must be read take 49 us at
// 256^3 at the copy bandwidth, its 100 FP32 instructions (51 of them in the
// compensated sums of a node outside the bubbles) 45 us at one per cycle and
// scheduler, of about 180 in all.  Measured, lbm_stats_noalloc with its fold,
// 256^3: 368 -> 123 us, 128^3 35, 32^3 78 -> 12 us, against one thread per
// node reading 19 points, with 15 FP64 values per thread reduced over the block
// (FP64 runs at a 60th of the FP32 rate: that reduction was most of a small
// box's time).  Also measured at 256^3: one column a thread 145 us (223
// instructions a node), two nodes a thread in f32x2 147 (the packed operations
// issue at half rate and their constants take register pairs), the planes
// staged by cp.async 133.
template <int WY>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
stats_kernel(Box b, StatsConst c, const float *__restrict__ phi, const float *__restrict__ rho,
             const float *__restrict__ ux, const float *__restrict__ uy, const float *__restrict__ uz,
             double *__restrict__ partials, const float *__restrict__ phi_lo, const float *__restrict__ phi_hi, int kz,
             int items)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ntx = (b.nx + SX - 1) / SX, nty = (b.ny + 2 * WY - 1) / (2 * WY);
    const unsigned nx = (unsigned)b.nx, nxy = (unsigned)b.nxy;
    Sum2 s_phi, s_rho, s_mx, s_my, s_mz, s_ux, s_uy, s_uz, s_in, s_out;
    unsigned cnt_in = 0, cnt_all = 0, cnt_bad = 0;
    float umax_c = 0.f, umax_all = 0.f;

    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int tile = it % (ntx * nty), z0 = (it / (ntx * nty) * (kWarps / WY) + warp / WY) * kz;
        const int x = (tile % ntx) * SX + lane, y = (tile / ntx) * 2 * WY + 2 * (warp % WY);
        if (x >= b.nx || y >= b.ny || z0 >= b.nz) continue;   // (no barrier in this loop)
        const bool two = y + 1 < b.ny;          // the row y + 1 is in the box
        const bool x_in = x >= 1 && x <= b.nx - 2;
        const bool in_a = x_in && y >= 1 && y <= b.ny - 2, in_b = x_in && y + 1 <= b.ny - 2;
        const int n_z = min(kz, b.nz - z0);
        // rows y - 1 .. y + 2, clamped to the box (a clamped row is not used)
        const unsigned o0 = (unsigned)y * nx + (unsigned)x;
        const unsigned om = y > 0 ? o0 - nx : o0, o1 = two ? o0 + nx : o0, o2 = y + 2 < b.ny ? o0 + 2 * nx : o0;

        // phi around the two nodes on plane z (one past the box: its periodic or ghost neighbour)
        float c4[4], e4[4], w4[4];
        auto load_phi = [&](int z) {
            const float *p = phi;
            unsigned t = 0;
            if (z < 0 && phi_lo) p = phi_lo;
            else if (z >= b.nz && phi_hi) p = phi_hi;
            else t = (unsigned)(z < 0 ? b.nz - 1 : (z >= b.nz ? 0 : z)) * nxy;
            const float *const rows[4] = {p + (t + om), p + (t + o0), p + (t + o1), p + (t + o2)};
#pragma unroll
            for (int k = 0; k < 4; k++) c4[k] = __ldg(rows[k]);
            if (x_in) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    e4[k] = __ldg(rows[k] + 1);
                    w4[k] = __ldg(rows[k] - 1);
                }
            }
        };
        auto derive = [&](int k) -> Plane {   // of row k of the four
            Plane p;
            const float f4 = (e4[k] + w4[k]) + (c4[k + 1] + c4[k - 1]);
            const float d1 = e4[k + 1] - w4[k - 1], d2 = e4[k - 1] - w4[k + 1];
            p.c = c4[k];
            p.fx = e4[k] - w4[k];
            p.fy = c4[k + 1] - c4[k - 1];
            p.a = fmaf(2.f, p.c, f4);
            p.mid = fmaf(2.f, fmaf(-12.f, p.c, f4), (e4[k + 1] + w4[k - 1]) + (e4[k - 1] + w4[k + 1]));
            p.gx = fmaf(2.f, p.fx, d1 + d2);
            p.gy = fmaf(2.f, p.fy, d1 - d2);
            return p;
        };
        struct Fields {
            float rho, ux, uy, uz;
        };
        Fields fa, fb;
        auto load_fields = [&](int z) {
            const unsigned ta = (unsigned)z * nxy + o0, tb = (unsigned)z * nxy + o1;
            fa = Fields{__ldg(rho + ta), __ldg(ux + ta), __ldg(uy + ta), __ldg(uz + ta)};
            fb = Fields{__ldg(rho + tb), __ldg(ux + tb), __ldg(uy + tb), __ldg(uz + tb)};
        };
        // one node: cur its plane, top and (a_b, fx_b, fy_b) the ones above and below
        auto node = [&](const Plane &cur, const Plane &top, float a_b, float fx_b, float fy_b, const Fields &f,
                        bool region) {
            const float ph = cur.c;
            // 0 * x summed over the fields is 0 if all are finite, else NaN
            const float t =
                fmaf(0.f, f.uz, fmaf(0.f, f.uy, fmaf(0.f, f.ux, fmaf(0.f, f.rho, __fmul_rn(0.f, ph)))));
            if (t != 0.f) {   // NaN
                cnt_bad++;
                return;
            }
            const float u2 = fmaf(f.uz, f.uz, fmaf(f.uy, f.uy, f.ux * f.ux));
            s_phi.add(ph);
            s_rho.add(f.rho);
            s_mx.add_product(f.rho, f.ux);
            s_my.add_product(f.rho, f.uy);
            s_mz.add_product(f.rho, f.uz);
            const bool heavy = ph >= 0.f;
            cnt_all += heavy;
            umax_all = fmaxf(umax_all, u2);
            if (!region) return;
            umax_c = fmaxf(umax_c, u2);
            const float lap = ((cur.mid + top.a) + a_b) * kInv6;
            // 12 grad; z: 2 (ct - cb) + f4t - f4b, with a = f4 + 2 c
            const float gx = cur.gx + (top.fx + fx_b), gy = cur.gy + (top.fy + fy_b), gz = top.a - a_b;
            const float ph2 = ph * ph;
            const float bulk = fmaf(ph2, fmaf(3.f, ph2, -2.f * c.phiStarSq), -c.phiStarSq * c.phiStarSq);
            const float g2 = fmaf(gz, gz, fmaf(gy, gy, gx * gx));
            const float surf = fmaf(-0.5f * kInv12 * kInv12, g2, ph * lap);
            const float pres = fmaf(kCsSq, f.rho, fmaf(c.alpha, bulk, -c.kappa * surf));
            if (heavy) {
                cnt_in++;
                s_ux.add(f.ux);
                s_uy.add(f.uy);
                s_uz.add(f.uz);
                s_in.add(pres);
            } else {
                s_out.add(pres);
            }
        };

#pragma unroll
        for (int k = 0; k < 4; k++) e4[k] = w4[k] = 0.f;   // (outside the region: not used)
        load_phi(z0 - 1);
        Plane p = derive(1), q = derive(2);
        float a_a = p.a, fx_a = p.fx, fy_a = p.fy, a_b = q.a, fx_b = q.fx, fy_b = q.fy;
        load_phi(z0);
        Plane cur_a = derive(1), cur_b = derive(2);
        load_phi(z0 + 1);
        load_fields(z0);
#pragma unroll 2
        for (int k = 0; k < n_z; k++) {
            const Plane top_a = derive(1), top_b = derive(2);
            const Fields f0 = fa, f1 = fb;
            if (k + 1 < n_z) {
                load_phi(z0 + k + 2);
                load_fields(z0 + k + 1);
            }
            node(cur_a, top_a, a_a, fx_a, fy_a, f0, in_a);
            if (two) node(cur_b, top_b, a_b, fx_b, fy_b, f1, in_b);
            a_a = cur_a.a;
            fx_a = cur_a.fx;
            fy_a = cur_a.fy;
            a_b = cur_b.a;
            fx_b = cur_b.fx;
            fy_b = cur_b.fy;
            cur_a = top_a;
            cur_b = top_b;
        }
    }

    // The block's sums: the threads' ten float pairs as three floats each through
    // a recursive halving over the warp (16 value slots: after offsets 16, 8, 4, 2
    // a lane holds one value of 16 lanes, then offset 1), 16 additions per thread
    // in place of 50, and FP64 from one value per warp on.  Three floats keep more
    // than FP64's 53 bits (two kept 48).  A warp with a sum of 2^122 or more is
    // scaled by 2^-6, so that no sum over it leaves FP32's range; what that can
    // shift out is 2^-149.  With FP64 from each thread on, whose additions run at
    // a 60th of the rate, 32^3, 64^3 and 128^3 took 13.6, 22.8 and
    // 37.5 us, so 11.5, 18.7 and 35.2 (as two floats 11.5, 16.7 and 35.2).
    const Sum2 *const all[10] = {&s_ux, &s_uy, &s_uz, &s_in, &s_out, &s_phi, &s_rho, &s_mx, &s_my, &s_mz};
    float most = 0.f;
#pragma unroll
    for (int v = 0; v < 10; v++) most = fmaxf(most, fabsf(all[v]->hi));
    const bool wide = __reduce_max_sync(0xffffffffu, __float_as_uint(most)) >= __float_as_uint(0x1p122f);
    const float scale = wide ? 0x1p-6f : 1.f;
    Sum3 t[16];
#pragma unroll
    for (int v = 0; v < 16; v++)
        t[v] = v < 10 ? Sum3{all[v < 10 ? v : 0]->hi * scale, all[v < 10 ? v : 0]->lo * scale, 0.f} : Sum3{0.f, 0.f, 0.f};
#pragma unroll
    for (int half = 8; half >= 1; half >>= 1) {
        const bool up = lane & (2 * half);
#pragma unroll
        for (int v = 0; v < half; v++) {
            if (v >= 10) continue;   // (both slots of the pair are empty)
            const Sum3 give = up ? t[v] : t[v + half];
            t[v] = up ? t[v + half] : t[v];
            t[v].add(give.shuffled(2 * half));
        }
    }
    t[0].add(t[0].shuffled(1));
    cnt_in = __reduce_add_sync(0xffffffffu, cnt_in);
    cnt_all = __reduce_add_sync(0xffffffffu, cnt_all);
    cnt_bad = __reduce_add_sync(0xffffffffu, cnt_bad);
    // |u|^2 >= 0: floats order like their bits
    const unsigned mx_c = __reduce_max_sync(0xffffffffu, __float_as_uint(umax_c));
    const unsigned mx_a = __reduce_max_sync(0xffffffffu, __float_as_uint(umax_all));
    __shared__ double red[kWarps][kStatsValues];
    // lane 2 v (of each pair of lanes) holds sum v: result entries 2..6 and 7..11
    if ((lane & 1) == 0 && lane < 20) red[warp][2 + (lane >> 1)] = t[0].value() * (wide ? 64.0 : 1.0);
    if (lane == 31) {
        red[warp][0] = __uint_as_float(mx_c);
        red[warp][1] = cnt_in;
        red[warp][12] = cnt_all;
        red[warp][13] = __uint_as_float(mx_a);
        red[warp][14] = cnt_bad;
        red[warp][15] = 0.0;
    }
    __syncthreads();
    if (threadIdx.x < kStatsValues) {
        const int v = threadIdx.x;
        double s = red[0][v];
        for (int w = 1; w < kWarps; w++) s = is_max(v) ? fmax(s, red[w][v]) : s + red[w][v];
        partials[(size_t)blockIdx.x * kStatsValues + v] = s;
    }
}

// The blocks' partials in a fixed order: thread (row group, value) sums every
// 16th row, then the 16 groups in order.
__global__ void __launch_bounds__(kThreads) fold_kernel(const double *__restrict__ partials, int nparts,
                                                        double *__restrict__ out)
{
    constexpr int kGroups = kThreads / kStatsValues;
    __shared__ double red[kGroups][kStatsValues];
    const int v = threadIdx.x % kStatsValues, grp = threadIdx.x / kStatsValues;
    double acc = 0.0;
#pragma unroll 4
    for (int p = grp; p < nparts; p += kGroups) {
        const double x = partials[(size_t)p * kStatsValues + v];
        acc = is_max(v) ? fmax(acc, x) : acc + x;
    }
    red[grp][v] = acc;
    __syncthreads();
    if (grp == 0) {
        for (int g = 1; g < kGroups; g++) acc = is_max(v) ? fmax(acc, red[g][v]) : acc + red[g][v];
        out[v] = acc;
    }
}

// Pressure of every node (src/vtksave.c:63-127): the same float expression as
// the stats, periodic neighbours.  One thread per node of a row-major grid.
__global__ void __launch_bounds__(kThreads) pressure_kernel(Box b, StatsConst c, const float *__restrict__ phi,
                                                            const float *__restrict__ rho, float *__restrict__ out)
{
    const int nx = b.nx, ny = b.ny, nz = b.nz;
    const int rows = ny * nz;
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const int k = r / ny, j = r - k * ny;
        const int jn = j == ny - 1 ? 0 : j + 1, js = j == 0 ? ny - 1 : j - 1;
        const int kt = k == nz - 1 ? 0 : k + 1, kb = k == 0 ? nz - 1 : k - 1;
        const size_t row_c = (size_t)r * nx;
        const size_t row_n = ((size_t)kk_row(jn, k, ny)) * nx, row_s = ((size_t)kk_row(js, k, ny)) * nx;
        const size_t row_t = ((size_t)kk_row(j, kt, ny)) * nx, row_b = ((size_t)kk_row(j, kb, ny)) * nx;
        const size_t row_nt = ((size_t)kk_row(jn, kt, ny)) * nx, row_sb = ((size_t)kk_row(js, kb, ny)) * nx;
        const size_t row_nb = ((size_t)kk_row(jn, kb, ny)) * nx, row_st = ((size_t)kk_row(js, kt, ny)) * nx;
        for (int i = threadIdx.x; i < nx; i += blockDim.x) {
            const size_t t = row_c + i;
            const float ph = phi[t];
            const int ie = i == nx - 1 ? 0 : i + 1, iw = i == 0 ? nx - 1 : i - 1;
            const float p01 = phi[row_c + ie], p02 = phi[row_c + iw], p03 = phi[row_n + i], p04 = phi[row_s + i];
            const float p05 = phi[row_t + i], p06 = phi[row_b + i], p07 = phi[row_n + ie], p08 = phi[row_s + iw];
            const float p09 = phi[row_s + ie], p10 = phi[row_n + iw], p11 = phi[row_t + ie], p12 = phi[row_b + iw];
            const float p13 = phi[row_b + ie], p14 = phi[row_t + iw], p15 = phi[row_nt + i], p16 = phi[row_sb + i];
            const float p17 = phi[row_nb + i], p18 = phi[row_st + i];
            const float lap = (p07 + p08 + p09 + p10 + p11 + p12 + p13 + p14 + p15 + p16 + p17 + p18
                               + 2.f * (p01 + p02 + p03 + p04 + p05 + p06 - 12.f * ph)) * kInv6;
            const float gx = (2.f * (p01 - p02) + p07 - p08 + p09 - p10 + p11 - p12 + p13 - p14) * kInv12;
            const float gy = (2.f * (p03 - p04) + p07 - p08 + p10 - p09 + p15 - p16 + p17 - p18) * kInv12;
            const float gz = (2.f * (p05 - p06) + p11 - p12 + p14 - p13 + p15 - p16 + p18 - p17) * kInv12;
            const float ph2 = ph * ph;
            out[t] = c.alpha * (ph2 * (3.f * ph2 - 2.f * c.phiStarSq) - c.phiStarSq * c.phiStarSq)
                     - c.kappa * (ph * lap - 0.5f * (gx * gx + gy * gy + gz * gz)) + kCsSq * rho[t];
        }
    }
}

// How a box is cut: wy warps of a block side by side in y (8, 4 or 2, no more
// than the box's row pairs fill), and items of one tile and 8 / wy runs of
// kz planes, the deepest (up to 16) that still give every resident block four of
// them, so that uneven items even out; a small box takes single planes.  With
// all eight warps in y a box of 3 or 4 rows used two of them: 2048 x 3 x 2048
// 371 -> 128 us, 4096 x 4 x 1024 380 -> 136, 5 x 5 x 100000 251 -> 177
// (before the marching columns 216, 271 and 2652).
struct Cut {
    int wy, kz, items, blocks;
};
Cut stats_cut(const Box &b)
{
    int wy = kWarps;
    while (wy > 2 && 2 * (wy / 2) >= b.ny) wy /= 2;
    const int runs = kWarps / wy;
    const long long tiles = (long long)((b.nx + SX - 1) / SX) * ((b.ny + 2 * wy - 1) / (2 * wy));
    auto items_of = [&](int kz) { return tiles * ((b.nz + kz * runs - 1) / (kz * runs)); };
    int kz = 16;
    while (kz > 1 && items_of(kz) < 4 * kMaxBlocks) kz /= 2;
    const long long items = items_of(kz);
    return Cut{wy, kz, (int)items, (int)std::min<long long>(items, kMaxBlocks)};
}

cudaError_t launch_stats_kernels(const Box &b, const StatsConst &c, const float *const f[5], const float *phi_lo,
                                 const float *phi_hi, double *partials, double *result, cudaStream_t s)
{
    const Cut k = stats_cut(b);
    auto launch = [&](auto kernel) {
        kernel<<<(unsigned)k.blocks, kThreads, 0, s>>>(b, c, f[0], f[1], f[2], f[3], f[4], partials, phi_lo, phi_hi,
                                                       k.kz, k.items);
    };
    if (k.wy == 8) launch(stats_kernel<8>);
    else if (k.wy == 4) launch(stats_kernel<4>);
    else launch(stats_kernel<2>);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    fold_kernel<<<1, kThreads, 0, s>>>(partials, k.blocks, result);
    return cudaGetLastError();
}

}  // namespace

size_t stats_partial_count(const Box &b) { return (size_t)stats_cut(b).blocks; }

cudaError_t launch_stats(const Box &b, const lbm_derived &d, const float *mom, double *partials,
                         size_t partial_count, double *result, cudaStream_t s, const float *phi_lo,
                         const float *phi_hi)
{
    if (partial_count < stats_partial_count(b)) return cudaErrorInvalidValue;
    const float *f[5];
    for (int a = 0; a < 5; a++) f[a] = mom + (size_t)a * b.n;
    return launch_stats_kernels(b, StatsConst{d.alpha, d.kappa, d.phiStarSq}, f, phi_lo, phi_hi, partials, result, s);
}

cudaError_t launch_pressure(const Box &b, const lbm_derived &d, const float *mom, float *out, cudaStream_t s)
{
    StatsConst c{d.alpha, d.kappa, d.phiStarSq};
    long long blocks = (long long)b.ny * b.nz;
    if (blocks > 152 * 16) blocks = 152 * 16;
    pressure_kernel<<<(unsigned)blocks, kThreads, 0, s>>>(b, c, mom, mom + b.n, out);
    return cudaGetLastError();
}

}  // namespace lbm

// ---------------------------------------------------------------------------
// lbm_stats_noalloc: the same reduction for callers that must not allocate
// device memory.
//
// Who needs it: code that inspects the fields of a simulation it does not own
// -- an in-situ analysis or monitoring hook called from inside another
// program's time loop.  There the device memory usually belongs to the host
// application's own pool allocator, and cudaMalloc / cudaFree are off limits:
// they would take memory outside the application's budget and they
// synchronise the whole device, stalling the work already queued.  Such a
// caller hands over the five field arrays and a 16-double output buffer it
// already owns; this entry point adds nothing to them.
//
// The per-block partial sums live in a fixed array in the library's static
// device memory (38 KiB, one row per resident block, reserved on every GPU that
// loads the library until the process exits).  Boxes of more than 512^3 nodes
// are rejected (LBM_NOALLOC_MAX_NODES).  Every row the final fold reads is
// written earlier in the same call, so no part of the array has to be cleared
// between calls.  All calls share the array: two calls
// whose kernels overlap on the GPU (different streams, or different host
// threads on one device) race on it and must be ordered by the caller.
// ---------------------------------------------------------------------------
#include <mutex>

#include "per_device.h"

namespace lbm {
namespace {

constexpr long long kNoAllocMaxNodes = LBM_NOALLOC_MAX_NODES;

static __device__ __align__(256) double g_noalloc_partials[kMaxBlocks * kStatsValues];

std::mutex g_noalloc_mutex;
double *g_noalloc_ptr[kMaxDevices] = {};

// Device address of the scratch array on `device` (which must be current).
// Looked up on the first call per device; later calls reuse it.  A
// cudaDeviceReset of that device ends the context that holds the array, so a
// process that resets a device must not call lbm_stats_noalloc on it again.
cudaError_t noalloc_scratch(int device, double **out)
{
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[device]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[device] = static_cast<double *>(p);
    }
    *out = g_noalloc_ptr[device];
    return cudaSuccess;
}

}  // namespace
}  // namespace lbm

extern "C" int lbm_stats_noalloc(const lbm_params *p, const float *phi, const float *rho, const float *ux,
                                 const float *uy, const float *uz, double *raw_out, void *stream)
{
    if (!p || !phi || !rho || !ux || !uy || !uz || !raw_out) {
        lbm::set_error("lbm_stats_noalloc: NULL argument");
        return LBM_EINVAL;
    }
    if (p->nx < 3 || p->ny < 3 || p->nz < 3) {
        lbm::set_error("lbm_stats_noalloc: box must be at least 3 nodes in each direction");
        return LBM_EINVAL;
    }
    const long long n = (long long)p->nx * p->ny * p->nz;
    if (n > lbm::kNoAllocMaxNodes) {
        lbm::set_error("lbm_stats_noalloc: box of " + std::to_string(n) +
                       " nodes exceeds the no-allocation limit of LBM_NOALLOC_MAX_NODES = 512^3 nodes");
        return LBM_EINVAL;
    }
    if (p->device < 0 || p->device >= lbm::kMaxDevices) {
        lbm::set_error("lbm_stats_noalloc: device ordinal out of range");
        return LBM_EINVAL;
    }
    if (const char *why = lbm::physics_error(*p)) {
        lbm::set_error(std::string("lbm_stats_noalloc: ") + why);
        return LBM_EINVAL;
    }
    // the caller's current device is given back on return (when it can be read)
    int prev = 0;
    const bool have_prev = cudaGetDevice(&prev) == cudaSuccess;
    const bool switch_device = !have_prev || prev != p->device;
    cudaError_t e = switch_device ? cudaSetDevice(p->device) : cudaSuccess;
    double *scratch = nullptr;
    if (e == cudaSuccess) e = lbm::noalloc_scratch(p->device, &scratch);
    if (e == cudaSuccess) {
        lbm_derived d;
        lbm::derive(*p, d);
        lbm::Box b;
        b.nx = p->nx;
        b.ny = p->ny;
        b.nz = p->nz;
        b.nxy = (long long)p->nx * p->ny;
        b.n = n;
        const float *f[5] = {phi, rho, ux, uy, uz};
        e = lbm::launch_stats_kernels(b, lbm::StatsConst{d.alpha, d.kappa, d.phiStarSq}, f, nullptr, nullptr, scratch,
                                      raw_out, static_cast<cudaStream_t>(stream));
    }
    if (switch_device && have_prev) cudaSetDevice(prev);
    if (e != cudaSuccess) {
        lbm::set_error(std::string("lbm_stats_noalloc: ") + cudaGetErrorString(e));
        return LBM_ECUDA;
    }
    return LBM_OK;
}
