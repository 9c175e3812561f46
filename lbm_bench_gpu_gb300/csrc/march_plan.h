// march_plan.h -- planes per block of the kernels whose blocks march in z, and
// the step kernel's staging geometry (host code, no CUDA).
#pragma once

namespace lbm {

// Planes per block of a kernel whose blocks march `planes` planes on `tiles`
// column tiles, per_sm of them resident on each of sms SMs.  A block's time is
// about (tz + prologue) plane-times, and r blocks that share an SM slow each
// other down by share[r] (less than r: a lone block is bound by its own
// latencies).  The launch takes as many full rounds of resident blocks as there
// are, then a last, partly filled one, which overlaps the end of the others:
// x blocks per SM of it add tail[x] (interpolated; tail[0] is what the first of
// them adds) of their time, which is that of the last, shorter run of planes
// if there are no others among them.  hidden: plane-times of that last round
// that pass beside the others' end.  drift: the share that each plane past 22
// adds, where neighbouring blocks drift apart and share fewer halo rows in L2.
// The depth up to `deepest` that minimises the sum is taken; cost is in
// plane-times of a lone block.
struct MarchCost {
    int deepest;
    double prologue;
    double share[9], tail[9];
    double hidden = 0.0, drift = 0.0;
};
struct Depth {
    int tz;
    double cost;
};
inline Depth march_depth(long long tiles, int planes, int sms, int per_sm, const MarchCost &m)
{
    const long long slots = (long long)sms * per_sm;
    Depth best = {1, -1.0};
    for (int tz = 1; tz <= m.deepest; tz++) {
        const int runs = (planes + tz - 1) / tz, last = planes - (runs - 1) * tz;
        const long long blocks = tiles * runs, full = blocks / slots, rest = blocks % slots;
        double cost = (double)full * m.share[per_sm] * (tz + m.prologue);
        if (full == 0) {
            cost = m.share[(rest + sms - 1) / sms] * (tz + m.prologue);
        } else if (rest > 0) {
            const long long i = rest / sms;   // < per_sm
            const double t = m.tail[i] + (m.tail[i + 1] - m.tail[i]) * (double)(rest - i * sms) / (double)sms;
            const double tail = t * ((rest <= tiles ? last : tz) + m.prologue) - m.hidden;
            cost += tail > 0.0 ? tail : 0.0;
        }
        if (tz > 22) cost *= 1.0 + m.drift * (tz - 22);
        if (best.cost < 0.0 || cost < best.cost) best = {tz, cost};
    }
    return best;
}

// Staging geometry (FP32 storage) and planes per block of a step launch.
//
// Fitted to forced depths 1 .. 60 of each geometry on 222 boxes from 64 x 40 x 6
// to 512 x 512 x 256, most of them drawn at random, a third of them flat, with
// the boxes of up to 256 x 256 columns and 26 planes or more weighted 2.5 fold.
// On those the plan taken is within 1.2 % of the best one measured on average
// (at most 8.6 % FP32, 384 x 448 x 11 16 % 16-bit). Before, with constants
// fitted to boxes of up to 1.2 million nodes and at most 24 planes, it was 3.0 and
// 2.1 %, and flat boxes lost against the single geometry with its older rule:
// FP32 384 x 320 x 40 194 us by the older rule, 203 before, 191 now; 384 x 384
// x 32 181, 188, 179; 32 x 104 x 72 12.9, 14.6, 12.0; FP16 448 x 256 x 30 81.3,
// 85.6, 78.2; 352 x 480 x 14 62.5, 67.9, 61.0.  On 216 boxes of other draws no
// plan is slower than the older rule's by more than 0.5 %.
struct StepPlan {
    bool deep;
    int tz;
};
inline StepPlan step_plan_16bit(long long tiles, int planes, int sms, int per_sm)
{
    constexpr MarchCost cost = {22, 0.854, {0.0, 1.0, 1.356, 2.344, 2.371}, {0.431, 1.257, 1.978, 1.982, 2.385}, 0.182};
    return {false, march_depth(tiles, planes, sms, per_sm, cost).tz};
}
inline StepPlan step_plan_fp32(long long tiles, int planes, int sms, int per_sm_deep, int per_sm_dense)
{
    constexpr MarchCost deep = {60, 1.531, {0.0, 1.0, 1.62}, {0.884, 1.799, 1.836}, 1.825, 0.002};
    constexpr MarchCost dense = {60, 1.402, {0.0, 1.0, 1.589, 1.755}, {0.880, 1.531, 1.738, 2.126}, 1.741, 0.037};
    const Depth d = march_depth(tiles, planes, sms, per_sm_deep, deep);
    const Depth e = march_depth(tiles, planes, sms, per_sm_dense, dense);
    // the two costs in one unit: a plane of the dense geometry takes a lone block
    // 1.35 times as long
    if (d.cost <= 1.355 * e.cost - 0.644) return {true, d.tz};
    return {false, e.tz};
}

}  // namespace lbm
