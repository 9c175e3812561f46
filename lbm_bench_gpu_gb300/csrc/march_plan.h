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
// Fitted to forced depths 1 .. 60 of each geometry on 379 boxes from 64 x 40 x 6
// to 512 x 512 x 512, most of them drawn at random, a third of them flat, with
// more weight on boxes of up to 256 x 256 columns and 26 planes or more and on
// large ones.  The plan taken is within 1.0 % of the best one measured on average.
// Before, with constants fitted to boxes of up to 1.2 million nodes and at most
// 24 planes, it was 3.0 (FP32) and 1.9 % (16-bit), and 52 and 18 of the boxes took
// longer than with the single geometry and its older rule, by up to 17 and 12 %;
// now 5 and 3, by up to 3.1 and 5.4 % (the worst are FP32 160 x 232 x 41 60.6 ->
// 62.5 us, FP16 384 x 448 x 11 51.7 -> 54.5).  On 81 boxes of another draw one is slower than
// by the older rule (288 x 520 x 32 FP32, 0.8 %).  Older rule, before, now: FP32 384 x
// 320 x 40 194, 203, 191 us; 32 x 104 x 72 12.9, 14.6, 12.0; 256^3 615, 604, 607;
// FP16 448 x 256 x 30 81.3, 85.6, 78.2; 352 x 480 x 14 62.5, 67.9, 61.0.
struct StepPlan {
    bool deep;
    int tz;
};
inline StepPlan step_plan_16bit(long long tiles, int planes, int sms, int per_sm)
{
    constexpr MarchCost cost = {22, 0.87, {0.0, 1.0, 1.398, 2.292, 2.459}, {0.588, 1.168, 1.729, 2.125, 2.569}, 0.438};
    return {false, march_depth(tiles, planes, sms, per_sm, cost).tz};
}
inline StepPlan step_plan_fp32(long long tiles, int planes, int sms, int per_sm_deep, int per_sm_dense)
{
    constexpr MarchCost deep = {60, 1.52, {0.0, 1.0, 1.618}, {0.891, 1.816, 1.838}, 1.863, 0.002};
    constexpr MarchCost dense = {60, 1.383, {0.0, 1.0, 1.653, 1.757}, {0.888, 1.438, 1.825, 2.112}, 1.724, 0.032};
    const Depth d = march_depth(tiles, planes, sms, per_sm_deep, deep);
    const Depth e = march_depth(tiles, planes, sms, per_sm_dense, dense);
    // the two costs in one unit: a plane of the dense geometry takes a lone block
    // 1.35 times as long
    if (d.cost <= 1.354 * e.cost - 0.642) return {true, d.tz};
    return {false, e.tz};
}

}  // namespace lbm
