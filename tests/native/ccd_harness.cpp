// Host build of the contact classification, the axis gap and the CCD's far limit
// (pamo_b200/csrc/distance.cuh) for the CPU tests.  Compiled by the test itself.
#include <cmath>
using std::fmax;
using std::fmin;
using std::sqrt;
#include "../../pamo_b200/csrc/distance.cuh"

using namespace pamo::s3;

extern "C" {

// n blocks of four vertices x and their steps p (float, 12 each): the classified
// float distance d, the float axis gap, and the first step slack (d - th) / lv of the
// FP64 class (infinite where lv is nothing)
void h_blocks(const float *x, const float *p, long long n, int kind, float ee_thres, double slack, double th, float *d,
              float *gap, double *first)
{
    for (long long b = 0; b < n; ++b) {
        F3 xf[4];
        D3 xd[4], v[4];
        for (int a = 0; a < 4; ++a) {
            const float *q = x + 12 * b + 3 * a, *s = p + 12 * b + 3 * a;
            xf[a] = {q[0], q[1], q[2]};
            xd[a] = {q[0], q[1], q[2]};
            v[a] = {s[0], s[1], s[2]};
        }
        const int t = classify(kind, xf, ee_thres);
        d[b] = classified_distance(kind, t, xf);
        gap[b] = axis_gap(kind, t, xf);
        const D3 avg = 0.25 * (v[0] + v[1] + v[2] + v[3]);
        for (int a = 0; a < 4; ++a) v[a] = v[a] - avg;
        const double lv = kind == KIND_PT ? len(v[0]) + fmax(len(v[1]), fmax(len(v[2]), len(v[3])))
                                          : fmax(len(v[0]), len(v[1])) + fmax(len(v[2]), len(v[3]));
        const double dd = classified_distance(kind, classify(kind, xd, (double)ee_thres), xd);
        first[b] = lv < 1e-12 ? INFINITY : slack * fmax(dd - th, 0.0) / lv;
    }
}

float h_ccd_far(float step_bound, float slack, float thick, int max_iters)
{
    return ccd_far(step_bound, slack, thick, max_iters);
}
}
