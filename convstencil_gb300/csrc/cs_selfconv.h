// cs_selfconv.h — kernels of several steps, on the host.
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

namespace cs {

// Kernel of `steps` steps of a (2r+1)^dims kernel (dims 1 or 2) at the centre
// of a (2R+1)^dims array: the self-convolution, every sum carried in two
// doubles (products by fma, sums by TwoSum) and rounded once at the end, what
// rounding leaves of one weight carried to the next so that their sum keeps
// its value (see f64_slice_weights). False when the weights' size could
// take a power of them out of range (such plans keep single steps, or fewer
// steps): the taps add up to at most (sum |w|)^steps in size, and every tap
// that weighs 2^-60 of that, with the rounding errors of its products, is a
// normal number while that lies within 2^+-900.
inline bool selfconv(const double *w, int dims, int r, int steps, int R, double *out)
{
    const int k = 2 * r + 1, K = 2 * R + 1, n = dims == 2 ? k * k : k, N = dims == 2 ? K * K : K;
    double sum = 0.0;
    for (int i = 0; i < n; ++i) sum += std::fabs(w[i]);
    if (steps * r > R) return false;
    if (steps > 1 && !(sum > 0x1p-64 && sum < 0x1p64 && std::fabs(std::log2(sum)) * steps < 900.0)) return false;
    std::vector<double> h(N, 0.0), l(N, 0.0), h2(N), l2(N);
    const int c = dims == 2 ? R * K + R : R;
    h[c] = 1.0;
    for (int s = 0; s < steps; ++s) {
        std::fill(h2.begin(), h2.end(), 0.0);
        std::fill(l2.begin(), l2.end(), 0.0);
        for (int i = 0; i < N; ++i) {
            if (h[i] == 0.0 && l[i] == 0.0) continue;
            for (int t = 0; t < n; ++t) {
                if (w[t] == 0.0) continue;
                const int j = i + (dims == 2 ? (t / k - r) * K + t % k - r : t - r);
                const double p = h[i] * w[t], pe = std::fma(h[i], w[t], -p) + l[i] * w[t];
                const double a = h2[j] + p, b = a - h2[j];
                l2[j] += (h2[j] - (a - b)) + (p - b) + pe;
                h2[j] = a;
            }
        }
        h.swap(h2);
        l.swap(l2);
    }
    double carry = 0.0;
    for (int i = 0; i < N; ++i) {
        out[i] = 0.0;
        if (h[i] == 0.0 && l[i] == 0.0) continue;
        out[i] = h[i] + (l[i] + carry);
        carry += (h[i] - out[i]) + l[i];
    }
    return true;
}

}  // namespace cs
