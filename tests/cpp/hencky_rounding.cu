// FP32 coefficients of StVK-Hencky (iso_coefficients) against FP64 and against
// the same quotients divided in FP32, on the host.  Prints per coefficient the
// two root-mean-square errors.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../ziran2019_b200/csrc/models.cuh"

using namespace zmpm;

int main()
{
    const double E = 5e4, nu = 0.35, mu = E / (2 * (1 + nu)), lam = E * nu / ((1 + nu) * (1 - 2 * nu));
    const double amps[] = { 0.01, 0.2, 0.6 };
    for (double amp : amps) {
        std::mt19937 rng(7);
        std::normal_distribution<double> nd(0, amp);
        double mine[12] = {}, plain[12] = {}, norm[12] = {};
        for (int n = 0; n < 200000; ++n) {
            float s[3], psi[3], c[12];
            for (float& v : s) v = (float)std::exp(nd(rng));
            const double sd[3] = { s[0], s[1], s[2] };
            double psid[3], cd[12];
            iso_coefficients<double>(ZMPM_MODEL_STVK_HENCKY_ISOTROPIC, mu, lam, sd, psid, cd);
            iso_coefficients<float>(ZMPM_MODEL_STVK_HENCKY_ISOTROPIC, (float)mu, (float)lam, s, psi, c);
            const float m = (float)mu, l = (float)lam, g = 2 * m + l;
            float L[3];
            for (int d = 0; d < 3; ++d) L[d] = std::log(std::fabs(s[d]));
            const float sum = L[0] + L[1] + L[2];
            float q[12];
            for (int d = 0; d < 3; ++d) q[d] = (2 * m * L[d] + l * sum) / s[d];
            const int o[3][2] = { { 1, 2 }, { 0, 2 }, { 0, 1 } }, pr[3][2] = { { 0, 1 }, { 0, 2 }, { 1, 2 } };
            for (int d = 0; d < 3; ++d) {
                q[3 + d] = (g * (1 - L[d]) - l * (L[o[d][0]] + L[o[d][1]])) / (s[d] * s[d]);
                const float x = s[pr[d][0]], y = s[pr[d][1]];
                q[6 + d] = l / (x * y);
                q[9 + d] = -(l * sum + 2 * m * diff_interlock_log_over_diff(x, y, L[pr[d][1]], 1e-6f)) / (x * y);
            }
            for (int k = 0; k < 12; ++k) {
                const double ref = k < 3 ? psid[k] : cd[k - 3], val = k < 3 ? psi[k] : c[k - 3];
                mine[k] += (val - ref) * (val - ref);
                plain[k] += (q[k] - ref) * (q[k] - ref);
                norm[k] += ref * ref;
            }
        }
        for (int k = 0; k < 12; ++k) std::printf("%g %d %.6e %.6e\n", amp, k, std::sqrt(mine[k] / norm[k]), std::sqrt(plain[k] / norm[k]));
    }
    return 0;
}
