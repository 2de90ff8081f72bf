// Set-up of the one-element-per-thread stage kernels (see lane.h).
#include "lane.h"

#include <algorithm>
#include <cmath>

namespace hgg {

bool tensor_lane_setup(const HostOperators &op, TensorLaneGeom &g, std::vector<int32_t> &nbr) {
    const int d = op.dim, np = op.np, ns = 2 * d;
    if (!op.tensor || !tensor_lane_order(d, op.order) || np != op.order + 1) return false;
    if (op.trace_pos[0] != 0 || op.trace_pos[1] != 1) return false;
    const double *a0 = op.elem_geo.data(), *s0 = op.t_sigma.data();
    const int8_t *m0 = op.t_mode.data();
    double abig = 0.0, sbig = 0.0;
    for (int c = 0; c < d; ++c) abig = std::max(abig, std::fabs(a0[c]));
    for (int s = 0; s < ns; ++s) sbig = std::max(sbig, std::fabs(s0[s]));
    const double atol = std::ldexp(abig, -40), stol = std::ldexp(sbig, -40);
    if (!std::isfinite(abig) || !std::isfinite(sbig)) return false;
    for (int64_t e = 0; e < op.nE; ++e) {
        for (int c = 0; c < d; ++c)
            if (!(std::fabs(op.elem_geo[e * d + c] - a0[c]) <= atol)) return false;
        for (int s = 0; s < ns; ++s)
            if (op.t_mode[e * ns + s] != m0[s] || !(std::fabs(op.t_sigma[e * ns + s] - s0[s]) <= stol)) return false;
    }
    g = TensorLaneGeom{};
    for (int i = 0; i < np * np; ++i) g.D1[i] = (float)op.D1[i];
    for (int sd = 0; sd < 2; ++sd)
        for (int a = 0; a < np; ++a) g.lift[sd][a] = (float)op.lift[(size_t)sd * np + a];
    for (int c = 0; c < d; ++c) {
        double *E = g.E + c * np * np, *L = g.L + c * np;
        for (int i = 0; i < np * np; ++i) E[i] = a0[c] * op.D1[i];
        g.side[c] = -1;
        g.ahat[c] = (float)a0[c];
        for (int sd = 0; sd < 2; ++sd) {
            const double sigma = s0[2 * c + sd];
            g.sigma[c][sd] = (float)sigma;
            const double *lift = &op.lift[(size_t)sd * np];
            switch (m0[2 * c + sd]) {
                case MODE_NONE: break;
                case MODE_SELF:
                    g.outflow[c] |= 1 << sd;
                    for (int a = 0; a < np; ++a) E[a * np + op.trace_pos[sd]] -= sigma * lift[a];
                    break;
                case MODE_NBR:
                    if (g.side[c] >= 0) return false;
                    g.side[c] = sd;
                    for (int a = 0; a < np; ++a) L[a] = -sigma * lift[a];
                    break;
                default:  // the average of a face along the flow: no flux when sigma is zero
                    if (sigma != 0.0) return false;
            }
        }
    }
    const int64_t tiles = (op.nE + 31) / 32;
    if (tiles > INT32_MAX) return false;
    g.n_tiles = (int32_t)tiles;
    nbr.assign((size_t)tiles * d * 32, 0);
    for (int64_t e = 0; e < op.nE; ++e)
        for (int c = 0; c < d; ++c)
            if (g.side[c] >= 0) nbr[((e >> 5) * d + c) * 32 + (e & 31)] = op.t_nbr[e * ns + 2 * c + g.side[c]];
    return true;
}

}  // namespace hgg
