// Which elements the lane kernels' set-up takes as equal (host code only).
// arguments: cells along each axis, upper corner, triangular, order, physics (0, 1),
// fp32, axis of the nodes to move (-1: none; dim: each node by its own amount along each
// axis), by how much (relative to a cell; every other node plane).  Prints: "tensor <accepted>" or "groups <accepted> <number of groups>
// <largest deviation of an element's geometry from its group's, relative to its own entry>
// <padding slots> <those that are their own neighbour across every face> <smallest face
// normal among the wave's plain tables' padding slots, 0 for other forms>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <sstream>
#include <string>

#include "lane.h"
#include "setup.h"

using namespace hgg;

int main(int argc, char **argv) {
    int at = 1;
    const int dim = std::atoi(argv[at++]);
    std::vector<int> n;
    std::vector<double> lower, upper;
    for (int i = 0; i < dim; ++i) n.push_back(std::atoi(argv[at++]));
    for (int i = 0; i < dim; ++i) lower.push_back(std::atof(argv[at++]));
    for (int i = 0; i < dim; ++i) upper.push_back(std::atof(argv[at++]));
    const bool tri = std::atoi(argv[at++]);
    const int order = std::atoi(argv[at++]), physics = std::atoi(argv[at++]);
    const bool fp32 = std::atoi(argv[at++]);
    const int axis = std::atoi(argv[at++]);
    const double by = std::atof(argv[at++]);
    StructuredDescription sd;
    sd.n.assign(n.begin(), n.end());
    sd.lower = lower;
    sd.upper = upper;
    sd.triangular = tri;
    sd.periodic.assign(dim, true);
    Mesh m = structured_mesh(sd);
    if (axis == dim) {
        for (size_t v = 0; v < m.nodes.size(); ++v) {
            uint64_t r = (uint64_t)m.nodes[v] * 0x9E3779B97F4A7C15ull;
            for (int c = 0; c < dim; ++c) {
                r = (r ^ (r >> 29)) * 0xBF58476D1CE4E5B9ull;
                m.coords[v * dim + c] += by * ((double)(r >> 11) * 0x1p-53 - 0.5) * (upper[c] - lower[c]) / n[c];
            }
        }
    } else if (axis >= 0) {
        const double h = (upper[axis] - lower[axis]) / n[axis];
        for (size_t v = 0; v < m.coords.size() / dim; ++v) {
            double &x = m.coords[v * dim + axis];
            if (std::lround((x - lower[axis]) / h) % 2) x += by * h;
        }
    }
    const double a[3] = {0.7, -0.4, 0.5}, cinv[1] = {0.8};
    StructuredProblem P = build_problem(std::move(m), order, physics, physics ? cinv : a, "RK4_4");
    hgg_problem_desc d{};
    d.dim = dim;
    d.shape = P.mesh.shape;
    d.order = order;
    d.n_vars = P.n_vars;
    d.physics = physics;
    for (int i = 0; i < 3; ++i) d.advection[i] = P.advection[i];
    d.c_inv = P.c_inv;
    d.n_elements = P.mesh.n_elements;
    d.n_basis = P.n_basis;
    d.n_quad = P.rule.size();
    d.quad_weights = P.rule.weights.data();
    d.basis_values = P.basis_values.data();
    d.basis_grads = P.basis_grads.data();
    d.n_face_quad = P.face_rule.size();
    d.face_weights = P.face_rule.weights.data();
    d.n_face_tabs = P.n_face_tabs;
    d.face_tabs = P.face_tabs.data();
    d.jacobians = P.jacobians.data();
    d.n_faces = P.mesh.n_faces();
    d.face_elements = P.mesh.face_elements.data();
    d.face_local = P.mesh.face_local.data();
    d.face_tab_index = P.face_tab_index.data();
    d.face_normals = P.normals.data();
    const HostOperators op = build_operators(d);
    if (op.tensor) {
        TensorLaneGeom g{};
        std::vector<int32_t> nbr;
        std::printf("tensor %d\n", (int)tensor_lane_setup(d, op, fp32, g, nbr));
        return 0;
    }
    LaneMesh lm;
    if (!lane_mesh(d, op, 148, 1, !fp32, 64, 1 << 20, lm)) {
        std::printf("groups 0 0 0 0 0 0\n");
        return 0;
    }
    std::vector<int32_t> group(lm.n_slots / 32);
    for (const LaneChunk &c : lm.chunks)
        for (int i = 0; i < c.tiles; ++i) group[c.tile0 + i] = c.group;
    double worst = 0.0;
    const int eg = (int)(op.elem_geo.size() / op.nE), fg = (int)(op.face_geo.size() / op.nE);
    for (int64_t e = 0; e < op.nE; ++e) {
        const int64_t r = lm.representative[group[lm.slot[e] >> 5]];
        auto compare = [&](double x, double y) {
            if (std::fabs(y) > 1e-9 && x != y) worst = std::max(worst, std::fabs(x - y) / std::fabs(y));
        };
        for (int i = 0; i < eg; ++i) compare(op.elem_geo[e * eg + i], op.elem_geo[r * eg + i]);
        for (int i = 0; i < fg; ++i) compare(op.face_geo[e * fg + i], op.face_geo[r * fg + i]);
    }
    std::vector<uint8_t> used(lm.n_slots, 0);
    for (int32_t s : lm.slot) used[s] = 1;
    double least = 0.0;
    LaneTables t;
    if (physics && fp32 && lane_wave_tables(op, lm, false, 4, t)) least = 1e300;
    int padding = 0, own = 0;
    for (int64_t s = 0; s < lm.n_slots; ++s) {
        if (used[s]) continue;
        ++padding;
        bool itself = true;
        for (int f = 0; f < op.nfl; ++f) itself &= lm.nbr[((s >> 5) * op.nfl + f) * 32 + (s & 31)] == s;
        own += itself;
        for (int f = 0; f < op.nfl && !t.geometry.empty(); ++f) {
            double q = 0.0;
            for (int c = 0; c < dim; ++c) {
                const double nu = t.geometry[((s >> 5) * (eg + fg) + eg + f * dim + c) * 32 + (s & 31)];
                q += nu * nu;
            }
            least = std::min(least, std::sqrt(q));
        }
    }
    std::printf("groups 1 %d %.3g %d %d %.3g\n", (int)lm.representative.size(), worst, padding, own, least);
    return 0;
}
