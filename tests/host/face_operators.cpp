// Which face operators are merged, and which trial functions vanish on a face (host code
// only).  arguments: dim, simplices, order, relative change of every second face
// tabulation, value added to every function that vanishes on a face.  Prints the number of
// pair operators, of distinct ones, and of trial functions that do not vanish.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "operators.h"
#include "setup.h"

using namespace hgg;

int main(int, char **argv) {
    const int dim = std::atoi(argv[1]);
    const bool tri = std::atoi(argv[2]);
    const int order = std::atoi(argv[3]);
    const double change = std::atof(argv[4]), value = std::atof(argv[5]);
    StructuredDescription sd;
    sd.n.assign(dim, 4);
    sd.lower.assign(dim, 0.0);
    sd.upper.assign(dim, 1.0);
    sd.triangular = tri;
    sd.periodic.assign(dim, true);
    const double cinv[1] = {0.8};
    StructuredProblem P = build_problem(structured_mesh(sd), order, 1, cinv, "RK4_4");
    const int nB = P.n_basis, nQ = P.face_rule.size();
    for (int t = 0; t < P.n_face_tabs; ++t)
        for (int j = 0; j < nB; ++j) {
            double most = 0.0;
            for (int q = 0; q < nQ; ++q) most = std::max(most, std::fabs(P.face_tabs[((size_t)t * nQ + q) * nB + j]));
            for (int q = 0; q < nQ; ++q) {
                double &v = P.face_tabs[((size_t)t * nQ + q) * nB + j];
                if (t % 2) v *= 1.0 + change;
                if (most < 1e-14) v += value;
            }
        }
    hgg_problem_desc d{};
    d.dim = dim;
    d.shape = P.mesh.shape;
    d.order = order;
    d.n_vars = P.n_vars;
    d.physics = 1;
    d.c_inv = P.c_inv;
    d.n_elements = P.mesh.n_elements;
    d.n_basis = nB;
    d.n_quad = P.rule.size();
    d.quad_weights = P.rule.weights.data();
    d.basis_values = P.basis_values.data();
    d.basis_grads = P.basis_grads.data();
    d.n_face_quad = nQ;
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
    int distinct = 0, trace = 0;
    for (int p = 0; p < op.n_pairs; ++p) {
        distinct += op.pair_same[p] == p;
        for (int j = 0; j < nB; ++j) trace += op.pair_trace[(size_t)p * nB + j];
    }
    std::printf("%d %d %d\n", op.n_pairs, distinct, trace);
    return 0;
}
