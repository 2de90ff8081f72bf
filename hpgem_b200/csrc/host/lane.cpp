// Set-up of the one-element-per-thread stage kernels (see lane.h).
#include "lane.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <optional>

#include "refshapes.h"

namespace hgg {

// The extent of the mesh along each axis bounds its coordinates' magnitude (a box that lies
// within a few times its own size of the origin, as meshes do).  The descriptor has no
// coordinates: the elements' places follow from their Jacobians, face by face, breadth
// first, so that periodic images stay within one period of the start.
GeometryRounding::GeometryRounding(const hgg_problem_desc &dsc, const HostOperators &o) : desc(dsc), op(o) {
    const int d = op.dim, nf = op.nfl;
    const ShapeInfo &si = shape_info(op.shape);
    const int fv = d == 1 ? 1 : si.face_vertices;
    double centre[3] = {0.0, 0.0, 0.0}, to_face[6][3] = {};  // face centres seen from the element's
    for (int k = 0; k < si.n_vertices; ++k)
        for (int c = 0; c < d; ++c) centre[c] += si.vertices[k][c] / si.n_vertices;
    for (int f = 0; f < nf; ++f)
        for (int c = 0; c < d; ++c) {
            for (int k = 0; k < fv; ++k) to_face[f][c] += si.vertices[si.faces[f][k]][c] / fv;
            to_face[f][c] -= centre[c];
        }
    std::vector<int8_t> other((size_t)op.nE * nf, 0);  // the neighbour's local face
    for (int64_t f = 0; f < desc.n_faces; ++f)
        for (int s = 0; s < 2; ++s)
            other[desc.face_elements[2 * f + s] * nf + desc.face_local[2 * f + s]] = (int8_t)desc.face_local[2 * f + 1 - s];
    std::vector<double> place((size_t)op.nE * d, 0.0);
    std::vector<uint8_t> seen(op.nE, 0);
    std::vector<int32_t> queue;
    queue.reserve(op.nE);
    double lo[3] = {0.0, 0.0, 0.0}, hi[3] = {0.0, 0.0, 0.0};
    for (int64_t start = 0; start < op.nE; ++start) {
        if (seen[start]) continue;
        seen[start] = 1;
        queue.push_back((int32_t)start);
        for (size_t at = queue.size() - 1; at < queue.size(); ++at) {
            const int64_t e = queue[at];
            const double *J = desc.jacobians + e * d * d, *x = &place[e * d];
            for (int r = 0; r < d; ++r) {
                double half = 0.0;  // (an element lies within |J_rc| of its centre, summed over c)
                for (int c = 0; c < d; ++c) half += std::fabs(J[r * d + c]);
                lo[r] = std::min(lo[r], x[r] - half);
                hi[r] = std::max(hi[r], x[r] + half);
            }
            for (int f = 0; f < nf; ++f) {
                const int32_t n = op.nbr[e * nf + f];
                if (seen[n]) continue;
                seen[n] = 1;
                const double *Jn = desc.jacobians + (int64_t)n * d * d;
                const double *a = to_face[f], *b = to_face[other[e * nf + f]];
                for (int r = 0; r < d; ++r) {
                    double y = x[r];
                    for (int c = 0; c < d; ++c) y += J[r * d + c] * a[c] - Jn[r * d + c] * b[c];
                    place[(int64_t)n * d + r] = y;
                }
                queue.push_back(n);
            }
        }
    }
    // a coordinate is off by half a unit in the last place (2^-54 of [0, L]'s upper half, twice
    // that where the box starts at L), a difference of two by twice as much, and two
    // elements' differences by four times
    for (int r = 0; r < d; ++r) eps[r] = 0x1p-51 * (hi[r] - lo[r]);
}

// With J' = J + dJ, |dJ_kl| <= eps_k, the inverse changes by J^{-1} dJ J^{-1}.  The rest is
// linear in it: ahat = J^{-1} a, G = J^{-T}, and n / |J| = J^{-T} m with m the reference
// element's face normal (Nanson's formula).
std::vector<double> GeometryRounding::bounds(int64_t e) const {
    const int d = op.dim, nf = op.nfl;
    const bool wave = op.physics != HGG_PHYSICS_ADVECTION;
    const ShapeInfo &si = shape_info(op.shape);
    double inv[9], t[9];  // J^{-1}, the bound of its change
    invert_matrix(d, desc.jacobians + e * d * d, inv);
    for (int c = 0; c < d; ++c)
        for (int r = 0; r < d; ++r) {
            double rows = 0.0, columns = 0.0;
            for (int k = 0; k < d; ++k) {
                rows += std::fabs(inv[c * d + k]) * eps[k];
                columns += std::fabs(inv[k * d + r]);
            }
            t[c * d + r] = rows * columns;
        }
    std::vector<double> out;
    double along[3] = {0.0, 0.0, 0.0};  // ... of ahat
    for (int c = 0; c < d; ++c)
        for (int r = 0; r < d; ++r) along[c] += t[c * d + r] * std::fabs(desc.advection[r]);
    if (wave)
        for (int r = 0; r < d; ++r)
            for (int c = 0; c < d; ++c) out.push_back(t[c * d + r]);
    else out.insert(out.end(), along, along + d);
    for (int f = 0; f < nf; ++f) {
        const int *v = si.faces[f];
        double m[3] = {1.0, 0.0, 0.0};
        if (d == 2) {
            m[0] = 0.5 * (si.vertices[v[1]][1] - si.vertices[v[0]][1]);
            m[1] = 0.5 * (si.vertices[v[1]][0] - si.vertices[v[0]][0]);
        } else if (d == 3) {
            const double scale = si.face_vertices == 4 ? 0.25 : 1.0;  // reference faces of area 4 and 1/2
            for (int c = 0; c < 3; ++c) {
                const int i = (c + 1) % 3, j = (c + 2) % 3;
                const double *x = si.vertices[v[0]], *y = si.vertices[v[1]], *z = si.vertices[v[2]];
                m[c] = scale * ((y[i] - x[i]) * (z[j] - x[j]) - (y[j] - x[j]) * (z[i] - x[i]));
            }
        }
        double sigma = 0.0;
        for (int c = 0; c < d; ++c) sigma += std::fabs(m[c]) * along[c];
        if (!wave) out.push_back(sigma);
        for (int r = 0; r < d && wave; ++r) {
            double nu = 0.0;
            for (int c = 0; c < d; ++c) nu += 0.5 * std::fabs(m[c]) * t[c * d + r];
            out.push_back(nu);
        }
    }
    return out;
}

bool tensor_lane_setup(const hgg_problem_desc &desc, const HostOperators &op, bool fp32, TensorLaneGeom &g,
                       std::vector<int32_t> &nbr) {
    const int d = op.dim, np = op.np, ns = 2 * d;
    if (!op.tensor || !tensor_lane_order(d, op.order) || np != op.order + 1) return false;
    if (op.trace_pos[0] != 0 || op.trace_pos[1] != 1) return false;
    const double *a0 = op.elem_geo.data(), *s0 = op.t_sigma.data();
    const int8_t *m0 = op.t_mode.data();
    // (a hypercube's sigma is +-ahat of its axis: the same bound)
    const std::vector<double> bound = GeometryRounding(desc, op).bounds(0);
    auto equal = [&](double v, double v0, int axis) {
        return std::isfinite(v) && std::fabs(v - v0) <= bound[axis] && (!fp32 || (float)v == (float)v0);
    };
    for (int64_t e = 0; e < op.nE; ++e) {
        for (int c = 0; c < d; ++c)
            if (!equal(op.elem_geo[e * d + c], a0[c], c)) return false;
        for (int s = 0; s < ns; ++s)
            if (op.t_mode[e * ns + s] != m0[s] || !equal(op.t_sigma[e * ns + s], s0[s], s / 2)) return false;
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

// ---- simplices and the wave -------------------------------------------------------

bool lane_mesh(const hgg_problem_desc &desc, const HostOperators &op, int num_sms, int chunk_tiles_max, bool folded,
               int coefficient_bytes, int spare_bytes, LaneMesh &m) {
    const int nf = op.nfl, d = op.dim, R = op.V * op.nB;
    const bool wave = op.physics != 0;
    // (plain tables hold no geometry: their kernels read every element's own)
    const int eg = !folded ? 0 : wave ? d * d : d, fg = !folded ? 0 : wave ? d : 1;
    // A group: elements with the same pair operators and upwind modes whose geometry differs
    // from the first one's by no more than the rounding of vertex coordinates, entry by
    // entry; all of them step with that one's values.  The hash key has the operators, the
    // modes, and the geometry rounded to 2^-20 of its largest entry (a filter only).
    // (the plain tables' results depend on their operators' last bits: no merging there)
    std::vector<int32_t> same = op.pair_same;
    if (!folded)
        for (int p = 0; p < op.n_pairs; ++p) same[p] = p;
    m = LaneMesh{};
    std::vector<int32_t> group(op.nE);
    std::vector<int64_t> count;
    const int words = 2 * nf + eg + nf * fg + 2;
    std::vector<uint64_t> key(words), keys;  // of one element, of the groups
    std::vector<int32_t> table(1024, -1);    // open addressing: groups by hash
    auto put = [&](uint64_t *dst, const double *v, int n) {
        double big = 0.0;
        for (int i = 0; i < n; ++i) big = std::max(big, std::fabs(v[i]));
        if (!std::isfinite(big)) return false;
        int e = 0;
        std::frexp(big, &e);
        // adding 1.5 * 2^52 rounds to a whole number (the scaled values are below 2^20)
        const double scale = big > 0.0 ? std::ldexp(1.0, 20 - e) : 0.0, magic = 0x1.8p52;
        for (int i = 0; i < n; ++i) {
            const volatile double r = v[i] * scale + magic;
            const double q = r;
            std::memcpy(&dst[i], &q, sizeof(q));
        }
        dst[n] = (uint64_t)(int64_t)e;
        return true;
    };
    const size_t most = (size_t)op.nE / 10 + 2 * num_sms;  // more groups than this take too much padding
    std::optional<GeometryRounding> rounding;
    if (folded) rounding.emplace(desc, op);
    std::vector<double> bounds;  // [group][eg + nf fg]
    const int ng = eg + nf * fg;
    auto equal = [&](int64_t e, int32_t g) {
        const int64_t r = m.representative[g];
        const double *b = &bounds[(size_t)g * ng];
        bool same_geo = true;
        for (int i = 0; i < eg; ++i) same_geo &= std::fabs(op.elem_geo[e * eg + i] - op.elem_geo[r * eg + i]) <= b[i];
        for (int i = 0; i < nf * fg; ++i)
            same_geo &= std::fabs(op.face_geo[e * nf * fg + i] - op.face_geo[r * nf * fg + i]) <= b[eg + i];
        return same_geo;
    };
    const int most_alike = 64;  // groups of one key: elements that vary by less than the filter sees
    for (int64_t e = 0; e < op.nE; ++e) {
        uint64_t *k = key.data();
        for (int f = 0; f < nf; ++f) {
            *k++ = (uint64_t)(uint32_t)same[op.self_pair[e * nf + f]] << 32 | (uint32_t)same[op.nbr_pair[e * nf + f]];
            *k++ = (uint64_t)op.mode[e * nf + f];
        }
        if (!put(k, &op.elem_geo[e * eg], eg) || !put(k + eg + 1, &op.face_geo[e * nf * fg], nf * fg)) return false;
        uint64_t hash = 0;
        for (uint64_t w : key) {
            hash = (hash ^ w) * 0x9E3779B97F4A7C15ull;
            hash ^= hash >> 29;
        }
        size_t at = hash & (table.size() - 1);
        for (int alike = 0; table[at] >= 0; at = (at + 1) & (table.size() - 1)) {
            if (!std::equal(key.begin(), key.end(), keys.begin() + (size_t)table[at] * words)) continue;
            if (!folded || equal(e, table[at])) break;
            if (++alike >= most_alike) return false;
        }
        if (table[at] < 0) {
            if (count.size() >= most || count.size() * 2 >= table.size()) return false;
            table[at] = (int32_t)count.size();
            keys.insert(keys.end(), key.begin(), key.end());
            m.representative.push_back(e);
            if (folded) {
                const std::vector<double> b = rounding->bounds(e);
                bounds.insert(bounds.end(), b.begin(), b.end());
            }
            count.push_back(0);
        }
        group[e] = table[at];
        count[group[e]]++;
    }
    int64_t tiles = 0;
    for (int64_t c : count) tiles += (c + 31) / 32;
    const int64_t pad = tiles * 32 - op.nE;
    // padded slots cost idle lanes and memory in every vector: at most twice as many as
    // elements (a full tile's element costs a third of the general kernels') unless all
    // tiles run at once, and within spare_bytes per element and 4 MB.  (A tile of one element
    // is then still the faster: 128 triangles that all differ, advection at p = 3 12.1 us per
    // RK4 step against 24.9, the wave at p = 1 12.7 against 32.8.)
    m.sparse = pad > 2 * op.nE;
    if (m.sparse && tiles > 2 * num_sms) return false;
    if ((double)pad * R * coefficient_bytes > (double)spare_bytes * (double)op.nE + 4e6) return false;
    if (tiles > INT32_MAX / 32) return false;
    m.n_slots = tiles * 32;
    // chunks of a group in element order, then all chunks by their first element, so that
    // neighbours in other groups run at about the same time
    const int per = 32 * chunk_tiles_max;
    std::vector<std::vector<int64_t>> members(count.size());
    for (size_t g = 0; g < count.size(); ++g) members[g].reserve(count[g]);
    for (int64_t e = 0; e < op.nE; ++e) members[group[e]].push_back(e);
    struct Piece {
        int64_t first;
        int32_t group;
        int64_t at;
    };
    std::vector<Piece> pieces;
    for (size_t g = 0; g < members.size(); ++g)
        for (int64_t at = 0; at < count[g]; at += per) pieces.push_back({members[g][at], (int32_t)g, at});
    std::sort(pieces.begin(), pieces.end(), [](const Piece &a, const Piece &b) { return a.first < b.first; });
    m.slot.assign(op.nE, 0);
    int32_t tile = 0;
    for (const Piece &p : pieces) {
        const int64_t n = std::min<int64_t>(per, count[p.group] - p.at);
        const int32_t nt = (int32_t)((n + 31) / 32);
        m.chunks.push_back({tile, nt, p.group, 0});
        for (int64_t i = 0; i < n; ++i) m.slot[members[p.group][p.at + i]] = tile * 32 + (int32_t)i;
        tile += nt;
    }
    // (a padding slot is its own neighbour: it starts at zero and stays there)
    m.nbr.resize((size_t)tiles * nf * 32);
    for (size_t i = 0; i < m.nbr.size(); ++i) m.nbr[i] = (int32_t)(i / (32 * nf) * 32 + i % 32);
    for (int64_t e = 0; e < op.nE; ++e)
        for (int f = 0; f < nf; ++f)
            m.nbr[((size_t)(m.slot[e] >> 5) * nf + f) * 32 + (m.slot[e] & 31)] = m.slot[op.nbr[e * nf + f]];
    return true;
}

namespace {

// functions of a face operator's trial side that do not vanish on the face; false when
// there are more than `most`
bool trace_columns(const HostOperators &op, int32_t pair, int most, std::vector<int32_t> &cols) {
    cols.clear();
    for (int j = 0; j < op.nB; ++j)
        if (op.pair_trace[(size_t)pair * op.nB + j]) cols.push_back(j);
    return (int)cols.size() <= most;
}

// appends to a group's table
struct Writer {
    std::vector<unsigned char> bytes;
    template <typename T>
    void put(T v) {
        const unsigned char *p = reinterpret_cast<const unsigned char *>(&v);
        bytes.insert(bytes.end(), p, p + sizeof(T));
    }
    // a value, or a column, of the contraction type
    void number(int elem_bytes, double v) {
        if (elem_bytes == 8) put(v);
        else put((float)v);
    }
    void plain_column(int elem_bytes, const double *A, int nb, int j, int r0, int rb, int rbp) {
        if (elem_bytes == 8) column<double>(A, nb, j, r0, rb, rbp, 1.0);
        else column<float>(A, nb, j, r0, rb, rbp, 1.0);
    }
    // column j of A ([nb][nb], scaled): rows r0 .. r0 + rb, padded with zeros
    template <typename T>
    void column(const double *A, int nb, int j, int r0, int rb, int rbp, double scale) {
        for (int i = 0; i < rbp; ++i)
            put((T)(i < rb && r0 + i < nb && A ? scale * A[(size_t)(r0 + i) * nb + j] : 0.0));
    }
};

// pads the group's table to 16 bytes, `tail` (a whole number of words) at its end
void finish_group(LaneTables &t, Writer &w, const std::vector<int32_t> &tail = {}) {
    while ((w.bytes.size() + 4 * tail.size()) % 16) w.put((unsigned char)0);
    for (int32_t v : tail) w.put(v);
    t.column_words = (int)tail.size();
    if (t.group_bytes && t.group_bytes != w.bytes.size()) w.bytes.resize(t.group_bytes, 0);
    t.group_bytes = w.bytes.size();
    t.data.insert(t.data.end(), w.bytes.begin(), w.bytes.end());
}

// every element's geometry in its slot: [tile][element's values, faces' values][32] (a
// padding slot has that of its group's first element: the upwind wave divides by the faces'
// normals)
void lane_geometry(const HostOperators &op, const LaneMesh &m, std::vector<double> &geo) {
    const size_t eg = op.elem_geo.size() / op.nE, fg = op.face_geo.size() / op.nE, q = eg + fg;
    geo.resize((size_t)m.n_slots * q);
    auto put = [&](int64_t slot, int64_t e) {
        double *g = &geo[(size_t)(slot >> 5) * q * 32 + (slot & 31)];
        for (size_t i = 0; i < eg; ++i) g[32 * i] = op.elem_geo[e * eg + i];
        for (size_t i = 0; i < fg; ++i) g[32 * (eg + i)] = op.face_geo[e * fg + i];
    };
    for (const LaneChunk &c : m.chunks)  // the last tile of a chunk may have padding
        for (int i = 0; i < 32; ++i) put(32 * (int64_t)(c.tile0 + c.tiles - 1) + i, m.representative[c.group]);
    for (int64_t e = 0; e < op.nE; ++e) put(m.slot[e], e);
}

}  // namespace

bool lane_wave_tables(const HostOperators &op, const LaneMesh &m, bool folded, int elem_bytes, LaneTables &t) {
    const int nb = op.nB, d = op.dim, nf = op.nfl, nfc = lane_trace(d, nf, op.order);
    const size_t nn = (size_t)nb * nb;
    const int most = lane_wave_rows(folded);
    const int rw = lane_warps(nb, most), rb = lane_rows(nb, most);
    const double invc = 1.0 / op.c_inv;
    const double c = op.physics == HGG_PHYSICS_WAVE_UPWIND ? 1.0 / std::sqrt(op.c_inv) : 0.0;
    t = LaneTables{};
    t.folded = folded;
    t.elem_bytes = elem_bytes;
    if (!folded) lane_geometry(op, m, t.geometry);
    for (int64_t e : m.representative) {
        const double *G = &op.elem_geo[e * d * d];  // G[dir][c]
        Writer w;
        // trace functions of both sides of every face: [face][own, neighbour][nfc], -1 past the last
        std::vector<int32_t> cs, cn, columns, neighbour_columns;
        for (int f = 0; f < nf && folded; ++f) {
            if (!trace_columns(op, op.self_pair[e * nf + f], nfc, cs) ||
                !trace_columns(op, op.nbr_pair[e * nf + f], nfc, cn))
                return false;
            for (auto *v : {&cs, &cn}) {
                const size_t have = v->size();
                for (int i = 0; i < nfc; ++i) columns.push_back(i < (int)have ? (*v)[i] : -1);
            }
            for (int i = 0; i < nfc; ++i) neighbour_columns.push_back(32 * std::max(columns[(2 * f + 1) * nfc + i], 0));
        }
        if (folded) {
            // physical derivatives D_dir = sum_c G[dir][c] vol_c
            std::vector<double> D(d * nn, 0.0);
            for (int a = 0; a < d; ++a)
                for (int k = 0; k < d; ++k)
                    for (size_t i = 0; i < nn; ++i) D[a * nn + i] += G[a * d + k] * op.vol[k * nn + i];
            const int rbp = lane_pad(rb, 8);
            for (int r = 0; r < rw; ++r) {
                for (int j = 0; j < nb; ++j)
                    for (int a = 0; a < d; ++a) w.column<double>(&D[a * nn], nb, j, r * rb, rb, rbp, 1.0);
                for (int f = 0; f < nf; ++f) {
                    const double *S = &op.pairs[op.self_pair[e * nf + f] * nn];
                    const double *N = &op.pairs[op.nbr_pair[e * nf + f] * nn];
                    for (int i = 0; i < nfc; ++i) {
                        const int js = columns[(f * 2) * nfc + i], jn = columns[(f * 2 + 1) * nfc + i];
                        w.column<double>(js >= 0 ? S : nullptr, nb, js, r * rb, rb, rbp, 1.0);
                        w.column<double>(jn >= 0 ? N : nullptr, nb, jn, r * rb, rb, rbp, 1.0);
                    }
                }
            }
            for (int f = 0; f < nf; ++f) {
                const double *nu = &op.face_geo[(e * nf + f) * d];
                double q = 0.0;
                for (int a = 0; a < d; ++a) q += nu[a] * nu[a];
                const double len = std::sqrt(q);
                for (int a = 0; a < d; ++a) w.put(nu[a]);
                w.put(c * len);
                for (int a = 0; a < d; ++a) w.put(invc * nu[a]);
                for (int a = 0; a < d; ++a) w.put(c == 0.0 ? 0.0 : c * (nu[a] / len));
            }
            w.put(invc);
            for (int f = 0; f < nf; ++f)
                for (int i = 0; i < nfc; ++i) w.put((int32_t)(32 * std::max(columns[2 * f * nfc + i], 0)));
        } else {
            const int rbp = lane_pad(rb, elem_bytes);
            for (int r = 0; r < rw; ++r) {
                for (int j = 0; j < nb; ++j)
                    for (int a = 0; a < d; ++a) w.plain_column(elem_bytes, &op.vol[a * nn], nb, j, r * rb, rb, rbp);
                for (int f = 0; f < nf; ++f)
                    for (int j = 0; j < nb; ++j) {
                        w.plain_column(elem_bytes, &op.pairs[op.self_pair[e * nf + f] * nn], nb, j, r * rb, rb, rbp);
                        w.plain_column(elem_bytes, &op.pairs[op.nbr_pair[e * nf + f] * nn], nb, j, r * rb, rb, rbp);
                    }
            }
            w.number(elem_bytes, c);
            w.number(elem_bytes, invc);
        }
        finish_group(t, w, neighbour_columns);
    }
    return true;
}

bool lane_advection_tables(const HostOperators &op, const LaneMesh &m, bool folded, int elem_bytes, LaneTables &t) {
    const int nb = op.nB, d = op.dim, nf = op.nfl, nfc = lane_trace(d, nf, op.order);
    const size_t nn = (size_t)nb * nb;
    const int rw = lane_warps(nb, kLaneAdvRows), rb = lane_rows(nb, kLaneAdvRows);
    t = LaneTables{};
    t.folded = folded;
    t.elem_bytes = elem_bytes;
    if (!folded) {  // a face along the flow has no flux (the plain kernel has no average)
        for (size_t i = 0; i < op.mode.size(); ++i)
            if (op.mode[i] == MODE_AVG && op.face_geo[i] != 0.0) return false;
        lane_geometry(op, m, t.geometry);
    }
    for (int64_t e : m.representative) {
        const double *ahat = &op.elem_geo[e * d], *sigma = &op.face_geo[e * nf];
        const int8_t *mode = &op.mode[e * nf];
        Writer w;
        if (folded) {
            // own matrix: volume and the faces the element's own trace leaves through
            std::vector<double> A(nn, 0.0);
            std::vector<int32_t> faces, columns, cols;
            std::vector<double> weight;
            for (int k = 0; k < d; ++k)
                for (size_t i = 0; i < nn; ++i) A[i] += ahat[k] * op.vol[k * nn + i];
            for (int f = 0; f < nf; ++f) {
                if (mode[f] == MODE_NONE || sigma[f] == 0.0) continue;
                const double s = mode[f] == MODE_AVG ? 0.5 * sigma[f] : sigma[f];
                if (mode[f] != MODE_NBR) {
                    const double *S = &op.pairs[op.self_pair[e * nf + f] * nn];
                    for (size_t i = 0; i < nn; ++i) A[i] -= s * S[i];
                }
                if (mode[f] != MODE_SELF) {
                    if (!trace_columns(op, op.nbr_pair[e * nf + f], nfc, cols)) return false;
                    faces.push_back(f);
                    weight.push_back(-s);
                    const size_t have = cols.size();
                    for (int i = 0; i < nfc; ++i) columns.push_back(i < (int)have ? cols[i] : -1);
                }
            }
            const int rbp = lane_pad(rb, 8);
            for (int r = 0; r < rw; ++r) {
                for (int j = 0; j < nb; ++j) w.column<double>(A.data(), nb, j, r * rb, rb, rbp, 1.0);
                for (int k = 0; k < nf; ++k)
                    for (int i = 0; i < nfc; ++i) {
                        const int j = k < (int)faces.size() ? columns[k * nfc + i] : -1;
                        const double *N = j >= 0 ? &op.pairs[op.nbr_pair[e * nf + faces[k]] * nn] : nullptr;
                        w.column<double>(N, nb, j, r * rb, rb, rbp, j >= 0 ? weight[k] : 0.0);
                    }
            }
            w.put((int32_t)faces.size());
            for (int k = 0; k < nf; ++k) w.put((int32_t)(k < (int)faces.size() ? faces[k] : 0));
            for (int k = 0; k < nf * nfc; ++k)
                w.put((int32_t)(k < (int)columns.size() ? 32 * std::max(columns[k], 0) : 0));
        } else {
            const int rbp = lane_pad(rb, elem_bytes);
            for (int r = 0; r < rw; ++r) {
                for (int j = 0; j < nb; ++j)
                    for (int a = 0; a < d; ++a) w.plain_column(elem_bytes, &op.vol[a * nn], nb, j, r * rb, rb, rbp);
                for (int f = 0; f < nf; ++f) {
                    const int32_t pair = mode[f] == MODE_SELF ? op.self_pair[e * nf + f] : op.nbr_pair[e * nf + f];
                    for (int j = 0; j < nb; ++j) w.plain_column(elem_bytes, &op.pairs[pair * nn], nb, j, r * rb, rb, rbp);
                }
            }
            for (int f = 0; f < nf; ++f) w.put((int32_t)(mode[f] == MODE_AVG ? MODE_NONE : mode[f]));
        }
        finish_group(t, w);
    }
    return true;
}

}  // namespace hgg
