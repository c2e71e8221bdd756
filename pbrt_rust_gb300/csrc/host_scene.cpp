// host_scene.cpp - primitive refinement, reference BVH build and device
// layout.  Compiled with -ffp-contract=off: every f32 expression follows
// the reference's operation order so the tree, the primitive edges and
// the camera matrices are the reference's bit for bit.
#include "host_scene.h"

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cstdio>
#include <cstring>

namespace pbrt {

// ------------------------------------------------------------------ boxes --
Box box_empty() { return Box{v3(FLT_MAX, FLT_MAX, FLT_MAX), v3(-FLT_MAX, -FLT_MAX, -FLT_MAX)}; }
// src/bbox.rs:170-183
Box box_union(const Box& a, const Box& b) {
    return Box{v3(std::fmin(a.lo.x, b.lo.x), std::fmin(a.lo.y, b.lo.y), std::fmin(a.lo.z, b.lo.z)),
               v3(std::fmax(a.hi.x, b.hi.x), std::fmax(a.hi.y, b.hi.y), std::fmax(a.hi.z, b.hi.z))};
}
// src/bbox.rs:155-168
Box box_union(const Box& a, V3 p) {
    return Box{v3(std::fmin(a.lo.x, p.x), std::fmin(a.lo.y, p.y), std::fmin(a.lo.z, p.z)),
               v3(std::fmax(a.hi.x, p.x), std::fmax(a.hi.y, p.y), std::fmax(a.hi.z, p.z))};
}
// src/bbox.rs:73-78
float box_area(const Box& b) {
    float dx = std::fmax(b.hi.x - b.lo.x, 0.0f);
    float dy = std::fmax(b.hi.y - b.lo.y, 0.0f);
    float dz = std::fmax(b.hi.z - b.lo.z, 0.0f);
    return 2.0f * (dx * dy + dx * dz + dy * dz);
}
// src/bbox.rs:87-96
int box_max_extent(const Box& b) {
    V3 d = b.hi - b.lo;
    if (d.x > d.y && d.x > d.z) return 0;
    if (d.y > d.z) return 1;
    return 2;
}

// --------------------------------------------------------------- matrices --
M4 m4_identity() {
    M4 r;
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j) r.m[i][j] = i == j ? 1.0f : 0.0f;
    return r;
}
// src/transform/matrix4x4.rs:167-182
M4 m4_mul(const M4& a, const M4& b) {
    M4 r;
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j)
            r.m[i][j] = a.m[i][0] * b.m[0][j] + a.m[i][1] * b.m[1][j] + a.m[i][2] * b.m[2][j] + a.m[i][3] * b.m[3][j];
    return r;
}
// src/transform/matrix4x4.rs:66-160: scaled partial pivoting where a row
// swap exchanges only columns k..3; the inverse's column c solves A x = e_c.
bool m4_inverse(const M4& a, M4* out) {
    float scale[4];
    for (int i = 0; i < 4; ++i) {
        float s = 0.0f;
        for (int j = 0; j < 4; ++j) s = std::fmax(std::fabs(a.m[i][j]), s);
        scale[i] = s;
    }
    M4 lu = a;
    int piv[4] = {0, 1, 2, 3};
    for (int k = 0; k < 3; ++k) {
        float best = 0.0f;
        int p = k;
        for (int i = k; i < 4; ++i) {
            float c = std::fabs(lu.m[i][k] / scale[i]);
            if (c > best) {
                best = c;
                p = i;
            }
        }
        piv[k] = p;
        if (best == 0.0f) return false;
        if (p != k)
            for (int j = k; j < 4; ++j) std::swap(lu.m[k][j], lu.m[p][j]);
        for (int i = k + 1; i < 4; ++i) {
            float f = lu.m[i][k] / lu.m[k][k];
            lu.m[i][k] = f;
            for (int j = k + 1; j < 4; ++j) lu.m[i][j] = lu.m[i][j] - f * lu.m[k][j];
        }
    }
    if (std::fabs(lu.m[3][3]) < 1.0e-6f) return false;
    M4 inv;
    for (int c = 0; c < 4; ++c) {
        float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        x[c] = 1.0f;
        for (int k = 0; k < 3; ++k) {
            if (piv[k] != k) std::swap(x[piv[k]], x[k]);
            for (int i = k + 1; i < 4; ++i) x[i] = x[i] - lu.m[i][k] * x[k];
        }
        x[3] = x[3] / lu.m[3][3];
        for (int i = 2; i >= 0; --i) {
            float acc = 0.0f;
            for (int j = i + 1; j < 4; ++j) acc = acc + lu.m[i][j] * x[j];
            x[i] = (x[i] - acc) / lu.m[i][i];
        }
        for (int r = 0; r < 4; ++r) inv.m[r][c] = x[r];
    }
    *out = inv;
    return true;
}
V3 m4_point(const M4& m, V3 p) {
    float xt = m.m[0][0] * p.x + m.m[0][1] * p.y + m.m[0][2] * p.z + m.m[0][3];
    float yt = m.m[1][0] * p.x + m.m[1][1] * p.y + m.m[1][2] * p.z + m.m[1][3];
    float zt = m.m[2][0] * p.x + m.m[2][1] * p.y + m.m[2][2] * p.z + m.m[2][3];
    float w = m.m[3][0] * p.x + m.m[3][1] * p.y + m.m[3][2] * p.z + m.m[3][3];
    if (w != 1.0f) return v3(xt / w, yt / w, zt / w);
    return v3(xt, yt, zt);
}
V3 m4_vector(const M4& m, V3 v) {
    return v3(m.m[0][0] * v.x + m.m[0][1] * v.y + m.m[0][2] * v.z, m.m[1][0] * v.x + m.m[1][1] * v.y + m.m[1][2] * v.z,
              m.m[2][0] * v.x + m.m[2][1] * v.y + m.m[2][2] * v.z);
}
bool m4_swaps_handedness(const M4& m) {
    float det = m.m[0][0] * (m.m[1][1] * m.m[2][2] - m.m[1][2] * m.m[2][1]) -
                m.m[0][1] * (m.m[1][0] * m.m[2][2] - m.m[1][2] * m.m[2][0]) +
                m.m[0][2] * (m.m[1][0] * m.m[2][1] - m.m[1][1] * m.m[2][0]);
    return 0.0f > det;
}
Xf xf_from_desc(const PbrtTransform& t) {
    Xf x;
    std::memcpy(x.m.m, t.m, sizeof(x.m.m));
    std::memcpy(x.mi.m, t.m_inv, sizeof(x.mi.m));
    return x;
}
Xf xf_mul(const Xf& a, const Xf& b) { return Xf{m4_mul(a.m, b.m), m4_mul(b.mi, a.mi)}; }
Xf xf_inverse(const Xf& a) { return Xf{a.mi, a.m}; }
static Xf xf_scale(float x, float y, float z) {
    Xf t{m4_identity(), m4_identity()};
    t.m.m[0][0] = x;
    t.m.m[1][1] = y;
    t.m.m[2][2] = z;
    t.mi.m[0][0] = 1.0f / x;
    t.mi.m[1][1] = 1.0f / y;
    t.mi.m[2][2] = 1.0f / z;
    return t;
}
static Xf xf_translate(float x, float y, float z) {
    Xf t{m4_identity(), m4_identity()};
    t.m.m[0][3] = x;
    t.m.m[1][3] = y;
    t.m.m[2][3] = z;
    t.mi.m[0][3] = -x;
    t.mi.m[1][3] = -y;
    t.mi.m[2][3] = -z;
    return t;
}

// ------------------------------------------------------------------ shapes --
// transform.rs:248-263 (eight-corner box transform)
static Box xf_box(const M4& m, const Box& b) {
    V3 tx = m4_vector(m, v3(b.hi.x - b.lo.x, 0.0f, 0.0f));
    V3 ty = m4_vector(m, v3(0.0f, b.hi.y - b.lo.y, 0.0f));
    V3 tz = m4_vector(m, v3(0.0f, 0.0f, b.hi.z - b.lo.z));
    V3 tp = m4_point(m, b.lo);
    Box r{tp, tp};
    r = box_union(r, tp + tx);
    r = box_union(r, tp + ty);
    r = box_union(r, tp + tz);
    r = box_union(r, (tp + tx) + ty);
    r = box_union(r, (tp + tx) + tz);
    r = box_union(r, (tp + ty) + tz);
    r = box_union(r, ((tp + tx) + ty) + tz);
    return r;
}

static float clampf(float x, float lo, float hi) {
    if (x < lo) x = lo;
    if (x > hi) x = hi;
    return x;
}

int parse_split_method(const char* s) {
    if (!s || !std::strcmp(s, "sah")) return PBRT_SPLIT_SAH;
    if (!std::strcmp(s, "middle")) return PBRT_SPLIT_MIDDLE;
    if (!std::strcmp(s, "equal")) return PBRT_SPLIT_EQUAL;
    std::fprintf(stderr, "Warning: BVH split method %s unknown. Using \"SAH\"\n", s);  // bvh.rs:345-348
    return PBRT_SPLIT_SAH;
}

// -------------------------------------------------------------- BVH build --
namespace {

// src/utils/mod.rs:112-169 over a slice of primitive indices keyed by a
// centroid coordinate (median-of-three pivot, three-way scan, recursion on
// the side holding the middle).
void partition_by_key(uint32_t* v, size_t n, const float* key) {
    while (true) {
        if (n < 3) {
            if (n == 2 && key[v[1]] < key[v[0]]) std::swap(v[0], v[1]);
            return;
        }
        float a = key[v[0]], b = key[v[n / 2]], c = key[v[n - 1]];
        float pivot = (a < b && b < c) ? b : ((b < a && a < c) ? a : c);
        size_t ls = 0, np = 0;
        for (size_t i = 0; i < n; ++i) {
            float k = key[v[i]];
            if (k < pivot) {
                std::swap(v[ls + np], v[i]);
                std::swap(v[ls + np], v[ls]);
                ++ls;
            } else if (k == pivot) {
                std::swap(v[ls + np], v[i]);
                ++np;
            }
        }
        size_t pi = std::max<size_t>(ls, 1);
        if (pi + np <= n / 2) {
            v += pi;
            n -= pi;
        } else if (pi >= n / 2) {
            n = pi;
        } else {
            return;
        }
    }
}

inline size_t f32_to_usize(float f) {  // Rust `as usize`: saturating, NaN -> 0
    if (!(f > 0.0f)) return 0;
    if (f >= 18446744073709551615.0f) return SIZE_MAX;
    return (size_t)f;
}

struct Task {
    uint32_t lo, hi;
    int32_t parent;  // node whose second-child offset is this node, or -1
    uint32_t depth;
};

}  // namespace

Box prim_bounds(const HostBVH& H, size_t i, V3* centroid) {
    const HostPrim& p = H.prims[i];
    Box b;
    if (p.kind == PBRT_SHAPE_TRIANGLE_MESH) {
        b = box_union(box_union(box_union(box_empty(), p.p1), p.p2), p.p3);  // mesh.rs:196-205
    } else {
        const SphereRec& s = H.spheres[p.sphere];
        M4 o2w;
        std::memcpy(o2w.m, s.o2w, sizeof(o2w.m));
        if (s.kind == kQuadInstance) {
            // transformed.rs:62-65: motion_bounds of a static transform =
            // the definition's bound through primitive-to-world
            b = xf_box(o2w, H.insts[s.instance].nodes[0].box);  // definitions are not empty
        } else {
            b = xf_box(o2w, Box{v3(-s.radius, -s.radius, s.z_min), v3(s.radius, s.radius, s.z_max)});
        }
    }
    *centroid = (b.lo + b.hi) * 0.5f;  // bvh.rs:77
    return b;
}

static int build_tree(HostBVH& H, uint32_t mp, int split, std::string* err) {
    const size_t n = H.prims.size();
    H.nodes.clear();
    H.ordered.resize(n);
    if (n == 0) return PBRT_OK;
    RawVec<Box> bounds(n);
    RawVec<float> cx(n), cy(n), cz(n);
    host_parallel(n, [&](size_t, size_t lo, size_t hi) {
        for (size_t i = lo; i < hi; ++i) {
            V3 c;
            bounds[i] = prim_bounds(H, i, &c);
            cx[i] = c.x;
            cy[i] = c.y;
            cz[i] = c.z;
            H.ordered[i] = (uint32_t)i;
        }
    });
    const float* cent[3] = {cx.data(), cy.data(), cz.data()};
    uint32_t* idx = H.ordered.data();
    H.nodes.reserve(2 * n);
    std::vector<Task> stack;
    stack.push_back(Task{0, (uint32_t)n, -1, 1});
    std::vector<uint32_t> scratch;
    H.depth = 0;
    const size_t NB = 12;
    while (!stack.empty()) {
        Task t = stack.back();
        stack.pop_back();
        uint32_t k = (uint32_t)H.nodes.size();
        if (t.parent >= 0) H.nodes[t.parent].offset = k;
        H.depth = std::max(H.depth, t.depth);
        const size_t cnt = t.hi - t.lo;
        Box bbox = box_empty();
        for (uint32_t i = t.lo; i < t.hi; ++i) bbox = box_union(bbox, bounds[idx[i]]);
        FlatNode node{bbox, true, t.lo, (uint32_t)cnt};
        uint32_t mid = 0;
        bool split_it = false;
        int dim = 0;
        if (cnt > 1) {
            Box cb = box_empty();
            for (uint32_t i = t.lo; i < t.hi; ++i) cb = box_union(cb, v3(cx[idx[i]], cy[idx[i]], cz[idx[i]]));
            dim = box_max_extent(cb);
            float cmin = axis_of(cb.lo, dim), cmax = axis_of(cb.hi, dim);
            const float* key = cent[dim];
            if (cmin != cmax) {
                auto equal_counts = [&]() {  // bvh.rs:92-103
                    partition_by_key(idx + t.lo, cnt, key);
                    mid = t.lo + (uint32_t)(cnt / 2);
                    split_it = true;
                };
                auto stable_split = [&](auto pred) {
                    scratch.clear();
                    uint32_t w = t.lo;
                    for (uint32_t i = t.lo; i < t.hi; ++i) {
                        if (pred(idx[i]))
                            idx[w++] = idx[i];
                        else
                            scratch.push_back(idx[i]);
                    }
                    mid = w;
                    std::copy(scratch.begin(), scratch.end(), idx + w);
                    split_it = true;
                };
                if (split == PBRT_SPLIT_MIDDLE) {  // bvh.rs:86-90
                    float p_mid = 0.5f * (cmin + cmax);
                    stable_split([&](uint32_t p) { return key[p] < p_mid; });
                } else if (split == PBRT_SPLIT_EQUAL) {
                    equal_counts();
                } else if (cnt <= 4) {  // bvh.rs:111-113
                    equal_counts();
                } else {  // bvh.rs:115-185
                    float dist = cmax - cmin;
                    auto bucket = [&](uint32_t p) {
                        float pdist = key[p] - cmin;
                        size_t b = f32_to_usize((float)NB * (pdist / dist));
                        return b == NB ? NB - 1 : b;
                    };
                    size_t bc[12] = {0};
                    Box bb[12];
                    for (size_t i = 0; i < NB; ++i) bb[i] = box_empty();
                    for (uint32_t i = t.lo; i < t.hi; ++i) {
                        size_t b = bucket(idx[i]);
                        bc[b] += 1;
                        bb[b] = box_union(bb[b], bounds[idx[i]]);
                    }
                    float tsa = box_area(bbox);
                    size_t best = 0;
                    float best_cost = FLT_MAX;
                    for (size_t s = 0; s + 1 < NB; ++s) {
                        size_t c0 = 0, c1 = 0;
                        Box b0 = box_empty(), b1 = box_empty();
                        for (size_t j = 0; j <= s; ++j) {
                            c0 += bc[j];
                            b0 = box_union(b0, bb[j]);
                        }
                        for (size_t j = s + 1; j < NB; ++j) {
                            c1 += bc[j];
                            b1 = box_union(b1, bb[j]);
                        }
                        float cost = 0.125f * ((float)c0 * box_area(b0) + (float)c1 * box_area(b1)) / tsa;
                        if (cost < best_cost) {
                            best_cost = cost;
                            best = s;
                        }
                    }
                    if (mp < cnt || f32_to_usize(best_cost) < cnt)
                        stable_split([&](uint32_t p) { return bucket(p) <= best; });
                }
            }
        }
        if (split_it) {
            if (mid == t.lo || mid == t.hi) {
                *err = "BVH build: empty partition (the reference asserts at bvh.rs:237-238)";
                return PBRT_ERR_BUILD;
            }
            node.leaf = false;
            node.offset = 0;
            node.count = (uint32_t)dim;
            H.nodes.push_back(node);
            stack.push_back(Task{mid, t.hi, (int32_t)k, t.depth + 1});
            stack.push_back(Task{t.lo, mid, -1, t.depth + 1});
        } else {
            H.nodes.push_back(node);
        }
    }
    // Inner bounds are the union of the two children (bvh.rs:247).
    for (size_t k = H.nodes.size(); k-- > 0;) {
        FlatNode& nd = H.nodes[k];
        if (!nd.leaf) nd.box = box_union(H.nodes[k + 1].box, H.nodes[nd.offset].box);
    }
    return PBRT_OK;
}

static void set_flags(PrimRec& r, uint32_t f) {
    uint32_t v;
    std::memcpy(&v, &r.r2[3], 4);
    v |= f;
    std::memcpy(&r.r2[3], &v, 4);
}

// The binary layout, and with it the primitive flags of the 4-wide walk, the
// leaf boxes they refer to, and whether the tree can have the 4-wide layout
// at all.
static void fill_device_layout(HostBVH& H) {
    const size_t m = H.nodes.size();
    // pairs are numbered in the pre-order of their parents
    RawVec<uint32_t> pair_of(m);
    std::vector<size_t> inner(host_parts(m) + 1, 0);  // inner nodes before each part
    host_parallel(m, [&](size_t part, size_t lo, size_t hi) {
        for (size_t k = lo; k < hi; ++k) inner[part + 1] += !H.nodes[k].leaf;
    });
    for (size_t p = 1; p < inner.size(); ++p) inner[p] += inner[p - 1];
    host_parallel(m, [&](size_t part, size_t lo, size_t hi) {
        uint32_t np = (uint32_t)inner[part];
        for (size_t k = lo; k < hi; ++k) pair_of[k] = H.nodes[k].leaf ? 0xffffffffu : np++;
    });
    auto rec = [&](size_t k) {
        const FlatNode& nd = H.nodes[k];
        ChildRec c;
        c.lo_x = nd.box.lo.x;
        c.lo_y = nd.box.lo.y;
        c.lo_z = nd.box.lo.z;
        c.hi_x = nd.box.hi.x;
        c.hi_y = nd.box.hi.y;
        c.hi_z = nd.box.hi.z;
        if (nd.leaf) {
            c.a = nd.offset;
            c.b = kLeafBit | nd.count;
        } else {
            c.a = pair_of[k];
            c.b = nd.count;
        }
        return c;
    };
    H.pairs.resize(inner.back());
    if (m) H.root = rec(0);
    H.recs.resize(H.ordered.size() + 1);  // and the null record
    std::memset(&H.recs.back(), 0, sizeof(PrimRec));
    set_flags(H.recs.back(), kPrimLastBit);
    auto usable = [](float v) { return std::fabs(v) <= kWideReach; };  // false for NaN
    auto usable3 = [&](V3 v) { return usable(v.x) && usable(v.y) && usable(v.z); };
    struct Part {
        bool wide = true;
        bool boxed = false;  // some leaf's box goes to the table
        double area = 0.0, length = 0.0;
    };
    std::vector<Part> parts(host_parts(m));
    host_parallel(m, [&](size_t part, size_t lo, size_t hi) {
        Part& A = parts[part];
        for (size_t k = lo; k < hi; ++k) {
            const FlatNode& nd = H.nodes[k];
            const V3 e = nd.box.hi - nd.box.lo;
            A.area += (double)e.x * e.y + (double)e.y * e.z + (double)e.z * e.x;
            A.length += (double)e.x + e.y + e.z;
            if (!nd.leaf) {
                NodePair& p = H.pairs[pair_of[k]];
                p.c[0] = rec(k + 1);
                p.c[1] = rec(nd.offset);
                continue;
            }
            A.wide = A.wide && usable3(nd.box.lo) && usable3(nd.box.hi);
            bool tri = false;
            for (uint32_t i = 0; i < nd.count; ++i) {
                const uint32_t ref = H.ordered[nd.offset + i];
                const HostPrim& p = H.prims[ref];
                PrimRec& r = H.recs[nd.offset + i];
                std::memset(&r, 0, sizeof(r));
                uint32_t id = H.flat_id.empty() ? ref : H.flat_id[ref];
                tri = p.kind == PBRT_SHAPE_TRIANGLE_MESH;
                if (tri) {
                    r.r0[0] = p.p1.x;
                    r.r0[1] = p.p1.y;
                    r.r0[2] = p.p1.z;
                    r.r1[0] = p.p2.x;
                    r.r1[1] = p.p2.y;
                    r.r1[2] = p.p2.z;
                    r.r2[0] = p.p3.x;
                    r.r2[1] = p.p3.y;
                    r.r2[2] = p.p3.z;
                    A.wide = A.wide && usable3(p.p1) && usable3(p.p2) && usable3(p.p3);
                } else {
                    const uint32_t si = (uint32_t)p.sphere;
                    id |= kSphereBit;
                    std::memcpy(&r.r1[3], &si, 4);
                }
                std::memcpy(&r.r0[3], &id, 4);
            }
            if (nd.count == 0) continue;
            set_flags(H.recs[nd.offset + nd.count - 1], kPrimLastBit);
            if (nd.count == 1 && tri)
                set_flags(H.recs[nd.offset], kPrimOwnBox);
            else
                A.boxed = true;
        }
    });
    H.wide = H.ordered.size() < 0x7ffffff0u && H.pairs.size() < (1u << kQuadAxisShift);
    H.leaf_boxes.clear();
    bool boxed = false;
    double area = 0.0, length = 0.0;
    for (const Part& A : parts) {
        H.wide = H.wide && A.wide;
        boxed = boxed || A.boxed;
        area += A.area;
        length += A.length;
    }
    tree_margins(H, area, length);
    for (size_t k = 0; boxed && k < m; ++k) {
        const FlatNode& nd = H.nodes[k];
        if (!nd.leaf || nd.count == 0) continue;
        const HostPrim& first = H.prims[H.ordered[nd.offset]];
        if (nd.count == 1 && first.kind == PBRT_SHAPE_TRIANGLE_MESH) continue;
        const bool entry = nd.count > 1 || H.spheres[first.sphere].kind == kQuadInstance;
        if (H.leaf_boxes.size() >= (1u << (32u - kPrimBoxShift))) {
            H.wide = false;
            break;
        }
        set_flags(H.recs[nd.offset], entry ? kPrimBoxEntry : kPrimHitBox);
        for (uint32_t i = 0; i < nd.count; ++i)
            set_flags(H.recs[nd.offset + i], (uint32_t)H.leaf_boxes.size() << kPrimBoxShift);
        const Box& b = nd.box;
        H.leaf_boxes.push_back(LeafBox{{b.lo.x, b.lo.y, b.lo.z, 0.0f}, {b.hi.x, b.hi.y, b.hi.z, 0.0f}});
    }
}

// A margin of m moves each of a box's planes outwards by m, so that it is met
// as often as a box of half area A + 4 m L + 12 m^2, A its own and L the sum
// of its edges.  A ray whose margins make that kFarVisits times the visits of
// the tree's nodes is better walked over the binary layout, whose boxes are
// exact.  With m taken as two thirds of the three axes' sum, that is where the
// measured times cross (100000 rays from 1000 / 3000 / 10000 extents away, us,
// 4-wide without the rule and binary: terrain of 980000 triangles 92 / 145 /
// 446 and 130 / 128 / 146, of 180000 107 / 127 / 137 and 168 / 168 / 117,
// 200000 random triangles 175 / 178 / 203 and 347 / 343 / 358).
constexpr double kFarVisits = 3.0;

void tree_margins(HostBVH& H, double area, double length) {
    H.quad_root = 0;
    if (H.nodes.empty()) return;
    auto axis = [](float lo, float hi, float* middle, float* half, float* spread) {
        *middle = (float)(0.5 * ((double)lo + (double)hi));
        const double last = std::max(std::fabs(lo), std::fabs(hi)) * 0x1p-22;
        *half = (float)(1.000001 * (std::max((double)hi - *middle, *middle - (double)lo) + last));
        *spread = std::max(kTreeMargin * *half, 0x1p-71f);  // the margins stay normal numbers
    };
    const Box& rb = H.nodes[0].box;
    axis(rb.lo.x, rb.hi.x, &H.middle.x, &H.half.x, &H.spread.x);
    axis(rb.lo.y, rb.hi.y, &H.middle.y, &H.half.y, &H.spread.y);
    axis(rb.lo.z, rb.hi.z, &H.middle.z, &H.half.z, &H.spread.z);
    const double a = 12.0 * (double)H.nodes.size(), b = 4.0 * length, c = (kFarVisits - 1.0) * area;
    const double m = c > 0.0 ? 2.0 * c / (b + std::sqrt(b * b + 4.0 * a * c)) : 0.0;
    // never so near that rays within the tree's own extent are meant, nor so
    // far (|c - o| of 2^41) that a plane's distance could overflow
    const float spread = H.spread.x + H.spread.y + H.spread.z;
    H.far = std::min(std::max((float)(1.5 * m), 2.0f * spread), spread + 0x1p41f * kFarMargin);
    if (H.nodes[0].leaf) H.quad_root = kNode4Leaf | H.nodes[0].offset;
}

// Where the 4-wide nodes start (two binary levels each, see layout.h:
// QuadNode).
static void fill_quad_layout(HostBVH& H) {
    const size_t m = H.nodes.size();
    H.quad_of.resize(H.pairs.size());
    H.n_quads = 0;
    H.stack4_bound = 0;
    if (m == 0 || H.nodes[0].leaf) return;
    // pairs are numbered in pre-order, so a node's 4-wide start is decided
    // before its grandchildren's
    RawVec<uint32_t> deferred(H.pairs.size());       // entries the walk may hold above a start
    std::vector<uint8_t> starts(H.pairs.size(), 0);  // split axis + 1 of a start
    starts[0] = (uint8_t)(H.nodes[0].count + 1);
    deferred[0] = 0;
    for (size_t p = 0; p < H.pairs.size(); ++p) {
        if (!starts[p]) {
            H.quad_of[p] = kNoQuad;
            continue;
        }
        H.quad_of[p] = H.n_quads++ | ((uint32_t)(starts[p] - 1) << kQuadAxisShift);
        uint32_t slots = 0;
        for (const ChildRec& c : H.pairs[p].c) slots += (c.b & kLeafBit) ? 1u : 2u;
        const uint32_t here = deferred[p] + slots - 1;
        H.stack4_bound = std::max(H.stack4_bound, here);
        for (const ChildRec& c : H.pairs[p].c) {
            if (c.b & kLeafBit) continue;
            for (const ChildRec& g : H.pairs[c.a].c) {
                if (g.b & kLeafBit) continue;
                starts[g.a] = (uint8_t)(g.b + 1);
                deferred[g.a] = here;
            }
        }
    }
}

void fill_host_layout(HostBVH& H) {
    const bool wide = H.wide;  // as created: the definitions' limits are in them
    const uint32_t bound = H.stack4_bound;
    fill_device_layout(H);
    fill_quad_layout(H);
    H.wide = wide;
    H.stack4_bound = bound;
}

int build_host_bvh(const PbrtShapeDesc* shapes, uint32_t n_shapes, uint32_t max_prims, const char* split_method,
                   HostBVH* out, std::string* err, bool on_device, const PbrtInstanceDesc* defs, uint32_t n_defs) {
    HostBVH& H = *out;
    H = HostBVH();
    // the definitions' BVHs, built like the scene's (the instance aggregate
    // of ObjectInstance uses the scene's accelerator, main.rs:735-763)
    H.insts.resize(n_defs);
    for (uint32_t k = 0; k < n_defs; ++k) {
        for (uint32_t i = 0; i < defs[k].n_shapes; ++i)
            if (defs[k].shapes[i].kind == PBRT_SHAPE_INSTANCE || defs[k].shapes[i].area_light >= 0) {
                *err = "instance definitions hold neither instances nor area lights";
                return PBRT_ERR_UNSUPPORTED;
            }
        int st = build_host_bvh(defs[k].shapes, defs[k].n_shapes, max_prims, split_method, &H.insts[k], err,
                                on_device);
        if (st) return st;
        if (H.insts[k].prims.empty()) {
            *err = "instance definition without shapes";
            return PBRT_ERR_INVALID_ARGUMENT;
        }
        if (H.insts[k].stack4_bound > 96) {  // kInstStack of the nested walk
            *err = "instance definition BVH too deep for the nested traversal stack (96 entries)";
            return PBRT_ERR_UNSUPPORTED;
        }
    }
    // Full refinement: primitive/mod.rs:47-63, mesh.rs:298-338.
    for (uint32_t si = 0; si < n_shapes; ++si) {
        const PbrtShapeDesc& d = shapes[si];
        Xf o2w = xf_from_desc(d.object_to_world);
        bool flip = (d.reverse_orientation != 0) != m4_swaps_handedness(o2w.m);
        if (d.kind == PBRT_SHAPE_TRIANGLE_MESH) {
            if (d.n_indices % 3 != 0 || (d.n_indices && (!d.indices || !d.points))) {
                *err = "triangle mesh: index count must be a multiple of 3 with points and indices given";
                return PBRT_ERR_INVALID_ARGUMENT;
            }
            RawVec<V3> wp(d.n_points);
            host_parallel(d.n_points, [&](size_t, size_t lo, size_t hi) {
                for (size_t i = lo; i < hi; ++i)
                    wp[i] = m4_point(o2w.m, v3(d.points[3 * i], d.points[3 * i + 1], d.points[3 * i + 2]));
            });
            const size_t first = H.prims.size(), nt = d.n_indices / 3;
            H.prims.resize(first + nt);
            std::atomic<bool> bad{false};
            host_parallel(nt, [&](size_t, size_t lo, size_t hi) {
                for (size_t k = lo; k < hi; ++k) {
                    uint32_t i0 = d.indices[3 * k], i1 = d.indices[3 * k + 1], i2 = d.indices[3 * k + 2];
                    if (i0 >= d.n_points || i1 >= d.n_points || i2 >= d.n_points) {
                        bad = true;
                        return;
                    }
                    HostPrim p{};
                    p.kind = PBRT_SHAPE_TRIANGLE_MESH;
                    p.shape = (int)si;
                    p.material = d.material;
                    p.area_light = d.area_light;
                    p.p1 = wp[i2];  // refine pops indices: v = (i2, i1, i0)
                    p.p2 = wp[i1];
                    p.p3 = wp[i0];
                    p.flip = flip;
                    p.sphere = -1;
                    H.prims[first + k] = p;
                }
            });
            if (bad) {
                *err = "triangle mesh: vertex index out of range";
                return PBRT_ERR_INVALID_ARGUMENT;
            }
        } else if (d.kind == PBRT_SHAPE_SPHERE) {
            if (!(d.radius > 0.0f)) {
                *err = "sphere: radius must be positive";
                return PBRT_ERR_INVALID_ARGUMENT;
            }
            // sphere.rs:28-44
            SphereRec s{};
            std::memcpy(s.o2w, o2w.m.m, sizeof(s.o2w));
            std::memcpy(s.w2o, o2w.mi.m, sizeof(s.w2o));
            float rad = d.radius;
            s.radius = rad;
            s.z_min = clampf(std::fmin(d.z0, d.z1), -rad, rad);
            s.z_max = clampf(std::fmax(d.z0, d.z1), -rad, rad);
            s.theta_min = std::acos(s.z_min / rad);
            s.theta_max = std::acos(s.z_max / rad);
            s.phi_max = clampf(d.phi_max_deg, 0.0f, 360.0f) * 3.14159265358979323846f / 180.0f;
            // With z_min = -r, z_max = r and phi_max >= 2*pi (f32) the clip
            // test of sphere.rs:88-92 can never reject: atan2 + 2*pi stays
            // <= 2*pi in f32.
            s.full = (s.z_min <= -rad && s.z_max >= rad && s.phi_max >= 2.0f * 3.14159265358979323846f) ? 1u : 0u;
            s.flip = flip ? 1u : 0u;
            s.kind = kQuadSphere;
            HostPrim p{};
            p.kind = PBRT_SHAPE_SPHERE;
            p.shape = (int)si;
            p.material = d.material;
            p.area_light = d.area_light;
            p.flip = flip;
            p.sphere = (int)H.spheres.size();
            H.spheres.push_back(s);
            H.prims.push_back(p);
            H.has_spheres = true;
        } else if (d.kind == PBRT_SHAPE_INSTANCE) {
            if (d.instance < 0 || (uint32_t)d.instance >= n_defs) {
                *err = "instance: definition index out of range";
                return PBRT_ERR_INVALID_ARGUMENT;
            }
            SphereRec s{};
            std::memcpy(s.o2w, o2w.m.m, sizeof(s.o2w));   // primitive to world
            std::memcpy(s.w2o, o2w.mi.m, sizeof(s.w2o));  // world to primitive
            s.kind = kQuadInstance;
            s.instance = (uint32_t)d.instance;
            HostPrim p{};
            p.kind = PBRT_SHAPE_SPHERE;  // one analytic-style primitive
            p.shape = (int)si;
            p.material = d.material;
            p.area_light = -1;
            p.flip = false;
            p.sphere = (int)H.spheres.size();
            H.spheres.push_back(s);
            H.prims.push_back(p);
            H.has_spheres = true;
        } else if (d.kind == PBRT_SHAPE_DISK || d.kind == PBRT_SHAPE_CYLINDER) {
            SphereRec s{};
            std::memcpy(s.o2w, o2w.m.m, sizeof(s.o2w));
            std::memcpy(s.w2o, o2w.mi.m, sizeof(s.w2o));
            s.radius = d.radius;
            s.phi_max = clampf(d.phi_max_deg, 0.0f, 360.0f) * 3.14159265358979323846f / 180.0f;
            if (d.kind == PBRT_SHAPE_DISK) {  // disk.rs:24-34: radii unclamped
                s.kind = kQuadDisk;
                s.height = d.height;
                s.inner_radius = d.inner_radius;
                s.z_min = s.z_max = d.height;
            } else {  // cylinder.rs:26-36
                s.kind = kQuadCylinder;
                s.z_min = std::fmin(d.z0, d.z1);
                s.z_max = std::fmax(d.z0, d.z1);
            }
            // phi = atan2 (+ 2 pi when negative) stays <= 2 pi in f32, so a
            // full turn never rejects on phi
            s.full = s.phi_max >= 2.0f * 3.14159265358979323846f ? 1u : 0u;
            s.flip = flip ? 1u : 0u;
            HostPrim p{};
            p.kind = PBRT_SHAPE_SPHERE;  // refined like a sphere: one analytic primitive
            p.shape = (int)si;
            p.material = d.material;
            p.area_light = d.area_light;
            p.flip = flip;
            p.sphere = (int)H.spheres.size();
            H.spheres.push_back(s);
            H.prims.push_back(p);
            H.has_spheres = true;
        } else {
            *err = "unknown shape kind";
            return PBRT_ERR_INVALID_ARGUMENT;
        }
    }
    bool any_instance = false;
    for (const SphereRec& s : H.spheres) any_instance |= s.kind == kQuadInstance;
    if (any_instance) {
        H.flat_id.resize(H.prims.size());
        uint64_t next = 0;
        for (size_t i = 0; i < H.prims.size(); ++i) {
            H.flat_id[i] = (uint32_t)next;
            const HostPrim& p = H.prims[i];
            const bool inst = p.sphere >= 0 && H.spheres[p.sphere].kind == kQuadInstance;
            next += inst ? H.insts[H.spheres[p.sphere].instance].prims.size() : 1u;
            if (next > 0x7fffffffull) {
                *err = "more than 2^31 - 1 primitives with the instances counted out";
                return PBRT_ERR_UNSUPPORTED;
            }
        }
        H.n_flat = next;
    } else {
        H.n_flat = H.prims.size();
    }
    const int split = parse_split_method(split_method);
    // equal-counts splits of large ranges use the sequential partition_by
    // (utils/mod.rs:112-169), which stays on the host
    int st = (on_device && split != PBRT_SPLIT_EQUAL) ? device_build_tree(H, max_prims, split, err)
                                                      : build_tree(H, max_prims, split, err);
    if (st) return st;
    if (!H.layout) {
        fill_device_layout(H);
        fill_quad_layout(H);
    }
    for (const HostBVH& I : H.insts) H.wide = H.wide && I.wide;
    if (!H.insts.empty()) {
        // the 4-wide walk enters a definition with two more entries (the
        // rest of the leaf, the exit word) on top of the scene's stack
        uint32_t inner = 0;
        for (const HostBVH& I : H.insts) inner = std::max(inner, I.stack4_bound);
        H.stack4_bound += 2 + inner;
        if (H.ordered.size() >= 0x7ffffffeu) {  // leaf words stay clear of the exit word
            *err = "too many primitives for a scene with instances";
            return PBRT_ERR_UNSUPPORTED;
        }
    }
    return PBRT_OK;
}

// -------------------------------------------------------------- camera ----
// Camera::perspective (camera/mod.rs:105-135): persp = scale(1/tan(fov/2))
// * P with n = 1e-2, f = 1000; Projection::new (projective.rs:48-72):
// raster_to_camera = inverse(persp) * inverse(screen_to_raster).
void camera_matrices(const PbrtCameraDesc& cam, float r2c_out[16], float c2w_out[16]) {
    const float znear = 1e-2f, zfar = 1000.0f;
    M4 pm = m4_identity();
    pm.m[2][2] = zfar / (zfar - znear);
    pm.m[2][3] = -(zfar * znear) / (zfar - znear);
    pm.m[3][2] = 1.0f;
    pm.m[3][3] = 0.0f;
    M4 pmi;
    if (!m4_inverse(pm, &pmi)) pmi = m4_identity();
    Xf p{pm, pmi};
    float rad = cam.fov_deg * 3.14159265358979323846f / 180.0f;
    float inv_tan = 1.0f / std::tan(rad / 2.0f);
    Xf persp = xf_mul(xf_scale(inv_tan, inv_tan, 1.0f), p);
    const float* sw = cam.screen_window;
    Xf s2r = xf_mul(xf_mul(xf_scale((float)cam.x_res, (float)cam.y_res, 1.0f),
                           xf_scale(1.0f / (sw[1] - sw[0]), 1.0f / (sw[2] - sw[3]), 1.0f)),
                    xf_translate(-sw[0], -sw[3], 0.0f));
    Xf r2c = xf_mul(xf_inverse(persp), xf_inverse(s2r));
    std::memcpy(r2c_out, r2c.m.m, sizeof(float) * 16);
    std::memcpy(c2w_out, cam.camera_to_world.m, sizeof(float) * 16);
}

}  // namespace pbrt

namespace pbrt {

// ------------------------------------------------------------------ filter ---
namespace {

// utils/mod.rs:207-217
float sinc_1d(float x, float tau) {
    float v = std::fabs(x);
    if (v < 1e-5f) return 1.0f;
    if (v >= 1.0f) return 0.0f;
    v *= 3.14159265358979323846f;
    const float vt = v * tau;
    const float s = std::sin(vt) / vt;
    return s * std::sin(v) / v;
}

// filter.rs:87-124 (Filter::evaluate) for the kinds of PBRT_FILTER_*
float filter_eval(int kind, float xw, float yw, float p0, float p1, float x, float y) {
    const float ixw = 1.0f / xw, iyw = 1.0f / yw;
    switch (kind) {
        case PBRT_FILTER_TRIANGLE: {
            const float dx = (xw - std::fabs(x)) * ixw, dy = (yw - std::fabs(y)) * iyw;
            return std::fmax(dx, 0.0f) * std::fmax(dy, 0.0f);
        }
        case PBRT_FILTER_GAUSSIAN: {  // filter.rs:55-64: exp_x / exp_y fixed at construction
            const float ex = std::exp(-p0 * xw * xw), ey = std::exp(-p0 * yw * yw);
            const float gx = std::fmax(std::exp(-p0 * x * x) - ex, 0.0f);
            const float gy = std::fmax(std::exp(-p0 * y * y) - ey, 0.0f);
            return gx * gy;
        }
        case PBRT_FILTER_MITCHELL: {
            const float b = p0, c = p1;
            auto m = [&](float v) {
                const float t = std::fabs(v * 2.0f);
                float r;
                if (t >= 2.0f)
                    r = 0.0f;
                else if (t > 1.0f)
                    r = (-b - 6.0f * c) * t * t * t + (6.0f * b + 30.0f * c) * t * t + (-12.0f * b - 48.0f * c) * t +
                        (8.0f * b + 24.0f * c);
                else
                    r = (12.0f - 9.0f * b - 6.0f * c) * t * t * t + (-18.0f + 12.0f * b + 6.0f * c) * t * t +
                        (6.0f - 2.0f * b);
                return (1.0f / 6.0f) * r;
            };
            return m(x * ixw) * m(y * iyw);
        }
        case PBRT_FILTER_LANCZOS:
            return sinc_1d(x * ixw, p0) * sinc_1d(y * iyw, p0);
        default:  // PBRT_FILTER_BOX: Filter::mean
            return 1.0f;
    }
}

}  // namespace

int filter_table(const PbrtCameraDesc& cam, float table[256]) {
    if (cam.filter_kind < PBRT_FILTER_BOX || cam.filter_kind > PBRT_FILTER_LANCZOS) return PBRT_ERR_INVALID_ARGUMENT;
    const float xw = cam.filter_x_width, yw = cam.filter_y_width;
    for (int y = 0; y < 16; ++y) {
        const float fy = ((float)y + 0.5f) * yw / 16.0f;
        for (int x = 0; x < 16; ++x) {
            const float fx = ((float)x + 0.5f) * xw / 16.0f;
            table[y * 16 + x] = filter_eval(cam.filter_kind, xw, yw, cam.filter_p0, cam.filter_p1, fx, fy);
        }
    }
    return PBRT_OK;
}

}  // namespace pbrt
