// host_scene.h - host-side scene preparation for the device path.
//
// f32 math with the reference's operation order (no FMA: this file is
// compiled with -ffp-contract=off), primitive refinement, the reference
// SAH/middle/equal BVH build, its depth-first flattening, and the
// conversion to the device pair layout of layout.h.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <memory>
#include <string>
#include <thread>
#include <utility>
#include <vector>

#include "../../include/pbrt_gpu.h"
#include "layout.h"

namespace pbrt {

// A vector whose resize leaves new elements uninitialised: the arrays of a
// scene are written element by element right after, by several threads
// (zeroing them first costs one thread's pass and all their page faults).
template <class T>
struct RawAlloc : std::allocator<T> {
    template <class U>
    struct rebind {
        using other = RawAlloc<U>;
    };
    RawAlloc() = default;
    template <class U>
    RawAlloc(const RawAlloc<U>&) {}
    template <class U>
    void construct(U* p) noexcept {
        ::new (static_cast<void*>(p)) U;
    }
    template <class U, class... A>
    void construct(U* p, A&&... a) {
        ::new (static_cast<void*>(p)) U(std::forward<A>(a)...);
    }
};
template <class T>
using RawVec = std::vector<T, RawAlloc<T>>;

// f(part, lo, hi) over [0, n) cut into host_parts(n) equal parts, each on its
// own thread; f must not throw.  A part has at least 16384 items, so small
// scenes stay on the caller's thread.  Creating a terrain of 180000 triangles
// with the device build took 18.2 ms with the host's loops on one thread and 11.9
// ms with eight (6.6 ms since its layout is made on the device).
inline size_t host_parts(size_t n) {
    const size_t cores = std::max(1u, std::thread::hardware_concurrency());
    return std::max<size_t>(1, std::min(std::min<size_t>(8, cores), n / 16384));
}
template <class F>
void host_parallel(size_t n, F f) {
    const size_t parts = host_parts(n);
    auto at = [&](size_t p) { return n / parts * p + std::min(p, n % parts); };
    std::vector<std::thread> others;
    size_t next = 1;
    try {
        others.reserve(parts - 1);
        for (; next < parts; ++next)
            others.emplace_back([&f, &at, next] { f(next, at(next), at(next + 1)); });
    } catch (...) {  // no thread to be had: the caller takes the remaining parts
    }
    f((size_t)0, (size_t)0, at(1));
    for (size_t p = next; p < parts; ++p) f(p, at(p), at(p + 1));
    for (std::thread& t : others) t.join();
}

struct V3 {
    float x, y, z;
};
inline V3 v3(float x, float y, float z) { return V3{x, y, z}; }
inline V3 operator+(V3 a, V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
inline V3 operator-(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
inline V3 operator*(V3 a, float f) { return v3(a.x * f, a.y * f, a.z * f); }
inline float dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
inline V3 cross3(V3 a, V3 b) {
    return v3((a.y * b.z) - (a.z * b.y), (a.z * b.x) - (a.x * b.z), (a.x * b.y) - (a.y * b.x));
}
inline float len3(V3 a) { return std::sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }
inline V3 normalize3(V3 a) {  // geometry/normal.rs:181-186: v * (1 / |v|)
    float r = 1.0f / len3(a);
    return a * r;
}
inline float axis_of(V3 a, int i) { return i == 0 ? a.x : (i == 1 ? a.y : a.z); }

struct Box {
    V3 lo, hi;
};
Box box_empty();
Box box_union(const Box& a, const Box& b);
Box box_union(const Box& a, V3 p);
float box_area(const Box& b);
int box_max_extent(const Box& b);

struct M4 {
    float m[4][4];
};
M4 m4_identity();
M4 m4_mul(const M4& a, const M4& b);
bool m4_inverse(const M4& a, M4* out);  // src/transform/matrix4x4.rs:66-160
V3 m4_point(const M4& m, V3 p);          // src/transform/transform.rs:195-208
V3 m4_vector(const M4& m, V3 v);         // src/transform/transform.rs:210-218
bool m4_swaps_handedness(const M4& m);   // src/transform/transform.rs:176-183

struct Xf {
    M4 m, mi;
};
Xf xf_from_desc(const PbrtTransform& t);
Xf xf_mul(const Xf& a, const Xf& b);
Xf xf_inverse(const Xf& a);

// One primitive of the fully refined list.
struct HostPrim {
    int kind;  // PBRT_SHAPE_TRIANGLE_MESH (triangle) or PBRT_SHAPE_SPHERE
    int shape;
    int material;
    int area_light;
    V3 p1, p2, p3;  // triangle vertices in refined order
    bool flip;
    int sphere;  // index into spheres
};

// Flattened reference node (PackedBVHNode, bvh.rs:260-272).
struct FlatNode {
    Box box;
    bool leaf;
    uint32_t offset;  // leaf: first prim; inner: second child
    uint32_t count;   // leaf: prim count; inner: axis
};

// A tree's arrays on the device where it was built (device_fill_layout).
struct DeviceLayout {
    int device = 0;
    NodePair* pairs = nullptr;
    PrimRec* prims = nullptr;
    LeafBox* boxes = nullptr;
    QuadNode* quads = nullptr;
    size_t n_pairs = 0, n_boxes = 0;
    DeviceLayout() = default;
    DeviceLayout(const DeviceLayout&) = delete;
    DeviceLayout& operator=(const DeviceLayout&) = delete;
    ~DeviceLayout();
};

struct HostBVH {
    RawVec<HostPrim> prims;
    std::vector<SphereRec> spheres;
    RawVec<FlatNode> nodes;
    RawVec<uint32_t> ordered;  // ordered_prims: refined input index
    uint32_t depth = 0;
    // device layout: the arrays below, or `layout`, which has them on the device
    std::shared_ptr<DeviceLayout> layout;
    ChildRec root{};
    RawVec<NodePair> pairs;
    RawVec<PrimRec> recs;
    bool has_spheres = false;
    // 4-wide layout (layout.h: QuadNode; same tree, two binary levels per
    // node), encoded on the device from the pairs: quad_of[pair] = index of
    // the 4-wide node that starts at the pair's node | its split axis <<
    // kQuadAxisShift, kNoQuad for the pairs in between
    RawVec<uint32_t> quad_of;
    uint32_t n_quads = 0;
    uint32_t quad_root = 0;           // the root's child word
    std::vector<LeafBox> leaf_boxes;  // leaf boxes the records' flags refer to
    // the tree has the 4-wide layout: every coordinate is finite and at most
    // kWideReach away from the origin
    bool wide = false;
    // its margins (tree_margins): the middle of the root's box, half its
    // extent and 2^-22 of its coordinates, kTreeMargin times that, and the sum
    // of the axes' margins up to which the 4-wide walk is the one to take
    V3 middle{}, half{}, spread{};
    float far = 0.0f;
    uint32_t stack4_bound = 0;  // most children a 4-wide traversal can defer (trace4.cuh: the stack)
    // instance definitions: one BVH each, shared by all their instances
    std::vector<HostBVH> insts;
    // With instances, the id a hit reports: refined primitives numbered in
    // order with each instance taking as many ids as its definition has
    // refined primitives (the ids of the same scene with every instance
    // copied out).  flat_id[i] = first id of refined primitive i; empty
    // without instances (id = refined index).
    std::vector<uint32_t> flat_id;
    uint64_t n_flat = 0;
};

constexpr uint32_t kNoQuad = 0xffffffffu;
constexpr uint32_t kQuadAxisShift = 30u;
constexpr float kWideReach = 1.099511627776e12f;  // 2^40

// Fully refine shapes, build and flatten the BVH, and fill the device
// layout.  Returns a PbrtStatus; *err gets a message on failure.
int build_host_bvh(const PbrtShapeDesc* shapes, uint32_t n_shapes, uint32_t max_prims, const char* split_method,
                   HostBVH* out, std::string* err, bool on_device = false, const PbrtInstanceDesc* defs = nullptr,
                   uint32_t n_defs = 0);

// H.middle, H.half, H.spread, H.far and H.quad_root of the nodes, whose boxes' half
// areas and edge lengths add up to `area` and `length`.
void tree_margins(HostBVH& H, double area, double length);

// The layout arrays on the host (after build_host_bvh left them on a device).
void fill_host_layout(HostBVH& H);

// Bounds (mesh.rs:196-205, sphere.rs:111-126) and centroid (bvh.rs:77) of
// refined primitive i.
Box prim_bounds(const HostBVH& H, size_t i, V3* centroid);

// The tree of build_tree (H.nodes, H.ordered, H.depth) built on the current
// CUDA device (bvh_build.cu): identical nodes and primitive order.  The
// layout is made there too (H.layout) unless a leaf is too large for a thread.
int device_build_tree(HostBVH& H, uint32_t max_prims, int split, std::string* err);

// The layout of a tree whose nodes (m) and primitive order are on the current
// device too, made there (quads.cu): the same arrays as fill_host_layout's.
// d_prims: H.prims on the device, or null.  Leaves H.layout null if the
// device's memory does not suffice.
void device_fill_layout(HostBVH& H, const FlatNode* d_nodes, uint32_t m, const uint32_t* d_ordered,
                        const HostPrim* d_prims);

int parse_split_method(const char* s);

// Camera set-up (src/camera/mod.rs:105-135, projective.rs:48-72): the
// raster-to-camera and camera-to-world matrices, row-major.
void camera_matrices(const PbrtCameraDesc& cam, float raster_to_camera[16], float camera_to_world[16]);

// The film's filter table (camera/film.rs:89-97, filter.rs:44-124); returns
// PBRT_ERR_INVALID_ARGUMENT for an unknown filter kind.
int filter_table(const PbrtCameraDesc& cam, float table[256]);

}  // namespace pbrt
