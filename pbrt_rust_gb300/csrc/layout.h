// layout.h - device data layout of a flattened BVH scene (host + device).
//
// The reference keeps a depth-first array of PackedBVHNode
// (src/primitive/aggregates/bvh.rs:260-326): first child at n+1, second
// child at second_child_offset.  On the device the same tree is stored as
// sibling PAIRS: every inner node owns one 64-byte pair holding its two
// children's 32-byte records (child1 first), so one visit fetches both
// child boxes.  Pairs are numbered in the depth-first pre-order of their
// parents.  The root's own record travels in the kernel arguments.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define PBRT_HD __host__ __device__ __forceinline__
#else
#define PBRT_HD inline
#endif

namespace pbrt {

// 32-byte child record: box + two words.
//   inner child: a = index of its own children's pair, b = its split axis
//   leaf child:  a = first ordered primitive,        b = kLeafBit | count
struct alignas(16) ChildRec {
    float lo_x, lo_y, lo_z;
    uint32_t a;
    float hi_x, hi_y, hi_z;
    uint32_t b;
};
static_assert(sizeof(ChildRec) == 32, "child record is 32 bytes");

struct alignas(64) NodePair {
    ChildRec c[2];
};
static_assert(sizeof(NodePair) == 64, "node pair is 64 bytes");

constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kCountMask = 0x7fffffffu;

// 4-wide node, two levels of the reference's binary tree with the four
// grandchildren's boxes on an 8-bit grid of the node's own extent.  For a
// binary inner node N with children L (first) and R (second): slot 0/1 = L's
// first/second child (slot 0 = L itself if L is a leaf, slot 1 then empty),
// slot 2/3 = the same for R.
//
// Why 64 bytes: a divergent warp pays one L1 wavefront per lane and 32-byte
// load, and with full-precision boxes (128 bytes, four loads) that pipe was
// the limit once the box arithmetic had been cut (80 % busy on 2^20 rays
// into 4096 random triangles).  Two loads halve it.
//
// Grid: plane code c (one byte) stands for the coordinate
//   org + v(c) * scale,  v(c) = 128 + c for c < 128, 2 c for c >= 128
// because v(c) is the float with bits 0x43000000 | c << 16: one byte permute
// decodes a plane.  Lower planes are rounded down and upper planes up, so a
// node's boxes contain the exact ones; the exact box of a leaf is tested when
// one of its primitives is hit (trace4.cuh says why that gives the
// reference's walk).
//   sxy    scale of x as a float whose low 16 bits are the top half of the
//          scale of y (a bfloat16)
//   sz     scale of z
//   order  3 bits per ray octant (bit i of the octant: the ray's direction is
//          negative on axis i), at 3 * octant: bit 0 / 1 = L's / R's children
//          swap places in the visit, bit 2 = L and R do
//   lo/hi  one byte per slot
//   ref    kNode4Leaf | first primitive, or the index of the child's own
//          node; an empty slot refers to the leaf of the null primitive that
//          ends the primitive array
struct alignas(64) QuadNode {
    float org_x, org_y, org_z;
    uint32_t sxy;
    float sz;
    uint32_t order;
    uint32_t lo_x, hi_x;
    uint32_t lo_y, hi_y, lo_z, hi_z;
    uint32_t ref[4];
};
static_assert(sizeof(QuadNode) == 64, "4-wide node is 64 bytes");
constexpr uint32_t kNode4Leaf = 0x80000000u;

// 48-byte primitive record in BVH (ordered) order; one null record (a
// triangle of zeros that no ray hits) follows the last.  Triangle: its
// vertices; the edges p2 - p1 and p3 - p1 are the f32 subtractions the
// reference does per test (src/shape/mesh.rs:45-46).
//   r0 = (p1.xyz, id)  id = refined input index | kSphereBit if analytic
//   r1 = (p2.xyz, analytic record's index)
//   r2 = (p3.xyz, flags)
// Flags (4-wide walk): kPrimLastBit on the last primitive of a leaf; and, for
// the exact box of the leaf,
//   kPrimBoxEntry  first primitive of a leaf of several, or an instance: the
//                  box in the table at flags >> kPrimBoxShift, tested before
//                  the leaf's primitives
//   kPrimOwnBox    a leaf of one triangle: the bounds of its vertices, tested
//                  when the triangle is hit
//   kPrimHitBox    a leaf of one analytic shape: the box in the table, tested
//                  when the shape is hit
// Every record of a leaf with a box in the table carries the box's index.
struct alignas(16) PrimRec {
    float r0[4];
    float r1[4];
    float r2[4];
};
static_assert(sizeof(PrimRec) == 48, "primitive record is 48 bytes");
constexpr uint32_t kSphereBit = 0x80000000u;
constexpr uint32_t kPrimLastBit = 1u;
constexpr uint32_t kPrimBoxEntry = 2u;
constexpr uint32_t kPrimOwnBox = 4u;
constexpr uint32_t kPrimHitBox = 8u;
constexpr uint32_t kPrimBoxShift = 4u;

// The 4-wide walk's margins (trace4.cuh), u = 2^-24: kFarMargin (6 u) per
// distance of the origin, kTreeMargin (32 u) per half extent of the tree.
constexpr float kFarMargin = 3.57627868652343750e-07f;
constexpr float kTreeMargin = 1.90734863281250e-06f;

// A leaf's exact box in the table of leaf boxes.
struct alignas(32) LeafBox {
    float lo[4], hi[4];
};

// An analytic shape - sphere (src/shape/sphere.rs:16-25), disk
// (src/shape/disk.rs:16-22) or cylinder (src/shape/cylinder.rs:16-23) -
// with its world-to-object and object-to-world matrix rows.  A disk keeps
// its height in z_min = z_max (its object bound, disk.rs:70-74).
// An instance (TransformedPrimitive) uses the same record: w2o / o2w are
// its world-to-primitive / primitive-to-world matrices and `instance`
// selects the definition's BVH.
enum { kQuadSphere = 0, kQuadDisk = 1, kQuadCylinder = 2, kQuadInstance = 3 };
struct alignas(16) SphereRec {
    float w2o[16];      // row-major world_to_object.m
    float o2w[16];      // row-major object_to_world.m
    float radius, z_min, z_max, phi_max;
    float theta_min, theta_max;
    uint32_t full;      // the phi (and for spheres the z) clip cannot reject
    uint32_t flip;      // reverse_orientation ^ transform_swaps_handedness
    uint32_t kind;      // kQuad*
    float height, inner_radius;
    uint32_t instance;  // kQuadInstance: definition index
};
static_assert(sizeof(SphereRec) == 176, "analytic shape record is 176 bytes");

}  // namespace pbrt
