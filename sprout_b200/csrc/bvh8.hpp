// Host-side BVH construction for the GPU cast: binned-SAH binary tree, greedy collapse to an
// 8-wide tree, and encoding into 96-byte nodes with 8-bit quantized child boxes.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

namespace spb {

// One 8-wide node, 96 bytes, loaded with three 256-bit loads.
//   origin.xyz, tri_valid | imask << 24, child_base, tri_base, scale.x, scale.y
//   x planes, y planes
//   z planes, scale.z
// Planes of an axis: byte 4 j + 2 c + s is the low (s = 0) or high (1) plane of child 2 j + c.
// Child slot i has the box origin + [lo, hi] * scale per axis, scale a power of two.  imask bit i
// marks an internal child; bits 3 i .. 3 i + 2 of tri_valid the triangles (1 to 3) of a leaf.  A
// node's triangles are stored contiguously from tri_base in the order of those bits, its internal
// children from child_base in slot order.
struct alignas(32) Wide_node {
    float    origin[3];
    uint32_t masks;
    uint32_t child_base;
    uint32_t tri_base;
    float    scale_xy[2];
    uint8_t  planes[3][8][2];  // axis, child, low / high
    float    scale_z;
    uint32_t pad[3];
};
static_assert(sizeof(Wide_node) == 96, "Wide_node must be 96 bytes");

// One triangle, 64 bytes, of which 48 are read (two loads): vertex a, edges b - a and c - a (exactly the values the
// Möller-Trumbore test computes first), the caller's triangle index and a class word the
// traversal can filter on (the path tracer marks participating-medium boundaries).
struct alignas(64) Wide_triangle {
    float    a[3];
    uint32_t id;
    float    e1[3];
    uint32_t tri_class;
    float    e2[3];
    uint32_t pad[5];
};
static_assert(sizeof(Wide_triangle) == 64, "Wide_triangle must be 64 bytes");

struct Wide_bvh {
    std::vector<Wide_node>     nodes;
    std::vector<Wide_triangle> triangles;
    uint32_t                   num_leaves = 0;
    uint32_t                   max_depth  = 0;
    double                     sah_cost   = 0.;
    float                      hit_margin = 0.f;  // see hit_margin_for
    // Bounds of all triangles widened by 2^-10 of the scene size (rounded outward): a ray that
    // misses this box cannot hit a triangle (scene_box_pad).
    float                      scene_lo[3] = {0.f, 0.f, 0.f};
    float                      scene_hi[3] = {0.f, 0.f, 0.f};
};

// Padding of the scene box a ray is first tested against: 2^-10 * max(scene extent, largest
// coordinate magnitude), 128 times the hit margin, so that no ray whose hit point the
// traversal accepts (within the hit margin of a triangle) falls outside it.
double scene_box_pad(double extent, double magnitude);

// Margin around a triangle's bounds within which a hit point must lie:
// 2^-17 * max(scene extent, largest coordinate magnitude), at least FLT_MIN.  extent and
// magnitude come from the float bounds of all triangle vertices, converted to double.
float hit_margin_for(double extent, double magnitude);

// Deepest tree the traversal kernels accept (their stack holds one entry per level).
constexpr uint32_t Max_wide_depth = 48;

// Builds the 8-wide tree.  Returns false (with a message) if the input is unusable.
// tri_class (optional, one word per triangle) is stored with each triangle.  min_margin: the hit
// margin is at least this (for a tree over some of a scene's triangles that is to answer as the
// whole scene's tree does).
bool build_wide_bvh(uint32_t num_vertices, uint32_t num_triangles, float const* positions,
                    uint32_t const* indices, uint32_t num_threads, Wide_bvh& out,
                    std::string& error, uint32_t const* tri_class = nullptr,
                    float min_margin = 0.f);

// Builds a top-level 8-wide tree over instance boxes (6 floats each: lo.xyz, hi.xyz).  Its leaf
// records carry the instance index in Wide_triangle::id and instance_class in tri_class; their
// vertex fields are unused.
bool build_wide_instances(uint32_t num_instances, float const* boxes_lo_hi, uint32_t instance_class,
                          uint32_t num_threads, Wide_bvh& out, std::string& error);

}  // namespace spb
