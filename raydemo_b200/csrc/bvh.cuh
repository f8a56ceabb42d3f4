// GPU BVH construction for one mesh.
#pragma once

#include <vector>

#include "common.cuh"

namespace rg {

struct MeshBvh {
    WideNode *nodes = nullptr;  // node 0 is the root
    uint32_t node_count = 0;
    TriRec *leaf_tris = nullptr; // leaf order; .mi = triangle index within the mesh
    uint32_t tri_count = 0;
    uint32_t depth = 0;          // wide levels on the longest root-to-leaf path
    float bmin[3] = {0, 0, 0}, bmax[3] = {0, 0, 0};
};

void free_mesh_bvh(MeshBvh &b);

// PreprocessTri (src/Ray/internal/Core.cpp:162-214) for n triangles given as
// 9 floats each (three vertex positions), plus their axis-aligned boxes.
// mat: 3 words per triangle (front material, back material, solid flag).
cudaError_t launch_preprocess_tris(const float *verts, const uint32_t *mat, uint32_t n, TriRec *tris_out, float *aabb_out,
                                   cudaStream_t st);

// Builds the wide BVH over n preprocessed triangles (Ref order) with boxes
// aabb (6 floats each): LBVH over 64-bit Morton keys, greedy collapse to
// 8-wide nodes, quantised child boxes. Allocates out.nodes / out.leaf_tris.
// Returns RAY_OK or a RAY_ERR_* code (message through set_error).
// Its scratch arrays lie in `scratch`, which is kept from mesh to mesh.
struct DeviceBuf;
int build_mesh_bvh(const TriRec *tris_ref, const float *aabb, uint32_t n, MeshBvh &out, DeviceBuf &scratch, cudaStream_t st);

// The instance tree: an LBVH over the instances' world boxes (Morton codes
// of the box centres, the same radix sort, binary radix tree and collapse as
// a mesh's build) as wide nodes with one instance per leaf slot, so that the
// traversal tests it with the mesh nodes' own step (1,024 instances, 262,144
// rays on B200: 0.84 ms; a binary tree of float boxes with its own stack in
// local memory took 1.86). slot_src keeps what each
// slot of a node holds; a refit (after instances moved) recomputes the boxes
// over the same topology, a level of nodes per launch from the deepest up. A
// build is needed when the instance count changed.
struct InstTree {
    uint32_t n = 0;              // instances of the current topology (0: none built)
    float *aabb = nullptr;       // 6 floats per instance: world box
    uint32_t *order = nullptr;   // leaf entry -> instance index
    WideNode *nodes = nullptr;   // node 0 is the root; a level's nodes are contiguous
    uint32_t *slot_src = nullptr; // 8 per node: INST_LEAF | instance, child node, or INST_EMPTY
    float *box = nullptr;        // 6 floats per node
    uint32_t count = 0;          // nodes
    std::vector<uint32_t> level; // first node of each level, then the node count
    uint32_t depth() const { return level.empty() ? 0u : (uint32_t)level.size() - 1u; }
};
void free_inst_tree(InstTree &t);
// boxes: n world boxes (6 floats each) in host memory. refit: keep the
// topology (requires t.n == n). Returns RAY_OK or a RAY_ERR_* code.
int build_inst_tree(const float *boxes, uint32_t n, bool refit, InstTree &t, cudaStream_t st);

} // namespace rg
