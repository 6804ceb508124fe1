// Internal layout of a u26_lbvh (one tree over vertices, edges or faces).
// Mirrors LbvhData (lbvh.h:77-150) with device-sorted Morton keys instead of the host copy.
#pragma once
#include "u26_internal.h"

namespace u26
{
	// A part of a DevBuf.
	struct DevView
	{
		void* ptr = nullptr;
		template <typename T>
		T* as() const { return static_cast<T*>(ptr); }
	};
} // namespace u26

struct u26_lbvh
{
	u26_ctx* ctx = nullptr;
	int type = U26_TREE_FACE;
	uint32_t n = 0; // leaves
	u26::DevBuf morton_sorted;		 // uint64[n]
	u26::DevBuf sorted_get_original; // uint32[n]
	u26::DevBuf parent;				 // uint32[2n-1]
	u26::DevBuf children;			 // uint32[2n-1][2]
	u26::DevBuf object_idx;			 // uint32[2n-1]
	u26::DevBuf node_aabb;			 // NodeBox[2n-1]
	u26::DevBuf block_aabb;			 // float[blocks][6] of the global AABB's reduction, then its arrival count
	u26::DevBuf global_aabb;		 // float[6]
	u26::DevBuf node_range;			 // uint32[max(n-1,1)]: inner node i covers leaves [min(i, r), max(i, r)], r = node_range[i]
	// refit plan, prepared by construct_tree (one per topology; its counts stay on the device): parts of one
	// allocation
	u26::DevBuf plan;
	u26::DevView plan_info;		 // uint32[4]: top nodes m, treelets nt, chunks, the tree's height (leaves 0)
	u26::DevView plan_words;		 // uint32[max(n-1,1)]: chunk-local child slots and height of each inner node
	u26::DevView chunk_lo;		 // uint32[chunks + 1]: first leaf of each refit chunk, then n
	u26::DevView chunk_tb;		 // uint32[chunks + 1]: first treelet of each chunk, then nt
	u26::DevView roots;			 // uint32[nt]: treelet roots (maximal subtrees of <= 1024 leaves) in leaf order
	u26::DevView root_height;	 // uint8[nt]: their heights
	u26::DevView root_slot;		 // uint32[nt]: 2 x the parent's place in top_nodes + the side
	u26::DevView root_box;		 // float[2m][6]: their boxes of the last refit, by root_slot
	u26::DevView top_nodes;		 // uint32[m]: nodes of more than 1024 leaves, by height
	u26::DevView top_links;		 // uint2[m]: their children as compact ids (top j, or 0x80000000 | treelet b)
	u26::DevView level_end;		 // uint32[65]: end of each height's run in top_nodes
	u26::DevView plan_scratch;	 // construction scratch (about 2 B per leaf)
	u26::DevBuf leaf_prims;			 // uint32[n][K]: the primitive table in leaf order (edge / face trees)
	const uint32_t* leaf_prims_src = nullptr; // the table leaf_prims was permuted from
	u26::DevBuf health;				 // uint32[1]: 1 healthy
	u26::RadixSorter sorter;
	// inputs of the last reduce_aabb (construct_tree reads them, as the reference
	// keeps sa_leaf_center from the reduce pass)
	const float* last_x = nullptr;
	const uint32_t* last_prims = nullptr;
	// 0: the reference's second-pass block count ceil(num_verts/256) (parity mode);
	// 1: all leaf blocks (the true global AABB, better Morton spread)
	int full_global_aabb = 0;
	uint32_t last_num_verts = 0;
	bool built = false; // construct_tree has run (parent / children / node_range are valid)

	uint32_t num_inner() const { return n > 0 ? n - 1 : 0; }
	uint32_t num_nodes() const { return n > 0 ? 2 * n - 1 : 0; }
};

namespace u26
{
	// Traversal view handed to the query kernels.
	struct TreeView
	{
		const NodeBox* __restrict__ boxes;
		const uint2* __restrict__ children;
		const uint32_t* __restrict__ object_idx;
		const uint32_t* __restrict__ health;
		const uint32_t* __restrict__ height;
		uint32_t n;
	};
	inline TreeView tree_view(const u26_lbvh* t)
	{
		return TreeView{ t->node_aabb.as<NodeBox>(), t->children.as<uint2>(), t->object_idx.as<uint32_t>(),
			t->health.as<uint32_t>(), t->plan_info.as<uint32_t>() + 3, t->n };
	}
} // namespace u26
