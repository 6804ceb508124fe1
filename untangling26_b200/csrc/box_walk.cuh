// Box queries of a warp against one tree (broad phase, fused EF detection): the traversal of
// query_template2 (lbvh.cpp:295-363, 780-894) for 32 queries, a stack per lane.
//
// What a query does at its leaves (counting and storing a pair, the EF test) runs with the few lanes that
// stand at one when a thread does it in its walk. Here the leaves met go into a queue
// in shared memory as (primitive, lane) entries, from which the caller takes full batches of 32. A
// step loads both children's boxes (32 bytes each) and links at once, one dependent latency per level, and goes
// on with a child in registers; the stack holds only the other one.
// (Measured against it and dropped: the warp walking the union of its queries' paths with broadcast loads. It
// visits three times the nodes of one query, one after the other: fused detection 5.7 ms against 4.4 ms on
// 3.9 M edges, 0.122 ms against 0.087 ms on 24,066.)
//
// Visit order, the 32-entry stack and the 100,000 step bound are the reference's, per query: a query whose
// stack is full, or that has taken its steps, stops and raises the flag; what it met before counts.
// Query sets too small to fill the chip are split into the parts of the tree below its first levels, where
// neither bound can be met (walk_split_log2, walk_part), since a part would not see another part's stop.
#pragma once
#include "lbvh_internal.h"

namespace u26
{
	constexpr uint32_t kLeafDrain = 64; // entries from which the queue is emptied to a batch's rest
	constexpr uint32_t kLeafQueue = 128;
	static_assert(kLeafDrain - 1 + 2 * 32 <= kLeafQueue, "a step adds two leaves a lane to a queue below the drain mark");
	constexpr uint32_t kQueryStack = 32;
	constexpr uint32_t kQuerySteps = 100000u;

	struct LeafQueue
	{
		uint32_t prim[kLeafQueue];
		uint8_t lane[kLeafQueue];
	};

	// Parts per query warp: doubled until 64 warps per SM are there, at most 32 (24,066 edges in 16 parts:
	// 0.087 ms; four times as many warps 0.094 ms). One part when the tree has more inner nodes than a query may
	// take steps.
	inline uint32_t walk_split_log2(uint32_t num_queries, uint32_t num_leaves)
	{
		const uint32_t warps = div_up(num_queries, 32);
		uint32_t s = 0;
		if (num_leaves <= kQuerySteps + 1u)
			while (s < 5 && (uint64_t(warps) << s) < 148u * 64u)
				s++;
		return s;
	}
	// The depth of this part's split, known on the device only; false when the part has no walk. A node whose
	// two children are stacked lies at most height - 2 below the root, and each node above it holds
	// at most one entry: a tree of height 32 never fills the stack. (Meshes of 100,000 triangles are 20 to 30 high;
	// several scenes in one tree up to 40.)
	__device__ __forceinline__ bool walk_part(const TreeView& tv, uint32_t part, uint32_t& split_log2)
	{
		if (__ldg(tv.height) <= kQueryStack)
			return true;
		split_log2 = 0u;
		return part == 0u;
	}

	// accept(prim): per lane, whether the leaf counts. flush(prim, lane, n): all lanes call it; lane k < n
	// holds entry k (the primitive and the lane of the query that met it). visited: boxes tested
	// by this lane's query.
	template <class Accept, class Flush>
	__device__ __forceinline__ void box_walk(const TreeView& tv, bool valid, f3 mn, f3 mx, uint32_t part, uint32_t split_log2, LeafQueue& lq,
		uint32_t& visited, uint32_t* __restrict__ dev_err, Accept accept, Flush flush)
	{
		constexpr uint32_t kAll = 0xFFFFFFFFu;
		const uint32_t lane = threadIdx.x & 31u;
		const uint32_t ni = tv.n - 1u;
		uint32_t count = 0; // queue entries (uniform)
		auto drain = [&](uint32_t keep)
		{
			__syncwarp();
			while (count > keep)
			{
				const uint32_t n = min(count, 32u);
				count -= n;
				const uint32_t k = count + min(lane, n - 1u);
				flush(lq.prim[k], uint32_t(lq.lane[k]), n);
			}
			__syncwarp();
		};
		auto push_leaf = [&](bool hit, uint32_t prim)
		{
			const uint32_t m = __ballot_sync(kAll, hit);
			if (hit)
			{
				const uint32_t k = count + __popc(m & ((1u << lane) - 1u));
				lq.prim[k] = prim;
				lq.lane[k] = uint8_t(lane);
			}
			count += __popc(m);
		};
		auto meets = [&](uint32_t c)
		{
			// one 32-byte load (boxes start on 32-byte boundaries)
			NodeBox b;
			asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
				: "=f"(b.mn.x), "=f"(b.mn.y), "=f"(b.mn.z), "=f"(b.mn.w), "=f"(b.mx.x), "=f"(b.mx.y), "=f"(b.mx.z), "=f"(b.mx.w)
				: "l"(tv.boxes + c));
			return overlap_strict(b, mn, mx);
		};

		// the start: the root, or the part's node below the first levels
		uint2 cur = __ldg(tv.children); // the children of the node that the lane stands at
		bool on = valid;
		for (uint32_t l = split_log2; l > 0 && __any_sync(kAll, on); l--)
		{
			const bool right = (part >> (l - 1)) & 1u;
			const bool mine = (part & ((1u << (l - 1)) - 1u)) == 0u; // the part that counts this step
			const uint32_t c = right ? cur.y : cur.x;
			const bool hit = on && meets(c);
			visited += on && mine ? 1u : 0u;
			const uint2 next = __ldg(tv.children + c);
			on = hit;
			if (c >= ni) // (uniform)
			{
				if (mine)
					push_leaf(hit && accept(next.x), next.x);
				on = false;
			}
			cur = next;
		}

		uint2 stack[kQueryStack]; // the children of the nodes to visit
		uint32_t top = 0, steps = 0;
		while (__any_sync(kAll, on))
		{
			bool hx = false, hy = false;
			uint2 nx = cur, ny = cur;
			if (on)
			{
				nx = __ldg(tv.children + cur.x);
				ny = __ldg(tv.children + cur.y);
				hx = meets(cur.x);
				hy = meets(cur.y);
				visited += 2u;
			}
			const bool leaf_x = cur.x >= ni, leaf_y = cur.y >= ni;
			bool go_x = hx && !leaf_x, go_y = hy && !leaf_y;
			if (go_x && top >= kQueryStack)
			{
				atomicOr(dev_err, U26_DEVERR_STACK_OVERFLOW);
				go_x = go_y = hy = on = false;
				visited--; // the second child is not tested
			}
			else if (go_y && top + (go_x ? 1u : 0u) >= kQueryStack)
			{
				atomicOr(dev_err, U26_DEVERR_STACK_OVERFLOW);
				go_x = go_y = on = false;
			}
			push_leaf(hx && leaf_x && accept(nx.x), nx.x);
			push_leaf(hy && leaf_y && accept(ny.x), ny.x);
			if (on)
			{
				if (++steps > kQuerySteps)
				{
					atomicOr(dev_err, U26_DEVERR_ITERATION_CAP);
					on = false;
				}
				else if (go_y)
				{
					// the second child first, as the last one stacked
					if (go_x)
						stack[top++] = nx;
					cur = ny;
				}
				else if (go_x)
					cur = nx;
				else if (top > 0u)
					cur = stack[--top];
				else
					on = false;
			}
			if (count >= kLeafDrain)
				drain(31u);
		}
		drain(0u);
	}
} // namespace u26
