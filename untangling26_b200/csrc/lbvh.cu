// LBVH build / refit / broad-phase query on sm_100a.
//
// Reference: Solver/CollisionDetector/lbvh.cpp. Construction: global AABB
// (372-452, 454-496, 988-1021), Morton keys (84-135, 512-528), sort (1037-1040, here a
// device radix sort), Karras emission (206-293, 546-601), check (603-616). Refit:
// leaf AABBs (621-688) and the bottom-up union (694-758), here height by height from a plan
// that construction prepares, instead of the reference's float-CAS flags and spin-waits: no
// thread waits on another outside its block's barriers. Query: stack-32
// traversal with strict overlap (295-363, 780-894), in the reference's visit order so
// that the stack-overflow cut-off drops the same pairs.
#include <algorithm>

#include "box_walk.cuh"
#include "lbvh_internal.h"

namespace u26
{
	namespace
	{
		template <int TYPE>
		__device__ __forceinline__ void prim_center_aabb(const float* __restrict__ x, const uint32_t* __restrict__ prims, uint32_t lid,
			f3& c, f3& mn, f3& mx)
		{
			if constexpr (TYPE == U26_TREE_FACE)
			{
				const uint32_t a = __ldg(prims + 3 * lid), b = __ldg(prims + 3 * lid + 1), d = __ldg(prims + 3 * lid + 2);
				const f3 pa = ld3(x, a), pb = ld3(x, b), pd = ld3(x, d);
				c = 0.333333f * ((pa + pb) + pd);
				mn = vmin(pa, vmin(pb, pd));
				mx = vmax(pa, vmax(pb, pd));
			}
			else if constexpr (TYPE == U26_TREE_EDGE)
			{
				const uint32_t a = __ldg(prims + 2 * lid), b = __ldg(prims + 2 * lid + 1);
				const f3 pa = ld3(x, a), pb = ld3(x, b);
				c = 0.5f * (pa + pb);
				mn = vmin(pa, pb);
				mx = vmax(pa, pb);
			}
			else
			{
				c = ld3(x, lid);
				mn = c;
				mx = c;
			}
		}

		__device__ __forceinline__ float warp_min(float v)
		{
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
				v = fminf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
			return v;
		}
		__device__ __forceinline__ float warp_max(float v)
		{
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
				v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
			return v;
		}

		// Global AABB of the first n primitives (fn_reduce_*_tree_global_aabb and fn_reduce_aabb_2_pass: minima and
		// maxima, so any grouping gives the same values). One launch: every block reduces its
		// stride, the last block to finish the blocks' results. arrivals is zero on entry
		// and left zero.
		constexpr uint32_t kReduceBlocks = 148u * 4u;
		__device__ __forceinline__ void block_aabb_reduce(float (&v)[6], float (*s)[8])
		{
			for (int k = 0; k < 6; k++)
				v[k] = k < 3 ? warp_min(v[k]) : warp_max(v[k]);
			const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
			if (lane == 0)
				for (int k = 0; k < 6; k++)
					s[k][warp] = v[k];
			__syncthreads();
			if (warp == 0)
				for (int k = 0; k < 6; k++)
				{
					const float t = lane < 8 ? s[k][lane] : (k < 3 ? INFINITY : -INFINITY);
					v[k] = k < 3 ? warp_min(t) : warp_max(t);
				}
		}
		template <int TYPE>
		__global__ void __launch_bounds__(256) reduce_aabb_kernel(const float* __restrict__ x, const uint32_t* __restrict__ prims,
			uint32_t n, float* __restrict__ block_aabb, uint32_t* __restrict__ arrivals, float* __restrict__ out)
		{
			__shared__ float s[6][8];
			__shared__ bool s_last;
			float v[6] = { INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY };
			for (uint64_t lid = uint64_t(blockIdx.x) * 256u + threadIdx.x; lid < n; lid += uint64_t(gridDim.x) * 256u)
			{
				f3 c, mn, mx;
				prim_center_aabb<TYPE>(x, prims, uint32_t(lid), c, mn, mx);
				const float p[6] = { mn.x, mn.y, mn.z, mx.x, mx.y, mx.z };
				for (int k = 0; k < 6; k++)
					v[k] = k < 3 ? fminf(v[k], p[k]) : fmaxf(v[k], p[k]);
			}
			block_aabb_reduce(v, s);
			if (threadIdx.x == 0)
			{
				for (int k = 0; k < 6; k++)
					block_aabb[6 * blockIdx.x + k] = v[k];
				__threadfence();
				s_last = atomicAdd(arrivals, 1u) == gridDim.x - 1u;
			}
			__syncthreads();
			if (!s_last)
				return;
			__threadfence();
			for (int k = 0; k < 6; k++)
				v[k] = k < 3 ? INFINITY : -INFINITY;
			for (uint32_t b = threadIdx.x; b < gridDim.x; b += 256u)
				for (int k = 0; k < 6; k++)
					v[k] = k < 3 ? fminf(v[k], __ldcg(block_aabb + 6 * b + k)) : fmaxf(v[k], __ldcg(block_aabb + 6 * b + k));
			block_aabb_reduce(v, s);
			if (threadIdx.x == 0)
			{
				for (int k = 0; k < 6; k++)
					out[k] = v[k];
				*arrivals = 0u;
			}
		}

		__device__ __forceinline__ uint32_t expand_bits(uint32_t v)
		{
			v = (v | (v << 16)) & 0x030000FFu;
			v = (v | (v << 8)) & 0x0300F00Fu;
			v = (v | (v << 4)) & 0x030C30C3u;
			return (v | (v << 2)) & 0x09249249u;
		}

		__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }

		__device__ __forceinline__ uint32_t morton32(f3 p)
		{
			const float x = clampf(p.x * 1024.0f, 0.0f, 1023.0f);
			const float y = clampf(p.y * 1024.0f, 0.0f, 1023.0f);
			const float z = clampf(p.z * 1024.0f, 0.0f, 1023.0f);
			return (expand_bits(uint32_t(x)) << 2) | (expand_bits(uint32_t(y)) << 1) | expand_bits(uint32_t(z));
		}

		// fn_compute_mortons: key = morton32(normalised centre) << 32 | leaf id; value = leaf id.
		template <int TYPE>
		__global__ void __launch_bounds__(256) morton_kernel(const float* __restrict__ x, const uint32_t* __restrict__ prims, uint32_t n,
			const float* __restrict__ gaabb, uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t* __restrict__ health)
		{
			const uint32_t lid = blockIdx.x * blockDim.x + threadIdx.x;
			if (lid == 0)
				*health = 1u;
			if (lid >= n)
				return;
			const f3 mn = mk3(gaabb[0], gaabb[1], gaabb[2]);
			const f3 mx = mk3(gaabb[3], gaabb[4], gaabb[5]);
			const f3 ext = vmax(mx - mn, mk3(1e-6f));
			const f3 inv = mk3(1.0f / ext.x, 1.0f / ext.y, 1.0f / ext.z);
			f3 c, a, b;
			prim_center_aabb<TYPE>(x, prims, lid, c, a, b);
			const f3 np = (c - mn) * inv;
			keys[lid] = (uint64_t(morton32(np)) << 32) | uint64_t(lid);
			vals[lid] = lid;
		}

		__device__ __forceinline__ int cp_ij(const uint64_t* __restrict__ keys, uint64_t mi, int j, int n)
		{
			if (j < 0 || j >= n)
				return -1;
			return __clzll(mi ^ __ldg(keys + j));
		}

		constexpr uint32_t kTreelet = 1024;
		constexpr uint32_t kTopRoot = 0x80000000u;
		constexpr uint32_t kMaxHeight = 64;
		// Device state of the refit plan while construct_tree makes it (one memset clears head and
		// root_bits). Entry capacities: cap, see plan_capacity.
		struct Plan
		{
			uint32_t* head;		  // [0] top nodes, [1] treelets, [2] chunks
			uint32_t* root_bits;  // a bit per leaf: a treelet starts here
			uint2* root_at;		  // by first leaf: the treelet's root node (then its index) and its parent's place in top_list
			uint32_t* top_at;	  // by node: a top node's place in top_list
			uint32_t* top_list;	  // top nodes, in no order
			uint2* top_raw;		  // their children: a node, or kTopRoot | a treelet's first leaf
			uint32_t* lo;		  // [cap + 1] the treelets' first leaves, then n
			uint32_t* jump[2];	  // [cap + 1]
			uint32_t* flag;		  // [cap + 1]
			uint32_t cap;
		};

		// fn_reset_tree, fn_apply_sorted and fn_build_inner_nodes: determineRange + findSplit (Karras
		// 2012) over unique keys. A thread per leaf: the leaf's links and primitive (the table in
		// leaf order, for the refits' coalesced reads), and inner node i. A node of more than kTreelet
		// leaves joins the top nodes and marks its children of at most kTreelet leaves as treelets.
		template <int K>
		__global__ void __launch_bounds__(256) karras_kernel(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ sorted_vals, uint32_t n,
			const uint32_t* __restrict__ prims, uint32_t* __restrict__ leaf_prims, uint2* __restrict__ children, uint32_t* __restrict__ object_idx,
			uint32_t* __restrict__ parent, uint32_t* __restrict__ node_range, Plan plan)
		{
			const int nid = blockIdx.x * blockDim.x + threadIdx.x;
			const int num_inner = int(n) - 1;
			if (nid >= int(n))
				return;
			{
				const uint32_t orig = sorted_vals[nid];
				children[num_inner + nid] = make_uint2(orig, orig);
				object_idx[num_inner + nid] = orig;
				if (K > 0)
				{
#pragma unroll
					for (int k = 0; k < K; k++)
						leaf_prims[size_t(K) * nid + k] = prims[size_t(K) * orig + k];
				}
			}
			if (nid == 0)
				parent[0] = kInvalid;
			if (nid >= num_inner)
				return;
			object_idx[nid] = kInvalid;
			int i = 0, j = num_inner;
			if (nid != 0)
			{
				const uint64_t mi = keys[nid];
				const int cl = cp_ij(keys, mi, nid - 1, int(n));
				const int cr = cp_ij(keys, mi, nid + 1, int(n));
				const int d = cl < cr ? 1 : -1;
				const int cp_min = min(cl, cr);
				int lmax = 2;
				while (cp_ij(keys, mi, nid + lmax * d, int(n)) > cp_min)
					lmax <<= 1;
				int l = 0;
				for (int t = lmax >> 1; t >= 1; t >>= 1)
					if (cp_ij(keys, mi, nid + (l + t) * d, int(n)) > cp_min)
						l += t;
				i = nid;
				j = nid + l * d;
			}
			int lo = i, hi = j;
			if (!(i < j))
			{
				lo = j;
				hi = i;
			}
			const uint64_t mlo = keys[lo], mhi = keys[hi];
			int split;
			if (mlo == mhi)
				split = (lo + hi) >> 1;
			else
			{
				const int cp_node = __clzll(mlo ^ mhi);
				int t = hi - lo;
				split = lo;
				for (;;)
				{
					t = (t + 1) >> 1;
					const int ns = split + t;
					if (ns < hi && __clzll(mlo ^ __ldg(keys + ns)) > cp_node)
						split = ns;
					if (!(t > 1))
						break;
				}
			}
			int c_left = (lo == split) ? num_inner + split : split;
			int c_right = (hi == split + 1) ? num_inner + split + 1 : split + 1;
			if (hi - lo + 1 > int(kTreelet))
			{
				const uint32_t k = atomicAdd(plan.head, 1u);
				auto child = [&](int first, int last, int c)
				{
					if (last - first + 1 > int(kTreelet))
						return uint32_t(c);
					atomicOr(plan.root_bits + (first >> 5), 1u << (first & 31));
					plan.root_at[first] = make_uint2(uint32_t(c), k);
					return kTopRoot | uint32_t(first);
				};
				uint2 raw = make_uint2(child(lo, split, c_left), child(split + 1, hi, c_right));
				if (c_right >= num_inner)
					raw = make_uint2(raw.y, raw.x); // as the links below
				plan.top_at[nid] = k;
				if (k < plan.cap)
				{
					plan.top_list[k] = uint32_t(nid);
					plan.top_raw[k] = raw;
				}
			}
			else if (nid == 0)
			{
				plan.root_bits[0] = 1u;
				plan.root_at[0] = make_uint2(0u, kInvalid);
			}
			if (c_right >= num_inner)
			{
				const int tmp = c_left;
				c_left = c_right;
				c_right = tmp;
			}
			parent[c_left] = uint32_t(nid);
			parent[c_right] = uint32_t(nid);
			children[nid] = make_uint2(uint32_t(c_left), uint32_t(c_right));
			node_range[nid] = uint32_t(j);
		}

		// ld3 as an 8-byte and a 4-byte load (which two words share 8 bytes depends on the vertex): a gather's L1
		// wavefronts are its lanes' lines times its loads.
		__device__ __forceinline__ f3 ld3_pair(const float* __restrict__ p, uint32_t i)
		{
			const float* v = p + 3 * i;
			const bool low = (reinterpret_cast<uintptr_t>(v) & 4u) == 0u; // (x, y), z; else x, (y, z)
			const float2 two = __ldg(reinterpret_cast<const float2*>(low ? v : v + 1));
			const float one = __ldg(low ? v + 2 : v);
			return low ? mk3(two.x, two.y, one) : mk3(one, two.x, two.y);
		}

		template <int TYPE>
		__device__ __forceinline__ void leaf_box(const float* __restrict__ x0, const float* __restrict__ x1, const float* __restrict__ thickness,
			const uint32_t* __restrict__ prims, uint32_t pid, f3& mn, f3& mx)
		{
			uint32_t first;
			// x_start == x_end (a refit at one state): min(v, v) = v, so one set of loads gives the
			// same box bit for bit
			const bool same = x0 == x1;
			if constexpr (TYPE == U26_TREE_FACE)
			{
				const uint32_t a = __ldg(prims + 3 * pid), b = __ldg(prims + 3 * pid + 1), c = __ldg(prims + 3 * pid + 2);
				const f3 s0 = ld3_pair(x0, a), s1 = ld3_pair(x0, b), s2 = ld3_pair(x0, c);
				if (same)
				{
					mn = vmin(s0, vmin(s1, s2));
					mx = vmax(s0, vmax(s1, s2));
				}
				else
				{
					const f3 e0 = ld3_pair(x1, a), e1 = ld3_pair(x1, b), e2 = ld3_pair(x1, c);
					mn = vmin(vmin(s0, vmin(s1, s2)), vmin(e0, vmin(e1, e2)));
					mx = vmax(vmax(s0, vmax(s1, s2)), vmax(e0, vmax(e1, e2)));
				}
				first = a;
			}
			else if constexpr (TYPE == U26_TREE_EDGE)
			{
				const uint32_t a = __ldg(prims + 2 * pid), b = __ldg(prims + 2 * pid + 1);
				const f3 s0 = ld3_pair(x0, a), s1 = ld3_pair(x0, b);
				if (same)
				{
					mn = vmin(s0, s1);
					mx = vmax(s0, s1);
				}
				else
				{
					const f3 e0 = ld3_pair(x1, a), e1 = ld3_pair(x1, b);
					mn = vmin(vmin(s0, s1), vmin(e0, e1));
					mx = vmax(vmax(s0, s1), vmax(e0, e1));
				}
				first = a;
			}
			else
			{
				const f3 s0 = ld3_pair(x0, pid);
				if (same)
				{
					mn = s0;
					mx = s0;
				}
				else
				{
					const f3 e0 = ld3_pair(x1, pid);
					mn = vmin(s0, e0);
					mx = vmax(s0, e0);
				}
				first = pid;
			}
			const float t = __ldg(thickness + first);
			mn = mn - mk3(t);
			mx = mx + mk3(t);
		}

		// fn_update_*_tree_leave_aabb_v2: flags (0, 1) as in the reference.
		template <int TYPE>
		__global__ void __launch_bounds__(256) leaf_update_kernel(const uint32_t* __restrict__ sorted_get_original, NodeBox* __restrict__ boxes,
			const float* __restrict__ x0, const float* __restrict__ x1, const float* __restrict__ thickness,
			const uint32_t* __restrict__ prims, uint32_t n)
		{
			const uint32_t lid = blockIdx.x * blockDim.x + threadIdx.x;
			if (lid >= n)
				return;
			f3 mn, mx;
			leaf_box<TYPE>(x0, x1, thickness, prims, __ldg(sorted_get_original + lid), mn, mx);
			NodeBox b;
			b.mn = make_float4(mn.x, mn.y, mn.z, 0.0f);
			b.mx = make_float4(mx.x, mx.y, mx.z, 1.0f);
			boxes[n - 1 + lid] = b;
		}

		// Bottom-up union (fn_refit_tree_aabb, lbvh.cpp:694-758) without atomics or waits, level
		// by level. construct_tree prepares, once per topology and without a host round trip:
		//  * treelets: the maximal subtrees of at most kTreelet leaves (each a contiguous leaf
		//    range, Karras 2012), packed in leaf order into chunks of at most kTreelet leaves;
		//  * for every inner node of a chunk one word: both children as chunk-local slots and
		//    its height (1 + the larger child height, leaves 0; a Karras tree over unique
		//    64-bit keys is at most 64 deep);
		//  * the top nodes (more than kTreelet leaves) sorted by height, their children as
		//    compact ids (top node j, or 0x80000000 | treelet b).
		// refit_chunk_kernel: one block per chunk. Leaf boxes and the chunk's inner nodes'
		// boxes live in shared memory, the nodes' words in registers; the nodes of height h are
		// united in step h, after a barrier, so every union reads finished children without
		// atomics or fences. Boxes go out coalesced.
		// refit_top_kernel: one block for the top tree, height by height, in shared memory when
		// it fits, else through L2.
		// Unions keep the (first child, second child) operand order of the reference.
		// The plan's counts stay on the device and its arrays have their upper bounds' sizes from
		// the start, so a construction is 5 to 10 kernels (4 of them in the sort of more than 8,192 keys) without an allocation or a host read (heights by
		// device atomics over the whole tree, two sorts and two host reads made it 53 to 61). Face and edge
		// tree constructed and refit: 3,844 triangles 1.80 ms, 0.18 ms now (host and launch latency); 130,050
		// 1.85 ms, 0.29 ms; 2.6 M 3.5 ms, 1.45 ms (0.43 ms of it the sorts, 0.31 ms the one-block kernels).
		constexpr size_t kChunkSmem = 2 * 24 * kTreelet;

		// Top nodes lie above nodes of more than kTreelet leaves, disjoint at every depth, and a tree over
		// 30 Morton bits and the leaf id bits has at most 62 depths with one: at most 62 n / 1025 < n / 16
		// top nodes, and one more treelet.
		inline uint32_t plan_capacity(uint32_t n) { return n / 16u + 64u; }
		// Two consecutive chunks hold more than kTreelet leaves together.
		inline uint32_t chunk_bound(uint32_t n) { return 2u * (n / kTreelet) + 2u; }

		// ---- construction: treelets and chunks (one block)
		__device__ __forceinline__ uint32_t block_scan1024(uint32_t v, uint32_t* warp_sum, uint32_t& total)
		{
			const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
			uint32_t s = v;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1)
			{
				const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, s, o);
				s += lane >= uint32_t(o) ? t : 0u;
			}
			if (lane == 31u)
				warp_sum[warp] = s;
			__syncthreads();
			uint32_t w = warp_sum[lane];
			total = __reduce_add_sync(0xFFFFFFFFu, w);
			w = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? w : 0u);
			__syncthreads();
			return w + s - v;
		}
		// Treelets in leaf order, then packed greedily into chunks of at most kTreelet leaves. The greedy
		// chain (a chunk ends where the next treelet does not fit) is followed by doubling: jump[b] is the
		// first treelet after a chunk that begins at b, and after round r every chunk start within
		// 2^(r + 1) chunks of the first is flagged. (One thread walking the treelets took 0.3 ms for 3,913
		// of them.)
		constexpr uint32_t kChainShared = 12u * 1024u; // treelets and their end (192 KB)
		__global__ void __launch_bounds__(1024) plan_chunks_kernel(Plan plan, uint32_t n, uint32_t* __restrict__ roots, uint32_t* __restrict__ chunk_lo,
			uint32_t* __restrict__ chunk_tb, uint32_t max_chunks, uint32_t* __restrict__ info, uint32_t* __restrict__ health)
		{
			extern __shared__ __align__(16) uint32_t s_chain[]; // [4][treelets + 1]
			__shared__ uint32_t s_sum[32];
			const uint32_t t = threadIdx.x;
			const uint32_t words = (n + 31u) / 32u;
			uint32_t nt = 0;
			constexpr uint32_t kPer = 8; // 16-byte loads a thread
			for (uint32_t w0 = 0; w0 < words; w0 += 4096u * kPer)
			{
				uint4 w[kPer];
				uint32_t sum = 0;
#pragma unroll
				for (uint32_t k = 0; k < kPer; k++)
				{
					const uint32_t i = w0 + (t * kPer + k) * 4u;
					w[k] = i < words ? *reinterpret_cast<const uint4*>(plan.root_bits + i) : make_uint4(0u, 0u, 0u, 0u); // zero past the last leaf
					sum += __popc(w[k].x) + __popc(w[k].y) + __popc(w[k].z) + __popc(w[k].w);
				}
				uint32_t total;
				uint32_t at = nt + block_scan1024(sum, s_sum, total);
				nt += total;
				if (sum)
				{
#pragma unroll
					for (uint32_t k = 0; k < kPer; k++)
#pragma unroll
						for (uint32_t q = 0; q < 4; q++)
						{
							const uint32_t i = w0 + (t * kPer + k) * 4u + q;
							for (uint32_t m = q == 0 ? w[k].x : q == 1 ? w[k].y : q == 2 ? w[k].z : w[k].w; m; m &= m - 1u, at++)
								if (at < plan.cap)
									plan.lo[at] = 32u * i + uint32_t(__ffs(m) - 1);
						}
				}
			}
			const uint32_t m = plan.head[0];
			if (nt == 0u || nt > plan.cap || m > plan.cap)
			{
				// more nodes than a tree over distinct keys has: the refits find no chunk
				if (t == 0)
				{
					info[0] = info[1] = info[2] = 0u;
					atomicExch(health, 0u);
				}
				return;
			}
			if (t == 0)
				plan.lo[nt] = n;
			__syncthreads();
			for (uint32_t b = t; b < nt; b += 1024u)
			{
				const uint32_t first = plan.lo[b];
				roots[b] = plan.root_at[first].x;
				plan.root_at[first].x = b;
			}
			// the chain's arrays in shared memory when they fit
			const uint32_t len = nt + 1u;
			const bool fits = len <= kChainShared;
			uint32_t* lo_ = fits ? s_chain : plan.lo;
			uint32_t* jump = fits ? s_chain + len : plan.jump[0];
			uint32_t* next = fits ? s_chain + 2u * len : plan.jump[1];
			uint32_t* flag = fits ? s_chain + 3u * len : plan.flag;
			if (fits)
				for (uint32_t b = t; b <= nt; b += 1024u)
					lo_[b] = plan.lo[b];
			__syncthreads();
			for (uint32_t b = t; b <= nt; b += 1024u)
			{
				// the last treelet b' > b with lo[b'] <= lo[b] + kTreelet
				uint32_t lo = b, hi = nt + 1u;
				const uint32_t end = b < nt ? lo_[b] + kTreelet : 0u;
				if (b < nt)
					while (hi - lo > 1u)
					{
						const uint32_t mid = (lo + hi) >> 1;
						if (lo_[mid] <= end)
							lo = mid;
						else
							hi = mid;
					}
				jump[b] = b < nt ? max(lo, b + 1u) : nt;
				flag[b] = b == 0u ? 1u : 0u;
			}
			__syncthreads();
			for (uint32_t reach = 1; reach < nt; reach <<= 1)
			{
				for (uint32_t b = t; b < nt; b += 1024u)
					if (flag[b])
						flag[jump[b]] = 1u;
				for (uint32_t b = t; b <= nt; b += 1024u)
					next[b] = jump[jump[b]];
				__syncthreads();
				uint32_t* x = jump;
				jump = next;
				next = x;
			}
			uint32_t k0 = 0;
			for (uint32_t b0 = 0; b0 < nt; b0 += 1024u)
			{
				const uint32_t b = b0 + t;
				const bool head = b < nt && flag[b];
				uint32_t total;
				const uint32_t k = k0 + block_scan1024(head ? 1u : 0u, s_sum, total);
				k0 += total;
				if (head && k < max_chunks)
				{
					chunk_lo[k] = lo_[b];
					chunk_tb[k] = b;
				}
			}
			if (t == 0)
			{
				const uint32_t k = min(k0, max_chunks);
				chunk_lo[k] = n;
				chunk_tb[k] = nt;
				info[0] = m;
				info[1] = nt;
				info[2] = k;
			}
		}
		// The words of a chunk's inner nodes: child slots (10 bits and a leaf bit each) and the height, 0 for a
		// node whose leaves are not all in the chunk. Heights: a thread per leaf climbs inside the chunk; the
		// first arrival at a node stops, the second stores 1 + the larger child height. Checks the
		// parent links (fn_check_construction).
		constexpr uint32_t kChunkThreads = 512;
		__global__ void __launch_bounds__(kChunkThreads) plan_words_kernel(const uint32_t* __restrict__ parent, const uint2* __restrict__ children,
			const uint32_t* __restrict__ node_range, uint32_t n, const uint32_t* __restrict__ chunk_lo, const uint32_t* __restrict__ chunk_tb,
			uint32_t* __restrict__ info, const uint32_t* __restrict__ roots, uint32_t* __restrict__ words, uint8_t* __restrict__ root_height,
			uint32_t* __restrict__ health)
		{
			__shared__ uint32_t s_word[kTreelet], s_parent[kTreelet], s_leaf_parent[kTreelet], s_count[kTreelet];
			__shared__ volatile uint8_t s_height[kTreelet];
			if (blockIdx.x >= info[2])
				return;
			const uint32_t base = chunk_lo[blockIdx.x], cnt = chunk_lo[blockIdx.x + 1] - base;
			const uint32_t ni = n - 1u, t = threadIdx.x;
			if (cnt > kTreelet || base + cnt > n)
			{
				if (t == 0)
					atomicExch(health, 0u);
				return;
			}
			for (uint32_t k = t; k < cnt; k += kChunkThreads)
			{
				const uint32_t x = base + k;
				uint32_t word = 0, par = kInvalid;
				if (x < ni)
				{
					const uint32_t r = __ldg(node_range + x);
					if (min(x, r) >= base && max(x, r) < base + cnt)
					{
						// children of a node inside the chunk are inside it too (checked, not assumed)
						const uint2 c = __ldg(children + x);
						const uint32_t ia = c.x >= ni ? c.x - ni - base : c.x - base, ib = c.y >= ni ? c.y - ni - base : c.y - base;
						if (ia < cnt && ib < cnt)
						{
							word = 0x80000000u | (ia | (c.x >= ni ? 0x400u : 0u)) | ((ib | (c.y >= ni ? 0x400u : 0u)) << 11);
							par = __ldg(parent + x);
						}
						else
							atomicExch(health, 0u);
					}
				}
				s_word[k] = word;
				s_parent[k] = par;
				s_leaf_parent[k] = __ldg(parent + ni + x);
				s_count[k] = 0u;
				s_height[k] = 0;
			}
			__syncthreads();
			for (uint32_t k = t; k < cnt; k += kChunkThreads)
			{
				const uint32_t w = s_word[k], a = w & 0x7FFu, b = (w >> 11) & 0x7FFu;
				if (w && ((a & 0x400u ? s_leaf_parent[a & 0x3FFu] : s_parent[a]) != base + k || (b & 0x400u ? s_leaf_parent[b & 0x3FFu] : s_parent[b]) != base + k))
					atomicExch(health, 0u);
				uint32_t node = s_leaf_parent[k];
				for (uint32_t steps = 0; steps < kMaxHeight; steps++)
				{
					const uint32_t i = node - base; // kInvalid and nodes outside wrap past cnt
					if (node == kInvalid || i >= cnt || s_word[i] == 0u)
						break;
					__threadfence_block();
					if (atomicAdd(&s_count[i], 1u) == 0u)
						break;
					__threadfence_block();
					const uint32_t w = s_word[i], a = w & 0x7FFu, b = (w >> 11) & 0x7FFu;
					const uint32_t ha = (a & 0x400u) ? 0u : s_height[a & 0x3FFu], hb = (b & 0x400u) ? 0u : s_height[b & 0x3FFu];
					s_height[i] = uint8_t(1u + max(ha, hb));
					node = s_parent[i];
				}
			}
			__syncthreads();
			for (uint32_t k = t; k < cnt; k += kChunkThreads)
				if (base + k < ni)
				{
					const uint32_t w = s_word[k];
					if (w && s_height[k] == 0)
						atomicExch(health, 0u); // unreached
					words[base + k] = w ? (w & 0x3FFFFFu) | (uint32_t(s_height[k]) << 22) : 0u;
				}
			const uint32_t tb0 = chunk_tb[blockIdx.x], tb1 = chunk_tb[blockIdx.x + 1];
			for (uint32_t b = tb0 + t; b < tb1; b += kChunkThreads)
			{
				const uint32_t x = roots[b];
				const uint32_t k = x >= ni ? x - ni - base : x - base;
				root_height[b] = x < ni && k < cnt ? s_height[k] : uint8_t(0);
				if (x == 0u && k < cnt)
					info[3] = s_height[k]; // the tree's root
				if (k >= cnt)
					atomicExch(health, 0u);
			}
		}
		// The top nodes sorted by height with their children's compact ids (one block): heights climb from the treelet
		// roots as in plan_words_kernel, then a counting sort over the heights.
		struct TopScratch // words per top node
		{
			uint32_t height, count, parent, place;
		};
		constexpr uint32_t kTopScratchShared = 12u * 1024u; // top nodes whose scratch fits in shared memory (192 KB)
		__global__ void __launch_bounds__(1024) plan_top_kernel(Plan plan, const uint32_t* __restrict__ parent, const uint2* __restrict__ children,
			uint32_t* __restrict__ info, const uint8_t* __restrict__ root_height, TopScratch* __restrict__ scratch,
			uint32_t* __restrict__ top_nodes, uint2* __restrict__ top_links, uint32_t* __restrict__ root_slot,
			uint32_t* __restrict__ level_end, uint32_t* __restrict__ health)
		{
			extern __shared__ __align__(16) unsigned char s_raw[];
			__shared__ uint32_t s_level[kMaxHeight + 2];
			const uint32_t t = threadIdx.x;
			const uint32_t m = info[0], nt = info[1];
			TopScratch* S = m <= kTopScratchShared ? reinterpret_cast<TopScratch*>(s_raw) : scratch;
#pragma unroll 4
			for (uint32_t j = t; j < m; j += 1024u)
			{
				const uint32_t x = plan.top_list[j];
				const uint2 c = children[x];
				const uint32_t p = parent[x];
				S[j] = TopScratch{ 0u, 0u, p == kInvalid ? kInvalid : plan.top_at[p], 0u };
				if (parent[c.x] != x || parent[c.y] != x)
					atomicExch(health, 0u);
			}
			if (t < kMaxHeight + 2)
				s_level[t] = 0u;
			__syncthreads();
#pragma unroll 4
			for (uint32_t b = t; b < nt; b += 1024u)
			{
				uint32_t j = m ? plan.root_at[plan.lo[b]].y : kInvalid;
				uint32_t h = root_height[b];
				for (uint32_t steps = 0; j < m && steps <= kMaxHeight; steps++)
				{
					h++;
					atomicMax(&S[j].height, h);
					__threadfence_block();
					if (atomicAdd(&S[j].count, 1u) == 0u)
						break;
					__threadfence_block();
					h = atomicMax(&S[j].height, 0u);
					j = S[j].parent;
				}
			}
			__syncthreads();
			for (uint32_t j = t; j < m; j += 1024u)
			{
				const uint32_t h = S[j].height;
				if (h == 0u || h > kMaxHeight)
					atomicExch(health, 0u);
				atomicAdd(&s_level[min(h, kMaxHeight) + 1u], 1u);
			}
			__syncthreads();
			if (t == 0)
				for (uint32_t h = 1; h < kMaxHeight + 2; h++)
					s_level[h] += s_level[h - 1]; // s_level[h]: first place of height h
			__syncthreads();
			if (t <= kMaxHeight)
				level_end[t] = s_level[t + 1];
			__syncthreads();
			for (uint32_t j = t; j < m; j += 1024u)
				S[j].place = atomicAdd(&s_level[min(S[j].height, kMaxHeight)], 1u);
			__syncthreads();
#pragma unroll 4
			for (uint32_t j = t; j < m; j += 1024u)
			{
				const uint32_t place = S[j].place;
				auto compact = [&](uint32_t v, uint32_t side)
				{
					if (!(v & kTopRoot))
						return S[min(plan.top_at[v], m - 1u)].place;
					const uint32_t r = plan.root_at[v & ~kTopRoot].x;
					root_slot[min(r, nt - 1u)] = 2u * place + side;
					return kTopRoot | r;
				};
				if (S[j].parent == kInvalid)
					info[3] = S[j].height; // the tree's root
				const uint2 raw = plan.top_raw[j];
				top_links[place] = make_uint2(compact(raw.x, 0u), compact(raw.y, 1u));
				top_nodes[S[j].place] = plan.top_list[j];
			}
		}

		// ---- refit
		// a box in shared memory: six floats on an 8-byte boundary (three 8-byte accesses)
		struct __align__(8) SBox
		{
			float2 v[3]; // (mn.x, mn.y), (mn.z, mx.x), (mx.y, mx.z)
		};
		__device__ __forceinline__ SBox sbox(f3 mn, f3 mx)
		{
			return SBox{ { make_float2(mn.x, mn.y), make_float2(mn.z, mx.x), make_float2(mx.y, mx.z) } };
		}
		__device__ __forceinline__ SBox unite_s(const SBox& a, const SBox& b)
		{
			return SBox{ { make_float2(fminf(a.v[0].x, b.v[0].x), fminf(a.v[0].y, b.v[0].y)),
				make_float2(fminf(a.v[1].x, b.v[1].x), fmaxf(a.v[1].y, b.v[1].y)),
				make_float2(fmaxf(a.v[2].x, b.v[2].x), fmaxf(a.v[2].y, b.v[2].y)) } };
		}
		__device__ __forceinline__ void store_sbox(NodeBox* p, const SBox& b)
		{
			__stcg(&p->mn, make_float4(b.v[0].x, b.v[0].y, b.v[1].x, 0.0f));
			__stcg(&p->mx, make_float4(b.v[1].y, b.v[2].x, b.v[2].y, 1.0f));
		}
		// One 512-thread block per chunk of at most 1024 leaves, two leaves and two inner-node
		// slots per thread, so that four chunks share an SM and one chunk's loads overlap another's
		// height steps. Bound by L1: the position gathers' wavefronts (82 % of its peak; 2.6 M faces, two position
		// arrays: 110 us, where the bytes alone would take 45).
		template <int TYPE, bool FUSED>
		__global__ void __launch_bounds__(kChunkThreads, 4) refit_chunk_kernel(const uint32_t* __restrict__ sorted_get_original,
			NodeBox* __restrict__ boxes, const float* __restrict__ x0, const float* __restrict__ x1, const float* __restrict__ thickness,
			const uint32_t* __restrict__ prims, bool prims_in_leaf_order, const uint32_t* __restrict__ words,
			const uint32_t* __restrict__ info, const uint32_t* __restrict__ chunk_lo, uint32_t n,
			const uint32_t* __restrict__ chunk_tb, const uint32_t* __restrict__ roots, const uint32_t* __restrict__ root_slot,
			SBox* __restrict__ root_box, uint32_t* __restrict__ health)
		{
			// dynamic shared memory (kChunkSmem bytes, four blocks per SM): leaf boxes, inner boxes
			extern __shared__ __align__(16) unsigned char s_raw[];
			SBox* s_leaf = reinterpret_cast<SBox*>(s_raw);
			SBox* s_inner = s_leaf + kTreelet;
			__shared__ uint32_t s_hmax;
			const uint32_t t = threadIdx.x;
			if (t == 0)
				s_hmax = 0u;
			__syncthreads();
			// (the chunk's bounds are read beside the number of chunks, not after it: the list has an entry for
			// every block)
			const uint32_t nchunks = __ldg(info + 2), base = __ldg(chunk_lo + blockIdx.x), next = __ldg(chunk_lo + blockIdx.x + 1);
			if (blockIdx.x >= nchunks)
				return;
			const uint32_t cnt = next - base;
			const uint32_t ni = n - 1;
			if (cnt > kTreelet || base + cnt > n)
			{
				// a plan that does not match the tree: nothing is read or written
				if (t == 0)
					atomicExch(health, 0u);
				return;
			}
			// inner nodes base + t and base + t + 512 (0: not all of their leaves are in the chunk)
			uint32_t w[2] = { 0u, 0u };
#pragma unroll
			for (int q = 0; q < 2; q++)
			{
				const uint32_t tq = t + q * kChunkThreads, x = base + tq;
				if (tq < cnt && x < ni)
					w[q] = __ldg(words + x);
			}
#pragma unroll
			for (int q = 0; q < 2; q++)
			{
				const uint32_t tq = t + q * kChunkThreads, lid = base + tq;
				if (tq < cnt)
				{
					f3 mn, mx;
					if constexpr (FUSED)
					{
						if (prims_in_leaf_order)
							leaf_box<TYPE>(x0, x1, thickness, prims, lid, mn, mx);
						else
							leaf_box<TYPE>(x0, x1, thickness, prims, __ldg(sorted_get_original + lid), mn, mx);
					}
					else
					{
						const float4 a = __ldcg(&boxes[ni + lid].mn), b = __ldcg(&boxes[ni + lid].mx);
						mn = mk3(a.x, a.y, a.z);
						mx = mk3(b.x, b.y, b.z);
					}
					s_leaf[tq] = sbox(mn, mx);
				}
			}
			const uint32_t wmax = __reduce_max_sync(0xFFFFFFFFu, max(w[0], w[1])) >> 22;
			if ((t & 31) == 0 && wmax)
				atomicMax(&s_hmax, wmax);
			__syncthreads();
			const uint32_t hmax = s_hmax;
			for (uint32_t lv = 1; lv <= hmax; lv++)
			{
#pragma unroll
				for (int q = 0; q < 2; q++)
				{
					if (w[q] >> 22 != lv)
						continue;
					const uint32_t ca = w[q] & 0x7FFu, cb = (w[q] >> 11) & 0x7FFu;
					// the leaf bit is the slot's place behind the inner boxes' (s_inner follows s_leaf)
					s_inner[t + q * kChunkThreads] = unite_s(s_leaf[ca ^ 0x400u], s_leaf[cb ^ 0x400u]);
				}
				__syncthreads();
			}
#pragma unroll
			for (int q = 0; q < 2; q++)
			{
				const uint32_t tq = t + q * kChunkThreads;
				if (tq < cnt)
				{
					store_sbox(boxes + ni + base + tq, s_leaf[tq]);
					if (w[q])
						store_sbox(boxes + base + tq, s_inner[tq]);
				}
			}
			// the chunk's treelet roots' boxes, also in the compact array that the top-tree launch reads (two per
			// top node, at the place of the child that they are)
			if (root_box)
			{
				const uint32_t tb0 = chunk_tb[blockIdx.x], tb1 = chunk_tb[blockIdx.x + 1];
				for (uint32_t b = tb0 + t; b < tb1; b += kChunkThreads)
				{
					const uint32_t x = roots[b];
					const uint32_t k = x >= ni ? x - ni - base : x - base;
					if (k < cnt)
						root_box[root_slot[b]] = x >= ni ? s_leaf[k] : s_inner[k];
					else
						atomicExch(health, 0u);
				}
			}
		}

		// The top tree in one block, height by height. Up to kTopShared top nodes, their boxes and links are in
		// shared memory: first every node takes its treelet children's boxes (one pass of independent
		// loads), a height step reads and writes shared memory only, and the boxes go out at the end. Otherwise
		// boxes and links go through L2 (the block's barrier orders its own stores before the next height's loads).
		constexpr uint32_t kTopShared = 7u * 1024u;
		constexpr size_t kTopSmem = (sizeof(SBox) + sizeof(uint2)) * kTopShared;
		__global__ void __launch_bounds__(1024) refit_top_kernel(NodeBox* __restrict__ boxes, const uint32_t* __restrict__ top_nodes,
			const uint2* __restrict__ top_links, const uint32_t* __restrict__ level_end, const uint32_t* __restrict__ info,
			const SBox* __restrict__ root_box, uint32_t room, uint32_t* __restrict__ health)
		{
			extern __shared__ __align__(16) unsigned char s_raw[]; // boxes and links of `room` top nodes
			SBox* s_box = reinterpret_cast<SBox*>(s_raw);
			uint2* s_link = reinterpret_cast<uint2*>(s_box + room);
			__shared__ uint32_t s_end[kMaxHeight + 1];
			const uint32_t t = threadIdx.x;
			// the first 1,024 nodes' data are read beside the counts, not after them (the arrays hold `room` nodes)
			const bool in = t < room;
			const uint2 link0 = in ? top_links[t] : make_uint2(0u, 0u);
			const uint32_t node0 = in ? top_nodes[t] : 0u;
			SBox first0 = SBox{}, second0 = SBox{};
			if (in)
			{
				first0 = root_box[2u * t];
				second0 = root_box[2u * t + 1u];
			}
			if (t <= kMaxHeight)
				s_end[t] = level_end[t];
			const uint32_t m = info[0], nt = info[1];
			const bool shared = m <= room;
			auto valid = [&](uint32_t id, uint32_t j) { return (id & kTopRoot) ? (id & ~kTopRoot) < nt : id < j; };
			if (shared)
			{
				auto place = [&](uint32_t j, uint2 l, const SBox& first, const SBox& second)
				{
					if (!valid(l.x, j) || !valid(l.y, j))
					{
						// a plan that does not match the tree
						atomicExch(health, 0u);
						l = make_uint2(kTopRoot, kTopRoot);
					}
					s_link[j] = l;
					const bool rx = (l.x & kTopRoot) != 0u, ry = (l.y & kTopRoot) != 0u;
					if (rx && ry)
						s_box[j] = unite_s(first, second);
					else if (rx || ry)
						s_box[j] = rx ? first : second;
				};
				if (t < m)
					place(t, link0, first0, second0);
#pragma unroll 4
				for (uint32_t j = t + 1024u; j < m; j += 1024u)
					place(j, top_links[j], root_box[2u * j], root_box[2u * j + 1u]);
			}
			__syncthreads();
			uint32_t begin = 0;
			for (uint32_t h = 1; h <= kMaxHeight && begin < m; h++)
			{
				const uint32_t end = min(s_end[h], m);
				for (uint32_t j = begin + t; j < end; j += 1024u)
				{
					SBox u;
					if (shared)
					{
						const uint2 l = s_link[j];
						const bool rx = (l.x & kTopRoot) != 0u, ry = (l.y & kTopRoot) != 0u;
						u = s_box[j];
						if (!rx || !ry)
							s_box[j] = unite_s(rx ? u : s_box[l.x], ry ? u : s_box[l.y]);
						continue;
					}
					else
					{
						const uint2 l = top_links[j];
						if (!valid(l.x, j) || !valid(l.y, j))
						{
							atomicExch(health, 0u);
							continue;
						}
						auto child = [&](uint32_t id, uint32_t side)
						{
							if (id & kTopRoot)
								return root_box[2u * j + side];
							const NodeBox* p = boxes + top_nodes[id];
							const float4 a = __ldcg(&p->mn), b = __ldcg(&p->mx);
							return sbox(mk3(a.x, a.y, a.z), mk3(b.x, b.y, b.z));
						};
						u = unite_s(child(l.x, 0u), child(l.y, 1u));
					}
					store_sbox(boxes + top_nodes[j], u);
				}
				if (end > begin)
				{
					begin = end;
					__syncthreads();
				}
			}
			if (shared)
			{
				if (t < m)
					store_sbox(boxes + node0, s_box[t]);
#pragma unroll 4
				for (uint32_t j = t + 1024u; j < m; j += 1024u)
					store_sbox(boxes + top_nodes[j], s_box[j]);
			}
		}

		// query_template2 for a warp of queries (box_walk.cuh): full batches of 32 pairs go out with one
		// counter atomic and coalesced stores. Bound by the latency of its dependent, divergent node loads.
		// Folded 256 x 256 sheet, 195,585 edges in id order, 4.4 M pairs: 1.19 ms with a thread per query
		// and an atomic per pair, 0.37 ms now; five stacked 512 x 512 sheets, 90 M pairs: 13.0 ms, 3.3 ms.
		template <int MODE>
		__global__ void __launch_bounds__(128) query_kernel(TreeView tv, const float* __restrict__ xb, const float* __restrict__ xe,
			const uint32_t* __restrict__ edges, uint32_t nq, const float* __restrict__ d_hat,
			const float* __restrict__ thickness, uint32_t* __restrict__ count, uint32_t* __restrict__ pairs,
			uint32_t max_pairs, uint32_t split_log2, uint32_t* __restrict__ dev_err)
		{
			__shared__ LeafQueue s_queue[4];
			const uint32_t lane = threadIdx.x & 31u;
			const uint32_t warps = (nq + 31u) / 32u;
			const uint64_t wi = uint64_t(blockIdx.x) * 4u + (threadIdx.x >> 5);
			if (wi >= uint64_t(warps) << split_log2 || *tv.health == 0u)
				return;
			const uint32_t part = uint32_t(wi / warps), q0 = uint32_t(wi - uint64_t(part) * warps) * 32u;
			if (!walk_part(tv, part, split_log2))
				return;
			const bool valid = q0 + lane < nq;
			const uint32_t q = valid ? q0 + lane : nq - 1u;
			f3 mn, mx;
			float pad;
			if constexpr (MODE == U26_QUERY_VERTS)
			{
				const f3 a = ld3(xb, q), b = ld3(xe, q);
				mn = vmin(a, b);
				mx = vmax(a, b);
				pad = __ldg(thickness + q) + __ldg(d_hat + q);
			}
			else
			{
				const uint32_t e0 = __ldg(edges + 2 * q), e1 = __ldg(edges + 2 * q + 1);
				const f3 p1 = ld3(xb, e0), p2 = ld3(xb, e1), p3 = ld3(xe, e0), p4 = ld3(xe, e1);
				mn = vmin(vmin(p1, p2), vmin(p3, p4));
				mx = vmax(vmax(p1, p2), vmax(p3, p4));
				pad = __ldg(thickness + e0) + __ldg(d_hat + e0);
			}
			mn = mn - mk3(pad);
			mx = mx + mk3(pad);
			uint32_t visited = 0;
			box_walk(
				tv, valid, mn, mx, part, split_log2, s_queue[threadIdx.x >> 5], visited, dev_err,
				[&](uint32_t prim) { return MODE != U26_QUERY_EDGES || q < prim; },
				[&](uint32_t prim, uint32_t from, uint32_t n)
				{
					uint32_t base = 0;
					if (lane == 0)
						base = atomicAdd(count, n);
					const uint64_t slot = uint64_t(__shfl_sync(0xFFFFFFFFu, base, 0)) + lane;
					if (lane < n && slot < max_pairs)
					{
						pairs[2 * slot] = q0 + from;
						pairs[2 * slot + 1] = prim;
					}
				});
		}

	} // namespace

	// ---- host side ------------------------------------------------------------------

	static u26_status lbvh_alloc(u26_lbvh* t)
	{
		u26_ctx* ctx = t->ctx;
		const uint32_t n = t->n;
		const uint32_t nn = 2 * n - 1;
		U26_CUDA(ctx, t->morton_sorted.reserve(sizeof(uint64_t) * n));
		U26_CUDA(ctx, t->sorted_get_original.reserve(sizeof(uint32_t) * n));
		U26_CUDA(ctx, t->parent.reserve(sizeof(uint32_t) * nn));
		U26_CUDA(ctx, t->children.reserve(sizeof(uint2) * nn));
		U26_CUDA(ctx, t->object_idx.reserve(sizeof(uint32_t) * nn));
		U26_CUDA(ctx, t->node_aabb.reserve(sizeof(NodeBox) * nn));
		U26_CUDA(ctx, t->block_aabb.reserve(sizeof(float) * 6 * kReduceBlocks + sizeof(uint32_t)));
		U26_CUDA(ctx, cudaMemsetAsync(t->block_aabb.ptr, 0, sizeof(float) * 6 * kReduceBlocks + sizeof(uint32_t), ctx->stream));
		U26_CUDA(ctx, t->global_aabb.reserve(sizeof(float) * 6));
		U26_CUDA(ctx, t->node_range.reserve(sizeof(uint32_t) * std::max<uint32_t>(n - 1, 1)));
		const uint32_t cap = plan_capacity(n), chunks = chunk_bound(n), words = div_up(n, 32);
		// construction scratch in words: head [64], root_bits, top_raw [cap][2], top scratch
		// (when it does not fit in shared memory), top_list [cap], lo, jump x 2, flag [cap + 1 each]
		const uint64_t w4 = (words + 3u) & ~3u, c2 = (uint64_t(cap) + 1u) & ~uint64_t(1);
		const uint64_t scratch = 64u + w4 + 2u * c2 + (cap > kTopScratchShared ? 4u * c2 : 0u) + 5u * uint64_t(cap + 1u);
		// the refit plan and its scratch: one allocation, every part on a 256-byte boundary
		struct Part
		{
			DevView* view;
			uint64_t bytes;
		};
		const Part parts[] = { { &t->plan_words, sizeof(uint32_t) * uint64_t(std::max<uint32_t>(n - 1, 1)) }, { &t->plan_info, sizeof(uint32_t) * 4 },
			{ &t->chunk_lo, sizeof(uint32_t) * uint64_t(chunks + 1) }, { &t->chunk_tb, sizeof(uint32_t) * uint64_t(chunks + 1) },
			{ &t->roots, sizeof(uint32_t) * uint64_t(cap) }, { &t->root_slot, sizeof(uint32_t) * uint64_t(cap) },
			{ &t->root_box, 2u * sizeof(SBox) * uint64_t(cap) }, { &t->root_height, cap },
			{ &t->top_nodes, sizeof(uint32_t) * uint64_t(cap) }, { &t->top_links, sizeof(uint2) * uint64_t(cap) },
			{ &t->level_end, sizeof(uint32_t) * (kMaxHeight + 1) }, { &t->plan_scratch, sizeof(uint32_t) * scratch } };
		uint64_t total = 0;
		for (const Part& q : parts)
			total += (q.bytes + 255u) & ~uint64_t(255);
		U26_CUDA(ctx, t->plan.reserve(total));
		total = 0;
		for (const Part& q : parts)
		{
			q.view->ptr = static_cast<unsigned char*>(t->plan.ptr) + total;
			total += (q.bytes + 255u) & ~uint64_t(255);
		}
		U26_CUDA(ctx, cudaMemsetAsync(t->plan_info.ptr, 0, sizeof(uint32_t) * 4, ctx->stream));
		if (t->type != U26_TREE_VERT)
			U26_CUDA(ctx, t->leaf_prims.reserve(sizeof(uint32_t) * (t->type == U26_TREE_FACE ? 3u : 2u) * size_t(n)));
		U26_CUDA(ctx, t->health.reserve(sizeof(uint32_t)));
		U26_CUDA(ctx, cudaMemsetAsync(t->health.ptr, 0, sizeof(uint32_t), ctx->stream));
		U26_CUDA(ctx, cudaMemsetAsync(t->node_aabb.ptr, 0, sizeof(NodeBox) * nn, ctx->stream));
		return U26_OK;
	}
} // namespace u26

using namespace u26;

#define U26_DISPATCH_TYPE(type, KERNEL, GRID, BLOCK, STREAM, ...)                        \
	do                                                                                   \
	{                                                                                    \
		if ((type) == U26_TREE_FACE)                                                     \
			KERNEL<U26_TREE_FACE><<<(GRID), (BLOCK), 0, (STREAM)>>>(__VA_ARGS__);        \
		else if ((type) == U26_TREE_EDGE)                                                \
			KERNEL<U26_TREE_EDGE><<<(GRID), (BLOCK), 0, (STREAM)>>>(__VA_ARGS__);        \
		else                                                                             \
			KERNEL<U26_TREE_VERT><<<(GRID), (BLOCK), 0, (STREAM)>>>(__VA_ARGS__);        \
	}                                                                                    \
	while (0)

U26_API u26_status u26_lbvh_create(u26_ctx* ctx, int tree_type, uint32_t num_leaves, u26_lbvh** out)
{
	if (!ctx || !out)
		return U26_ERR_INVALID_INPUT;
	*out = nullptr;
	if (tree_type < U26_TREE_VERT || tree_type > U26_TREE_EDGE)
		return set_error(ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_create: bad tree type %d", tree_type);
	if (num_leaves == 0 || num_leaves > 0x7FFFFFFFu)
		return set_error(ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_create: num_leaves %u out of range", num_leaves);
	U26_CUDA(ctx, cudaSetDevice(ctx->device));
	u26_lbvh* t = new u26_lbvh();
	t->ctx = ctx;
	t->type = tree_type;
	t->n = num_leaves;
	const u26_status st = lbvh_alloc(t);
	if (st != U26_OK)
	{
		u26_lbvh_destroy(t);
		return st;
	}
	*out = t;
	return U26_OK;
}

U26_API void u26_lbvh_destroy(u26_lbvh* t)
{
	if (!t)
		return;
	t->morton_sorted.release();
	t->sorted_get_original.release();
	t->parent.release();
	t->children.release();
	t->object_idx.release();
	t->node_aabb.release();
	t->block_aabb.release();
	t->global_aabb.release();
	t->node_range.release();
	t->plan.release();
	t->leaf_prims.release();
	t->health.release();
	t->sorter.release();
	delete t;
}

U26_API u26_status u26_lbvh_reduce_aabb(u26_lbvh* t, const float* x, uint32_t num_verts, const uint32_t* prims)
{
	if (!t || !x || (t->type != U26_TREE_VERT && !prims))
		return t ? set_error(t->ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_reduce_aabb: null input") : U26_ERR_INVALID_INPUT;
	u26_ctx* ctx = t->ctx;
	// lbvh.cpp:999-1021: the edge/face trees reduce ceil(num_verts/256) blocks of 256 primitives in the second pass.
	const uint32_t nb_leaf = div_up(t->n, 256);
	const uint32_t nb = (t->type == U26_TREE_VERT || t->full_global_aabb) ? nb_leaf : std::max(std::min(nb_leaf, div_up(num_verts, 256)), 1u);
	const uint32_t count = nb == nb_leaf ? t->n : nb * 256u;
	float* blocks = t->block_aabb.as<float>();
	U26_DISPATCH_TYPE(t->type, reduce_aabb_kernel, std::min(nb, kReduceBlocks), 256, ctx->stream, x, prims, count, blocks,
		reinterpret_cast<uint32_t*>(blocks + 6 * kReduceBlocks), t->global_aabb.as<float>());
	U26_TRY(after_launch(ctx, "reduce_aabb_kernel"));
	t->last_x = x;
	t->last_prims = prims;
	t->last_num_verts = num_verts;
	return U26_OK;
}

// The kernels' dynamic shared memory (above the 48 KB default), set once per context.
static u26_status size_plan_kernels(u26_ctx* ctx)
{
	if (ctx->sized_plan.load(std::memory_order_acquire))
		return U26_OK;
	const void* chunk_kernels[] = { (const void*)refit_chunk_kernel<U26_TREE_VERT, false>, (const void*)refit_chunk_kernel<U26_TREE_VERT, true>,
		(const void*)refit_chunk_kernel<U26_TREE_EDGE, false>, (const void*)refit_chunk_kernel<U26_TREE_EDGE, true>,
		(const void*)refit_chunk_kernel<U26_TREE_FACE, false>, (const void*)refit_chunk_kernel<U26_TREE_FACE, true> };
	for (const void* k : chunk_kernels)
		U26_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kChunkSmem)));
	U26_CUDA(ctx, cudaFuncSetAttribute(refit_top_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTopSmem)));
	U26_CUDA(ctx, cudaFuncSetAttribute(plan_chunks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(uint32_t) * 4u * kChainShared)));
	U26_CUDA(ctx, cudaFuncSetAttribute(plan_top_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(TopScratch) * kTopScratchShared)));
	ctx->sized_plan.store(true, std::memory_order_release);
	return U26_OK;
}

U26_API u26_status u26_lbvh_construct_tree(u26_lbvh* t)
{
	if (!t)
		return U26_ERR_INVALID_INPUT;
	u26_ctx* ctx = t->ctx;
	if (!t->last_x)
		return set_error(ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_construct_tree: call u26_lbvh_reduce_aabb first");
	const uint32_t n = t->n;
	U26_TRY(size_plan_kernels(ctx));
	uint64_t* keys = t->morton_sorted.as<uint64_t>();
	uint32_t* vals = t->sorted_get_original.as<uint32_t>();
	uint32_t* health = t->health.as<uint32_t>();
	const uint32_t cap = plan_capacity(n), words = div_up(n, 32), w4 = (words + 3u) & ~3u;
	const uint64_t c2 = (uint64_t(cap) + 1u) & ~uint64_t(1);
	// the sort's other buffers are free after it
	U26_CUDA(ctx, t->sorter.keys_alt.reserve(sizeof(uint64_t) * n));
	U26_CUDA(ctx, t->sorter.vals_alt.reserve(sizeof(uint32_t) * n));
	uint32_t* sc = t->plan_scratch.as<uint32_t>();
	auto take = [&](uint64_t count)
	{
		uint32_t* p = sc;
		sc += count;
		return p;
	};
	// (every region up to the top scratch starts on a 16-byte boundary)
	Plan plan;
	plan.cap = cap;
	plan.head = take(64);
	plan.root_bits = take(w4);
	plan.root_at = t->sorter.keys_alt.as<uint2>();
	plan.top_at = t->sorter.vals_alt.as<uint32_t>();
	TopScratch* top_scratch = cap > kTopScratchShared ? reinterpret_cast<TopScratch*>(take(4u * c2)) : nullptr;
	plan.top_raw = reinterpret_cast<uint2*>(take(2u * c2));
	plan.top_list = take(cap);
	plan.lo = take(cap + 1u);
	plan.jump[0] = take(cap + 1u);
	plan.jump[1] = take(cap + 1u);
	plan.flag = take(cap + 1u);
	U26_CUDA(ctx, cudaMemsetAsync(plan.head, 0, sizeof(uint32_t) * (64u + w4), ctx->stream));
	U26_DISPATCH_TYPE(t->type, morton_kernel, div_up(n, 256), 256, ctx->stream, t->last_x, t->last_prims, n,
		t->global_aabb.as<float>(), keys, vals, health);
	U26_TRY(after_launch(ctx, "morton_kernel"));
	// Keys are unique and values start as the identity: a stable sort of the Morton bits
	// [32, 62) reproduces the 64-bit key order.
	U26_TRY(t->sorter.sort(ctx, keys, vals, n, 32, 62));
	// (leaf_prims: the mesh topology is fixed between constructions; a refit given another
	// table gathers)
	t->leaf_prims_src = nullptr;
	auto karras = [&](auto* kernel)
	{
		kernel<<<div_up(n, 256), 256, 0, ctx->stream>>>(keys, vals, n, t->last_prims, t->leaf_prims.as<uint32_t>(), t->children.as<uint2>(),
			t->object_idx.as<uint32_t>(), t->parent.as<uint32_t>(), t->node_range.as<uint32_t>(), plan);
	};
	if (t->type == U26_TREE_FACE)
		karras(&karras_kernel<3>);
	else if (t->type == U26_TREE_EDGE)
		karras(&karras_kernel<2>);
	else
		karras(&karras_kernel<0>);
	U26_TRY(after_launch(ctx, "karras_kernel"));
	if (t->type != U26_TREE_VERT)
		t->leaf_prims_src = t->last_prims;
	if (n > 1)
	{
		uint32_t* info = t->plan_info.as<uint32_t>();
		const uint32_t chunks = chunk_bound(n);
		plan_chunks_kernel<<<1, 1024, sizeof(uint32_t) * 4u * std::min(cap + 1u, kChainShared), ctx->stream>>>(plan, n, t->roots.as<uint32_t>(), t->chunk_lo.as<uint32_t>(), t->chunk_tb.as<uint32_t>(),
			chunks, info, health);
		U26_TRY(after_launch(ctx, "plan_chunks_kernel"));
		plan_words_kernel<<<chunks, kChunkThreads, 0, ctx->stream>>>(t->parent.as<uint32_t>(), t->children.as<uint2>(), t->node_range.as<uint32_t>(),
			n, t->chunk_lo.as<uint32_t>(), t->chunk_tb.as<uint32_t>(), info, t->roots.as<uint32_t>(), t->plan_words.as<uint32_t>(),
			t->root_height.as<uint8_t>(), health);
		U26_TRY(after_launch(ctx, "plan_words_kernel"));
		if (n > kTreelet)
		{
			plan_top_kernel<<<1, 1024, sizeof(TopScratch) * std::min(cap, kTopScratchShared), ctx->stream>>>(plan, t->parent.as<uint32_t>(),
				t->children.as<uint2>(), info, t->root_height.as<uint8_t>(), top_scratch, t->top_nodes.as<uint32_t>(), t->top_links.as<uint2>(),
				t->root_slot.as<uint32_t>(), t->level_end.as<uint32_t>(), health);
			U26_TRY(after_launch(ctx, "plan_top_kernel"));
		}
	}
	t->built = true;
	return U26_OK;
}

U26_API u26_status u26_lbvh_update_leaves(u26_lbvh* t, const float* thickness, const float* x_start, const float* x_end,
	const uint32_t* prims)
{
	if (!t || !thickness || !x_start || !x_end || (t->type != U26_TREE_VERT && !prims))
		return t ? set_error(t->ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_update_leaves: null input") : U26_ERR_INVALID_INPUT;
	u26_ctx* ctx = t->ctx;
	U26_DISPATCH_TYPE(t->type, leaf_update_kernel, div_up(t->n, 256), 256, ctx->stream, t->sorted_get_original.as<uint32_t>(),
		t->node_aabb.as<NodeBox>(), x_start, x_end, thickness, prims, t->n);
	return after_launch(ctx, "leaf_update_kernel");
}

static u26_status refit_impl(u26_lbvh* t, bool fused, const float* thickness, const float* x0, const float* x1,
	const uint32_t* prims)
{
	u26_ctx* ctx = t->ctx;
	if (t->n <= 1)
	{
		if (fused)
			return u26_lbvh_update_leaves(t, thickness, x0, x1, prims);
		return U26_OK;
	}
	if (!t->built)
		return set_error(ctx, U26_ERR_INVALID_INPUT, "refit: call u26_lbvh_construct_tree first");
	const bool sorted = fused && prims && prims == t->leaf_prims_src;
	SBox* root_box = t->n > kTreelet ? t->root_box.as<SBox>() : nullptr;
	const uint32_t* lp = sorted ? t->leaf_prims.as<uint32_t>() : prims;
	const uint32_t* info = t->plan_info.as<uint32_t>();
	// (the chunk count stays on the device: blocks past it leave at once)
#define U26_REFIT(T, F)                                                                                                          \
	refit_chunk_kernel<T, F><<<chunk_bound(t->n), kChunkThreads, kChunkSmem, ctx->stream>>>(t->sorted_get_original.as<uint32_t>(), \
		t->node_aabb.as<NodeBox>(), x0, x1, thickness, lp, sorted, t->plan_words.as<uint32_t>(), info, t->chunk_lo.as<uint32_t>(),  \
		t->n, t->chunk_tb.as<uint32_t>(), t->roots.as<uint32_t>(), t->root_slot.as<uint32_t>(), root_box, t->health.as<uint32_t>())
	if (t->type == U26_TREE_FACE)
	{
		if (fused)
			U26_REFIT(U26_TREE_FACE, true);
		else
			U26_REFIT(U26_TREE_FACE, false);
	}
	else if (t->type == U26_TREE_EDGE)
	{
		if (fused)
			U26_REFIT(U26_TREE_EDGE, true);
		else
			U26_REFIT(U26_TREE_EDGE, false);
	}
	else if (fused)
		U26_REFIT(U26_TREE_VERT, true);
	else
		U26_REFIT(U26_TREE_VERT, false);
#undef U26_REFIT
	U26_TRY(after_launch(ctx, "refit_chunk_kernel"));
	if (t->n <= kTreelet)
		return U26_OK;
	const uint32_t room = std::min(kTopShared, plan_capacity(t->n));
	refit_top_kernel<<<1, 1024, (sizeof(SBox) + sizeof(uint2)) * room, ctx->stream>>>(t->node_aabb.as<NodeBox>(), t->top_nodes.as<uint32_t>(),
		t->top_links.as<uint2>(), t->level_end.as<uint32_t>(), info, t->root_box.as<SBox>(), room, t->health.as<uint32_t>());
	return after_launch(ctx, "refit_top_kernel");
}

U26_API u26_status u26_lbvh_refit(u26_lbvh* t)
{
	if (!t)
		return U26_ERR_INVALID_INPUT;
	return refit_impl(t, false, nullptr, nullptr, nullptr, nullptr);
}

U26_API u26_status u26_lbvh_update_and_refit(u26_lbvh* t, const float* thickness, const float* x_start, const float* x_end,
	const uint32_t* prims)
{
	if (!t || !thickness || !x_start || !x_end || (t->type != U26_TREE_VERT && !prims))
		return t ? set_error(t->ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_update_and_refit: null input") : U26_ERR_INVALID_INPUT;
	return refit_impl(t, true, thickness, x_start, x_end, prims);
}

U26_API u26_status u26_lbvh_query(u26_lbvh* t, int mode, const float* x_begin, const float* x_end, const uint32_t* edges,
	uint32_t num_queries, const float* d_hat, const float* thickness, uint32_t* count, uint32_t* pairs, uint32_t max_pairs)
{
	if (!t || !x_begin || !x_end || !d_hat || !thickness || !count || (!pairs && max_pairs))
		return t ? set_error(t->ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_query: null input") : U26_ERR_INVALID_INPUT;
	if (mode != U26_QUERY_VERTS && !edges)
		return set_error(t->ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_query: edges required for edge queries");
	if (num_queries == 0)
		return U26_OK;
	u26_ctx* ctx = t->ctx;
	const TreeView tv = tree_view(t);
	const uint32_t split = walk_split_log2(num_queries, t->n);
	const uint32_t grid = uint32_t(div_up64(uint64_t(div_up(num_queries, 32)) << split, 4));
	if (mode == U26_QUERY_VERTS)
		query_kernel<U26_QUERY_VERTS><<<grid, 128, 0, ctx->stream>>>(tv, x_begin, x_end, edges, num_queries, d_hat, thickness, count,
			pairs, max_pairs, split, ctx->dev_err);
	else if (mode == U26_QUERY_EDGES)
		query_kernel<U26_QUERY_EDGES><<<grid, 128, 0, ctx->stream>>>(tv, x_begin, x_end, edges, num_queries, d_hat, thickness, count,
			pairs, max_pairs, split, ctx->dev_err);
	else if (mode == U26_QUERY_EDGES_UNCULLED)
		query_kernel<U26_QUERY_EDGES_UNCULLED><<<grid, 128, 0, ctx->stream>>>(tv, x_begin, x_end, edges, num_queries, d_hat, thickness,
			count, pairs, max_pairs, split, ctx->dev_err);
	else
		return set_error(ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_query: bad mode %d", mode);
	return after_launch(ctx, "query_kernel");
}

U26_API u26_status u26_lbvh_check_health(u26_lbvh* t, int* healthy)
{
	if (!t || !healthy)
		return U26_ERR_INVALID_INPUT;
	u26_ctx* ctx = t->ctx;
	U26_CUDA(ctx, cudaMemcpyAsync(ctx->host_word, t->health.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
	U26_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
	*healthy = *ctx->host_word != 0u ? 1 : 0;
	return U26_OK;
}

U26_API u26_status u26_lbvh_arrays_get(const u26_lbvh* t, u26_lbvh_arrays* out)
{
	if (!t || !out)
		return U26_ERR_INVALID_INPUT;
	out->num_leaves = t->n;
	out->num_nodes = t->num_nodes();
	out->morton_sorted = t->morton_sorted.as<uint64_t>();
	out->sorted_get_original = t->sorted_get_original.as<uint32_t>();
	out->parent = t->parent.as<uint32_t>();
	out->children = t->children.as<uint32_t>();
	out->object_idx = t->object_idx.as<uint32_t>();
	out->node_aabb = t->node_aabb.as<float>();
	out->global_aabb = t->global_aabb.as<float>();
	return U26_OK;
}

U26_API u26_status u26_lbvh_set_option(u26_lbvh* t, int option, int value)
{
	if (!t)
		return U26_ERR_INVALID_INPUT;
	if (option == U26_LBVH_OPT_FULL_GLOBAL_AABB)
	{
		t->full_global_aabb = value != 0;
		return U26_OK;
	}
	return set_error(t->ctx, U26_ERR_INVALID_INPUT, "u26_lbvh_set_option: unknown option %d", option);
}
