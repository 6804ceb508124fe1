// Differentiation of the PRP objective over fixed supports S(r) on sm_100a.
//
// For each contour c with support S (the selected hits of u26_prp_resolve) and direction r:
//   delta_h(x, r) = (w_h . n_h) / (r . n_h)    (the ray distance of hit h)
//     VF: w = a - p, n = (b - a) x (c - a)   (vertex p along +r onto face abc)
//     FV: w = q - a, n = (b - a) x (c - a)   (vertex q along -r onto face abc)
//     EE: w = q0 - p0, n = (p1 - p0) x (q1 - q0)   (edge p0p1 swept along r onto q0q1)
//   J = (sum_h A_h) * D^2, D = max_h delta_h      (prp_eval_penetration_v2's objective,
//                                                   intersection_resolver2.cpp:1883-1954)
//   E = sum_h (delta_h + 3e-3)^2 / kappa_h         (its displacement cost; kappa_h the
//                                                   effective inverse mass, helper.cpp:611-645)
// The adjoint gives dJ/dr, dE/dr and dJ/dx, dE/dx: with g = 1 / (r . n), u = w - delta r,
//   d delta / dr = -delta n g
//   VF: d/dp = -n g, d/da = (n + u x (c - b)) g, d/db = ((c - a) x u) g, d/dc = (u x (b - a)) g
//   FV: d/dq =  n g, d/da = (-n + u x (c - b)) g, d/db, d/dc as VF
//   EE: d/dp0 = (-n - e2 x u) g, d/dp1 = (e2 x u) g, d/dq0 = (n - u x e1) g, d/dq1 = (u x e1) g
// (e1 = p1 - p0, e2 = q1 - q0). J's subgradient goes through the argmax hit (the first in
// key order among equal maxima); A_h and kappa_h are constants of the support (rest areas,
// masses and the stored barycentric coordinates). dE/dr is the gradient the reference's
// direction refinement builds (intersection_resolver2.cpp:1268-1320).
#include <algorithm>

#include <cooperative_groups.h>

#include "u26_internal.h"

namespace cg = cooperative_groups;

namespace u26
{
	namespace
	{
		struct HitGeo
		{
			f3 P[4];	   // the hit's vertices: VF p a b c, FV q a b c, EE p0 p1 q0 q1
			uint32_t V[4]; // their ids
			f3 n, w;
			float rn, delta;
		};

		__device__ __forceinline__ HitGeo hit_geo(const u26_prp_hit& h, const float* __restrict__ x, f3 r)
		{
			HitGeo G;
			if (h.type == 1u)
			{
				G.V[0] = h.src_verts[0];
				G.V[1] = h.src_verts[1];
				G.V[2] = h.dst_verts[0];
				G.V[3] = h.dst_verts[1];
			}
			else if (h.type == 0u)
			{
				G.V[0] = h.src_verts[0];
				G.V[1] = h.dst_verts[0];
				G.V[2] = h.dst_verts[1];
				G.V[3] = h.dst_verts[2];
			}
			else
			{
				G.V[0] = h.dst_verts[0];
				G.V[1] = h.src_verts[0];
				G.V[2] = h.src_verts[1];
				G.V[3] = h.src_verts[2];
			}
#pragma unroll
			for (int k = 0; k < 4; k++)
				G.P[k] = ld3(x, G.V[k]);
			if (h.type == 1u)
			{
				G.n = cross(G.P[1] - G.P[0], G.P[3] - G.P[2]);
				G.w = G.P[2] - G.P[0];
			}
			else
			{
				G.n = cross(G.P[2] - G.P[1], G.P[3] - G.P[1]);
				G.w = h.type == 0u ? G.P[1] - G.P[0] : G.P[0] - G.P[1];
			}
			G.rn = dot(r, G.n);
			G.delta = dot(G.w, G.n) / G.rn;
			return G;
		}

		// coefficient * d delta / d(vertex k), k = 0..3 in HitGeo order
		__device__ __forceinline__ void delta_vertex_grads(uint32_t type, const HitGeo& G, f3 r, float coef, f3 out[4])
		{
			const float g = coef / G.rn;
			const f3 u = G.w - r * G.delta;
			if (type == 1u)
			{
				const f3 e1 = G.P[1] - G.P[0], e2 = G.P[3] - G.P[2];
				const f3 e2u = cross(e2, u), ue1 = cross(u, e1);
				out[0] = (-G.n - e2u) * g;
				out[1] = e2u * g;
				out[2] = (G.n - ue1) * g;
				out[3] = ue1 * g;
				return;
			}
			const f3 A = G.P[1], B = G.P[2], C = G.P[3];
			const f3 sgn_n = type == 0u ? G.n : -G.n; // d w / d a: +1 for VF (w = a - p), -1 for FV (w = q - a)
			out[0] = (type == 0u ? -G.n : G.n) * g;
			out[1] = (sgn_n + cross(u, C - B)) * g;
			out[2] = cross(C - A, u) * g;
			out[3] = cross(u, B - A) * g;
		}

		__device__ __forceinline__ float hit_area(const u26_prp_hit& h, const float* __restrict__ va, const float* __restrict__ ea,
			const float* __restrict__ fa)
		{
			return h.type == 0u ? va[h.src_id] : (h.type == 1u ? ea[h.src_id] : fa[h.src_id]);
		}

		__device__ __forceinline__ float hit_kappa(const u26_prp_hit& h, const float* __restrict__ vert_mass)
		{
			auto im = [&](uint32_t v)
			{ return 1.0f / fmaxf(vert_mass[v], 1e-8f); };
			const float b0 = h.bary[0], b1 = h.bary[1];
			if (h.type == 0u)
			{
				const float bz = 1.0f - b0 - b1;
				return ((im(h.src_verts[0]) + b0 * b0 * im(h.dst_verts[0])) + b1 * b1 * im(h.dst_verts[1])) + bz * bz * im(h.dst_verts[2]);
			}
			if (h.type == 2u)
			{
				const float bz = 1.0f - b0 - b1;
				return ((b0 * b0 * im(h.src_verts[0]) + b1 * b1 * im(h.src_verts[1])) + bz * bz * im(h.src_verts[2])) + im(h.dst_verts[0]);
			}
			const float a1 = 1.0f - b0, c1 = 1.0f - b1;
			return ((b0 * b0 * im(h.src_verts[0]) + a1 * a1 * im(h.src_verts[1])) + b1 * b1 * im(h.dst_verts[0])) + c1 * c1 * im(h.dst_verts[1]);
		}

		__device__ __forceinline__ void add3(float* __restrict__ gx, uint32_t v, f3 g)
		{
			atomicAdd(gx + 3 * size_t(v), g.x);
			atomicAdd(gx + 3 * size_t(v) + 1, g.y);
			atomicAdd(gx + 3 * size_t(v) + 2, g.z);
		}

		// The deepest hit of some of a contour's hits: the deeper of two, the earlier of equals. A NaN
		// depth never wins, except that of the contour's first hit, which stays.
		struct Deepest
		{
			float depth;
			uint32_t hit; // kInvalid: none
		};
		__device__ __forceinline__ void deepest(Deepest& a, float depth, uint32_t hit, uint32_t first)
		{
			if (hit == kInvalid || (isnan(a.depth) && a.hit == first))
				return;
			if (a.hit == kInvalid || depth > a.depth || (depth == a.depth && hit < a.hit) || (isnan(depth) ? hit == first : isnan(a.depth)))
			{
				a.depth = depth;
				a.hit = hit;
			}
		}

		// A hit's terms of the two sums, its depth in the running deepest.
		struct HitTerms
		{
			float area, cost;
		};
		__device__ __forceinline__ HitTerms hit_terms(const u26_prp_hit& h, const float* __restrict__ x, f3 r, const float* __restrict__ va,
			const float* __restrict__ ea, const float* __restrict__ fa, const float* __restrict__ vm, Deepest& my, uint32_t i, uint32_t first)
		{
			const HitGeo G = hit_geo(h, x, r);
			const float kap = hit_kappa(h, vm);
			const float sd = G.delta + 3e-3f;
			deepest(my, G.delta, i, first);
			return HitTerms{ hit_area(h, va, ea, fa), kap > 1e-8f ? (sd * sd) / kap : 0.0f };
		}
		// A hit's part of the gradients for the upstream gradients gj, ge: dJ is gj 2 A D d(delta) of the deepest hit.
		__device__ __forceinline__ void hit_grads(const u26_prp_hit& h, const float* __restrict__ x, f3 r, const float* __restrict__ vm, bool deep,
			float gj, float ge, float sA, float D, double (&gr)[3], float* __restrict__ grad_x)
		{
			const HitGeo G = hit_geo(h, x, r);
			float coef = 0.0f;
			if (ge != 0.0f)
			{
				const float kap = hit_kappa(h, vm);
				if (kap > 1e-8f)
					coef = ge * (2.0f * (G.delta + 3e-3f) / kap);
			}
			if (deep && gj != 0.0f)
				coef = coef + gj * (2.0f * sA * D);
			if (coef == 0.0f)
				return;
			const f3 g = G.n * (-G.delta * coef / G.rn);
			gr[0] += double(g.x);
			gr[1] += double(g.y);
			gr[2] += double(g.z);
			if (grad_x)
			{
				f3 gv[4];
				delta_vertex_grads(h.type, G, r, coef, gv);
#pragma unroll
				for (int k = 0; k < 4; k++)
					add3(grad_x, G.V[k], gv[k]);
			}
		}

		constexpr uint32_t kWaveClusters = 64;	 // clusters of 8 x 256 threads that run at once
		constexpr uint32_t kManyContours = 148; // up to here a cluster of 8 blocks per contour, then a block
		constexpr uint32_t kShortClusters = 592; // blocks of 256 threads that the chip holds at 64 registers
		__device__ __forceinline__ f3 direction(const float* __restrict__ dirs, uint32_t c)
		{
			return mk3(dirs[3 * size_t(c)], dirs[3 * size_t(c) + 1], dirs[3 * size_t(c) + 2]);
		}

		// Hits that a warp takes alone: as many as one warp's rounds take no longer than a cluster's barriers (64; 128 where the
		// contours' clusters take more than one wave: 148 contours of 100 hits 35 + 51 us by clusters, 23 + 37 by warps),
		// or, with a chip full of contours, than about two thirds of all hits' time (0.12 us a hit in one warp's chain,
		// 55 ps of the whole chip: 3,000 contours of 500 hits 103 + 251 us by blocks, 86 + 252 by warps).
		__device__ __forceinline__ uint32_t few_hits(const uint32_t* __restrict__ off, uint32_t nc)
		{
			if (nc <= kManyContours)
				return nc > kWaveClusters ? 128u : 64u;
			const uint32_t all = off[nc] - off[0];
			return min(max(max(nc / 16u, all / 3000u), 64u), 1024u);
		}
		// The first contour of c, c + step, ... that has more (every warp finds the same one); kInvalid: none.
		__device__ __forceinline__ uint32_t next_long(const uint32_t* __restrict__ off, uint32_t nc, uint64_t c, uint32_t step)
		{
			const uint32_t few = few_hits(off, nc);
			for (; c < nc; c += 32ull * step)
			{
				const uint64_t cl = c + uint64_t(threadIdx.x & 31u) * step;
				const uint32_t h0 = cl < nc ? off[cl] : 0u, h1 = cl < nc ? off[cl + 1] : 0u;
				const uint32_t m = __ballot_sync(0xFFFFFFFFu, h1 > h0 && h1 - h0 > few);
				if (m)
					return uint32_t(c + uint64_t(__ffs(m) - 1) * step);
			}
			return kInvalid;
		}

		// The contours first, first + step, ... of at most `few` hits, one after the other by this warp. Out of line: the cluster's
		// loops keep their registers.
		__device__ __noinline__ void warp_contours(const float* __restrict__ x, const u26_prp_hit* __restrict__ hits, const uint32_t* __restrict__ off,
			uint32_t nc, const float* __restrict__ dirs, const float* __restrict__ va, const float* __restrict__ ea, const float* __restrict__ fa,
			const float* __restrict__ vm, float* __restrict__ J_out, float* __restrict__ E_out, const float* __restrict__ gJ,
			const float* __restrict__ gE, float* __restrict__ grad_dirs, float* __restrict__ grad_x, uint32_t few, uint32_t first, uint32_t step)
		{
			constexpr uint32_t kAll = 0xFFFFFFFFu;
			const int lane = threadIdx.x & 31;
			for (uint64_t c64 = first; c64 < nc; c64 += step)
			{
				const uint32_t c = uint32_t(c64), h0 = off[c], h1 = off[c + 1];
				if (h1 > h0 && h1 - h0 > few)
					continue;
				const f3 r = direction(dirs, c);
				Deepest my = { -INFINITY, kInvalid };
				float sA = 0.0f, sE = 0.0f;
#pragma unroll 1
				for (uint64_t i = uint64_t(h0) + lane; i < h1; i += 32u)
				{
					const u26_prp_hit h = hits[i];
					const HitTerms t = hit_terms(h, x, r, va, ea, fa, vm, my, uint32_t(i), h0);
					sA = sA + t.area;
					sE = sE + t.cost;
				}
#pragma unroll
				for (int o = 16; o >= 1; o >>= 1)
				{
					sA = sA + __shfl_xor_sync(kAll, sA, o);
					sE = sE + __shfl_xor_sync(kAll, sE, o);
					const float od = __shfl_xor_sync(kAll, my.depth, o);
					const uint32_t oi = __shfl_xor_sync(kAll, my.hit, o);
					deepest(my, od, oi, h0);
				}
				const float D = h1 > h0 ? my.depth : 0.0f;
				if (lane == 0)
				{
					if (J_out)
						J_out[c] = (sA * D) * D;
					if (E_out)
						E_out[c] = sE;
				}
				if (!grad_dirs && !grad_x)
					continue;
				const float gj = gJ ? gJ[c] : 0.0f, ge = gE ? gE[c] : 0.0f;
				double gr[3] = { 0.0, 0.0, 0.0 };
#pragma unroll 1
				for (uint64_t i = uint64_t(h0) + lane; i < h1; i += 32u)
				{
					// without a cost gradient only the deepest hit has one
					if (ge == 0.0f && uint32_t(i) != my.hit)
						continue;
					const u26_prp_hit h = hits[i];
					hit_grads(h, x, r, vm, uint32_t(i) == my.hit, gj, ge, sA, D, gr, grad_x);
				}
				if (grad_dirs)
#pragma unroll
					for (int k = 0; k < 3; k++)
					{
#pragma unroll
						for (int o = 16; o >= 1; o >>= 1)
							gr[k] += __shfl_xor_sync(kAll, gr[k], o);
						if (lane == 0)
							grad_dirs[3 * size_t(c) + k] = float(gr[k]);
					}
			}
		}

		// Forward J, E, then the vector-Jacobian products for the upstream gradients gJ, gE (when given).
		// Clusters of nb blocks (the rule is in u26_prp_adjoint); cluster q of nq takes the contours q, q + nq, ...
		// A contour of few hits is one warp's, whose chain of gather latencies is as short as a cluster's barriers; a longer
		// one is the whole cluster's. Forward and backward kernels with a warp for every contour, with a
		// cluster or block for every contour, and now:
		//   148 contours of 4 hits    13 + 15 us,        28 + 38 us,    15 + 17 us
		//   3,000 of 32               17 + 27,           47 + 74,       20 + 31
		//   20,000 of 32              41 + 96,           228 + 385,     48 + 113
		//   60 of 2,000               197 + 453,         41 + 56,       43 + 56
		//   3,000 of 1 to 4,000       359 + 759,         123 + 274,     121 + 271
		//   1 of 90,526               7,772 + 16,028,    120 + 253,     122 + 255
		// A hit costs one 48-byte record, four gathered vertices and about 250 flops. A long contour's hits are spread over
		// up to 8,192 threads; what stays serial is the canonical summation order of the areas
		// and costs (32 lanes striding over the hits, then an xor butterfly): the terms go to shared
		// memory, round by round, and two warps of the cluster add them up from there (distributed
		// shared memory, one add per 32 hits). No scratch memory, and the results
		// do not depend on timing, but for the order of grad_x's atomics (also within one contour). The gradients in the
		// direction are summed in double, in a fixed order.
		template <int NT>
		__global__ void __launch_bounds__(NT, 1024 / NT) adjoint_kernel(const float* __restrict__ x, const u26_prp_hit* __restrict__ hits,
			const uint32_t* __restrict__ off, uint32_t nc, const float* __restrict__ dirs, const float* __restrict__ va,
			const float* __restrict__ ea, const float* __restrict__ fa, const float* __restrict__ vm, float* __restrict__ J_out,
			float* __restrict__ E_out, const float* __restrict__ gJ, const float* __restrict__ gE, float* __restrict__ grad_dirs,
			float* __restrict__ grad_x)
		{
			constexpr uint32_t kAll = 0xFFFFFFFFu;
			constexpr int kWarps = NT / 32;
			constexpr uint32_t kSlice = 4 * NT; // a block's hits per round
			__shared__ Deepest s_warp[kWarps];
			__shared__ Deepest s_block;
			__shared__ float s_area[kSlice], s_cost[kSlice];
			__shared__ float s_sum[2];
			__shared__ double s_gr[kWarps][3];
			__shared__ double s_gr_block[3];
			cg::cluster_group cluster = cg::this_cluster();
			const uint32_t nb = cluster.num_blocks(), rank = cluster.block_rank();
			const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
			const uint32_t q = blockIdx.x / nb, nq = gridDim.x / nb;
			const bool own = nq == nc && nq <= kShortClusters; // a cluster has one contour, short or long
			for (uint32_t c = own ? q : next_long(off, nc, q, nq); c < nc; c = next_long(off, nc, uint64_t(c) + nq, nq))
			{
				const uint32_t h0 = off[c], h1 = off[c + 1];
				if (own && (h1 <= h0 || h1 - h0 <= few_hits(off, nc)))
					break;
				const uint32_t n = h1 - h0, round = nb * kSlice;
				const f3 r = direction(dirs, c);
				Deepest my = { -INFINITY, kInvalid };
				float sum = 0.0f; // lanes of the summing warps: 0 the areas, 1 the costs
				for (uint64_t q = 0; q < n; q += round)
				{
					const uint32_t left = uint32_t(min(uint64_t(round), n - q));
#pragma unroll 1
					for (uint32_t k = threadIdx.x; k < kSlice; k += NT)
					{
						if (rank * kSlice + k >= left)
							break;
						const uint32_t i = h0 + uint32_t(q) + rank * kSlice + k;
						const u26_prp_hit h = hits[i];
						const HitTerms t = hit_terms(h, x, r, va, ea, fa, vm, my, i, h0);
						s_area[k] = t.area;
						s_cost[k] = t.cost;
					}
					cluster.sync();
					if (rank == 0 && warp < 2)
					{
						// 32 loads in flight: a remote load's latency is about eight adds'
						for (uint32_t blk = 0; blk < nb && blk * kSlice < left; blk++)
						{
							const float* p = cluster.map_shared_rank(warp == 0 ? s_area : s_cost, blk);
							const uint32_t m = min(kSlice, left - blk * kSlice);
							uint32_t k = lane;
							for (; k - lane + 1024u <= m; k += 1024u)
							{
								float t[32];
#pragma unroll
								for (int u = 0; u < 32; u++)
									t[u] = p[k + 32 * u];
#pragma unroll
								for (int u = 0; u < 32; u++)
									sum = sum + t[u];
							}
							for (; k < m; k += 32u)
								sum = sum + p[k];
						}
					}
					cluster.sync(); // the terms are read before the next round's are written
				}
#pragma unroll
				for (int o = 16; o >= 1; o >>= 1)
				{
					const float od = __shfl_xor_sync(kAll, my.depth, o);
					const uint32_t oi = __shfl_xor_sync(kAll, my.hit, o);
					deepest(my, od, oi, h0);
					sum = sum + __shfl_xor_sync(kAll, sum, o);
				}
				if (lane == 0)
				{
					s_warp[warp] = my;
					if (warp < 2)
						s_sum[warp] = sum;
				}
				__syncthreads();
				if (threadIdx.x == 0)
				{
					for (int w = 1; w < kWarps; w++)
						deepest(my, s_warp[w].depth, s_warp[w].hit, h0);
					s_block = my;
				}
				cluster.sync();
				Deepest all = *cluster.map_shared_rank(&s_block, 0);
				for (uint32_t blk = 1; blk < nb; blk++)
				{
					const Deepest o = *cluster.map_shared_rank(&s_block, blk);
					deepest(all, o.depth, o.hit, h0);
				}
				const float sA = *cluster.map_shared_rank(s_sum, 0);
				const float D = all.depth;
				if (rank == 0 && threadIdx.x == 0)
				{
					if (J_out)
						J_out[c] = (sA * D) * D;
					if (E_out)
						E_out[c] = s_sum[1];
				}
				double gr[3] = { 0.0, 0.0, 0.0 };
				if (grad_dirs || grad_x)
				{
					const float gj = gJ ? gJ[c] : 0.0f, ge = gE ? gE[c] : 0.0f;
					// (64-bit: the index may pass 2^32 behind the last hit)
					for (uint64_t i = uint64_t(h0) + rank * NT + threadIdx.x; i < h1; i += nb * NT)
					{
						// without a cost gradient only the deepest hit has one
						if (ge == 0.0f && uint32_t(i) != all.hit)
							continue;
						const u26_prp_hit h = hits[i];
						hit_grads(h, x, r, vm, uint32_t(i) == all.hit, gj, ge, sA, D, gr, grad_x);
					}
				}
				if (grad_dirs)
				{
#pragma unroll
					for (int k = 0; k < 3; k++)
					{
#pragma unroll
						for (int o = 16; o >= 1; o >>= 1)
							gr[k] += __shfl_xor_sync(kAll, gr[k], o);
						if (lane == 0)
							s_gr[warp][k] = gr[k];
					}
					__syncthreads();
					if (threadIdx.x < 3)
					{
						double t = 0.0;
						for (int w = 0; w < kWarps; w++)
							t += s_gr[w][threadIdx.x];
						s_gr_block[threadIdx.x] = t;
					}
					cluster.sync();
					if (rank == 0 && threadIdx.x < 3)
					{
						double t = 0.0;
						for (uint32_t blk = 0; blk < nb; blk++)
							t += cluster.map_shared_rank(s_gr_block, blk)[threadIdx.x];
						grad_dirs[3 * size_t(c) + threadIdx.x] = float(t);
					}
				}
				cluster.sync(); // no block goes on or leaves while another reads its shared memory
				if (own)
					return;
			}
			// the short ones, by the last clusters (the first ones to start have long contours to do)
			const uint32_t ns = min(nq, kShortClusters);
			if (q >= nq - ns)
				warp_contours(x, hits, off, nc, dirs, va, ea, fa, vm, J_out, E_out, gJ, gE, grad_dirs, grad_x, few_hits(off, nc), q - (nq - ns) + (rank * kWarps + warp) * ns, nb * kWarps * ns);
		}

		template <int NT, class... Args>
		cudaError_t launch_adjoint(cudaStream_t st, uint32_t clusters, uint32_t blocks, Args... args)
		{
			cudaLaunchConfig_t cfg = {};
			cfg.gridDim = dim3(clusters * blocks);
			cfg.blockDim = dim3(NT);
			cfg.stream = st;
			cudaLaunchAttribute at[1];
			at[0].id = cudaLaunchAttributeClusterDimension;
			at[0].val.clusterDim.x = blocks;
			at[0].val.clusterDim.y = 1;
			at[0].val.clusterDim.z = 1;
			cfg.attrs = at;
			cfg.numAttrs = 1;
			return cudaLaunchKernelEx(&cfg, adjoint_kernel<NT>, args...);
		}
	} // namespace
} // namespace u26

using namespace u26;

U26_API u26_status u26_prp_adjoint(u26_ctx* ctx, const float* x, const u26_prp_hit* hits, const uint32_t* hit_offsets, uint32_t num_contours,
	const float* dirs, const float* vert_area, const float* edge_area, const float* face_area, const float* vert_mass, float* J, float* E,
	const float* grad_J, const float* grad_E, float* grad_dirs, float* grad_x)
{
	if (!ctx)
		return U26_ERR_INVALID_INPUT;
	if (num_contours == 0)
		return U26_OK;
	if (!x || !hits || !hit_offsets || !dirs || !vert_area || !edge_area || !face_area || !vert_mass)
		return set_error(ctx, U26_ERR_INVALID_INPUT, "u26_prp_adjoint: null input");
	// Threads per long contour by the number of contours (the hits per contour are known on the device only): 8 blocks of
	// 1,024 while all run at once (two such clusters in each of eight GPCs: 18 contours of 20,000 hits took 86 + 160
	// us so, 73 + 139 with blocks of 256), then 8 of 256 (148 of 20,000: 243 + 547 us; 64 clusters run at once),
	// then one block of 256 (149 of 2,000: 46 + 98 us, where 148 with eight blocks take 75 + 109; but a support
	// of 90,000 hits among 149 takes 1.2 + 2.6 ms).
	auto launch = [&](auto threads, uint32_t clusters, uint32_t blocks)
	{
		return launch_adjoint<decltype(threads)::value>(ctx->stream, clusters, blocks, x, hits, hit_offsets, num_contours, dirs, vert_area, edge_area,
			face_area, vert_mass, J, E, grad_J, grad_E, grad_dirs, grad_x);
	};
	cudaError_t e;
	if (num_contours <= 16u)
		e = launch(std::integral_constant<int, 1024>(), num_contours, 8u);
	else if (num_contours <= kManyContours)
		e = launch(std::integral_constant<int, 256>(), num_contours, 8u);
	else
		e = launch(std::integral_constant<int, 256>(), std::min(num_contours, 4u * kShortClusters), 1u);
	U26_CUDA(ctx, e);
	return after_launch(ctx, "adjoint_kernel");
}
