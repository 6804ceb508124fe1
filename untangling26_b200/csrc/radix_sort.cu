// Stable LSD radix sort of (uint64 key, uint32 value) pairs on the device.
//
// Replaces the host pdqsort + two PCIe copies of LBVH::construct_tree
// (lbvh.cpp:1037-1040). Only the live bits are sorted: for Morton keys
// (m32 << 32 | leaf id) with values starting as the identity, a stable sort of bits
// [32, 62) yields exactly the order of the full 64-bit key.
//
// RadixSorter::sort, 8-bit digits:
//  * up to 8,192 keys: one launch of one block, every digit pass in shared memory;
//  * more: one launch counts every pass's digits, then one launch per pass (onesweep): a tile of 3,072
//    keys is ranked with __match_any_sync peer masks and per-warp digit counters, its digit
//    counts are published and the counts of the earlier tiles looked up (decoupled look-back,
//    eight tiles at a time), and the keys go out in digit order from shared memory.
//  Each pass reads and writes every pair once. The three-launch form (below) reads the keys twice, writes
//  them uncoalesced and scans a count table in between; a sort of a few thousand keys is
//  nothing but its launches (12 to 20 for 4 passes, now 1 or 6). Device time: 782 keys in 4 passes
//  61 us, 10 us; 3,844 keys 58 us, 24 us; 2.6 M and 3.9 M keys in 4 passes each 0.90 ms, 0.42 ms (a pass's 24
//  bytes a pair would take 12 us of the 46; the rest is a tile's chain of ranking rounds).
// RadixSorter::sort_into (allocation-free callers: fixed scratch) and sorts of 2^30 keys and more (beyond
// the look-back words' 30-bit counts) run three launches per digit: (1) per-tile digit
// histogram, (2) exclusive scan of the digit-major count table (reduce / scan block sums /
// downsweep over 8192-word segments), (3) stable scatter: each tile is ranked in chunks
// of 256 with __match_any_sync peer masks and a per-warp digit table in shared memory.
#include <algorithm>

#include "u26_internal.h"

namespace u26
{
	namespace
	{
		constexpr int kThreads = 256;
		constexpr int kChunks = 8;
		constexpr int kTile = kThreads * kChunks; // 2048 keys per tile
		constexpr int kWarps = kThreads / 32;

		__global__ void __launch_bounds__(kThreads) radix_hist_kernel(const uint64_t* __restrict__ keys, uint32_t n, int shift, uint32_t mask,
			uint32_t* __restrict__ counts, uint32_t num_tiles)
		{
			__shared__ uint32_t hist[256];
			hist[threadIdx.x] = 0;
			__syncthreads();
			const uint32_t base = blockIdx.x * kTile;
#pragma unroll
			for (int c = 0; c < kChunks; c++)
			{
				const uint32_t i = base + c * kThreads + threadIdx.x;
				if (i < n)
				{
					const uint32_t d = uint32_t(keys[i] >> shift) & mask;
					atomicAdd(&hist[d], 1u);
				}
			}
			__syncthreads();
			counts[threadIdx.x * num_tiles + blockIdx.x] = hist[threadIdx.x];
		}

		// Exclusive scan of counts[0, total) in place by one block of 1024 threads.
		__global__ void __launch_bounds__(1024) radix_scan_kernel(uint32_t* __restrict__ counts, uint32_t total)
		{
			__shared__ uint32_t warp_sums[32];
			const uint32_t per = (total + blockDim.x - 1) / blockDim.x;
			const uint32_t begin = threadIdx.x * per;
			const uint32_t end = min(total, begin + per);
			uint32_t local = 0;
			for (uint32_t i = begin; i < end; i++)
				local += counts[i];
			// block exclusive scan of `local`
			const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
			uint32_t v = local;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1)
			{
				uint32_t t = __shfl_up_sync(0xFFFFFFFFu, v, o);
				if (lane >= o)
					v += t;
			}
			if (lane == 31)
				warp_sums[warp] = v;
			__syncthreads();
			if (warp == 0)
			{
				uint32_t w = warp_sums[lane];
#pragma unroll
				for (int o = 1; o < 32; o <<= 1)
				{
					uint32_t t = __shfl_up_sync(0xFFFFFFFFu, w, o);
					if (lane >= o)
						w += t;
				}
				warp_sums[lane] = w;
			}
			__syncthreads();
			uint32_t run = v - local + (warp > 0 ? warp_sums[warp - 1] : 0u);
			for (uint32_t i = begin; i < end; i++)
			{
				const uint32_t c = counts[i];
				counts[i] = run;
				run += c;
			}
		}

		// ---- device-wide exclusive scan of uint32 words: segments of kScanSeg words, each
		// thread owning kScanPer consecutive words
		constexpr int kScanThreads = 1024;
		constexpr int kScanPer = 8;
		constexpr uint32_t kScanSeg = kScanThreads * kScanPer;

		__device__ __forceinline__ void load8(const uint32_t* __restrict__ v, uint32_t i, uint32_t n, uint32_t (&w)[kScanPer])
		{
			if (i + kScanPer <= n)
			{
				const uint4 a = *reinterpret_cast<const uint4*>(v + i);
				const uint4 b = *reinterpret_cast<const uint4*>(v + i + 4);
				w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w, w[4] = b.x, w[5] = b.y, w[6] = b.z, w[7] = b.w;
			}
			else
			{
#pragma unroll
				for (int j = 0; j < kScanPer; j++)
					w[j] = i + j < n ? v[i + j] : 0u;
			}
		}

		// block-wide exclusive scan of one value per thread; returns the exclusive prefix and
		// writes the block total to *total (all threads)
		__device__ __forceinline__ uint32_t block_exclusive(uint32_t x, uint32_t* total)
		{
			__shared__ uint32_t ws[32];
			__shared__ uint32_t tot;
			const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
			uint32_t v = x;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1)
			{
				const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, v, o);
				if (lane >= o)
					v += t;
			}
			if (lane == 31)
				ws[warp] = v;
			__syncthreads();
			if (warp == 0)
			{
				uint32_t w = lane < int(blockDim.x >> 5) ? ws[lane] : 0u;
#pragma unroll
				for (int o = 1; o < 32; o <<= 1)
				{
					const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, w, o);
					if (lane >= o)
						w += t;
				}
				ws[lane] = w;
				if (lane == 31)
					tot = w;
			}
			__syncthreads();
			const uint32_t r = v - x + (warp > 0 ? ws[warp - 1] : 0u);
			*total = tot;
			__syncthreads();
			return r;
		}

		__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const uint32_t* __restrict__ v, uint32_t n, uint32_t* __restrict__ seg_sums)
		{
			uint32_t w[kScanPer];
			load8(v, blockIdx.x * kScanSeg + threadIdx.x * kScanPer, n, w);
			uint32_t s = 0;
#pragma unroll
			for (int j = 0; j < kScanPer; j++)
				s += w[j];
			s = __reduce_add_sync(0xFFFFFFFFu, s);
			__shared__ uint32_t ws[32];
			if ((threadIdx.x & 31) == 0)
				ws[threadIdx.x >> 5] = s;
			__syncthreads();
			if (threadIdx.x < 32)
			{
				uint32_t t = ws[threadIdx.x];
				t = __reduce_add_sync(0xFFFFFFFFu, t);
				if (threadIdx.x == 0)
					seg_sums[blockIdx.x] = t;
			}
		}

		// exclusive scan in place of each segment, offset by offsets[segment] (or 0)
		__global__ void __launch_bounds__(kScanThreads) scan_down_kernel(uint32_t* __restrict__ v, uint32_t n, const uint32_t* __restrict__ offsets)
		{
			uint32_t w[kScanPer];
			const uint32_t i = blockIdx.x * kScanSeg + threadIdx.x * kScanPer;
			load8(v, i, n, w);
			uint32_t s = 0;
#pragma unroll
			for (int j = 0; j < kScanPer; j++)
				s += w[j];
			uint32_t total;
			uint32_t run = block_exclusive(s, &total) + (offsets ? offsets[blockIdx.x] : 0u);
#pragma unroll
			for (int j = 0; j < kScanPer; j++)
			{
				const uint32_t c = w[j];
				w[j] = run;
				run += c;
			}
			if (i + kScanPer <= n)
			{
				*reinterpret_cast<uint4*>(v + i) = make_uint4(w[0], w[1], w[2], w[3]);
				*reinterpret_cast<uint4*>(v + i + 4) = make_uint4(w[4], w[5], w[6], w[7]);
			}
			else
			{
#pragma unroll
				for (int j = 0; j < kScanPer; j++)
					if (i + j < n)
						v[i + j] = w[j];
			}
		}

		__global__ void __launch_bounds__(kThreads) radix_scatter_kernel(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
			uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n, int shift, uint32_t mask,
			const uint32_t* __restrict__ offsets, uint32_t num_tiles)
		{
			__shared__ uint32_t warp_cnt[kWarps][256];
			__shared__ uint32_t base_run[256];
			const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
			base_run[tid] = offsets[tid * num_tiles + blockIdx.x];
			const uint32_t lanemask_lt = (1u << lane) - 1u;
			const uint32_t tile_base = blockIdx.x * kTile;
			for (int c = 0; c < kChunks; c++)
			{
#pragma unroll
				for (int w = 0; w < kWarps; w++)
					warp_cnt[w][tid] = 0;
				__syncthreads();
				const uint32_t i = tile_base + c * kThreads + tid;
				const bool valid = i < n;
				uint64_t k = 0;
				uint32_t v = 0, d = 0x100u + lane; // invalid lanes get unique digits
				if (valid)
				{
					k = keys_in[i];
					v = vals_in[i];
					d = uint32_t(k >> shift) & mask;
				}
				const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
				const uint32_t rank = __popc(peers & lanemask_lt);
				const int leader = __ffs(peers) - 1;
				if (valid && lane == leader)
					warp_cnt[warp][d] = __popc(peers);
				__syncthreads();
				{
					uint32_t run = base_run[tid];
#pragma unroll
					for (int w = 0; w < kWarps; w++)
					{
						const uint32_t t = warp_cnt[w][tid];
						warp_cnt[w][tid] = run;
						run += t;
					}
					base_run[tid] = run;
				}
				__syncthreads();
				if (valid)
				{
					const uint32_t pos = warp_cnt[warp][d] + rank;
					keys_out[pos] = k;
					vals_out[pos] = v;
				}
				__syncthreads();
			}
		}

		// ---- one block: all digit passes of up to kSmall keys in shared memory. NT threads: 256 up to 2,048 keys (the
		// digit table has a row per warp to clear and scan), else 1,024; every thread holds ceil(n / NT) keys.
		constexpr uint32_t kSmallItems = 8, kSmall = 1024 * kSmallItems, kSmallFew = 256 * kSmallItems;
		template <uint32_t NT>
		struct SmallSort
		{
			uint64_t keys[NT * kSmallItems];
			uint32_t vals[NT * kSmallItems];
			uint16_t cnt[NT / 32][256]; // per warp and digit
			uint32_t start[256];
			uint32_t warp_sum[8];
		};
		// exclusive scan over the first 256 threads' values (whole warps; the caller's barriers order
		// warp_sum's uses); every thread of the block calls it
		__device__ __forceinline__ uint32_t scan256(uint32_t v, uint32_t* warp_sum)
		{
			const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
			uint32_t s = v;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1)
			{
				const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, s, o);
				s += lane >= uint32_t(o) ? t : 0u;
			}
			if (warp < 8u && lane == 31u)
				warp_sum[warp] = s;
			__syncthreads();
			uint32_t base = 0;
#pragma unroll
			for (uint32_t w = 0; w < 7; w++)
				base += w < warp ? warp_sum[w] : 0u;
			return base + s - v;
		}
		template <uint32_t NT>
		__global__ void __launch_bounds__(NT) radix_small_kernel(uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n,
			int bit_lo, int bit_hi)
		{
			extern __shared__ __align__(16) unsigned char s_raw[];
			SmallSort<NT>& S = *reinterpret_cast<SmallSort<NT>*>(s_raw);
			const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
			const uint32_t lt = (1u << lane) - 1u;
			// a warp's keys are consecutive: item i of lane l is key 32 * (per * warp + i) + l
			const uint32_t per = (n + NT - 1u) / NT;
			const uint32_t first = warp * 32u * per + lane;
			uint64_t k[kSmallItems];
			uint32_t v[kSmallItems];
#pragma unroll
			for (uint32_t i = 0; i < kSmallItems; i++)
				if (i < per)
				{
					const uint32_t at = first + 32u * i;
					k[i] = at < n ? keys[at] : 0u;
					v[i] = at < n ? vals[at] : 0u;
				}
			for (int shift = bit_lo; shift < bit_hi; shift += 8)
			{
				const uint32_t mask = (1u << min(8, bit_hi - shift)) - 1u;
				for (uint32_t d = lane; d < 128u; d += 32u)
					reinterpret_cast<uint32_t*>(S.cnt[warp])[d] = 0u;
				__syncwarp();
				uint32_t rank[kSmallItems];
#pragma unroll
				for (uint32_t i = 0; i < kSmallItems; i++)
				{
					if (i >= per)
						break;
					const bool ok = first + 32u * i < n;
					const uint32_t d = ok ? uint32_t(k[i] >> shift) & mask : 0x100u + lane;
					const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
					uint32_t old = 0;
					if (ok)
						old = S.cnt[warp][d];
					__syncwarp();
					if (ok && (peers & lt) == 0u)
						S.cnt[warp][d] = uint16_t(old + __popc(peers));
					__syncwarp();
					rank[i] = old + __popc(peers & lt);
				}
				__syncthreads();
				uint32_t total = 0;
				if (tid < 256u)
				{
					uint32_t c[NT / 32];
#pragma unroll
					for (uint32_t w = 0; w < NT / 32; w++)
						c[w] = S.cnt[w][tid];
#pragma unroll
					for (uint32_t w = 0; w < NT / 32; w++)
					{
						S.cnt[w][tid] = uint16_t(total);
						total += c[w];
					}
				}
				const uint32_t start = scan256(total, S.warp_sum);
				if (tid < 256u)
					S.start[tid] = start;
				__syncthreads();
#pragma unroll
				for (uint32_t i = 0; i < kSmallItems; i++)
					if (i < per && first + 32u * i < n)
					{
						const uint32_t d = uint32_t(k[i] >> shift) & mask;
						const uint32_t at = S.start[d] + S.cnt[warp][d] + rank[i];
						S.keys[at] = k[i];
						S.vals[at] = v[i];
					}
				__syncthreads();
#pragma unroll
				for (uint32_t i = 0; i < kSmallItems; i++)
				{
					const uint32_t at = first + 32u * i;
					if (i < per && at < n)
					{
						k[i] = S.keys[at];
						v[i] = S.vals[at];
					}
				}
			}
#pragma unroll
			for (uint32_t i = 0; i < kSmallItems; i++)
			{
				const uint32_t at = first + 32u * i;
				if (i < per && at < n)
				{
					keys[at] = k[i];
					vals[at] = v[i];
				}
			}
		}

		// ---- onesweep
		constexpr uint32_t kSweepThreads = 256, kSweepItems = 12, kSweepTile = kSweepThreads * kSweepItems, kSweepWarps = 8, kMaxPasses = 8;
		// scratch words: digit counts [kMaxPasses][256], tickets [64], look-back words [passes][tiles][256]
		constexpr uint32_t kSweepHead = kMaxPasses * 256u + 64u;
		constexpr uint32_t kAggregate = 0x40000000u, kInclusive = 0x80000000u, kCountMask = 0x3FFFFFFFu;
		constexpr uint32_t kMaxPolls = 1u << 24;
		constexpr int kLookBack = 8; // tiles looked up at a time (32: the same time)

		// every pass's digit counts, and the look-back words cleared
		__global__ void __launch_bounds__(256) radix_count_kernel(const uint64_t* __restrict__ keys, uint32_t n, int bit_lo, int bit_hi,
			uint32_t* __restrict__ hist, uint32_t* __restrict__ status, uint64_t status_words)
		{
			__shared__ uint32_t h[kMaxPasses][256];
			const int passes = (bit_hi - bit_lo + 7) / 8;
			for (int p = 0; p < passes; p++)
				h[p][threadIdx.x] = 0u;
			const uint64_t id = uint64_t(blockIdx.x) * 256u + threadIdx.x, step = uint64_t(gridDim.x) * 256u;
			for (uint64_t i = id; i < status_words; i += step)
				status[i] = 0u;
			__syncthreads();
			const uint32_t lane = threadIdx.x & 31u;
			for (uint64_t i0 = id - lane; i0 < n; i0 += step) // whole warps
			{
				const bool ok = i0 + lane < n;
				const uint64_t k = ok ? keys[i0 + lane] : 0u;
				const uint32_t live = __ballot_sync(0xFFFFFFFFu, ok);
				for (int p = 0; p < passes; p++)
				{
					const int shift = bit_lo + 8 * p;
					const uint32_t mask = (1u << min(8, bit_hi - shift)) - 1u;
					const uint32_t d = uint32_t(k >> shift) & mask;
					// neighbouring keys often share their high digits: one add for the warp then
					const uint32_t d0 = __shfl_sync(0xFFFFFFFFu, d, 0);
					if (__all_sync(0xFFFFFFFFu, !ok || d == d0))
					{
						if (lane == 0)
							atomicAdd(&h[p][d0], uint32_t(__popc(live)));
					}
					else if (ok)
						atomicAdd(&h[p][d], 1u);
				}
			}
			__syncthreads();
			for (int p = 0; p < passes; p++)
				if (h[p][threadIdx.x])
					atomicAdd(hist + 256 * p + threadIdx.x, h[p][threadIdx.x]);
		}

		__global__ void __launch_bounds__(kSweepThreads, 3) radix_sweep_kernel(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
			uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n, int shift, uint32_t mask,
			const uint32_t* __restrict__ hist, uint32_t* __restrict__ ticket, uint32_t* __restrict__ status, uint32_t* __restrict__ dev_err)
		{
			__shared__ uint64_t s_keys[kSweepTile];
			__shared__ uint32_t s_vals[kSweepTile];
			__shared__ uint16_t s_cnt[kSweepWarps][256];
			__shared__ uint32_t s_start[256]; // of each digit in the tile
			__shared__ uint32_t s_base[256];  // global position of a digit's keys, less s_start
			__shared__ uint32_t s_sum[2][8];
			__shared__ uint32_t s_tile;
			const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
			const uint32_t lt = (1u << lane) - 1u;
			// tiles in the order the blocks start, so every earlier tile is running or done
			if (tid == 0)
				s_tile = atomicAdd(ticket, 1u);
			for (uint32_t d = lane; d < 128u; d += 32u)
				reinterpret_cast<uint32_t*>(s_cnt[warp])[d] = 0u;
			__syncthreads();
			const uint32_t tile = s_tile;
			const uint32_t begin = tile * kSweepTile;
			if (begin >= n)
				return;
			const uint32_t count = min(kSweepTile, n - begin);
			const uint32_t first = warp * 32u * kSweepItems + lane;
			uint64_t k[kSweepItems];
			uint32_t v[kSweepItems];
			uint16_t rank[kSweepItems];
#pragma unroll
			for (uint32_t i = 0; i < kSweepItems; i++)
			{
				const uint32_t at = first + 32u * i;
				k[i] = at < count ? keys_in[begin + at] : 0u;
				v[i] = at < count ? vals_in[begin + at] : 0u;
			}
#pragma unroll
			for (uint32_t i = 0; i < kSweepItems; i++)
			{
				const bool ok = first + 32u * i < count;
				const uint32_t d = ok ? uint32_t(k[i] >> shift) & mask : 0x100u + lane;
				const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
				uint32_t old = 0;
				if (ok)
					old = s_cnt[warp][d];
				__syncwarp();
				if (ok && (peers & lt) == 0u)
					s_cnt[warp][d] = uint16_t(old + __popc(peers));
				__syncwarp();
				rank[i] = uint16_t(old + __popc(peers & lt));
			}
			__syncthreads();
			// thread d: digit d
			uint32_t total = 0;
#pragma unroll
			for (uint32_t w = 0; w < kSweepWarps; w++)
			{
				const uint32_t t = s_cnt[w][tid];
				s_cnt[w][tid] = uint16_t(total);
				total += t;
			}
			volatile uint32_t* st = status + size_t(tile) * 256u + tid;
			*st = (tile == 0 ? kInclusive : kAggregate) | total;
			const uint32_t start = scan256(total, s_sum[0]);
			const uint32_t base = scan256(hist[tid], s_sum[1]);
			s_start[tid] = start;
			__syncthreads();
#pragma unroll
			for (uint32_t i = 0; i < kSweepItems; i++)
				if (first + 32u * i < count)
				{
					const uint32_t d = uint32_t(k[i] >> shift) & mask;
					const uint32_t at = s_start[d] + s_cnt[warp][d] + rank[i];
					s_keys[at] = k[i];
					s_vals[at] = v[i];
				}
			// look back over the earlier tiles' counts of the digit
			uint32_t before = 0, polls = 0;
			int64_t t = int64_t(tile) - 1;
			bool done = tile == 0;
			while (!done)
			{
				// (the first wave's tiles find no total but tile 0's and walk back to it)
				uint32_t w[kLookBack];
#pragma unroll
				for (int j = 0; j < kLookBack; j++)
					w[j] = t - j >= 0 ? *(volatile uint32_t*)(status + size_t(t - j) * 256u + tid) : uint32_t(kInclusive);
#pragma unroll
				for (int j = 0; j < kLookBack; j++)
				{
					if (done || w[j] == 0u)
						break;
					before += w[j] & kCountMask;
					t--;
					done = (w[j] & kInclusive) != 0u;
				}
				if (++polls > kMaxPolls)
				{
					atomicOr(dev_err, U26_DEVERR_ITERATION_CAP);
					done = true;
				}
			}
			if (tile != 0)
				*st = kInclusive | (before + total);
			s_base[tid] = base + before - start;
			__syncthreads();
			for (uint32_t j = tid; j < count; j += kSweepThreads)
			{
				const uint64_t key = s_keys[j];
				const uint32_t at = s_base[uint32_t(key >> shift) & mask] + j;
				if (at < n)
				{
					keys_out[at] = key;
					vals_out[at] = s_vals[j];
				}
			}
		}
	} // namespace

	// Exclusive scan of v[0, n) in place; tmp holds ceil(n / 8192) + 1 words of scratch. The
	// segment sums are scanned recursively, so any n that fits the words works.
	u26_status device_exclusive_scan(u26_ctx* ctx, uint32_t* v, uint32_t n, DevBuf& tmp)
	{
		if (n == 0)
			return U26_OK;
		const uint32_t segs = div_up(n, kScanSeg);
		if (segs == 1)
		{
			scan_down_kernel<<<1, kScanThreads, 0, ctx->stream>>>(v, n, nullptr);
			return after_launch(ctx, "scan_down_kernel");
		}
		// scratch for every recursion level: segs + segs/8192 + ... words, 4-word aligned
		size_t words = 0;
		for (uint32_t m = segs; m > 1; m = div_up(m, kScanSeg))
			words += (m + 3u) & ~3u;
		U26_CUDA(ctx, tmp.reserve(sizeof(uint32_t) * (words + 4)));
		uint32_t* sums = tmp.as<uint32_t>();
		std::vector<std::pair<uint32_t*, uint32_t>> levels; // (array, length) from v upwards
		levels.emplace_back(v, n);
		uint32_t* cur = sums;
		for (uint32_t m = n; div_up(m, kScanSeg) > 1;)
		{
			const uint32_t k = div_up(m, kScanSeg);
			scan_reduce_kernel<<<k, kScanThreads, 0, ctx->stream>>>(levels.back().first, m, cur);
			U26_TRY(after_launch(ctx, "scan_reduce_kernel"));
			levels.emplace_back(cur, k);
			cur += (k + 3u) & ~3u;
			m = k;
		}
		// the top level fits one segment
		scan_down_kernel<<<1, kScanThreads, 0, ctx->stream>>>(levels.back().first, levels.back().second, nullptr);
		U26_TRY(after_launch(ctx, "scan_down_kernel"));
		for (size_t l = levels.size() - 1; l > 0; l--)
		{
			const uint32_t m = levels[l - 1].second;
			scan_down_kernel<<<div_up(m, kScanSeg), kScanThreads, 0, ctx->stream>>>(levels[l - 1].first, m, levels[l].first);
			U26_TRY(after_launch(ctx, "scan_down_kernel"));
		}
		return U26_OK;
	}

	// Three launches per digit. scan_tmp: scratch of the multi-block scan; null: the count table is scanned by one
	// block, without allocating.
	static u26_status sort_three_launches(u26_ctx* ctx, uint64_t* keys, uint32_t* vals, uint32_t n, int bit_lo, int bit_hi, uint64_t* keys_alt,
		uint32_t* vals_alt, uint32_t* counts, DevBuf* scan_tmp)
	{
		const uint32_t num_tiles = div_up(n, kTile);
		uint64_t* k_src = keys;
		uint32_t* v_src = vals;
		uint64_t* k_dst = keys_alt;
		uint32_t* v_dst = vals_alt;
		for (int shift = bit_lo; shift < bit_hi; shift += 8)
		{
			const int bits = min(8, bit_hi - shift);
			const uint32_t mask = (1u << bits) - 1u;
			radix_hist_kernel<<<num_tiles, kThreads, 0, ctx->stream>>>(k_src, n, shift, mask, counts, num_tiles);
			U26_TRY(after_launch(ctx, "radix_hist_kernel"));
			if (scan_tmp)
				U26_TRY(device_exclusive_scan(ctx, counts, 256u * num_tiles, *scan_tmp));
			else
			{
				radix_scan_kernel<<<1, 1024, 0, ctx->stream>>>(counts, 256u * num_tiles);
				U26_TRY(after_launch(ctx, "radix_scan_kernel"));
			}
			radix_scatter_kernel<<<num_tiles, kThreads, 0, ctx->stream>>>(k_src, v_src, k_dst, v_dst, n, shift, mask, counts, num_tiles);
			U26_TRY(after_launch(ctx, "radix_scatter_kernel"));
			std::swap(k_src, k_dst);
			std::swap(v_src, v_dst);
		}
		if (k_src != keys)
		{
			U26_CUDA(ctx, cudaMemcpyAsync(keys, k_src, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, ctx->stream));
			U26_CUDA(ctx, cudaMemcpyAsync(vals, v_src, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, ctx->stream));
		}
		return U26_OK;
	}

	u26_status RadixSorter::sort(u26_ctx* ctx, uint64_t* keys, uint32_t* vals, uint32_t n, int bit_lo, int bit_hi)
	{
		if (n <= 1 || bit_hi <= bit_lo)
			return U26_OK;
		if (n <= kSmall)
		{
			// one block
			if (n <= kSmallFew)
				radix_small_kernel<256><<<1, 256, sizeof(SmallSort<256>), ctx->stream>>>(keys, vals, n, bit_lo, bit_hi);
			else
			{
				if (!ctx->sized_sort.load(std::memory_order_acquire))
				{
					U26_CUDA(ctx, cudaFuncSetAttribute(radix_small_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(SmallSort<1024>))));
					ctx->sized_sort.store(true, std::memory_order_release);
				}
				radix_small_kernel<1024><<<1, 1024, sizeof(SmallSort<1024>), ctx->stream>>>(keys, vals, n, bit_lo, bit_hi);
			}
			return after_launch(ctx, "radix_small_kernel");
		}
		U26_CUDA(ctx, keys_alt.reserve(sizeof(uint64_t) * n));
		U26_CUDA(ctx, vals_alt.reserve(sizeof(uint32_t) * n));
		const uint32_t passes = uint32_t(bit_hi - bit_lo + 7) / 8u;
		if (n >= kAggregate || passes > kMaxPasses)
		{
			U26_CUDA(ctx, counts.reserve(sizeof(uint32_t) * 256u * div_up(n, kTile)));
			return sort_three_launches(ctx, keys, vals, n, bit_lo, bit_hi, keys_alt.as<uint64_t>(), vals_alt.as<uint32_t>(),
				counts.as<uint32_t>(), &scan_tmp);
		}
		const uint32_t tiles = div_up(n, kSweepTile);
		const uint64_t words = uint64_t(passes) * tiles * 256u;
		U26_CUDA(ctx, counts.reserve(sizeof(uint32_t) * (kSweepHead + words)));
		uint32_t* hist = counts.as<uint32_t>();
		uint32_t* ticket = hist + kMaxPasses * 256u;
		uint32_t* status = hist + kSweepHead;
		U26_CUDA(ctx, cudaMemsetAsync(hist, 0, sizeof(uint32_t) * kSweepHead, ctx->stream));
		radix_count_kernel<<<std::min(div_up(n, 2048), 148u * 8u), 256, 0, ctx->stream>>>(keys, n, bit_lo, bit_hi, hist, status, words);
		U26_TRY(after_launch(ctx, "radix_count_kernel"));
		uint64_t* k_src = keys;
		uint32_t* v_src = vals;
		uint64_t* k_dst = keys_alt.as<uint64_t>();
		uint32_t* v_dst = vals_alt.as<uint32_t>();
		for (uint32_t p = 0; p < passes; p++)
		{
			const int shift = bit_lo + 8 * int(p);
			radix_sweep_kernel<<<tiles, kSweepThreads, 0, ctx->stream>>>(k_src, v_src, k_dst, v_dst, n, shift,
				(1u << std::min(8, bit_hi - shift)) - 1u, hist + 256u * p, ticket + p, status + size_t(p) * tiles * 256u, ctx->dev_err);
			U26_TRY(after_launch(ctx, "radix_sweep_kernel"));
			std::swap(k_src, k_dst);
			std::swap(v_src, v_dst);
		}
		if (k_src != keys)
		{
			U26_CUDA(ctx, cudaMemcpyAsync(keys, k_src, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, ctx->stream));
			U26_CUDA(ctx, cudaMemcpyAsync(vals, v_src, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, ctx->stream));
		}
		return U26_OK;
	}

	u26_status RadixSorter::sort_into(u26_ctx* ctx, uint64_t* keys, uint32_t* vals, uint32_t n, int bit_lo, int bit_hi,
		uint64_t* keys_alt, uint32_t* vals_alt, uint32_t* counts)
	{
		if (n <= 1 || bit_hi <= bit_lo)
			return U26_OK;
		return sort_three_launches(ctx, keys, vals, n, bit_lo, bit_hi, keys_alt, vals_alt, counts, nullptr);
	}
} // namespace u26
