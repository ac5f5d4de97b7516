// restir_trace: a fixed ray set through the BVH (bvh.sh:298-319). Each warp
// takes a part of the set (warptrace.cuh), with a ray per lane or per group of
// four lanes, or each thread one ray, by the size of the set and the scene; the
// lock-step and the watertight walks run one thread per ray.
// RESTIR_TRACE_CLOSEST_QUEUE always takes the parts, whose warps run the queue
// tracer's loop. Nothing is allocated: a warp's part is its queue.
#include "bvh.cuh"
#include "wavefront.cuh"
#include "watertight.cuh"

namespace restir
{
namespace
{

constexpr int kTraceBlock = 128;

// Which kernel traces a ray set, by its size n and the scene's nodes. Measured
// on random rays, 43 to 1.9M nodes, n 1 to 1M (us; 4: four lanes a ray, 1: one
// thread a ray, w: a warp's part, leaves tested together):
//   any hit, city of 1.9M nodes, n 1,000: 4 47, 1 81, w 87; 64,000: 4 127, 1 142,
//     w 127; 300,000: 4 250, 1 214, w 196; Cornell box, 16,000: 4 15, 1 21, w 23;
//     64,000: 4 23, 1 21, w 18; 500,000: 4 87, 1 60, w 53;
//   stackless, city of 47k nodes, 64,000: 4 158, 1 148, w 156; 200,000: 4 293,
//     1 251, w 263; of 1.9M, 1,000,000: 1 3,762, w 2,502; Cornell box, 300,000:
//     1 49, w 56; 500,000: 1 73, w 73;
//   closest (1r: one thread a ray, its re-walk by four lanes), city of 1.9M nodes,
//     1: 1 70, w 89; 1,000: 1 268, w 225; 1,000,000: 1 2,325, w 1,813; of 190k, 32:
//     1 101, w 115; 200,000: 1 396, w 410; of 47k, 16,000: 1 60, 1r 68, w 74;
//     300,000: 1 159, 1r 175, w 180; 500,000: 1 216, w 215; courtyard of 40k nodes,
//     16,000: 1 332, 1r 268, w 266; 300,000: 1 488, 1r 483, w 457; 1,000,000:
//     Cornell box 1 134, w 157; 3.9k nodes 1 403, w 403; 10k (city) 1 220, w 228,
//     (courtyard) 1 776, w 670.
// So walks take four lanes up to a group of them for each ray that the SMs hold
// at once (148 x 32 warps x 8), where they are latency-bound; then any hits take
// the warp's shared leaves, stackless nearest hits one thread each until every
// lane has two rays. Nearest hits take one thread each where a ray visits few
// nodes or the rays are few (below 128, and in scenes of up to 4,096 nodes), and
// past one ray a lane, where the parts' last warps leave the SMs idle; in scenes
// of up to 131,072 nodes with a lane for every ray the four-lane re-walk is the
// middle between the courtyard's long walks and the city's short ones.
constexpr uint32_t kResidentLanes = 148u * 32u * 32u;
constexpr uint32_t kFourLaneRays = kResidentLanes / 4u;
constexpr uint32_t kFewRays = 128u;
constexpr int kSmallScene = 4096;
constexpr int kMiddleScene = 131072;

enum class Nearest
{
	thread,
	threadGroupRewalk,
	part
};

Nearest nearestKernel(uint32_t n, int nodes)
{
	if (n < kFewRays || nodes <= kSmallScene)
	{
		return Nearest::thread;
	}
	if (nodes <= kMiddleScene && n <= kResidentLanes)
	{
		return Nearest::threadGroupRewalk;
	}
	const bool thread = n > kResidentLanes && n <= (nodes <= kMiddleScene ? 3u * kResidentLanes : kResidentLanes + kResidentLanes / 2u);
	return thread ? Nearest::thread : Nearest::part;
}

// A contiguous part of the ray set, one per warp: its lanes take the part's
// rays as theirs end, without an atomic.
template<int kKind, int kLanes>
struct PartSource
{
	static constexpr int kCount = kKind;
	RayArrays arrays;
	uint32_t next, end;

	__device__ __forceinline__ void take(bool idle, bool& more, Ray& r)
	{
		const unsigned mask = idleMask<kLanes>(idle);
		const uint32_t wanted = uint32_t(__popc(mask));
		const uint32_t left = end - next;
		const uint32_t rank = uint32_t(idleRank<kLanes>(mask));
		if (idle && rank < left)
		{
			arrays.load(next + rank, r);
		}
		next += min(wanted, left);
		more = left > wanted;
	}
	__device__ __forceinline__ void store(const Ray& r) const { arrays.store(r); }
};

__device__ __forceinline__ bool warpPart(uint32_t n, uint32_t part, uint32_t& first, uint32_t& end)
{
	const uint64_t at = (uint64_t(blockIdx.x) * (kTraceBlock / 32) + (threadIdx.x >> 5)) * part;
	first = uint32_t(at);
	end = uint32_t(min(at + part, uint64_t(n)));
	return at < n;
}

template<bool kWide>
__global__ void __launch_bounds__(kTraceBlock, 8) nearestPartsKernel(BvhView bvh, RayArrays arrays, uint32_t n, uint32_t part)
{
	__shared__ NearestStorage storage[kTraceBlock / 32];
	uint32_t first, end;
	if (!warpPart(n, part, first, end))
	{
		return; // whole warp
	}
	PartSource<RESTIR_COUNT_CLOSEST, 1> source{ arrays, first, end };
	traceNearest<kWide>(bvh, source, storage[threadIdx.x >> 5]);
	__syncwarp(); // the warp's stores
	MarkedSource<4> marked{ arrays, first, end, nullptr };
	traceGroupWalks<false, kWide>(bvh, marked);
}

// One thread per ray, and the rays whose short stack dropped entries by four
// lanes each afterwards: the re-walk is the longest part of such a ray, and in
// one thread it holds up its warp.
template<bool kWide>
__global__ void __launch_bounds__(kTraceBlock) nearestThreadsKernel(BvhView bvh, RayArrays arrays, uint32_t n)
{
	__shared__ int stack[kBvhShortStack * kTraceBlock];
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	const uint32_t first = i & ~31u;
	if (first >= n)
	{
		return; // whole warp
	}
	if (i < n)
	{
		Ray r;
		arrays.load(i, r);
		if (bvh.available())
		{
			TraceWork work;
			bool dropped;
			r.hit = walkShortStack(bvh, r.o, r.d, r.distance, stack + threadIdx.x, kTraceBlock, work, dropped);
			countWork(RESTIR_COUNT_CLOSEST, work.nodes, work.triangles);
			r.hit = dropped ? markedHit(r.hit) : r.hit;
		}
		arrays.store(r);
	}
	__syncwarp(); // the warp's stores
	MarkedSource<4> marked{ arrays, first, n - first > 32u ? first + 32u : n, nullptr };
	traceGroupWalks<false, kWide>(bvh, marked);
}

template<bool kAny, bool kWide, int kLanes>
__global__ void __launch_bounds__(kTraceBlock, 8) walkPartsKernel(BvhView bvh, RayArrays arrays, uint32_t n, uint32_t part)
{
	__shared__ LeafSlots slots[kLanes == 1 ? kTraceBlock / 32 : 1];
	uint32_t first, end;
	if (!warpPart(n, part, first, end))
	{
		return; // whole warp
	}
	PartSource<RESTIR_COUNT_ANY, kLanes> source{ arrays, first, end };
	if constexpr (kLanes == 1)
	{
		traceLaneWalks<kAny, kWide>(bvh, source, slots[threadIdx.x >> 5]);
	}
	else
	{
		traceGroupWalks<kAny, kWide>(bvh, source);
	}
}

// One thread per ray, a kernel per kind (each fetches its own kind's code only:
// 1,000 nearest hits in the Cornell box take 17 us against 21 us in one kernel
// for all kinds).
template<int kKind, bool kWide = false>
__global__ void __launch_bounds__(kTraceBlock) traceKernel(BvhView bvh, RayArrays arrays, uint32_t n)
{
	__shared__ int stack[kKind == RESTIR_TRACE_CLOSEST ? kBvhShortStack * kTraceBlock : 1];
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
	{
		return;
	}
	Ray r;
	arrays.load(i, r);
	const float length = r.distance;
	if (kKind == RESTIR_TRACE_CLOSEST)
	{
		r.hit = traceBvh(bvh, r.o, r.d, length, false, r.distance, stack + threadIdx.x, kTraceBlock);
	}
	else if (kKind == RESTIR_TRACE_CLOSEST_STACKLESS)
	{
		r.hit = traceBvh(bvh, r.o, r.d, length, false, r.distance, nullptr, 0);
	}
	else if (kKind == RESTIR_TRACE_ANY_WAVE)
	{
		r.hit = traceVisibility<true>(bvh, r.o, r.d, length, r.distance);
	}
	else
	{
		r.hit = traceWatertight<kWide>(bvh, r.o, r.d, r.distance);
	}
	arrays.store(r);
}

uint32_t threadBlocks(uint32_t n)
{
	return uint32_t((uint64_t(n) + kTraceBlock - 1) / kTraceBlock);
}

template<int kKind, bool kWide = false>
void launchThreads(const BvhView& bvh, const RayArrays& arrays, uint32_t n, cudaStream_t s)
{
	traceKernel<kKind, kWide><<<threadBlocks(n), kTraceBlock, 0, s>>>(bvh, arrays, n);
}

// Rays per warp: as few as fill the SMs once (148 x 32 warps resident), a
// multiple of the lanes' or groups' number, then four times that, so that
// lanes whose rays end early have more to take.
uint32_t partOf(uint32_t n, uint32_t takers)
{
	return n > kResidentLanes / 32u * takers ? 4u * takers : takers;
}

uint32_t partBlocks(uint32_t n, uint32_t part)
{
	const uint64_t warps = (uint64_t(n) + part - 1u) / part;
	return uint32_t((warps + kTraceBlock / 32 - 1) / (kTraceBlock / 32));
}

template<bool kAny, bool kWide>
void launchWalks(const BvhView& bvh, const RayArrays& arrays, uint32_t n, cudaStream_t s)
{
	if (n <= kFourLaneRays)
	{
		const uint32_t part = partOf(n, 8u);
		walkPartsKernel<kAny, kWide, 4><<<partBlocks(n, part), kTraceBlock, 0, s>>>(bvh, arrays, n, part);
	}
	else
	{
		const uint32_t part = partOf(n, 32u);
		walkPartsKernel<kAny, kWide, 1><<<partBlocks(n, part), kTraceBlock, 0, s>>>(bvh, arrays, n, part);
	}
}

template<bool kWide>
void launchParts(const BvhView& bvh, const RayArrays& arrays, uint32_t n, int kind, cudaStream_t s)
{
	if (kind == RESTIR_TRACE_CLOSEST || kind == RESTIR_TRACE_CLOSEST_QUEUE)
	{
		const uint32_t part = partOf(n, 32u);
		nearestPartsKernel<kWide><<<partBlocks(n, part), kTraceBlock, 0, s>>>(bvh, arrays, n, part);
	}
	else if (kind == RESTIR_TRACE_ANY)
	{
		launchWalks<true, kWide>(bvh, arrays, n, s);
	}
	else
	{
		launchWalks<false, kWide>(bvh, arrays, n, s);
	}
}

} // namespace
} // namespace restir

using namespace restir;

extern "C" int restir_bvh_wide_rows(const RestirScene* scene)
{
	return scene != nullptr && wideRows(makeBvhView(scene)) ? 1 : 0;
}

extern "C" int restir_trace(const RestirParams* params, const RestirScene* scene, const float* rays,
	int32_t* hit_triangle, float* hit_distance, uint32_t n, int kind, void* stream)
{
	(void)params;
	if (scene == nullptr || rays == nullptr || hit_triangle == nullptr || hit_distance == nullptr
		|| kind < RESTIR_TRACE_CLOSEST || kind > RESTIR_TRACE_ANY_WAVE)
	{
		return RESTIR_ERROR_INVALID_ARGUMENT;
	}
	if (n == 0u)
	{
		return RESTIR_OK;
	}
	BvhView bvh = makeBvhView(scene);
	cudaStream_t s = asStream(stream);
	const RayArrays arrays = { reinterpret_cast<const float4*>(rays), hit_triangle, hit_distance };
	const Nearest nearest = nearestKernel(n, bvh.nodeCount);
	if (kind == RESTIR_TRACE_ANY_WAVE)
	{
		launchThreads<RESTIR_TRACE_ANY_WAVE>(bvh, arrays, n, s);
	}
	else if (kind == RESTIR_TRACE_CLOSEST_WATERTIGHT)
	{
		if (wideRows(bvh))
		{
			launchThreads<RESTIR_TRACE_CLOSEST_WATERTIGHT, true>(bvh, arrays, n, s);
		}
		else
		{
			launchThreads<RESTIR_TRACE_CLOSEST_WATERTIGHT>(bvh, arrays, n, s);
		}
	}
	else if (kind == RESTIR_TRACE_CLOSEST && nearest == Nearest::thread)
	{
		launchThreads<RESTIR_TRACE_CLOSEST>(bvh, arrays, n, s);
	}
	else if (kind == RESTIR_TRACE_CLOSEST && nearest == Nearest::threadGroupRewalk)
	{
		(wideRows(bvh) ? nearestThreadsKernel<true> : nearestThreadsKernel<false>)<<<threadBlocks(n), kTraceBlock, 0, s>>>(bvh, arrays, n);
	}
	else if ((kind == RESTIR_TRACE_CLOSEST_STACKLESS && n > kFourLaneRays && n <= 2u * kResidentLanes)
		|| (bvh.nodeCount == 0 && kind != RESTIR_TRACE_CLOSEST_QUEUE)) // nothing to hit, and no ray to count
	{
		launchThreads<RESTIR_TRACE_CLOSEST_STACKLESS>(bvh, arrays, n, s);
	}
	else if (wideRows(bvh))
	{
		launchParts<true>(bvh, arrays, n, kind, s);
	}
	else
	{
		launchParts<false>(bvh, arrays, n, kind, s);
	}
	return launchStatus();
}
