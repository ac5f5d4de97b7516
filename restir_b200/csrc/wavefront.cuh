// Wavefront ray queues: a persistent traversal kernel that keeps every lane
// of a warp busy.
//
// A producer pass appends rays to a queue in global memory (a warp's lanes
// take consecutive slots: one __ballot_sync, one atomicAdd per warp). The
// tracer below runs one resident grid; each lane holds one ray (warptrace.cuh),
// and lanes whose rays have ended take the next unclaimed ones. Lanes therefore
// stay in the same traversal loop instead of idling behind the longest ray of
// their warp.
#pragma once

#include "warptrace.cuh"

namespace restir
{

// Queue layout: rays[2 * i] = (origin, tmax), rays[2 * i + 1] = (direction, 0)
// (restir_trace's ray format); results hitTriangle[i], hitDistance[i].
struct RayQueue
{
	float4* rays;
	int* hitTriangle;
	float* hitDistance;
	uint32_t* count;    // rays appended by the producer; null: capacity rays
	uint32_t* claimed;  // rays taken by the tracer; next to it, rays looked through by the re-walk
	uint32_t capacity;
};

// Appends this lane's ray when push is set; every lane of the warp must call
// it (it votes). Returns the slot, or -1.
__device__ __forceinline__ int queuePush(const RayQueue& q, bool push, V3 origin, float tmax, V3 direction)
{
	const unsigned lane = threadIdx.x & 31u;
	const unsigned mask = __ballot_sync(0xffffffffu, push);
	const int leader = mask != 0u ? __ffs(mask) - 1 : 0;
	uint32_t base = 0;
	if (mask != 0u && int(lane) == leader)
	{
		base = atomicAdd(q.count, uint32_t(__popc(mask)));
	}
	base = __shfl_sync(0xffffffffu, base, leader);
	if (!push)
	{
		return -1;
	}
	const uint32_t slot = base + uint32_t(__popc(mask & ((1u << lane) - 1u)));
	if (slot >= q.capacity)
	{
		raiseStatus(4u);
		return -1;
	}
	q.rays[2 * slot] = make_float4(origin.x, origin.y, origin.z, tmax);
	q.rays[2 * slot + 1] = make_float4(direction.x, direction.y, direction.z, 0.0f);
	return int(slot);
}

__device__ __forceinline__ uint32_t queuedRays(const RayQueue& q)
{
	return q.count != nullptr ? min(*q.count, q.capacity) : q.capacity;
}

// Rays and hits in restir_trace's layout.
struct RayArrays
{
	const float4* rays;
	int* hitTriangle;
	float* hitDistance;

	__device__ __forceinline__ void load(uint32_t i, Ray& r) const
	{
		const float4 a = rays[2 * size_t(i)];
		const float4 c = rays[2 * size_t(i) + 1];
		r.o = v3(a.x, a.y, a.z);
		r.d = v3(c.x, c.y, c.z);
		r.distance = a.w;
		r.hit = -1;
		r.index = i;
	}
	__device__ __forceinline__ void store(const Ray& r) const
	{
		hitTriangle[r.index] = r.hit;
		hitDistance[r.index] = r.distance;
	}
};

// A queue as a source: one atomicAdd per warp claims rays for all takers.
template<int kKind, int kLanes>
struct QueueSource
{
	static constexpr int kCount = kKind;
	const RayQueue& q;
	RayArrays arrays;
	uint32_t total;

	__device__ __forceinline__ explicit QueueSource(const RayQueue& queue)
		: q(queue), arrays{ queue.rays, queue.hitTriangle, queue.hitDistance }, total(queuedRays(queue))
	{
	}
	__device__ __forceinline__ void take(bool idle, bool& more, Ray& r) const
	{
		const unsigned mask = idleMask<kLanes>(idle);
		const uint32_t wanted = uint32_t(__popc(mask));
		uint32_t start = 0;
		if ((threadIdx.x & 31u) == 0u)
		{
			start = atomicAdd(q.claimed, wanted);
		}
		start = __shfl_sync(0xffffffffu, start, 0);
		more = start < total && total - start > wanted;
		const uint32_t mine = start + uint32_t(idleRank<kLanes>(mask));
		if (idle && mine >= start && mine < total)
		{
			arrays.load(mine, r);
		}
	}
	__device__ __forceinline__ void store(const Ray& r) const { arrays.store(r); }
};

// The marked rays (markedHit) among the first `end` of a ray set: a source for
// the walks. The warp looks through 32 consecutive rays at a time, the next
// ones no warp has claimed (claimed), or the next of its own part (null).
template<int kLanes>
struct MarkedSource
{
	static constexpr int kCount = -1;
	RayArrays arrays;
	uint32_t next, end;
	uint32_t* claimed;
	uint32_t base = 0u;
	unsigned pending = 0u; // marked rays from base on

	__device__ __forceinline__ void take(bool idle, bool& more, Ray& r)
	{
		const unsigned lane = threadIdx.x & 31u;
		unsigned mask = idleMask<kLanes>(idle);
		while (mask != 0u)
		{
			if (pending == 0u)
			{
				base = next;
				if (claimed != nullptr)
				{
					if (lane == 0u)
					{
						base = atomicAdd(claimed, 32u);
					}
					base = __shfl_sync(0xffffffffu, base, 0);
				}
				if (base >= end)
				{
					more = false;
					break;
				}
				next = base + min(32u, end - base);
				const uint32_t i = base + lane;
				pending = __ballot_sync(0xffffffffu, lane < end - base && arrays.hitTriangle[i] < -1);
				continue;
			}
			// The first idle group takes the first marked ray.
			if ((lane & ~unsigned(kLanes - 1)) == unsigned(__ffs(mask) - 1))
			{
				const uint32_t i = base + uint32_t(__ffs(pending) - 1);
				arrays.load(i, r);
				r.hit = markedHit(arrays.hitTriangle[i]);
				r.distance = arrays.hitDistance[i];
			}
			mask &= mask - 1u;
			pending &= pending - 1u;
		}
	}
	__device__ __forceinline__ void store(const Ray& r) const { arrays.store(r); }
};

// The persistent tracers over a queue, for grids of whole warps. Nearest hits
// take two launches: queueNearest marks the rays whose short stack dropped
// entries, queueRewalk finishes those. queueWalk traces nearest hits by the
// stackless walk alone (the fragment-shader passes).
template<bool kWide>
__device__ __forceinline__ void queueNearest(const BvhView& b, const RayQueue& q, NearestStorage* storage)
{
	QueueSource<RESTIR_COUNT_CLOSEST, 1> source(q);
	traceNearest<kWide>(b, source, storage[threadIdx.x >> 5]);
}

template<bool kWide>
__device__ __forceinline__ void queueRewalk(const BvhView& b, const RayQueue& q, LeafSlots* slots)
{
	MarkedSource<1> source{ { q.rays, q.hitTriangle, q.hitDistance }, 0u, queuedRays(q), q.claimed + 1 };
	traceLaneWalks<false, kWide>(b, source, slots[threadIdx.x >> 5]);
}

template<bool kWide, int kLanes>
__device__ __forceinline__ void queueWalk(const BvhView& b, const RayQueue& q, LeafSlots* slots)
{
	QueueSource<RESTIR_COUNT_ANY, kLanes> source(q);
	if constexpr (kLanes == 1)
	{
		traceLaneWalks<false, kWide>(b, source, slots[threadIdx.x >> 5]);
	}
	else
	{
		traceGroupWalks<false, kWide>(b, source);
	}
}

} // namespace restir
