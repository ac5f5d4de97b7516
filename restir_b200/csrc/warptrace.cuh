// Warp-cooperative BVH traversal. A ray's own sequence of nodes, tests and
// distances is that of bvh.cuh's walks (bvh.sh:140-174, 216-295), so its hit,
// its distance, its step count and the work counted are the same.
//
// A ray of the measured scenes passes into a leaf on 2-6% of its node visits.
// With a ray per lane and leaves tested as they are reached, one or two lanes
// run the triangle tests (200 instructions) after nearly every step while the
// other 30 wait: such walks kept 9 of 32 lanes busy. Here a ray that reaches a
// leaf waits for others, and four lanes test each waiting leaf, one triangle a
// lane.
//
#pragma once

#include "bvh.cuh"

namespace restir
{

// --- leaves --------------------------------------------------------------------

constexpr int kLeafSlots = 8;

// What a waiting lane hands to the four lanes that test its leaf.
struct LeafSlots
{
	float4 origin[kLeafSlots];     // w: first triangle
	float4 direction[kLeafSlots];  // w: number of triangles
	float distance[kLeafSlots];
};

// intersectTriangle (bvh.sh:44-71) without its early returns; t < 0 or NaN for none.
template<bool kWide>
__device__ __forceinline__ float leafTriangle(const BvhView& b, int t, V3 o, V3 d)
{
	const int row = b.triangleOffset + t * 4;
	V3 v0, v1, v2;
	if (kWide && !RESTIR_CHECKS)
	{
		F2 p, q, r, s;
		asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(p), "=l"(q), "=l"(r), "=l"(s) : "l"(b.rows + row));
		float unused;
		unpack2(p, v0.x, v0.y);
		unpack2(q, v0.z, unused);
		unpack2(r, v1.x, v1.y);
		unpack2(s, v1.z, unused);
	}
	else
	{
		v0 = b.row(row).xyz();
		v1 = b.row(row + 1).xyz();
	}
	v2 = b.row(row + 2).xyz();
	const V3 edge1 = v1 - v0;
	const V3 edge2 = v2 - v0;
	const V3 p = cross(d, edge2);
	const float determinant = dot(edge1, p);
	const float inverse = 1.0f / determinant;
	const V3 s = o - v0;
	const float u = dot(s, p) * inverse;
	const V3 q = cross(s, edge1);
	const float v = dot(d, q) * inverse;
	const bool outside = fabsf(determinant) < 1e-12f || u < 0.0f || u > 1.0f || v < 0.0f || u + v > 1.0f;
	return outside ? -1.0f : dot(edge2, q) * inverse;
}

// Tests up to kLeafSlots of the leaves of the lanes that wait for one. Every
// lane of the warp calls it. Returns true on the lanes whose leaf was tested;
// distance and hit are then what testing its triangles one by one leaves
// (intersectLeaf: the nearest below distance, the lower triangle of equals).
template<bool kWide>
__device__ __forceinline__ bool testLeaves(const BvhView& b, LeafSlots& slots, bool waiting, V3 o, V3 d, int first, int count,
	float& distance, int& hit)
{
	const unsigned lane = threadIdx.x & 31u;
	const unsigned mask = __ballot_sync(0xffffffffu, waiting);
	const int rank = __popc(mask & ((1u << lane) - 1u));
	const bool mine = waiting && rank < kLeafSlots;
	if (mine)
	{
		slots.origin[rank] = make_float4(o.x, o.y, o.z, __int_as_float(first));
		slots.direction[rank] = make_float4(d.x, d.y, d.z, __int_as_float(count));
		slots.distance[rank] = distance;
	}
	__syncwarp();
	const int slot = int(lane) >> 2;
	const bool used = slot < __popc(mask);
	V3 so = v3s(0.0f), sd = v3s(0.0f);
	int at = 0, end = 0;
	unsigned best = 0u; // the float's bits order distances, all of them >= 0
	if (used)
	{
		const float4 a = slots.origin[slot];
		const float4 c = slots.direction[slot];
		so = v3(a.x, a.y, a.z);
		sd = v3(c.x, c.y, c.z);
		at = __float_as_int(a.w);
		end = at + __float_as_int(c.w);
		best = __float_as_uint(slots.distance[slot]);
	}
	__syncwarp();
	int base = first;
	// One round for leaves of up to four triangles, nearly all of them.
	do
	{
		const int t = at + int(lane & 3u);
		float h = -1.0f;
		if (t < end)
		{
			h = leafTriangle<kWide>(b, t, so, sd);
		}
		const unsigned key = h > 0.0f && h < __uint_as_float(best) ? __float_as_uint(h) : 0xffffffffu;
		unsigned nearest = min(key, __shfl_xor_sync(0xffffffffu, key, 1));
		nearest = min(nearest, __shfl_xor_sync(0xffffffffu, nearest, 2));
		const unsigned winners = __ballot_sync(0xffffffffu, key == nearest && key != 0xffffffffu);
		const unsigned closer = __shfl_sync(0xffffffffu, nearest, (rank * 4) & 31);
		if (nearest != 0xffffffffu)
		{
			best = nearest;
		}
		const unsigned mineWon = (winners >> ((rank * 4) & 31)) & 15u;
		if (mine && mineWon != 0u)
		{
			distance = __uint_as_float(closer);
			hit = base + __ffs(mineWon) - 1;
		}
		base += 4;
		at += 4;
	} while (__any_sync(0xffffffffu, at < end));
	return mine;
}

// --- rays ----------------------------------------------------------------------
//
// traceNearest, traceLaneWalks and traceGroupWalks trace rays until their source has no more. Every
// lane of the warp calls them. A source gives
//   take(idle, more, r): called by the whole warp; an idle lane (traceGroupWalks:
//     the four lanes of an idle group) gets a ray in r, r.index stays kNoRay when
//     there is none for it, and more is cleared when there are none left;
//   store(r): the ray's hit and distance;
//   kCount: the kind of ray to count (-1: a ray counted before).

// A ray set has up to 2^32 - 1 rays (restir_trace's n), the last index is free.
constexpr uint32_t kNoRay = 0xffffffffu;

struct Ray
{
	V3 o, d;
	float distance;  // the nearest hit's, or the ray's length
	int hit;
	uint32_t index;  // kNoRay: none
};

// The lanes' takers: one per lane (kLanes 1) or one per group of kLanes lanes,
// ranked among the idle ones.
template<int kLanes>
__device__ __forceinline__ unsigned idleMask(bool idle)
{
	return __ballot_sync(0xffffffffu, idle && (threadIdx.x & (kLanes - 1)) == 0u);
}

template<int kLanes>
__device__ __forceinline__ int idleRank(unsigned mask)
{
	const unsigned leader = threadIdx.x & 31u & ~unsigned(kLanes - 1);
	return __popc(mask & ((1u << leader) - 1u));
}

// A hit index that marks a ray whose re-walk is still to come (and the same
// function back): below -1.
__device__ __forceinline__ int markedHit(int hit)
{
	return -3 - hit;
}

// The warp leaves its stepping loop to test leaves and to take new rays when
// this share (1 / n) of the lanes with a ray do not step; it takes new rays
// when so many lanes have none.
#ifndef RESTIR_TRACE_SHARE
#	define RESTIR_TRACE_SHARE 4
#endif
#ifndef RESTIR_TRACE_REFILL
#	define RESTIR_TRACE_REFILL 4
#endif
// Visits between two votes.
#ifndef RESTIR_TRACE_STEPS
#	define RESTIR_TRACE_STEPS 2
#endif

// The warp's shared memory of traceNearest.
struct NearestStorage
{
	LeafSlots leaves;
	uint2 stack[kBvhShortStack][32];
};

// Nearest hits with the short stack (bvh.sh:216-295), a ray per lane. A ray
// whose stack dropped entries is stored marked (markedHit): a walk finishes
// it. In one loop with the short stack, the re-walk would make the two halves
// of a warp wait for each other (18% of random rays in the 1M-triangle city
// drop entries, and their re-walk visits 142 nodes after 53). Bound by the L1's
// rate of 32-byte rows (its data pipe 69% busy on 1M random rays): those take
// 0.81 ms here and 0.84 ms in the re-walk, 2.36 ms in the one-lane state
// machine it replaces (9.4 of 32 lanes active there, 19.4 here); the GI
// candidates of a 1080p frame 0.48 + 0.39 ms, before 1.17 ms.
template<bool kWide, typename Source>
__device__ __forceinline__ void traceNearest(const BvhView& b, Source& source, NearestStorage& storage)
{
	const unsigned lane = threadIdx.x & 31u;
	constexpr unsigned kAll = 0xffffffffu;
	constexpr int kStep = 0, kLeaf = 1, kDone = 2;
	int mode = kDone;
	Ray r = {};
	r.index = kNoRay;
	SlabRay slab = {};
	// The node to visit: (node, -a) of an interior node or (a's bits, b) of a
	// leaf, told apart by the second word's sign, so that a child's words, read
	// with its box, are not read again when it is visited.
	int node = 0;
	float word = 0.0f;
	int step = 0;
	int stackTop = 0, stackCount = 0;
	bool dropped = false;
	int leafVisits = 0;
	uint32_t triangles = 0;
	bool more = true;

	// Goes on to the node in (node, word), unless the visits' cap is reached (bvh.sh:23).
	auto goOn = [&]()
	{
		mode = __float_as_int(word) >= 0 ? kLeaf : kStep;
		if (step >= kBvhMaxSteps)
		{
			reportTruncatedRay();
			mode = kDone;
		}
	};
	auto pop = [&]()
	{
		if (stackCount == 0)
		{
			mode = kDone;
			return;
		}
		--stackTop;
		--stackCount;
		const uint2 e = storage.stack[stackTop & (kBvhShortStack - 1)][lane];
		node = int(e.x);
		word = __uint_as_float(e.y);
		goOn();
	};
	auto visit = [&]()
	{
		const int left = node + 1;
		const int right = int(-word);
		const NodeRow leftRow = loadNode<kWide>(b, left);
		const NodeRow rightRow = loadNode<kWide>(b, right);
		float leftA, leftB, rightA, rightB;
		const float leftDistance = slabEnter(slab, leftRow, r.distance, leftA, leftB);
		const float rightDistance = slabEnter(slab, rightRow, r.distance, rightA, rightB);
		const bool visitLeft = leftDistance >= 0.0f;
		const bool visitRight = rightDistance >= 0.0f;
		const bool leftFirst = leftDistance <= rightDistance;
		const int leftNode = leftB >= 0.0f ? __float_as_int(leftA) : left;
		const float leftWord = leftB >= 0.0f ? leftB : -leftA;
		const int rightNode = rightB >= 0.0f ? __float_as_int(rightA) : right;
		const float rightWord = rightB >= 0.0f ? rightB : -rightA;
		++step;
		if (visitLeft && visitRight)
		{
			storage.stack[stackTop & (kBvhShortStack - 1)][lane] =
				make_uint2(uint32_t(leftFirst ? rightNode : leftNode), __float_as_uint(leftFirst ? rightWord : leftWord));
			++stackTop;
			dropped = dropped || stackCount == kBvhShortStack;
			stackCount = min(stackCount + 1, kBvhShortStack);
		}
		if (visitLeft || visitRight)
		{
			const bool goLeft = visitLeft && visitRight ? leftFirst : visitLeft;
			node = goLeft ? leftNode : rightNode;
			word = goLeft ? leftWord : rightWord;
			goOn();
		}
		else
		{
			pop();
		}
	};

	for (;;)
	{
		// Rays that have ended are stored, and lanes without one take the next.
		const unsigned done = __ballot_sync(kAll, mode == kDone && (r.index != kNoRay || more));
		if (__popc(done) >= RESTIR_TRACE_REFILL || (done != 0u && __all_sync(kAll, mode == kDone)))
		{
			if (mode == kDone && r.index != kNoRay)
			{
				// The root, and both children of each interior node visited.
				countWork(Source::kCount, 1u + 2u * uint32_t(step - leafVisits), triangles);
				r.hit = dropped ? markedHit(r.hit) : r.hit;
				source.store(r);
				r.index = kNoRay;
			}
			if (more)
			{
				const bool idle = r.index == kNoRay;
				source.take(idle, more, r);
				if (idle && r.index != kNoRay)
				{
					slab = slabRay(r.o, r.d);
					step = 0;
					triangles = 0;
					leafVisits = 0;
					stackTop = 0;
					stackCount = 0;
					dropped = false;
					if (b.available())
					{
						float a, w;
						if (slabEnter(slab, loadNode<kWide>(b, 0), r.distance, a, w) >= 0.0f)
						{
							node = w >= 0.0f ? __float_as_int(a) : 0;
							word = w >= 0.0f ? w : -a;
							mode = __float_as_int(word) >= 0 ? kLeaf : kStep;
						}
					}
				}
			}
		}
		const int active = __popc(__ballot_sync(kAll, r.index != kNoRay));
		if (active == 0 && !more)
		{
			break;
		}
		const int limit = active - (active + RESTIR_TRACE_SHARE - 1) / RESTIR_TRACE_SHARE;
		do
		{
#pragma unroll
			for (int k = 0; k < RESTIR_TRACE_STEPS; ++k)
			{
				if (mode == kStep)
				{
					visit();
				}
			}
		} while (__popc(__ballot_sync(kAll, mode == kStep)) > limit);
		if (__any_sync(kAll, mode == kLeaf))
		{
			const int count = int(word);
			if (testLeaves<kWide>(b, storage.leaves, mode == kLeaf, slabOrigin(slab), r.d, int(__int_as_float(node)), count,
					r.distance, r.hit))
			{
				triangles += uint32_t(count);
				++step;
				++leafVisits;
				pop();
			}
		}
	}
}

// The stackless walk (bvh.sh:140-174; kAny: to the first leaf with a hit), four
// lanes a ray. The layout is depth first and a walk goes on to the next node
// or over a subtree, so four consecutive nodes hold 2.3 of its visits on
// average (1M-triangle city; two hold 1.65, eight 2.7): the lanes of a group
// read and test one each (128 consecutive bytes), and the group follows the
// walk through the results. That divides a walk's chain of dependent loads by
// 2.3, for launches that its latency bounds (the longest walks, up to 2,048
// visits, end last): the specular rays of a 1283x717 frame take 0.51 ms, with a
// ray per lane 0.62 ms, 0.87 ms in the one-lane loop with unshared leaves.
template<bool kAny, bool kWide, typename Source>
__device__ __forceinline__ void traceGroupWalks(const BvhView& b, Source& source)
{
	const int lane = int(threadIdx.x & 31u);
	const int group = lane & 28;
	const int sub = lane & 3;
	constexpr unsigned kAll = 0xffffffffu;
	constexpr int kAtLeaf = 0x7fffffff;
	Ray r = {};
	r.index = kNoRay;
	SlabRay slab = {};
	int node = 0;           // the walk's next node
	int step = 0;
	uint32_t triangles = 0;
	bool go = false;        // walking
	bool waiting = false;   // at a leaf: the node of lane `turn`
	int turn = 0;
	float a = 0.0f, w = 0.0f;
	bool more = true;
	for (;;)
	{
		// Rays that have ended are stored, and groups without one take the next.
		if (__any_sync(kAll, !go && !waiting && (r.index != kNoRay || more)))
		{
			if (!go && !waiting && r.index != kNoRay)
			{
				if (sub == 0)
				{
					countWork(Source::kCount, uint32_t(step), triangles);
					source.store(r);
				}
				r.index = kNoRay;
			}
			if (more)
			{
				const bool take = r.index == kNoRay;
				source.take(take, more, r);
				if (take && r.index != kNoRay)
				{
					slab = slabRay(r.o, r.d);
					node = 0;
					step = 0;
					triangles = 0;
					go = b.available();
				}
			}
		}
		const int rays = __popc(__ballot_sync(kAll, r.index != kNoRay));
		if (rays == 0)
		{
			if (!more)
			{
				break;
			}
			continue;
		}
		const int limit = rays - max(rays / 3, 4);
		do
		{
			const int last = b.nodeCount - node;  // the walk ends at this lane
			float enter = -1.0f;
			if (go)
			{
				enter = slabEnter(slab, loadNode<kWide>(b, node + min(sub, last - 1)), r.distance, a, w);
			}
			const bool leaf = w >= 0.0f;
			const bool pass = enter >= 0.0f;
			// Where the walk does not go on to the next node: a box it misses, a
			// leaf it enters, the end.
			const bool turned = leaf == pass || sub >= last;
			const int away = leaf ? kAtLeaf : int(-w) - 1 - node;   // the skip target, from the first node
			const unsigned turns = __ballot_sync(kAll, turned) >> group & 15u;
			int at = turns != 0u ? __ffs(turns) - 1 : 4;
			int visits = at;
			// A subtree of three nodes missed at the first lane ends before the last.
			if (__shfl_sync(kAll, away, group) == 3 && at == 0)
			{
				at = (turns & 8u) != 0u ? 3 : 4;
				visits = at - 2;
			}
			const int target = __shfl_sync(kAll, away, group | (at & 3));
			if (go)
			{
				const bool end = at >= last;
				const bool missed = at < 4 && target != kAtLeaf;
				turn = at;
				waiting = !end && at < 4 && target == kAtLeaf;
				step += visits + (missed && !end ? 1 : 0);
				node += waiting ? 0 : (missed ? target : 4);
				go = !end && !waiting && node < b.nodeCount;
				if (step >= kBvhMaxSteps)
				{
					step = kBvhMaxSteps;
					go = false;
					waiting = false;
					if (sub == 0)
					{
						reportTruncatedRay();
					}
				}
			}
		} while (__popc(__ballot_sync(kAll, go)) > limit);
		if (__any_sync(kAll, waiting))
		{
			const int first = int(__shfl_sync(kAll, a, group | (turn & 3)));
			const float leafWord = __shfl_sync(kAll, w, group | (turn & 3));
			const int count = waiting ? int(leafWord) : 0;
			int t = 0;
			do
			{
				float h = -1.0f;
				if (t + sub < count)
				{
					h = leafTriangle<kWide>(b, first + t + sub, r.o, r.d);
				}
				const unsigned key = h > 0.0f && h < r.distance ? __float_as_uint(h) : kAll;
				unsigned nearest = min(key, __shfl_xor_sync(kAll, key, 1));
				nearest = min(nearest, __shfl_xor_sync(kAll, nearest, 2));
				const unsigned winners = __ballot_sync(kAll, key == nearest && key != kAll) >> group & 15u;
				if (winners != 0u)
				{
					r.distance = __uint_as_float(nearest);
					r.hit = first + t + __ffs(winners) - 1;
				}
				t += 4;
			} while (__any_sync(kAll, t < count));
			if (waiting)
			{
				triangles += uint32_t(count);
				waiting = false;
				++step;
				node += turn + 1;
				go = !(kAny && r.hit >= 0);
			}
		}
	}
}

// The same with a ray per lane and the leaves tested together, for launches with
// more rays than lanes: 1M any-hit rays in the city take 0.39 ms, 0.65 ms with
// unshared leaves (6 of 32 lanes active there, 21 here) and 0.74 ms with four
// lanes a ray; half of its instructions take rays and test leaves.
template<bool kAny, bool kWide, typename Source>
__device__ __forceinline__ void traceLaneWalks(const BvhView& b, Source& source, LeafSlots& slots)
{
	constexpr unsigned kAll = 0xffffffffu;
	Ray r = {};
	r.index = kNoRay;
	SlabRay slab = {};
	int node = 0;
	int step = 0;
	uint32_t triangles = 0;
	bool go = false;
	bool waiting = false;
	float a = 0.0f, w = 0.0f;
	bool more = true;
	for (;;)
	{
		if (__any_sync(kAll, !go && !waiting && (r.index != kNoRay || more)))
		{
			if (!go && !waiting && r.index != kNoRay)
			{
				if (step >= kBvhMaxSteps && !(kAny && r.hit >= 0))
				{
					reportTruncatedRay();
				}
				countWork(Source::kCount, uint32_t(step), triangles);
				source.store(r);
				r.index = kNoRay;
			}
			if (more)
			{
				const bool take = r.index == kNoRay;
				source.take(take, more, r);
				if (take && r.index != kNoRay)
				{
					slab = slabRay(r.o, r.d);
					node = 0;
					step = 0;
					triangles = 0;
					go = b.available();
				}
			}
		}
		const int rays = __popc(__ballot_sync(kAll, r.index != kNoRay));
		if (rays == 0)
		{
			if (!more)
			{
				break;
			}
			continue;
		}
		const int limit = rays - max(rays / 3, 1);
		do
		{
#pragma unroll
			for (int k = 0; k < 4; ++k)
			{
				if (go)
				{
					const bool pass = slabEnter(slab, loadNode<kWide>(b, node), r.distance, a, w) >= 0.0f;
					const bool leaf = w >= 0.0f;
					waiting = pass && leaf;
					const int next = pass || leaf ? node + 1 : int(-w) - 1;
					node = waiting ? node : next;
					step += waiting ? 0 : 1;
					go = !waiting && node < b.nodeCount && step < kBvhMaxSteps;
				}
			}
		} while (__popc(__ballot_sync(kAll, go)) > limit);
		if (__any_sync(kAll, waiting))
		{
			const int count = int(w);
			if (testLeaves<kWide>(b, slots, waiting, r.o, r.d, int(a), count, r.distance, r.hit))
			{
				triangles += uint32_t(count);
				waiting = false;
				++step;
				++node;
				go = !(kAny && r.hit >= 0) && node < b.nodeCount && step < kBvhMaxSteps;
			}
		}
	}
}

} // namespace restir
