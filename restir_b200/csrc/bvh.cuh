// BVH traversal over the reference's depth-first node layout (src/bvh.h:7-22):
// node i = float4 rows 2i, 2i+1: (min.xyz, a), (max.xyz, b); b >= 0 a leaf of
// triangles [a, a+b), b < 0 an interior node with right child a and skip
// link -b-1; triangle t = rows triangleOffset + 4t .. +3.
//
// Same algorithms and arithmetic as shaders/bvh.sh (slab test 32-41,
// Moeller-Trumbore 44-71, stackless walk 140-174, nearest-first short stack
// 216-295), so hit ids and distances are bit-identical to the CPU
// restatement. The walks of this file's first half read each row with one
// 16-byte read-only load; the packed tests below and warptrace.cuh's read a node
// or a triangle's first two rows with one of 32 bytes where the scene's rows
// start on that (wideRows).
#pragma once

#include "common.cuh"

namespace restir
{

#define kBvhShortStack 8
#define kBvhMaxSteps 2048

struct BvhView
{
	const float4* rows = nullptr;
	int nodeCount = 0;
	int triangleOffset = 0;
	int rowCount = 0;   // nodes x 2 + triangles x 4 (checked builds test indices against it)

	__device__ __forceinline__ bool available() const { return nodeCount > 0; }
	__device__ __forceinline__ V4 row(int i) const
	{
		if (!checkedIndex(uint32_t(i), uint32_t(rowCount)))
		{
			return { 0.0f, 0.0f, 0.0f, 0.0f };
		}
		float4 q = __ldg(rows + i);
		return { q.x, q.y, q.z, q.w };
	}
	__device__ __forceinline__ V3 vertex(int t, int corner) const { return row(triangleOffset + t * 4 + corner).xyz(); }
	__device__ __forceinline__ V3 albedo(int t) const { return row(triangleOffset + t * 4 + 3).xyz(); }
	__device__ __forceinline__ V3 emission(int t) const
	{
		int base = triangleOffset + t * 4;
		return v3(row(base + 1).w, row(base + 2).w, row(base + 3).w);
	}
};

__host__ __device__ inline BvhView makeBvhView(const RestirScene* s)
{
	BvhView b;
	if (s != nullptr && s->bvh != nullptr)
	{
		b.rows = reinterpret_cast<const float4*>(s->bvh);
		b.nodeCount = int(s->node_count);
		b.triangleOffset = int(s->triangle_offset);
		b.rowCount = int(s->triangle_offset + 4u * s->triangle_count);
	}
	return b;
}

// Node fetches and triangle tests of one ray, for the work counters.
struct TraceWork
{
	uint32_t nodes = 0;
	uint32_t triangles = 0;
};

__device__ __forceinline__ float intersectBox(V3 o, V3 inv, V3 bmin, V3 bmax, float maxDistance)
{
	V3 t0 = (bmin - o) * inv;
	V3 t1 = (bmax - o) * inv;
	V3 n = vmin(t0, t1);
	V3 f = vmax(t0, t1);
	float enter = fmaxf(fmaxf(n.x, n.y), fmaxf(n.z, 0.0f));
	float leave = fminf(fminf(f.x, f.y), fminf(f.z, maxDistance));
	return enter <= leave ? enter : -1.0f;
}

__device__ __forceinline__ float intersectTriangle(V3 o, V3 d, V3 v0, V3 v1, V3 v2)
{
	V3 edge1 = v1 - v0;
	V3 edge2 = v2 - v0;
	V3 p = cross(d, edge2);
	float determinant = dot(edge1, p);
	if (fabsf(determinant) < 1e-12f)
	{
		return -1.0f;
	}
	float inverse = 1.0f / determinant;
	V3 s = o - v0;
	float u = dot(s, p) * inverse;
	if (u < 0.0f || u > 1.0f)
	{
		return -1.0f;
	}
	V3 q = cross(s, edge1);
	float v = dot(d, q) * inverse;
	if (v < 0.0f || u + v > 1.0f)
	{
		return -1.0f;
	}
	return dot(edge2, q) * inverse;
}

__device__ __forceinline__ float safeInverse(float d)
{
	float s = fabsf(d) > 1e-8f ? d : (d >= 0.0f ? 1e-8f : -1e-8f);
	return 1.0f / s;
}

__device__ __forceinline__ V3 bvhInverseDirection(V3 d)
{
	return { safeInverse(d.x), safeInverse(d.y), safeInverse(d.z) };
}

__device__ __forceinline__ int intersectLeaf(const BvhView& b, V3 o, V3 d, int first, int count, float& distance, int hit,
	TraceWork& work)
{
	work.triangles += uint32_t(count);
#pragma unroll 1
	for (int t = first; t < first + count; ++t)
	{
		float h = intersectTriangle(o, d, b.vertex(t, 0), b.vertex(t, 1), b.vertex(t, 2));
		if (h > 0.0f && h < distance)
		{
			distance = h;
			hit = t;
		}
	}
	return hit;
}

// bvh.sh:140-174
__device__ inline int traceStacklessWalk(const BvhView& b, V3 o, V3 d, bool anyHit, float& distance, TraceWork& work)
{
	V3 inv = bvhInverseDirection(d);
	int hit = -1;
	int node = 0;
	int step = 0;
	for (; step < kBvhMaxSteps; ++step)
	{
		if (node >= b.nodeCount)
		{
			break;
		}
		++work.nodes;
		V4 node0 = b.row(node * 2);
		V4 node1 = b.row(node * 2 + 1);
		bool leaf = node1.w >= 0.0f;
		if (intersectBox(o, inv, node0.xyz(), node1.xyz(), distance) < 0.0f)
		{
			node = leaf ? node + 1 : int(-node1.w) - 1;
			continue;
		}
		if (leaf)
		{
			hit = intersectLeaf(b, o, d, int(node0.w), int(node1.w), distance, hit, work);
			if (anyHit && hit >= 0)
			{
				return hit;
			}
		}
		node = node + 1;
	}
	if (step == kBvhMaxSteps)
	{
		reportTruncatedRay();
	}
	return hit;
}

// traceBvhWave (bvh.sh:177-212), the visibility rays of the reference's
// Vulkan build: the lanes that call it walk the skip-link order in lock
// step. Each step the warp takes the smallest node any lane still needs
// (__reduce_min_sync; a finished lane asks for nodeCount), and the lanes at
// that node test it while the others wait, so lanes on the same part of the
// tree share every node fetch. A lane visits its nodes in the stackless
// walk's order, so its hit is the stackless walk's; only the step cap counts
// the warp's steps.
__device__ inline int traceStacklessWave(const BvhView& b, V3 o, V3 d, bool anyHit, float& distance, TraceWork& work)
{
	const unsigned mask = __activemask();
	V3 inv = bvhInverseDirection(d);
	const int nodeCount = b.nodeCount;
	int hit = -1;
	int node = 0;
	int step = 0;
	for (; step < kBvhMaxSteps; ++step)
	{
		const int waveNode = int(__reduce_min_sync(mask, unsigned(node)));
		if (waveNode >= nodeCount)
		{
			break;
		}
		if (node == waveNode)
		{
			++work.nodes;
			V4 node0 = b.row(waveNode * 2);
			V4 node1 = b.row(waveNode * 2 + 1);
			bool leaf = node1.w >= 0.0f;
			if (intersectBox(o, inv, node0.xyz(), node1.xyz(), distance) < 0.0f)
			{
				node = leaf ? node + 1 : int(-node1.w) - 1;
			}
			else
			{
				if (leaf)
				{
					hit = intersectLeaf(b, o, d, int(node0.w), int(node1.w), distance, hit, work);
				}
				node = anyHit && hit >= 0 ? nodeCount : node + 1;
			}
		}
	}
	if (step == kBvhMaxSteps)
	{
		reportTruncatedRay();
	}
	return hit;
}

// The nearest-first walk of bvh.sh:216-295 up to its re-walk, which is to follow
// when dropped. stack: this thread's kBvhShortStack entries, stride apart (shared
// memory, interleaved across the block's threads).
__device__ __forceinline__ int walkShortStack(const BvhView& b, V3 o, V3 d, float& distance, int* stack, int stride,
	TraceWork& work, bool& dropped)
{
	V3 inv = bvhInverseDirection(d);
	dropped = false;
	++work.nodes;
	if (intersectBox(o, inv, b.row(0).xyz(), b.row(1).xyz(), distance) < 0.0f)
	{
		return -1;
	}
	int stackTop = 0;
	int stackCount = 0;
	int hit = -1;
	int node = 0;
	int step = 0;
	for (; step < kBvhMaxSteps; ++step)
	{
		V4 node0 = b.row(node * 2);
		V4 node1 = b.row(node * 2 + 1);
		if (node1.w >= 0.0f)
		{
			hit = intersectLeaf(b, o, d, int(node0.w), int(node1.w), distance, hit, work);
		}
		else
		{
			int left = node + 1;
			int right = int(node0.w);
			work.nodes += 2u;
			float leftDistance = intersectBox(o, inv, b.row(left * 2).xyz(), b.row(left * 2 + 1).xyz(), distance);
			float rightDistance = intersectBox(o, inv, b.row(right * 2).xyz(), b.row(right * 2 + 1).xyz(), distance);
			bool visitLeft = leftDistance >= 0.0f;
			bool visitRight = rightDistance >= 0.0f;
			if (visitLeft && visitRight)
			{
				bool leftFirst = leftDistance <= rightDistance;
				stack[(stackTop & (kBvhShortStack - 1)) * stride] = leftFirst ? right : left;
				++stackTop;
				if (stackCount == kBvhShortStack)
				{
					dropped = true;
				}
				else
				{
					++stackCount;
				}
				node = leftFirst ? left : right;
				continue;
			}
			if (visitLeft || visitRight)
			{
				node = visitLeft ? left : right;
				continue;
			}
		}
		if (stackCount == 0)
		{
			break;
		}
		--stackTop;
		--stackCount;
		node = stack[(stackTop & (kBvhShortStack - 1)) * stride];
	}
	if (step == kBvhMaxSteps)
	{
		reportTruncatedRay();
	}
	return hit;
}

// bvh.sh:216-295.
__device__ inline int traceShortStack(const BvhView& b, V3 o, V3 d, float& distance, int* stack, int stride, TraceWork& work)
{
	bool dropped;
	int hit = walkShortStack(b, o, d, distance, stack, stride, work, dropped);
	if (dropped)
	{
		int stacklessHit = traceStacklessWalk(b, o, d, false, distance, work);
		if (stacklessHit >= 0)
		{
			hit = stacklessHit;
		}
	}
	return hit;
}

// traceBvh (bvh.sh:298-319). stack == nullptr: stackless for every ray (the
// passes without BVH_SHARED_STACK).
__device__ __forceinline__ int traceBvh(const BvhView& b, V3 o, V3 d, float maxDistance, bool anyHit, float& distance,
	int* stack, int stride)
{
	distance = maxDistance;
	if (!b.available())
	{
		return -1;
	}
	TraceWork work;
	int hit;
	int kind;
	if (stack != nullptr && !anyHit)
	{
		hit = traceShortStack(b, o, d, distance, stack, stride, work);
		kind = RESTIR_COUNT_CLOSEST;
	}
	else
	{
		hit = traceStacklessWalk(b, o, d, anyHit, distance, work);
		kind = RESTIR_COUNT_ANY;
	}
	countWork(kind, work.nodes, work.triangles);
	return hit;
}

// A visibility (any-hit) ray: traceBvh's stackless walk, or with kWave the
// warp-lock-step walk of the reference's Vulkan build (same hits). A template
// parameter, so that a kernel holds the code it runs and no other: both in one
// kernel made GI spatial 7,952 instructions instead of 7,184, DI temporal 4,840
// instead of 4,064.
template<bool kWave>
__device__ __forceinline__ int traceVisibility(const BvhView& b, V3 o, V3 d, float maxDistance, float& distance)
{
	if (!kWave)
	{
		return traceBvh(b, o, d, maxDistance, true, distance, nullptr, 0);
	}
	distance = maxDistance;
	if (!b.available())
	{
		return -1;
	}
	TraceWork work;
	const int hit = traceStacklessWave(b, o, d, true, distance, work);
	countWork(RESTIR_COUNT_ANY, work.nodes, work.triangles);
	return hit;
}

// --- packed node tests ---------------------------------------------------------
//
// A node is read with one 256-bit load where the buffer starts on 32 bytes
// (kWide; the layout's nodes are 32 bytes), else with two of 128 bits, and
// its slab test runs on packed pairs of floats (add and mul.rn.f32x2 round each
// half as the scalar operations do).

typedef unsigned long long F2;

__device__ __forceinline__ F2 pack2(float a, float b)
{
	F2 r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
	return r;
}

__device__ __forceinline__ void unpack2(F2 v, float& a, float& b)
{
	asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}

__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
	F2 r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}

__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
	F2 r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}

// --- nodes ---------------------------------------------------------------------

// A node's 32 bytes: (min.xy) (min.z, a) (max.xy) (max.z, b).
struct NodeRow
{
	F2 lo, loA, hi, hiB;
};

template<bool kWide>
__device__ __forceinline__ NodeRow loadNode(const BvhView& b, int node)
{
	NodeRow n;
	if (!checkedIndex(uint32_t(node) * 2u + 1u, uint32_t(b.rowCount)))
	{
		n.lo = n.loA = n.hi = n.hiB = 0ull;
		return n;
	}
	const float4* row = b.rows + size_t(node) * 2;
	if (kWide)
	{
		asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(n.lo), "=l"(n.loA), "=l"(n.hi), "=l"(n.hiB) : "l"(row));
	}
	else
	{
		asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(n.lo), "=l"(n.loA) : "l"(row));
		asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(n.hi), "=l"(n.hiB) : "l"(row + 1));
	}
	return n;
}

// A ray as the slab test takes it: the negated origin and the inverse direction.
struct SlabRay
{
	F2 negXY, invXY;
	float negZ, invZ;
};

__device__ __forceinline__ SlabRay slabRay(V3 o, V3 d)
{
	const V3 inv = bvhInverseDirection(d);
	SlabRay r;
	r.negXY = pack2(-o.x, -o.y);
	r.invXY = pack2(inv.x, inv.y);
	r.negZ = -o.z;
	r.invZ = inv.z;
	return r;
}

__device__ __forceinline__ V3 slabOrigin(const SlabRay& r)
{
	float x, y;
	unpack2(r.negXY, x, y);
	return v3(-x, -y, -r.negZ);
}

// intersectBox (bvh.sh:32-41); a and b are the node's two words. kConservative:
// the box's exit widened (traceNearestFirst). kSigns: the signs of the ray's
// direction when they are known (bit k: component k is negative), kAnySigns
// otherwise; with them the nearer plane of each pair is known, and the smaller
// and larger of the two products need no comparison (a box's bounds are
// ordered, and rounding keeps the order).
constexpr int kAnySigns = 8;

template<bool kConservative = false, int kSigns = kAnySigns>
__device__ __forceinline__ float slabEnter(const SlabRay& r, const NodeRow& n, float maxDistance, float& a, float& b)
{
	float loZ, hiZ;
	unpack2(n.loA, loZ, a);
	unpack2(n.hiB, hiZ, b);
	float t0x, t0y, t1x, t1y;
	unpack2(mul2(add2(n.lo, r.negXY), r.invXY), t0x, t0y);
	unpack2(mul2(add2(n.hi, r.negXY), r.invXY), t1x, t1y);
	const float t0z = (loZ + r.negZ) * r.invZ;
	const float t1z = (hiZ + r.negZ) * r.invZ;
	const float nearX = kSigns == kAnySigns ? fminf(t0x, t1x) : ((kSigns & 1) != 0 ? t1x : t0x);
	const float nearY = kSigns == kAnySigns ? fminf(t0y, t1y) : ((kSigns & 2) != 0 ? t1y : t0y);
	const float nearZ = kSigns == kAnySigns ? fminf(t0z, t1z) : ((kSigns & 4) != 0 ? t1z : t0z);
	const float farX = kSigns == kAnySigns ? fmaxf(t0x, t1x) : ((kSigns & 1) != 0 ? t0x : t1x);
	const float farY = kSigns == kAnySigns ? fmaxf(t0y, t1y) : ((kSigns & 2) != 0 ? t0y : t1y);
	const float farZ = kSigns == kAnySigns ? fmaxf(t0z, t1z) : ((kSigns & 4) != 0 ? t0z : t1z);
	const float enter = fmaxf(fmaxf(nearX, nearY), fmaxf(nearZ, 0.0f));
	const float leave = kConservative ? fminf(fminf(fminf(farX, farY), farZ) * 1.00000036f, maxDistance)
		: fminf(fminf(farX, farY), fminf(farZ, maxDistance));
	return enter <= leave ? enter : -1.0f;
}

// Whether a scene's nodes (two rows each) and the first two rows of its
// triangles (four rows each, from triangleOffset on) can be read 32 bytes at a
// time: both start on 32 bytes when the buffer does and the offset is even. The
// offset is the caller's, and any padding may lie before the triangles.
__host__ inline bool wideRows(const BvhView& b)
{
	return (reinterpret_cast<uintptr_t>(b.rows) & 31u) == 0u && (b.triangleOffset & 1) == 0;
}

// Nearest hit in (0, distance) among the triangles accept() lets through,
// ties to the lower triangle index, nearest child first with a full stack of
// 64 entries in local memory (the layout's depth is at most 40, bvh.h:49).
// test(t, distance) is the triangle test. With conservative set, a box's exit
// distance is widened by 1 + 2 gamma_3 (Ize, "Robust BVH Ray Traversal",
// JCGT 2(2), 2013), so that rounding in the slab test never culls a box
// whose triangle the watertight test hits.
template<bool kWide, bool kConservative, int kSigns, typename Test, typename Accept>
__device__ __forceinline__ int nearestFirstLoop(const BvhView& b, const SlabRay& slab, float& distance, Test& test, Accept& accept)
{
	TraceWork work;
	++work.nodes;
	// The words of the node to visit; a child's come with its box.
	float nodeA = 0.0f, nodeB = 0.0f;
	if (!b.available()
		|| slabEnter<kConservative, kSigns>(slab, loadNode<kWide>(b, 0), distance, nodeA, nodeB) < 0.0f)
	{
		countWork(RESTIR_COUNT_PRIMARY, b.available() ? work.nodes : 0u, work.triangles);
		return -1;
	}
	// Each entry keeps the box's entry distance: a box that passed its test
	// when pushed passes it again at the pop exactly when that distance is
	// still within the nearest hit (its own exit did not change), so the pop
	// needs no second fetch of the box.
	float2 stack[64];
	int top = 0;
	int hit = -1;
	int node = 0;
	for (int step = 0; step < (1 << 24); ++step)
	{
		if (nodeB >= 0.0f)
		{
			const int first = int(nodeA);
			const int count = int(nodeB);
			work.triangles += uint32_t(count);
#pragma unroll 1
			for (int t = first; t < first + count; ++t)
			{
				float h = test(t, distance);
				if (h > 0.0f && (h < distance || (h == distance && hit >= 0 && t < hit)) && accept(t))
				{
					distance = h;
					hit = t;
				}
			}
		}
		else
		{
			const int left = node + 1;
			const int right = int(nodeA);
			const NodeRow leftRow = loadNode<kWide>(b, left);
			const NodeRow rightRow = loadNode<kWide>(b, right);
			work.nodes += 2u;
			float leftA, leftB, rightA, rightB;
			const float leftDistance = slabEnter<kConservative, kSigns>(slab, leftRow, distance, leftA, leftB);
			const float rightDistance = slabEnter<kConservative, kSigns>(slab, rightRow, distance, rightA, rightB);
			const bool visitLeft = leftDistance >= 0.0f;
			const bool visitRight = rightDistance >= 0.0f;
			if (visitLeft || visitRight)
			{
				bool goLeft = visitLeft;
				if (visitLeft && visitRight)
				{
					goLeft = leftDistance <= rightDistance;
					if (top < 64)
					{
						stack[top] = goLeft ? make_float2(__int_as_float(right), rightDistance)
							: make_float2(__int_as_float(left), leftDistance);
						++top;
					}
					else
					{
						reportTruncatedRay();
					}
				}
				node = goLeft ? left : right;
				nodeA = goLeft ? leftA : rightA;
				nodeB = goLeft ? leftB : rightB;
				continue;
			}
		}
		// Pop, skipping subtrees that the nearest hit found since rules out.
		bool found = false;
		while (top > 0)
		{
			--top;
			const float2 e = stack[top];
			if (e.y <= distance)
			{
				node = __float_as_int(e.x);
				found = true;
				break;
			}
		}
		if (!found)
		{
			break;
		}
		nodeA = b.row(node * 2).w;
		nodeB = b.row(node * 2 + 1).w;
	}
	countWork(RESTIR_COUNT_PRIMARY, work.nodes, work.triangles);
	return hit;
}

// kSplit: the rays of a tile nearly always agree on the signs of their
// directions: a copy of the loop for each combination, and one for warps that
// disagree (G-buffer of the 1080p city frame 0.50 -> 0.43 ms with the words
// carried; the loop was bound by the ALU pipe, 69% busy, on which minima and
// maxima run).
template<bool kWide, bool kSplit, bool kConservative, typename Test, typename Accept>
__device__ inline int traceNearestFirst(const BvhView& b, V3 o, V3 d, float& distance, Test test, Accept accept)
{
	const SlabRay slab = slabRay(o, d);
	if constexpr (kSplit)
	{
		float ix, iy;
		unpack2(slab.invXY, ix, iy);
		const unsigned lanes = __activemask();
		const int signs = (ix < 0.0f ? 1 : 0) | (iy < 0.0f ? 2 : 0) | (slab.invZ < 0.0f ? 4 : 0);
		int same = 0;
		__match_all_sync(lanes, signs, &same);
		switch (same != 0 ? signs : kAnySigns)
		{
		case 0:
			return nearestFirstLoop<kWide, kConservative, 0>(b, slab, distance, test, accept);
		case 1:
			return nearestFirstLoop<kWide, kConservative, 1>(b, slab, distance, test, accept);
		case 2:
			return nearestFirstLoop<kWide, kConservative, 2>(b, slab, distance, test, accept);
		case 3:
			return nearestFirstLoop<kWide, kConservative, 3>(b, slab, distance, test, accept);
		case 4:
			return nearestFirstLoop<kWide, kConservative, 4>(b, slab, distance, test, accept);
		case 5:
			return nearestFirstLoop<kWide, kConservative, 5>(b, slab, distance, test, accept);
		case 6:
			return nearestFirstLoop<kWide, kConservative, 6>(b, slab, distance, test, accept);
		case 7:
			return nearestFirstLoop<kWide, kConservative, 7>(b, slab, distance, test, accept);
		default:
			break;
		}
	}
	return nearestFirstLoop<kWide, kConservative, kAnySigns>(b, slab, distance, test, accept);
}

// Moeller-Trumbore nearest hit among accepted triangles (the raster
// passes' ray casts).
template<bool kWide, bool kSplit, typename Accept>
__device__ inline int traceNearestFiltered(const BvhView& b, V3 o, V3 d, float& distance, Accept accept)
{
	return traceNearestFirst<kWide, kSplit, false>(b, o, d, distance,
		[&](int t, float) { return intersectTriangle(o, d, b.vertex(t, 0), b.vertex(t, 1), b.vertex(t, 2)); }, accept);
}

} // namespace restir
