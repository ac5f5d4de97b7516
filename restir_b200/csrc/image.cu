// Image-space passes: the SVGF denoiser (svgf.sh:26-36, fs_svgf_variance.sc:29-76,
// fs_svgf_atrous.sc:29-95) at GI resolution, and the composite
// (fs_composite.sc:48-143) at full resolution. One thread per pixel in 16x8
// tiles; the denoiser's stencils read their tile's texels from shared memory.
#include "bvh.cuh"
#include "gi.cuh"
#include "screen.cuh"

namespace restir
{
namespace
{

__device__ __forceinline__ V3 xyz4(const float4* p, int i)
{
	float4 q = __ldg(p + i);
	return v3(q.x, q.y, q.z);
}

constexpr int kFilterW = 16, kFilterH = 8;   // pixels per block

// A neighbour's texel for the geometry weight (svgf.sh:26-36), its normal
// normalised once for all pixels that read it.
struct GeometryTexel
{
	float4 position;  // w: free
	float4 normal;    // normalised; w: 1 where there is a surface, 0 where not, -1 outside the image
};

__device__ __forceinline__ GeometryTexel outsideTexel()
{
	return { make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, -1.0f) };
}

__device__ __forceinline__ GeometryTexel geometryTexel(const float4* __restrict__ receiver, const float4* __restrict__ normal, int j,
	float free)
{
	const V3 position = xyz4(receiver, j);
	V3 n = xyz4(normal, j);
	const bool surface = !(dot(n, n) < 0.5f);
	n = surface ? normalize(n) : n;
	return { make_float4(position.x, position.y, position.z, free), make_float4(n.x, n.y, n.z, surface ? 1.0f : 0.0f) };
}

__device__ __forceinline__ float geometryWeight(float planeScale, V3 p, V3 n, float4 tp, float4 tn)
{
	if (tn.w < 0.5f)
	{
		return 0.0f;
	}
	const float planeDistance = fabsf(dot(n, v3(tp.x, tp.y, tp.z) - p)) / planeScale;
	const float normalWeight = rn_pow64(fmaxf(dot(n, v3(tn.x, tn.y, tn.z)), 0.0f));
	return rn_exp(-planeDistance) * normalWeight;
}

// The spatial estimate of the variance, of the pixels with less than four
// frames of history: a block that has one reads its 22x14 texels to shared
// memory once. With 49 taps that each fetched 40 bytes and normalised a normal
// it took 0.135 ms on 960x540 pixels, a third of them short; now 0.069 ms.
constexpr int kVarianceTileW = kFilterW + 6, kVarianceTileH = kFilterH + 6;

__global__ void __launch_bounds__(128) varianceKernel(const RestirParams P, const uint16_t* __restrict__ color,
	const uint16_t* __restrict__ moments, const float4* __restrict__ receiver, const float4* __restrict__ normal, uint16_t* out)
{
	__shared__ GeometryTexel tile[kVarianceTileW * kVarianceTileH];
	__shared__ float secondMoment[kVarianceTileW * kVarianceTileH];
	const int w = int(P.gi_width), h = int(P.gi_height);
	const int firstX = int(blockIdx.x) * kFilterW, firstY = int(blockIdx.y) * kFilterH;
	const int lx = int(threadIdx.x) % kFilterW, ly = int(threadIdx.x) / kFilterW;
	const int px = firstX + lx, py = firstY + ly;
	const int i = py * w + px;
	bool spatial = false;
	float historyLength = 0.0f;
	V3 col = v3s(0.0f);
	if (px < w && py < h)
	{
		const V3 n = xyz4(normal, i);
		if (dot(n, n) < 0.5f)
		{
			storeH4(out, i, v4(0.0f, 0.0f, 0.0f, 0.0f));
		}
		else
		{
			col = loadH4(color, i).xyz();
			const V4 m = loadH4(moments, i);
			historyLength = m.z;
			spatial = !(historyLength >= 4.0f);
			if (!spatial)
			{
				storeH4(out, i, v4(col, fmaxf(m.y - m.x * m.x, 0.0f)));
			}
		}
	}
	if (__syncthreads_or(spatial) == 0)
	{
		return; // whole block
	}
	for (int k = int(threadIdx.x); k < kVarianceTileW * kVarianceTileH; k += 128)
	{
		const int x = firstX + k % kVarianceTileW - 3;
		const int y = firstY + k / kVarianceTileW - 3;
		GeometryTexel t = outsideTexel();
		float second = 0.0f;
		if (x >= 0 && x < w && y >= 0 && y < h)
		{
			const V4 m = loadH4(moments, y * w + x);
			t = geometryTexel(receiver, normal, y * w + x, m.x);
			second = m.y;
		}
		tile[k] = t;
		secondMoment[k] = second;
	}
	__syncthreads();
	if (!spatial)
	{
		return;
	}
	const int center = (ly + 3) * kVarianceTileW + lx + 3;
	const float4 p4 = tile[center].position;
	const float4 n4 = tile[center].normal;
	const V3 position = v3(p4.x, p4.y, p4.z);
	const V3 n = v3(n4.x, n4.y, n4.z);
	const float planeScale = 0.02f * P.scene_scale;
	float sumX = 0.0f, sumY = 0.0f;
	float weightSum = 0.0f;
#pragma unroll 1
	for (int y = -3; y <= 3; ++y)
	{
#pragma unroll
		for (int x = -3; x <= 3; ++x)
		{
			const int j = center + y * kVarianceTileW + x;
			const float4 tn = tile[j].normal;
			if (tn.w < 0.0f)
			{
				continue; // outside the image
			}
			const float4 tp = tile[j].position;
			const float weight = geometryWeight(planeScale, position, n, tp, tn);
			sumX += tp.w * weight;
			sumY += secondMoment[j] * weight;
			weightSum += weight;
		}
	}
	const float denominator = fmaxf(weightSum, 0.0001f);
	const float mx = sumX / denominator;
	const float my = sumY / denominator;
	const float variance = fmaxf(my - mx * mx, 0.0f) * (4.0f / fmaxf(historyLength, 1.0f));
	storeH4(out, i, v4(col, variance));
}

__device__ __forceinline__ float splineWeight(int offset)
{
	int d = offset < 0 ? -offset : offset;
	return d == 0 ? 0.375f : (d == 1 ? 0.25f : 0.0625f);
}

struct FilterTexel
{
	GeometryTexel geometry;  // position.w: luminance
	float4 color;            // w: variance
};

// What a tap at (x, y) reads.
__device__ __forceinline__ FilterTexel filterTexel(const uint16_t* __restrict__ input, const float4* __restrict__ receiver,
	const float4* __restrict__ normal, int w, int h, int x, int y)
{
	FilterTexel t = { outsideTexel(), make_float4(0.0f, 0.0f, 0.0f, 0.0f) };
	if (x >= 0 && x < w && y >= 0 && y < h)
	{
		const V4 color = loadH4(input, y * w + x);
		t.geometry = geometryTexel(receiver, normal, y * w + x, luminance(color.xyz()));
		t.color = make_float4(color.x, color.y, color.z, color.w);
	}
	return t;
}

// One a-trous level's pixel (px, py) from its own texel and its taps',
// tap(x, y) for offsets of -2 to 2 steps.
template<typename Tap>
__device__ __forceinline__ void filterPixel(const RestirParams& P, const uint16_t* __restrict__ input, uint16_t* out, int px, int py,
	const GeometryTexel& center, Tap tap)
{
	const int w = int(P.gi_width), h = int(P.gi_height);
	const int i = py * w + px;
	const float4 n4 = center.normal;
	if (n4.w < 0.5f)
	{
		storeH4(out, i, v4(0.0f, 0.0f, 0.0f, 0.0f));
		return;
	}
	const V3 n = v3(n4.x, n4.y, n4.z);
	const float4 p4 = center.position;
	const V3 position = v3(p4.x, p4.y, p4.z);
	const float centerLuminance = p4.w;
	float variance = 0.0f;
	for (int by = -1; by <= 1; ++by)
	{
		const int row = min(max(py + by, 0), h - 1) * w;
		for (int bx = -1; bx <= 1; ++bx)
		{
			float weight = (bx == 0 ? 0.5f : 0.25f) * (by == 0 ? 0.5f : 0.25f);
			variance += loadH4(input, row + min(max(px + bx, 0), w - 1)).w * weight;
		}
	}
	const float luminanceScale = 1.0f / (4.0f * sqrtf(fmaxf(variance, 0.0f)) + 0.0001f);
	const float planeScale = 0.02f * P.scene_scale;
	V3 colorSum = v3s(0.0f);
	float varianceSum = 0.0f;
	float weightSum = 0.0f;
#pragma unroll 1
	for (int y = -2; y <= 2; ++y)
	{
#pragma unroll
		for (int x = -2; x <= 2; ++x)
		{
			const FilterTexel& t = tap(x, y);
			const float4 tn = t.geometry.normal;
			if (tn.w < 0.0f)
			{
				continue; // outside the image
			}
			const float4 color = t.color;
			float weight = splineWeight(x) * splineWeight(y);
			if (x != 0 || y != 0)
			{
				const float4 tp = t.geometry.position;
				weight *= geometryWeight(planeScale, position, n, tp, tn);
				weight *= rn_exp(-fabsf(tp.w - centerLuminance) * luminanceScale);
			}
			colorSum = colorSum + v3(color.x, color.y, color.z) * weight;
			varianceSum += color.w * weight * weight;
			weightSum += weight;
		}
	}
	storeH4(out, i, v4(colorSum / weightSum, varianceSum / (weightSum * weightSum)));
}

// One a-trous level. A pixel's taps lie step texels apart, so the pixels of one
// residue (x mod step, y mod step) filter among themselves: a block takes 16x8
// of them and its 20x12 texels go to shared memory once, the
// normals normalised there. Every tap used to fetch 40 bytes and normalise the
// neighbour's normal (a square root and a division, 24 times per texel instead
// of 1.9) at 220 instructions a tap. Bound by issue (79% of the slots busy);
// five levels at 960x540 take 0.36 ms, before 0.52 ms; the rows are a loop, so
// that its 1,360 instructions stay in the instruction cache (unrolled: 0.42 ms).
constexpr int kFilterTileW = kFilterW + 4, kFilterTileH = kFilterH + 4;

__global__ void __launch_bounds__(128) atrousKernel(const RestirParams P, int step, int residuesX, int residuesY,
	int blocksX, const uint16_t* __restrict__ input, const float4* __restrict__ receiver, const float4* __restrict__ normal, uint16_t* out)
{
	__shared__ FilterTexel tile[kFilterTileW * kFilterTileH];
	const int w = int(P.gi_width), h = int(P.gi_height);
	// Neighbouring blocks take neighbouring residues: they read the same lines.
	const int blockX = int(blockIdx.x % uint32_t(blocksX)), blockY = int(blockIdx.x / uint32_t(blocksX));
	const int firstX = blockX % residuesX + blockX / residuesX * kFilterW * step;
	const int firstY = blockY % residuesY + blockY / residuesY * kFilterH * step;
	if (firstX >= w || firstY >= h)
	{
		return; // whole block
	}
	for (int k = int(threadIdx.x); k < kFilterTileW * kFilterTileH; k += 128)
	{
		tile[k] = filterTexel(input, receiver, normal, w, h, firstX + (k % kFilterTileW - 2) * step,
			firstY + (k / kFilterTileW - 2) * step);
	}
	__syncthreads();
	const int lx = int(threadIdx.x) % kFilterW, ly = int(threadIdx.x) / kFilterW;
	const int px = firstX + lx * step, py = firstY + ly * step;
	if (px >= w || py >= h)
	{
		return;
	}
	const int center = (ly + 2) * kFilterTileW + lx + 2;
	filterPixel(P, input, out, px, py, tile[center].geometry,
		[&](int x, int y) -> const FilterTexel& { return tile[center + y * kFilterTileW + x]; });
}

// The same with the taps read from the image: for steps so large that a
// residue's pixels leave most of a tile empty (restir_svgf_atrous).
__global__ void __launch_bounds__(128) atrousDirectKernel(const RestirParams P, int step, const uint16_t* __restrict__ input,
	const float4* __restrict__ receiver, const float4* __restrict__ normal, uint16_t* out)
{
	const int w = int(P.gi_width), h = int(P.gi_height);
	const int px = int(blockIdx.x) * kFilterW + int(threadIdx.x) % kFilterW;
	const int py = int(blockIdx.y) * kFilterH + int(threadIdx.x) / kFilterW;
	if (px >= w || py >= h)
	{
		return;
	}
	filterPixel(P, input, out, px, py, filterTexel(input, receiver, normal, w, h, px, py).geometry,
		[&](int x, int y) { return filterTexel(input, receiver, normal, w, h, px + x * step, py + y * step); });
}

// The split-sum specular albedo, brdf.sh:68-76 (Karis' analytic fit).
__device__ __forceinline__ V3 compositeSpecularAlbedo(V3 f0, float roughness, float normalView)
{
	const float rx = -1.0f * roughness + 1.0f, ry = -0.0275f * roughness + 0.0425f;
	const float rz = -0.572f * roughness + 1.04f, rw = 0.022f * roughness + -0.04f;
	const float a004 = fminf(rx * rx, rn_exp2(-9.28f * normalView)) * rx + ry;
	const float scale = -1.04f * a004 + rz, bias = 1.04f * a004 + rw;
	return f0 * scale + bias;
}

// fs_composite.sc:48-143 with the final view's options; the indirect
// specular when a specular target is given.
// Bound by the latency of its taps and divisions. kBlocks: blocks a SM; eight
// (64 registers, 40 bytes spilled) where 94 registers left five: 189 -> 144 us
// at 1920x1080 (courtyard), 75 -> 62 at 1280x720, 19 -> 15 at 480x270. Images of
// no more than five blocks a SM run in one wave either way and take the
// registers: 320x180 12.5 -> 10.6 (Cornell box), 256x256 with the specular target
// 14.5 -> 12.5.
template<int kBlocks>
__global__ void __launch_bounds__(128, kBlocks) compositeKernel(const RestirParams P, RestirGBuffer gb, const float* __restrict__ atlas,
	const uint16_t* __restrict__ gi, const uint16_t* __restrict__ diDiffuse, const uint16_t* __restrict__ diSpecular,
	const uint16_t* __restrict__ specularTarget, uint16_t* hdr)
{
	const int W = int(P.width), H = int(P.height);
	const int w = int(P.gi_width), h = int(P.gi_height);
	const int px = int(blockIdx.x * 16 + threadIdx.x % 16);
	const int py = int(blockIdx.y * 8 + threadIdx.x / 16);
	if (px >= W || py >= H)
	{
		return;
	}
	const int i = py * W + px;
	const V2 texel = v2(1.0f / float(W), 1.0f / float(H));
	const V2 uv = pixelUv(px, py, texel);
	const V3 camera = v3(P.camera_position[0], P.camera_position[1], P.camera_position[2]);
	const int c = texelIndex(uv, W, H);
	const float depth = loadF1(gb.depth, c);
	if (depth >= 0.99999f)
	{
		V3 farPosition = reconstructWorldPosition(P, uv, 1.0f);
		V3 direction = normalize(farPosition - camera);
		storeH4(hdr, i, skyEnabled(P) ? v4(skyRadiance(P, direction), 1.0f) : v4(0.0f, 0.0f, 0.0f, 0.0f));
		return;
	}
	const V4 albedoRoughness = loadU8(gb.albedo, c);
	const V4 normalMetallic = loadU8(gb.normal, c);
	const V3 albedo = albedoRoughness.xyz();
	const float roughness = fmaxf(albedoRoughness.w, 0.05f);
	const float metallic = normalMetallic.w;
	const V3 surfaceNormal = normalize(v3(normalMetallic.x * 2.0f - 1.0f, normalMetallic.y * 2.0f - 1.0f, normalMetallic.z * 2.0f - 1.0f));
	const V4 sh = loadU8(gb.shading_normal, c);
	const V3 normal = normalize(v3(sh.x * 2.0f - 1.0f, sh.y * 2.0f - 1.0f, sh.z * 2.0f - 1.0f));
	const V4 emissiveOcclusion = loadH4(gb.emissive, c);
	const V3 position = reconstructWorldPosition(P, uv, depth);
	const V3 viewDirection = normalize(camera - position);
	const V3 lightPosition = v3(P.light_position[0], P.light_position[1], P.light_position[2]);
	const V3 lightColor = v3(P.light_color[0], P.light_color[1], P.light_color[2]);
	const float s = P.scene_scale;
	const V3 toLight = lightPosition - position;
	const float distanceSquared = fmaxf(dot(toLight, toLight), 0.01f * s * s);
	const V3 lightDirection = toLight * inversesqrt(distanceSquared);

	// evaluateBrdf (brdf.sh:41-62)
	const float normalLight = fmaxf(dot(normal, lightDirection), 0.0f);
	const float normalView = fmaxf(dot(normal, viewDirection), 0.0f);
	const V3 halfway = normalize(viewDirection + lightDirection);
	const V3 f0 = mix(v3s(0.04f), albedo, metallic);
	const float cosine = clampf(dot(halfway, viewDirection), 0.0f, 1.0f);
	const V3 fresnel = f0 + (v3s(1.0f) - f0) * rn_pow5(1.0f - cosine);
	const float rough = fmaxf(roughness, 0.05f);
	const float alpha = rough * rough;
	const float alphaSquared = alpha * alpha;
	const float nh = fmaxf(dot(normal, halfway), 0.0f);
	const float dd = nh * nh * (alphaSquared - 1.0f) + 1.0f;
	const float distribution = alphaSquared / fmaxf(kPi * dd * dd, 0.0001f);
	const float k = (rough + 1.0f) * (rough + 1.0f) / 8.0f;
	const float gl = normalLight / fmaxf(normalLight * (1.0f - k) + k, 0.0001f);
	const float gv = normalView / fmaxf(normalView * (1.0f - k) + k, 0.0001f);
	const float geometry = gl * gv;
	const V3 specular = fresnel * (distribution * geometry) / fmaxf(4.0f * normalLight * normalView, 0.001f) * normalLight;
	const V3 diffuse = (v3s(1.0f) - fresnel) * (1.0f - metallic) * albedo / kPi * normalLight;

	float visibility = 0.0f;
	if (dot(normal, lightDirection) > 0.0f)
	{
		visibility = lightVisibilitySoft(P, atlas, position, surfaceNormal);
	}
	const V3 direct = (diffuse + specular) * (lightColor / distanceSquared) * visibility + loadH4(diDiffuse, c).xyz()
		+ loadH4(diSpecular, c).xyz();

	// upsampleIndirect (fs_composite.sc:48-80), diffuse part.
	const V2 texelCoord = v2(uv.x * float(w) - 0.5f, uv.y * float(h) - 0.5f);
	const V2 baseCoord = v2(floorf(texelCoord.x), floorf(texelCoord.y));
	const V2 blend = texelCoord - baseCoord;
	const V2 giTexel = v2(1.0f / float(w), 1.0f / float(h));
	V3 sum = v3s(0.0f);
	V3 specularSum = v3s(0.0f);
	float weightSum = 0.0f;
	for (int tapIndex = 0; tapIndex < 4; ++tapIndex)
	{
		const V2 offset = v2(float(tapIndex & 1), float(tapIndex >> 1));
		const V2 tapUv = v2((baseCoord.x + offset.x + 0.5f) * giTexel.x, (baseCoord.y + offset.y + 0.5f) * giTexel.y);
		const int t = texelIndex(tapUv, W, H);
		const float tapDepth = loadF1(gb.depth, t);
		if (tapDepth >= 0.99999f)
		{
			continue;
		}
		const V3 tapPosition = reconstructWorldPosition(P, tapUv, tapDepth);
		const V3 tapNormal = decodeNormal(gb.normal, t);
		const V2 bilinear = v2(mixf(1.0f - blend.x, blend.x, offset.x), mixf(1.0f - blend.y, blend.y, offset.y));
		const float weight = (bilinear.x * bilinear.y + 0.01f) * stepf(fabsf(dot(tapPosition - position, surfaceNormal)), 0.03f * s)
			* stepf(0.9f, dot(tapNormal, surfaceNormal));
		sum = sum + loadH4(gi, texelIndex(tapUv, w, h)).xyz() * weight;
		if (specularTarget != nullptr)
		{
			specularSum = specularSum + loadH4(specularTarget, texelIndex(tapUv, w, h)).xyz() * weight;
		}
		weightSum += weight;
	}
	const V3 irradiance = weightSum > 0.0f ? sum / weightSum : loadH4(gi, texelIndex(uv, w, h)).xyz();
	V3 indirect = irradiance
		* (P.composite_options[2] > 0.5f ? albedo * (1.0f - metallic) * emissiveOcclusion.w : v3s(1.0f));
	if (specularTarget != nullptr)
	{
		// fs_composite.sc:131-136
		const V3 specularRadiance = weightSum > 0.0f ? specularSum / weightSum
			: loadH4(specularTarget, texelIndex(uv, w, h)).xyz();
		indirect = indirect + specularRadiance * compositeSpecularAlbedo(f0, roughness, fmaxf(dot(normal, viewDirection), 0.001f))
			* emissiveOcclusion.w * P.composite_specular;
	}
	const V3 result = direct * P.composite_options[0] + indirect * P.composite_options[1]
		+ emissiveOcclusion.xyz() * P.composite_options[3];
	storeH4(hdr, i, v4(result, 1.0f));
}

int launchComposite(const RestirParams& params, const RestirGBuffer& gbuffer, const float* shadowAtlas, const uint16_t* gi,
	const uint16_t* diDiffuse, const uint16_t* diSpecular, const uint16_t* specular, uint16_t* hdr, cudaStream_t s)
{
	const dim3 grid((params.width + 15) / 16, (params.height + 7) / 8);
	const bool oneWave = uint64_t(grid.x) * grid.y <= 148u * 5u;
	(oneWave ? compositeKernel<5> : compositeKernel<8>)<<<grid, 128, 0, s>>>(params, gbuffer, shadowAtlas, gi, diDiffuse, diSpecular,
		specular, hdr);
	return launchStatus();
}

} // namespace
} // namespace restir

using namespace restir;

extern "C" int restir_svgf_variance(const RestirParams* params, const uint16_t* color, const uint16_t* moments,
	const float* receiver, const float* normal, uint16_t* output, void* stream)
{
	if (params == nullptr || color == nullptr || moments == nullptr || receiver == nullptr || normal == nullptr || output == nullptr
		|| params->gi_width == 0 || params->gi_height == 0)
	{
		return RESTIR_ERROR_INVALID_ARGUMENT;
	}
	dim3 grid((params->gi_width + 15) / 16, (params->gi_height + 7) / 8);
	varianceKernel<<<grid, 128, 0, asStream(stream)>>>(*params, color, moments, reinterpret_cast<const float4*>(receiver),
		reinterpret_cast<const float4*>(normal), output);
	return launchStatus();
}

extern "C" int restir_svgf_atrous(const RestirParams* params, int step, const uint16_t* input, const float* receiver,
	const float* normal, uint16_t* output, void* stream)
{
	if (params == nullptr || input == nullptr || receiver == nullptr || normal == nullptr || output == nullptr || step < 1
		|| params->gi_width == 0 || params->gi_height == 0 || input == output)
	{
		return RESTIR_ERROR_INVALID_ARGUMENT;
	}
	// All taps but the centre lie outside the image from the larger size on.
	const uint32_t s = min(uint32_t(step), max(params->gi_width, params->gi_height));
	// A residue has at most ceil(size / step) pixels per axis.
	const uint32_t residuesX = min(s, params->gi_width), residuesY = min(s, params->gi_height);
	const uint32_t blocksX = ((params->gi_width + s - 1u) / s + kFilterW - 1u) / kFilterW * residuesX;
	const uint32_t blocksY = ((params->gi_height + s - 1u) / s + kFilterH - 1u) / kFilterH * residuesY;
	// Tiles where the residues fill them well, or all blocks are in flight at once;
	// the farther the taps, the more of them lie outside the image, which a tile
	// does not gain from. us, tiles / taps from the image: 1920x1080, step 16 (88%
	// full) 283 / 324, 40 (84%) 274 / 320, 48 (78%) 311 / 311, 80 (63%) 348 / 298,
	// 96 (44%) 449 / 291, 256 (25%) 576 / 236; 960x540, 16 (79%) 84 / 92, 32 (66%)
	// 86 / 86, 48 (44%) 125 / 84; 640x360, 48 (78%) 49 / 41; 128x128, 28 (16%, 784
	// blocks) 18 / 23, 40 (8%, 1,600 blocks) 25 / 18.
	const uint64_t tilePixels = uint64_t(blocksX) * blocksY * (kFilterW * kFilterH);
	const uint64_t pixels = uint64_t(params->gi_width) * params->gi_height;
	const cudaStream_t queue = asStream(stream);
	if ((s < 48u && pixels * 10u >= tilePixels * 7u) || uint64_t(blocksX) * blocksY <= 148u * 8u)
	{
		atrousKernel<<<blocksX * blocksY, 128, 0, queue>>>(*params, int(s), int(residuesX), int(residuesY), int(blocksX),
			input, reinterpret_cast<const float4*>(receiver), reinterpret_cast<const float4*>(normal), output);
	}
	else
	{
		const dim3 grid((params->gi_width + kFilterW - 1) / kFilterW, (params->gi_height + kFilterH - 1) / kFilterH);
		atrousDirectKernel<<<grid, 128, 0, queue>>>(*params, int(s), input, reinterpret_cast<const float4*>(receiver),
			reinterpret_cast<const float4*>(normal), output);
	}
	return launchStatus();
}

extern "C" int restir_composite(const RestirParams* params, const RestirGBuffer* gbuffer, const float* shadow_atlas,
	const uint16_t* gi, const uint16_t* di_diffuse, const uint16_t* di_specular, uint16_t* hdr, void* stream)
{
	if (params == nullptr || gbuffer == nullptr || gbuffer->albedo == nullptr || gbuffer->normal == nullptr
		|| gbuffer->emissive == nullptr || gbuffer->shading_normal == nullptr || gbuffer->depth == nullptr
		|| shadow_atlas == nullptr || gi == nullptr || hdr == nullptr || params->width == 0 || params->height == 0)
	{
		return RESTIR_ERROR_INVALID_ARGUMENT;
	}
	return launchComposite(*params, *gbuffer, shadow_atlas, gi, di_diffuse, di_specular, nullptr, hdr, asStream(stream));
}

extern "C" int restir_composite_specular(const RestirParams* params, const RestirGBuffer* gbuffer, const float* shadow_atlas,
	const uint16_t* gi, const uint16_t* di_diffuse, const uint16_t* di_specular, const uint16_t* specular, uint16_t* hdr,
	void* stream)
{
	if (params == nullptr || gbuffer == nullptr || gbuffer->albedo == nullptr || gbuffer->normal == nullptr
		|| gbuffer->emissive == nullptr || gbuffer->shading_normal == nullptr || gbuffer->depth == nullptr
		|| shadow_atlas == nullptr || gi == nullptr || hdr == nullptr || params->width == 0 || params->height == 0)
	{
		return RESTIR_ERROR_INVALID_ARGUMENT;
	}
	return launchComposite(*params, *gbuffer, shadow_atlas, gi, di_diffuse, di_specular, specular, hdr, asStream(stream));
}
