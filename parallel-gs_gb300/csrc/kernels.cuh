// kernels.cuh -- sm_103a kernels of the GS backend.
//
//   setup_kernel     one thread per primitive: edge planes, reciprocal area,
//                    attribute deltas, bounding box (triangle_setup.comp)
//   bin_kernel       32 primitives per group, 1 to 16 CTAs each: per-coarse-tile
//                    membership and super-sampling flags (binning.comp), and
//                    the primitive's bit in the bitmask of every 8x8 sub-tile
//                    it may touch; the bitmask keeps primitive order without
//                    any sort
//   shade_kernel     one CTA per 8x8-pixel sub-tile of a coarse tile, one
//                    thread per pixel sample (256 threads at most, the rest
//                    in turn or, where the list is long, in CTAs of its own);
//                    walks the tile's primitives in order with the
//                    deferred-shading logic of ubershader.comp
//   upload_kernel    host->local and local->local transfers into swizzled VRAM
//   clut_kernel      CLUT instance load (clut_write.comp)
//
// All floating-point steps use explicit round-to-nearest intrinsics so that
// no multiply-add is contracted; the build also passes -fmad=false.
#pragma once

#include "gs_defs.h"
#include "pgs.h"

#include <cuda_runtime.h>
#include <stdint.h>

namespace pgs
{
// ---------------------------------------------------------------------------
// Device records.
struct __align__(16) PrimSetup
{
	int32_t a[3];
	float inv_area;
	int32_t b[3];
	float error_i;
	int32_t c[3];
	float error_j;
	int32_t bb[4];
	uint32_t z[4]; // depth at the first vertex, float differences to the others, inv_area again
};
static_assert(sizeof(PrimSetup) == 80, "PrimSetup layout");

// Interpolation terms per primitive: value at the first vertex and the
// differences to the other two, for S T Q FOG and for the unorm colour.
struct __align__(16) TransformedAttr
{
	float stqf0[4];
	float stqf1[4];
	float stqf2[4];
	float rgba0[4];
	float rgba1[4];
	float rgba2[4];
};
static_assert(sizeof(TransformedAttr) == 96, "TransformedAttr layout");

// Decoded framebuffer instance for the shading kernels.
struct DevInstance
{
	uint32_t fb_base, fb_stride, fb_psm;
	uint32_t zb_base, zb_psm; // zb_psm == 0xffffffff when not Z sensitive
	int32_t base_x, base_y;
	uint32_t tiles_w, tiles_h;
	uint32_t rate_x_log2, rate_y_log2;
	uint32_t preserve_samples;
	uint32_t instance;
	uint32_t prim_lo, prim_count; // primitive range of this dispatch
	uint32_t mask_words;          // bitmask words per 8x8 sub-tile (1 bit per primitive)
	uint32_t sub_w, sub_h;        // 8x8 sub-tiles per row / column
	int32_t snap_mask_y;          // raster snap of rows: half the sample pitch when field rendering
	uint32_t force_ss;            // field rendering: every covered tile super-sampled
	uint32_t blend_demote;        // primitives per coarse tile that demote a blended tile, 0 = off
	uint32_t split_count;         // primitives per coarse tile that split its sub-tiles (split_tile), 0 = never
	uint32_t split_first;         // CTAs for split parts in front of those of the sub-tiles
};

// Linear RGBA8 image decoded from swizzled VRAM + CLUT for one mip level of
// one texture of a pass (the role of the reference's texture cache,
// upload.comp:108-229); slot l of texture t is entry t * TEX_SLOTS + l: mip
// level l, or for a super-sampled texture layer l (0: single-sampled image,
// s + 1: sample s).
constexpr uint32_t TEX_LEVELS = 7;
constexpr uint32_t TEX_SLOTS = 17;
// Phase LUT of super-sampled texture filtering: 64 x 64 (x, y) pairs for
// bilinear, then 32 x 32 sample ids for nearest.
constexpr uint32_t PHASE_LUT_WORDS = 64 * 64 * 2 + 32 * 32;

// Mean position of the samples inside a pixel per sampling grid
// (get_average_sampling_offset, utils.h:108-126).
__host__ __device__ inline float average_sampling_offset(uint32_t rx, uint32_t ry)
{
	if (rx == ry)
		return ry == 0 ? 0.0f : (ry == 1 ? 0.25f : (ry == 2 ? 0.375f : 0.4375f));
	if (rx == 0 && ry == 1)
		return 0.25f;
	if (rx == 1 && ry == 2)
		return 0.375f;
	if (rx == 0 && ry == 2)
		return 0.375f;
	if (rx == 1 && ry == 3)
		return 0.4375f;
	return 0.0f;
}

__host__ __device__ inline uint32_t texture_slots(const pgs_texture_desc &t)
{
	return t.samples > 1 ? t.samples + 1 : (t.levels > 1 ? t.levels : 1u);
}

struct TexImage
{
	uint32_t offset; // first texel in PassParams::texels
	uint32_t ext_u, ext_v;
	uint32_t padding;
};

// How level 0 of a texture is sampled along one axis: a wrap mode as
// (v & and_mask | or_mask) clamped to [lo, hi], the scale to 1/16 texels, and
// the bounds of the coordinate there (the +-2047 of every coordinate and the
// sampler's own clamp).  `place` is the image's first texel on the U axis and
// its row length on the V axis.
struct __align__(16) TexAxis
{
	int32_t and_mask, or_mask, lo, hi;
	float clamp_lo, clamp_hi, scale;
	uint32_t place;
};

// Both axes, for texel and perspective coordinates (+ 2), each without and with
// the primitive's clamp bit (+ 1).
struct TexSampler
{
	TexAxis u[4], v[4];
};

// Flat-primitive depth buckets found by triangle setup in a super-sampled pass
// (SingleSampleHeuristic, gs/shaders/data_structures.h:190-195).  Each of the
// 256 buckets covers 2^16 (2^8 for 16-bit Z) depth values.
struct SsHeuristic
{
	uint32_t bucket_count;
	uint32_t active[8];
	uint32_t bucket[256];
};

// Per-instance depth quantisation for the heuristic
// (dispatch_single_sample_heuristic, gs/gs_renderer.cpp:1979-2039).
struct HeuristicParams
{
	uint32_t z_shift_bucket[8];
	uint32_t z_shift[8];
	uint32_t z_max[8];
	uint32_t instance_mask;
};

// Decision of the heuristic for one primitive, applied after every bucket has
// been evaluated against the states triangle setup produced.
constexpr uint8_t HEURISTIC_SET_SNAP_RASTER = 1;
constexpr uint8_t HEURISTIC_CLEAR_SNAP_ATTRIBUTE = 2;

struct PassParams
{
	// Textures [snap_limit[k - 1], snap_limit[k]) are decoded from
	// snap_vram[k], the rest from vram.
	const uint8_t *snap_vram[PGS_MAX_VRAM_SNAPSHOTS];
	uint32_t snap_limit[PGS_MAX_VRAM_SNAPSHOTS];
	uint32_t num_snaps;
	const pgs_vertex_position *pos;
	const pgs_vertex_attribute *attr;
	// Primitive words: setup reads them from prims_in and writes prims, which the
	// kernels after it use (the same array where a pass is run once).
	const pgs_primitive_attribute *prims_in;
	pgs_primitive_attribute *prims;
	const pgs_state_vector *states;
	const pgs_texture_desc *textures;
	const TexImage *tex_images;
	const TexSampler *samplers;
	uint32_t *texels;
	PrimSetup *setup;
	TransformedAttr *tattr;
	uint32_t num_prims;
	uint32_t num_states, num_textures;
	uint32_t max_tex_levels;      // largest slot count (mip levels or sample layers) of the pass's textures
	uint32_t rp_is_blur_mask;     // per instance: the pass looks like a blur kernel (render_pass_instance_is_deduced_blur)
	uint32_t force_linear_ss;     // FORCE_LINEAR_SUPER_SAMPLE: field rendering with super-sampled textures
	const uint32_t *phase_lut;    // PHASE_LUT_WORDS words
	uint32_t tile_size_log2;
	uint32_t has_aa1, has_scanmsk, has_ss_reference;
	uint32_t setup_rate_x_log2, setup_rate_y_log2;
	uint32_t opaque_fbmask[8];
	uint8_t *vram;
	// Depth reads come from this snapshot of all VRAM planes when set
	// (frame and depth buffer aliased), else from vram.
	const uint8_t *zcache;
	const uint16_t *clut;
	const float *rcp_float_lut;
	const float *unorm_lut;
	uint32_t *error_flags;
	unsigned long long *fragment_counter;
	// 4 bits per instance: flat-primitive bucket shift / 8 (z_shift_to_bucket,
	// gs/gs_renderer.cpp:1914-1934).
	uint32_t packed_z_shift;
	SsHeuristic *heuristic;
	uint8_t *heuristic_action;
};

// Per-tile flag bits written by bin_kernel.
constexpr uint32_t TILE_NONEMPTY = 1u << 0;
constexpr uint32_t TILE_REQ_SS = 1u << 1;
constexpr uint32_t TILE_REQ_SS_ZW = 1u << 2;
constexpr uint32_t TILE_HAS_ZW = 1u << 3;
// Primitives binned to the tile, counted from this bit for blend demotion, or by
// every eighth primitive for splitting.
constexpr uint32_t TILE_COUNT_SHIFT = 8;
constexpr uint32_t SPLIT_ALL = ~0u; // DevInstance::split_count: every tile

constexpr uint32_t ERROR_FLAG_TILE_OVERFLOW = 1u << 0;

__constant__ uint8_t c_rcp_tab[256];

// Largest shading CTA, as the sampling rate it holds a whole sub-tile of, and
// occupancy target of the shading kernels in 256-thread units per SM: 4 means at
// most 64 registers per thread.  Textured 4x frame of 52,000 primitives: 4 CTAs
// 618 us, 5 631 us, 6 642 us; 128 threads 596 us where 256 take 560.  Plain 1x
// frame at 10, 12, 16, 20, 24 CTAs of 64 threads: 55, 48.5, 47, 50, 64 us.
// Feedback frame of 100,000 primitives at 16x: 4 CTAs 2.74 ms (alone 3.28), 5
// 2.74 (3.33), 6 2.81 (3.48).
#ifndef PGS_SHADE_CTA_NS
#define PGS_SHADE_CTA_NS 4
#endif
#ifndef PGS_SHADE_OCC
#define PGS_SHADE_OCC 4
#endif
#define PGS_SHADE_MIN_BLOCKS(NS) (PGS_SHADE_OCC * 4 / ((NS) < PGS_SHADE_CTA_NS ? (NS) : PGS_SHADE_CTA_NS))

// ---------------------------------------------------------------------------
// Scalar helpers.
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float u2f(uint32_t u) { return __uint_as_float(u); }
__device__ __forceinline__ uint32_t f2u(float f) { return __float_as_uint(f); }

__device__ __forceinline__ int32_t idot3(const int32_t p[3], int32_t x, int32_t y)
{
	return int32_t(uint32_t(p[0]) * uint32_t(x) + uint32_t(p[1]) * uint32_t(y) + uint32_t(p[2]));
}

// Reciprocal of a 32-bit fixed-point area: table seed plus two Newton steps in
// 32-bit fixed point, quantised to FP32 (rcp_fixed, math_utils.h:27-61).
__device__ __forceinline__ float rcp_fixed(uint32_t b)
{
	int lz = __clz(b);
	uint32_t nb = b << lz;
	uint32_t rcp = uint32_t(c_rcp_tab[(nb >> 23) & 0xffu]) | 0x100u;
	uint32_t f = (rcp * rcp) << 14;
	uint32_t p = __umulhi(f, nb);
	rcp = (rcp << 23) - p;
	rcp <<= 1;
	p = __umulhi(rcp, nb);
	rcp = __umulhi(rcp, 0u - p);
	rcp = (rcp + 64u) >> 7;
	rcp -= 1u << 23;
	rcp += uint32_t(127 - 32 + lz) << 23;
	return u2f(rcp);
}

// Reciprocal by table seed + 4 Newton-Raphson steps (rcp_float, math_utils.h:65-101).
__device__ __forceinline__ float rcp_float(float v, const float *lut)
{
	uint32_t u = f2u(v);
	int e = int((u >> 23) & 0xffu);
	if (e == 0)
		return u2f(0x7f800000u);
	int shifted = 127 - e;
	float x = lut[(u >> 15) & 0xffu];
	u = (u & ((1u << 23) - 1u)) | (127u << 23);
	float a = u2f(u);
	#pragma unroll
	for (int it = 0; it < 4; it++)
	{
		float x2 = fmul(x, 2.0f);
		float xs = fmul(x, x);
		float xsa = fmul(xs, a);
		x = fsub(x2, xsa);
	}
	return ldexpf(x, shifted);
}

__device__ __forceinline__ bool tie_break(int32_t ex, int32_t ey) { return ey > 0 || (ey == 0 && ex < 0); }

__device__ __forceinline__ bool order_less(int32_t ax, int32_t ay, int32_t bx, int32_t by, uint32_t az, uint32_t bz)
{
	if (bz != az) return az < bz;
	if (by != ay) return ay < by;
	return ax < bx;
}

// Inclusive sum over the lanes of a warp.
__device__ __forceinline__ uint32_t warp_scan(uint32_t v, uint32_t lane)
{
	uint32_t x = v;
	#pragma unroll
	for (int o = 1; o < 32; o <<= 1)
	{
		const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
		if (lane >= uint32_t(o))
			x += y;
	}
	return x;
}

template <typename T>
__device__ __forceinline__ void dswap(T &a, T &b) { T t = a; a = b; b = t; }

// ---------------------------------------------------------------------------
// K1: triangle setup.
__device__ __forceinline__ float unorm8_lut(const float *lut, uint32_t c, int ch) { return __ldg(lut + ((c >> (8 * ch)) & 0xffu)); }

// Colour terms of the shading interpolation c0 + (c1 - c0) i + (c2 - c0) j,
// per channel in unorm floats.
__device__ __forceinline__ void set_color_terms(const PassParams &P, TransformedAttr &ta, uint32_t r0, uint32_t r1,
                                                uint32_t r2)
{
	#pragma unroll
	for (int k = 0; k < 4; k++)
	{
		const float c0 = unorm8_lut(P.unorm_lut, r0, k), c1 = unorm8_lut(P.unorm_lut, r1, k);
		const float c2 = unorm8_lut(P.unorm_lut, r2, k);
		ta.rgba0[k] = c0;
		ta.rgba1[k] = fsub(c1, c0);
		ta.rgba2[k] = fsub(c2, c0);
	}
}

__global__ void __launch_bounds__(128) setup_kernel(PassParams P)
{
	uint32_t index = blockIdx.x * blockDim.x + threadIdx.x;
	if (index >= P.num_prims)
		return;

	pgs_primitive_attribute pa = P.prims_in[index];
	PrimSetup out;
	TransformedAttr ta;
	const int sry = int(P.setup_rate_y_log2);

	int order0 = 0, order1 = 1, order2 = 2;
	uint32_t st = pa.state;
	bool parallelogram = (st >> STATE_BIT_PARALLELOGRAM) & 1;
	bool perspective = (st >> STATE_BIT_PERSPECTIVE) & 1;
	bool iip = (st >> STATE_BIT_IIP) & 1;
	bool fix = (st >> STATE_BIT_FIX) & 1;
	bool sprite = (st >> STATE_BIT_SPRITE) & 1;
	bool line = (st >> STATE_BIT_LINE) & 1;
	bool multisample = (st >> STATE_BIT_MULTISAMPLE) & 1;
	uint32_t provoking = (st >> STATE_PARALLELOGRAM_PROVOKING_OFFSET) & 3u;
	uint32_t opaque_fbmask = P.opaque_fbmask[(st >> STATE_VERTEX_RENDER_PASS_INSTANCE_OFFSET) & 7u];

	pgs_vertex_position v0 = P.pos[3 * index], v1 = P.pos[3 * index + 1], v2 = P.pos[3 * index + 2];
	int32_t ax = v0.x, ay = v0.y, bx = v1.x, by = v1.y, cx = v2.x, cy = v2.y;
	uint32_t za = v0.z, zb = v1.z, zc = v2.z;

	if (line)
	{
		bool sax = (ax & 15) == 0, say = (ay & 15) == 0, sbx = (bx & 15) == 0, sby = (by & 15) == 0;
		if ((sax || sbx) && bx > ax) { ax += 1; bx += 1; }
		if ((say || sby) && by > ay) { ay += 1; by += 1; }
	}

	if ((!parallelogram || line) && !fix)
	{
		if (!line && !order_less(bx, by, cx, cy, zb, zc))
		{
			dswap(order1, order2); dswap(bx, cx); dswap(by, cy); dswap(zb, zc);
		}
		if (!order_less(ax, ay, bx, by, za, zb))
		{
			dswap(order0, order1); dswap(ax, bx); dswap(ay, by); dswap(za, zb);
		}
	}
	else if (provoking == 1)
	{
		dswap(order0, order1); dswap(ax, bx); dswap(ay, by); dswap(za, zb);
	}
	else if (provoking == 2)
	{
		dswap(order0, order2); dswap(ax, cx); dswap(ay, cy); dswap(za, zc);
	}

	if (sprite)
	{
		cx = ax; cy = by;
		by = ay;
	}
	else if (line)
	{
		int32_t abx = bx - ax, aby = by - ay;
		if (abs(abx) >= abs(aby))
		{
			int32_t yd = -((abx > 0) - (abx < 0)) * 8;
			if (multisample) yd *= 2;
			cy = ay + yd; ay -= yd; by -= yd;
			if (!multisample) { ay += 1; by += 1; }
			cx = ax;
		}
		else
		{
			int32_t xd = ((aby > 0) - (aby < 0)) * 8;
			if (multisample) xd *= 2;
			cx = ax + xd; ax -= xd; bx -= xd;
			if (!multisample) { ax += 1; bx += 1; }
			cy = ay;
		}
	}

	int32_t abx = bx - ax, aby = by - ay, acx = cx - ax, acy = cy - ay;
	int64_t signed_area = int64_t(aby) * acx - int64_t(abx) * acy;
	if (signed_area == 0)
	{
		out.bb[0] = 0; out.bb[1] = 0; out.bb[2] = -1; out.bb[3] = -1;
		reinterpret_cast<int4 *>(&P.setup[index])[3] = make_int4(0, 0, -1, -1);
		if (sry != 0)
			pa.state = st | (1u << STATE_BIT_SNAP_ATTRIBUTE);
		P.prims[index] = pa;
		return;
	}

	uint32_t area;
	bool flipped = signed_area < 0;
	if (flipped)
	{
		area = uint32_t(0ull - uint64_t(signed_area));
		dswap(abx, acx); dswap(aby, acy);
		dswap(bx, cx); dswap(by, cy);
		dswap(zb, zc);
		dswap(order1, order2);
	}
	else
		area = uint32_t(uint64_t(signed_area));

	int32_t bcx = cx - bx, bcy = cy - by;
	int32_t cax = -acx, cay = -acy;
	int32_t dcdx = aby, dcdy = -abx;
	int32_t dadx = bcy, dady = -bcx;
	int32_t dbdx = cay, dbdy = -cax;
	int64_t const_c = int64_t(-ax) * dcdx - int64_t(ay) * dcdy;
	int64_t const_a = int64_t(-bx) * dadx - int64_t(by) * dady;
	int64_t const_b = int64_t(-cx) * dbdx - int64_t(cy) * dbdy;
	bool tba = tie_break(bcx, bcy), tbb = tie_break(cax, cay), tbc = tie_break(abx, aby);
	int32_t err_a = !tba, err_b = !tbb, err_c = !tbc;
	const_a -= err_a; const_b -= err_b; const_c -= err_c;
	err_a += int32_t(uint64_t(const_a) & 1u);
	err_b += int32_t(uint64_t(const_b) & 1u);
	err_c += int32_t(uint64_t(const_c) & 1u);
	int32_t flip_b = 0, flip_c = 0;
	if (parallelogram)
	{
		int32_t tbo = 1 - int32_t(tbb) - int32_t(tbc);
		flip_b = (tbo + err_b + err_a + 2) >> 1;
		flip_c = (tbo + err_c + err_a + 2) >> 1;
	}

	float inv_area = rcp_fixed(area);
	float inv_area_scaled = fmul(inv_area, 2.0f);
	float error_i = fmul(__int2float_rn(err_b), inv_area);
	float error_j = fmul(__int2float_rn(err_c), inv_area);

	if (sprite) { zb = za; zc = za; }
	else if (line) { zc = za; }
	if (fix || sprite) { order0 = 0; order1 = 1; order2 = 2; }

	pgs_vertex_attribute at0 = P.attr[3 * index + order0];
	pgs_vertex_attribute at1 = P.attr[3 * index + order1];
	pgs_vertex_attribute at2 = {};
	if (!sprite && !line)
		at2 = P.attr[3 * index + order2];

	float s0[4], s1[4], s2[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
	if (perspective)
	{
		s0[0] = at0.s; s0[1] = at0.t; s0[2] = at0.q; s0[3] = at0.fog;
		s1[0] = at1.s; s1[1] = at1.t; s1[2] = at1.q; s1[3] = at1.fog;
		if (!sprite && !line) { s2[0] = at2.s; s2[1] = at2.t; s2[2] = at2.q; s2[3] = at2.fog; }
	}
	else
	{
		s0[0] = fmul(float(at0.u), 0.0625f); s0[1] = fmul(float(at0.v), 0.0625f); s0[2] = at0.q; s0[3] = at0.fog;
		s1[0] = fmul(float(at1.u), 0.0625f); s1[1] = fmul(float(at1.v), 0.0625f); s1[2] = at1.q; s1[3] = at1.fog;
		if (!sprite && !line)
		{
			s2[0] = fmul(float(at2.u), 0.0625f); s2[1] = fmul(float(at2.v), 0.0625f); s2[2] = at2.q; s2[3] = at2.fog;
		}
	}

	if (sprite)
	{
		float o0x = s0[0], o0y = s0[1], o0z = s0[2], o0w = s0[3], o1x = s1[0], o1y = s1[1];
		if (flipped)
		{
			s2[0] = o1x; s2[1] = o0y; s2[2] = o0z; s2[3] = o0w;
			s1[0] = o0x; s1[1] = o1y; s1[2] = o0z; s1[3] = o0w;
		}
		else
		{
			s2[0] = o0x; s2[1] = o1y; s2[2] = o0z; s2[3] = o0w;
			s1[0] = o1x; s1[1] = o0y; s1[2] = o0z; s1[3] = o0w;
		}
	}
	else if (line)
	{
		s2[0] = s0[0]; s2[1] = s0[1]; s2[2] = s0[2]; s2[3] = s0[3];
	}

	if (perspective)
	{
		if (s0[2] < 0.0f)
		{
			s0[0] = -s0[0]; s0[1] = -s0[1]; s1[0] = -s1[0]; s1[1] = -s1[1]; s2[0] = -s2[0]; s2[1] = -s2[1];
		}
		s0[2] = fabsf(s0[2]); s1[2] = fabsf(s1[2]); s2[2] = fabsf(s2[2]);
		uint32_t qexp = (f2u(fmaxf(fmaxf(s0[2], s1[2]), s2[2])) >> 23) & 0xffu;
		s0[2] = u2f(f2u(s0[2]) & ~0xffu);
		s1[2] = u2f(f2u(s1[2]) & ~0xffu);
		s2[2] = u2f(f2u(s2[2]) & ~0xffu);
		uint32_t sexp = (f2u(fmaxf(fmaxf(fabsf(s0[0]), fabsf(s1[0])), fabsf(s2[0]))) >> 23) & 0xffu;
		uint32_t texp = (f2u(fmaxf(fmaxf(fabsf(s0[1]), fabsf(s1[1])), fabsf(s2[1]))) >> 23) & 0xffu;
		uint32_t schop = min(9u + max(sexp, qexp) - sexp, 23u);
		uint32_t tchop = min(9u + max(texp, qexp) - texp, 23u);
		uint32_t smask = ~((1u << schop) - 1u), tmask = ~((1u << tchop) - 1u);
		s0[0] = u2f(f2u(s0[0]) & smask); s1[0] = u2f(f2u(s1[0]) & smask); s2[0] = u2f(f2u(s2[0]) & smask);
		s0[1] = u2f(f2u(s0[1]) & tmask); s1[1] = u2f(f2u(s1[1]) & tmask); s2[1] = u2f(f2u(s2[1]) & tmask);
		bool needs_lod = (pa.tex2 & TEX2_FIXED_LOD_BIT) == 0;
		if (!needs_lod && s0[2] == s1[2] && s0[2] == s2[2])
		{
			float inv_q = rcp_float(s0[2], P.rcp_float_lut);
			s0[0] = fmul(s0[0], inv_q); s0[1] = fmul(s0[1], inv_q);
			s1[0] = fmul(s1[0], inv_q); s1[1] = fmul(s1[1], inv_q);
			s2[0] = fmul(s2[0], inv_q); s2[1] = fmul(s2[1], inv_q);
			s0[2] = 1.0f; s1[2] = 1.0f; s2[2] = 1.0f;
		}
	}

	float di[4], dj[4];
	#pragma unroll
	for (int k = 0; k < 4; k++)
	{
		di[k] = fix ? 0.0f : fsub(s1[k], s0[k]);
		dj[k] = fix ? 0.0f : fsub(s2[k], s0[k]);
		ta.stqf0[k] = s0[k];
		ta.stqf1[k] = di[k];
		ta.stqf2[k] = dj[k];
	}
	if (iip && !sprite)
	{
		uint32_t r0 = at0.rgba, r1 = at1.rgba, r2 = at2.rgba;
		if (fix) r1 = r0;
		if (fix || line) r2 = r0;
		set_color_terms(P, ta, r0, r1, r2);
	}
	else
	{
		uint32_t flat = P.attr[3 * index].rgba;
		set_color_terms(P, ta, flat, flat, flat);
	}

	int32_t pa0 = dadx, pa1 = dady, pa2 = int32_t(uint32_t(uint64_t(const_a) >> 1));
	int32_t pb0 = dbdx, pb1 = dbdy, pb2 = int32_t(uint32_t(uint64_t(const_b) >> 1));
	int32_t pc0 = dcdx, pc1 = dcdy, pc2 = int32_t(uint32_t(uint64_t(const_c) >> 1));
	uint32_t axw = (uint32_t(pa0) << 6) & ~1u;
	axw |= uint32_t(parallelogram);
	axw = (axw & ~(3u << 2)) | ((uint32_t(flip_b) & 3u) << 2);
	axw = (axw & ~(3u << 4)) | ((uint32_t(flip_c) & 3u) << 4);

	int32_t dx = parallelogram ? (bx + cx - ax) : cx;
	int32_t dy = parallelogram ? (by + cy - ay) : cy;

	int32_t di_r = 0, dj_r = 0;
	if (sprite)
	{
		int32_t xd = dx - ax, yd = dy - ay;
		if (xd > 0 && (xd & (xd - 1)) != 0) { di_r += pb0; dj_r += pc0; }
		if (yd > 0 && (yd & (yd - 1)) != 0) { di_r += pb1; dj_r += pc1; }
	}
	else if (parallelogram && !perspective)
	{
		bool nearest = (pa.tex & TEX_SAMPLER_MAG_LINEAR_BIT) == 0;
		bool npot_area = (area & (area - 1)) != 0;
		if (nearest && npot_area)
		{
			int32_t d0x = int32_t(at0.u) - ax, d0y = int32_t(at0.v) - ay;
			int32_t d1x = int32_t(at1.u) - bx, d1y = int32_t(at1.v) - by;
			int32_t d2x = int32_t(at2.u) - cx, d2y = int32_t(at2.v) - cy;
			if (d0x == d1x && d0y == d1y && d0x == d2x && d0y == d2y)
			{
				bool mis_x = (min(ax, dx) & 15) != 0, mis_y = (min(ay, dy) & 15) != 0;
				float dudx = fadd(fmul(di[0], float(pb0)), fmul(dj[0], float(pc0)));
				float dvdx = fadd(fmul(di[1], float(pb0)), fmul(dj[1], float(pc0)));
				float dudy = fadd(fmul(di[0], float(pb1)), fmul(dj[0], float(pc1)));
				float dvdy = fadd(fmul(di[1], float(pb1)), fmul(dj[1], float(pc1)));
				bool adj_x = mis_x && ((dudx > 0.0f && dvdx == 0.0f) || (dvdx > 0.0f && dudx == 0.0f));
				bool adj_y = mis_y && ((dudy > 0.0f && dvdy == 0.0f) || (dvdy > 0.0f && dudy == 0.0f));
				if (adj_x) { di_r -= pb0; dj_r -= pc0; }
				if (adj_y) { di_r -= pb1; dj_r -= pc1; }
			}
		}
	}
	float eighth = fmul(0.125f, inv_area_scaled);
	error_i = fadd(error_i, fmul(__int2float_rn(di_r), eighth));
	error_j = fadd(error_j, fmul(__int2float_rn(dj_r), eighth));

	out.a[0] = int32_t(axw); out.a[1] = pa1; out.a[2] = pa2;
	out.b[0] = pb0; out.b[1] = pb1; out.b[2] = pb2;
	out.c[0] = pc0; out.c[1] = pc1; out.c[2] = pc2;
	out.inv_area = inv_area_scaled;
	out.error_i = error_i;
	out.error_j = error_j;
	out.z[0] = za;
	out.z[1] = f2u(__uint2float_rn(zb - za));
	out.z[2] = f2u(__uint2float_rn(zc - za));
	out.z[3] = f2u(inv_area_scaled);

	int32_t lox = min(min(ax, bx), min(cx, dx)), loy = min(min(ay, by), min(cy, dy));
	int32_t hix = max(max(ax, bx), max(cx, dx)), hiy = max(max(ay, by), max(cy, dy));
	lox = (lox + (15 >> sry)) >> 4;
	loy = (loy + (15 >> sry)) >> 4;
	hix = (hix - 1) >> 4;
	hiy = (hiy - 1) >> 4;
	if (multisample && !line) { lox -= 1; loy -= 1; hix += 1; hiy += 1; }
	out.bb[0] = max(lox, int32_t(pa.bb[0]));
	out.bb[1] = max(loy, int32_t(pa.bb[1]));
	out.bb[2] = min(hix, int32_t(pa.bb[2]));
	out.bb[3] = min(hiy, int32_t(pa.bb[3]));

	uint32_t tex = pa.tex;
	if (sprite && !perspective)
	{
		int32_t u0x = int32_t(at0.u) - ax, u0y = int32_t(at0.v) - ay;
		int32_t u1x = int32_t(at1.u) - dx, u1y = int32_t(at1.v) - dy;
		int32_t mnx = min(u0x, u1x), mny = min(u0y, u1y), mxx = max(u0x, u1x), mxy = max(u0y, u1y);
		bool csx = (mnx & 15) == 8, csy = (mny & 15) == 8;
		bool nsx = (mxx & 15) == 9, nsy = (mxy & 15) == 9;
		int32_t ddx = abs(dx - ax), ddy = abs(dy - ay);
		nsx = nsx && (ddx & (ddx - 1)) != 0;
		nsy = nsy && (ddy & (ddy - 1)) != 0;
		bool no_interp = (mxx - mnx) <= 1 && (mxy - mny) <= 1;
		if ((nsx || csx) && (nsy || csy) && no_interp)
			tex &= ~TEX_SAMPLER_MAG_LINEAR_BIT;
	}

	uint32_t new_state = st;
	if (pa.fbmsk != opaque_fbmask && (new_state & (1u << STATE_BIT_OPAQUE)))
		new_state &= ~(1u << STATE_BIT_OPAQUE);

	// Super-sampled textures (triangle_setup.comp:677-825): nearest blits map
	// sample to sample, nearest downsamples and blur kernels fall back to the
	// single-sampled layer, linear upsamples read the resolved layer (with
	// FORCE_LINEAR_SUPER_SAMPLE, for field rendering, blur kernels read the
	// resolved layer linearly and linear downsamples and upsamples stay per
	// sample); what stays per-sample interpolates per sample around the
	// single-sampled mean position.
	if (sry != 0 && (tex & (TEX_PER_SAMPLE_BIT | TEX_SAMPLE_MAPPING_BIT)) == TEX_PER_SAMPLE_BIT)
	{
		const int32_t udx = abs(int32_t(at1.u) - int32_t(at0.u)), udy = abs(int32_t(at1.v) - int32_t(at0.v));
		const int32_t ddx = abs(dx - ax), ddy = abs(dy - ay);
		if ((tex & TEX_SAMPLER_MAG_LINEAR_BIT) == 0)
		{
			if (perspective)
				tex |= TEX_SAMPLE_MAPPING_BIT;
			else if (udx > ddx + 1 || udy > ddy + 1)
				tex &= ~TEX_PER_SAMPLE_BIT;
			else if (udx >= ddx - 16 || udy >= ddy - 16)
			{
				const uint32_t blend = P.states[min(st & STATE_INDEX_MASK, P.num_states - 1u)].blend_mode;
				const uint32_t inst = (st >> STATE_VERTEX_RENDER_PASS_INSTANCE_OFFSET) & 7u;
				const bool blur = ((P.rp_is_blur_mask >> inst) & 1u) && (blend & BLEND_MODE_ABE_BIT) &&
				                  !(st & (1u << STATE_BIT_Z_TEST)) &&
				                  ((blend >> BLEND_MODE_A_MODE_OFFSET) & 3u) == BLEND_RGB_SOURCE &&
				                  ((blend >> BLEND_MODE_B_MODE_OFFSET) & 3u) == BLEND_RGB_ZERO &&
				                  ((blend >> BLEND_MODE_D_MODE_OFFSET) & 3u) == BLEND_RGB_DEST;
				if (blur && P.force_linear_ss)
				{
					// Field rendering keeps blur kernels per sample: the
					// resolved layer, filtered linearly, with the mean sample
					// position moved to the texel centre
					// (triangle_setup.comp:729-746).
					tex |= TEX_SAMPLE_RESOLVED_BIT | TEX_SAMPLER_MAG_LINEAR_BIT;
					const int32_t avg_u = (int32_t(at0.u) + int32_t(at1.u)) >> 1;
					const int32_t avg_v = (int32_t(at0.v) + int32_t(at1.v)) >> 1;
					const int32_t ph_x = (avg_u - ((dx + ax) >> 1)) & 15, ph_y = (avg_v - ((dy + ay) >> 1)) & 15;
					ta.stqf0[0] = fadd(ta.stqf0[0], fsub(0.5f, fmul(__int2float_rn(ph_x), 0.0625f)));
					ta.stqf0[1] = fadd(ta.stqf0[1], fsub(0.5f, fmul(__int2float_rn(ph_y), 0.0625f)));
				}
				else if (blur)
					tex &= ~TEX_PER_SAMPLE_BIT;
				else
					tex |= TEX_SAMPLE_MAPPING_BIT;
			}
		}
		else if (!perspective)
		{
			if (udx > ddx + 1 && udy > ddy + 1)
			{
				if (!P.force_linear_ss)
					tex &= ~TEX_PER_SAMPLE_BIT;
			}
			else if (ddx >= 2 * udx && ddy >= 2 * udy)
			{
				if (!P.force_linear_ss)
					tex |= TEX_SAMPLE_RESOLVED_BIT;
			}
		}
		if ((tex & (TEX_PER_SAMPLE_BIT | TEX_SAMPLE_MAPPING_BIT)) == TEX_PER_SAMPLE_BIT)
		{
			new_state &= ~(1u << STATE_BIT_SNAP_ATTRIBUTE);
			const float corner = fmul(8.0f, average_sampling_offset(P.setup_rate_x_log2, P.setup_rate_y_log2));
			const float di_dcorner = fmul(__int2float_rn(pb0 + pb1), corner);
			const float dj_dcorner = fmul(__int2float_rn(pc0 + pc1), corner);
			out.error_i = fsub(out.error_i, fmul(di_dcorner, inv_area_scaled));
			out.error_j = fsub(out.error_j, fmul(dj_dcorner, inv_area_scaled));
		}
	}

	if (sry != 0 && !sprite)
	{
		bool per_sample = multisample;
		if (!per_sample && perspective)
			per_sample = di[2] != 0.0f || dj[2] != 0.0f;
		if (!per_sample)
			per_sample = za != zb || zb != zc;
		if (!per_sample)
		{
			// Flat primitive: snap attributes and register its depth bucket
			// for the single-sample heuristic (triangle_setup.comp:826-871).
			if (!line)
				new_state |= 1u << STATE_BIT_SNAP_ATTRIBUTE;
			uint32_t inst = (st >> STATE_VERTEX_RENDER_PASS_INSTANCE_OFFSET) & 7u;
			uint32_t z_shift = ((P.packed_z_shift >> (4 * inst)) & 15u) * 8u;
			uint32_t bucket = min(255u, z_shift >= 32 ? 0u : za >> z_shift);
			uint32_t old = atomicOr(&P.heuristic->active[bucket >> 5], 1u << (bucket & 31));
			if (((old >> (bucket & 31)) & 1u) == 0)
			{
				uint32_t slot = atomicAdd(&P.heuristic->bucket_count, 1u);
				P.heuristic->bucket[slot] = bucket;
			}
		}
	}

	P.setup[index] = out;
	P.tattr[index] = ta;
	pa.state = new_state;
	pa.tex = tex;
	P.prims[index] = pa;
}

// ---------------------------------------------------------------------------
// Single-sample heuristic (single_sample_heuristic.comp:148-291): for every
// depth bucket that holds a flat primitive, decide which flat primitives are
// UI elements to rasterise single-sampled (SNAP_RASTER) and which sit inside
// the 3D depth range and go back to full SSAA (SNAP_ATTRIBUTE cleared).
// One CTA per (bucket, instance); 3 x 64K-bit masks in shared memory.
// Decisions go to P.heuristic_action so that every bucket reads the states
// triangle setup wrote, whatever order the CTAs run in.

__device__ __forceinline__ uint32_t heuristic_hash_vertex(const pgs_vertex_position &v)
{
	// Three rounds of ((s >> 8) ^ s.yzx) * 1103515245 (:86-94).
	uint32_t x = uint32_t(v.x), y = uint32_t(v.y), z = v.z;
	#pragma unroll
	for (int r = 0; r < 3; r++)
	{
		uint32_t nx = ((x >> 8) ^ y) * 1103515245u;
		uint32_t ny = ((y >> 8) ^ z) * 1103515245u;
		uint32_t nz = ((z >> 8) ^ x) * 1103515245u;
		x = nx; y = ny; z = nz;
	}
	return x >> 16;
}

constexpr uint32_t HEURISTIC_MASK_WORDS = 65536 / 32;

__global__ void __launch_bounds__(1024) single_sample_heuristic_kernel(PassParams P, HeuristicParams H)
{
	const uint32_t inst = blockIdx.y;
	if (((H.instance_mask >> inst) & 1u) == 0)
		return;
	if (blockIdx.x >= P.heuristic->bucket_count)
		return;

	__shared__ uint32_t full3d[HEURISTIC_MASK_WORDS];
	__shared__ uint32_t candidate[HEURISTIC_MASK_WORDS];
	__shared__ uint32_t shared_vertex[HEURISTIC_MASK_WORDS];
	__shared__ uint32_t any_full3d, min_z, max_z;

	const uint32_t tid = threadIdx.x, nthreads = blockDim.x;
	for (uint32_t i = tid; i < HEURISTIC_MASK_WORDS; i += nthreads)
	{
		full3d[i] = 0;
		candidate[i] = 0;
		shared_vertex[i] = 0;
	}
	if (tid == 0)
	{
		any_full3d = 0;
		min_z = ~0u;
		max_z = 0;
	}
	__syncthreads();

	const uint32_t z_shift = H.z_shift[inst], z_max = H.z_max[inst];
	uint32_t zlo = P.heuristic->bucket[blockIdx.x];
	uint32_t zhi = ((zlo + 1) << H.z_shift_bucket[inst]) - 1;
	zlo <<= H.z_shift_bucket[inst];

	const uint32_t SA = 1u << STATE_BIT_SNAP_ATTRIBUTE, SR = 1u << STATE_BIT_SNAP_RASTER;
	const uint32_t LINE = 1u << STATE_BIT_LINE;
	const uint32_t NO_FULL_3D = (1u << STATE_BIT_SPRITE) | LINE | SA;
	const uint32_t n = P.num_prims;
	auto inst_of = [](uint32_t st) { return (st >> STATE_VERTEX_RENDER_PASS_INSTANCE_OFFSET) & 7u; };
	auto snap = [&](uint32_t z) { return min(z_max, z) >> z_shift; };

	// Pass 1: depth values used by 3D primitives, and flat candidates.
	uint32_t lmin = ~0u, lmax = 0, lany = 0;
	for (uint32_t i = tid; i < n; i += nthreads)
	{
		uint32_t st = P.prims[i].state;
		if (inst_of(st) != inst)
			continue;
		if ((st & NO_FULL_3D) == 0)
		{
			#pragma unroll
			for (int k = 0; k < 3; k++)
			{
				uint32_t z = P.pos[3 * i + k].z;
				lmin = min(lmin, z);
				lmax = max(lmax, z);
				uint32_t s = snap(z);
				if (s >= zlo && s <= zhi)
					atomicOr(&full3d[(s - zlo) >> 5], 1u << ((s - zlo) & 31));
			}
			lany = 1;
		}
		else if ((st & (SA | SR)) == SA || (st & LINE) != 0)
		{
			uint32_t s = snap(P.pos[3 * i].z);
			if (s >= zlo && s <= zhi)
				atomicOr(&candidate[(s - zlo) >> 5], 1u << ((s - zlo) & 31));
		}
	}
	lmin = __reduce_min_sync(0xffffffffu, lmin);
	lmax = __reduce_max_sync(0xffffffffu, lmax);
	lany = __reduce_or_sync(0xffffffffu, lany);
	if ((tid & 31) == 0)
	{
		atomicMin(&min_z, lmin);
		atomicMax(&max_z, lmax);
		if (lany)
			any_full3d = 1;
	}
	__syncthreads();

	// Pass 2: hash the vertices of 3D primitives whose depth is a candidate.
	for (uint32_t i = tid; i < n; i += nthreads)
	{
		uint32_t st = P.prims[i].state;
		if (inst_of(st) != inst || (st & NO_FULL_3D) != 0)
			continue;
		#pragma unroll
		for (int k = 0; k < 3; k++)
		{
			pgs_vertex_position v = P.pos[3 * i + k];
			uint32_t s = snap(v.z);
			if (s >= zlo && s <= zhi && ((candidate[(s - zlo) >> 5] >> ((s - zlo) & 31)) & 1u))
			{
				uint32_t h = heuristic_hash_vertex(v);
				atomicOr(&shared_vertex[h >> 5], 1u << (h & 31));
			}
		}
	}
	__syncthreads();

	// Pass 3: a flat candidate that shares a vertex with a 3D primitive at a
	// depth the 3D geometry uses keeps its depth out of demotion.
	for (uint32_t i = tid; i < n; i += nthreads)
	{
		uint32_t st = P.prims[i].state;
		if (inst_of(st) != inst || (st & (SA | SR)) != SA)
			continue;
		uint32_t s = snap(P.pos[3 * i].z);
		if (s < zlo || s > zhi)
			continue;
		uint32_t o = s - zlo;
		if (((full3d[o >> 5] >> (o & 31)) & 1u) == 0)
			continue;
		bool conflict = false;
		#pragma unroll
		for (int k = 0; k < 3; k++)
		{
			uint32_t h = heuristic_hash_vertex(P.pos[3 * i + k]);
			conflict |= ((shared_vertex[h >> 5] >> (h & 31)) & 1u) != 0;
		}
		if (conflict)
			atomicAnd(&candidate[o >> 5], ~(1u << (o & 31)));
	}
	__syncthreads();

	// Pass 4: decisions.
	const bool force_single_sample = any_full3d == 0;
	const uint32_t zmin3d = min_z, zmax3d = max_z;
	for (uint32_t i = tid; i < n; i += nthreads)
	{
		uint32_t z = P.pos[3 * i].z;
		uint32_t s = snap(z);
		if (s < zlo || s > zhi)
			continue;
		uint32_t st = P.prims[i].state;
		if (inst_of(st) != inst)
			continue;
		bool tri_candidate = (st & (SA | SR)) == SA;
		bool line_candidate = force_single_sample && (st & LINE) != 0;
		if (!tri_candidate && !line_candidate)
			continue;
		uint32_t o = s - zlo;
		if ((candidate[o >> 5] >> (o & 31)) & 1u)
			P.heuristic_action[i] = HEURISTIC_SET_SNAP_RASTER;
		else if ((st & ((1u << STATE_BIT_Z_TEST) | (1u << STATE_BIT_Z_WRITE))) != 0 && z > zmin3d && z < zmax3d)
			P.heuristic_action[i] = HEURISTIC_CLEAR_SNAP_ATTRIBUTE;
	}
}

// Applies and clears the heuristic's decisions.
__global__ void __launch_bounds__(256) heuristic_apply_kernel(PassParams P)
{
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= P.num_prims)
		return;
	uint8_t a = P.heuristic_action[i];
	if (a == 0)
		return;
	uint32_t st = P.prims[i].state;
	if (a == HEURISTIC_SET_SNAP_RASTER)
		st |= 1u << STATE_BIT_SNAP_RASTER;
	else
		st &= ~(1u << STATE_BIT_SNAP_ATTRIBUTE);
	P.prims[i].state = st;
	P.heuristic_action[i] = 0;
}

// ---------------------------------------------------------------------------
// Conservative tile test (intersect.h:24-81).
__device__ __forceinline__ bool intersects_tile(const PrimSetup &s, int32_t lo0, int32_t lo1, int32_t hi0, int32_t hi1,
                                                bool ms_tri)
{
	int32_t l0 = max(s.bb[0], lo0), l1 = max(s.bb[1], lo1);
	int32_t h0 = min(s.bb[2], hi0), h1 = min(s.bb[3], hi1);
	if (h0 < l0 || h1 < l1)
		return false;
	int32_t axw = s.a[0];
	bool par = (axw & 1) != 0;
	int32_t off_b = int32_t((uint32_t(axw) >> 2) & 3u) - 1;
	int32_t off_c = int32_t((uint32_t(axw) >> 4) & 3u) - 1;
	int32_t A[3] = { axw >> 6, s.a[1], s.a[2] };
	l0 <<= 3; l1 <<= 3;
	h0 = (h0 << 3) | 7; h1 = (h1 << 3) | 7;
	int32_t da = idot3(A, A[0] >= 0 ? h0 : l0, A[1] >= 0 ? h1 : l1);
	int32_t db = idot3(s.b, s.b[0] >= 0 ? h0 : l0, s.b[1] >= 0 ? h1 : l1);
	int32_t dc = idot3(s.c, s.c[0] >= 0 ? h0 : l0, s.c[1] >= 0 ? h1 : l1);
	if (ms_tri && !par)
	{
		da += 8 * max(abs(A[0]), abs(A[1]));
		db += 8 * max(abs(s.b[0]), abs(s.b[1]));
		dc += 8 * max(abs(s.c[0]), abs(s.c[1]));
	}
	bool ok = da >= 0 && db >= 0 && dc >= 0;
	if (par && !ok)
	{
		da = idot3(A, A[0] >= 0 ? h0 : l0, A[1] >= 0 ? h1 : l1);
		db = idot3(s.b, -s.c[0] >= 0 ? h0 : l0, -s.c[1] >= 0 ? h1 : l1);
		dc = idot3(s.c, -s.b[0] >= 0 ? h0 : l0, -s.b[1] >= 0 ? h1 : l1);
		db += da + off_b;
		dc += da + off_c;
		da = idot3(A, A[0] >= 0 ? l0 : h0, A[1] >= 0 ? l1 : h1);
		ok = (-1 >= da) && db >= 0 && dc >= 0;
	}
	return ok;
}

// ---------------------------------------------------------------------------
// K2: binning.  Coarse tiles (2^tile_size_log2 pixels) carry the reference's
// membership test and super-sampling flags (binning.comp:74-125); shading
// lists are kept per 8x8 sub-tile as bitmasks over the pass's primitive range
// so that ascending primitive order needs no sort.  The primitives of one mask
// word (32) are a group; its (primitive, tile) candidates, those of the coarse grid and then those of the
// sub-tile grid, are dealt out 32 at a time to the warps of gridDim.y CTAs, so
// that neither a primitive over the whole frame nor one over hundreds of coarse
// tiles holds a lane.
// Bound: latency (dependent loads, shuffles and reductions at under 20 % of the
// issue slots), hence many short chains: with one lane walking all coarse tiles
// of its primitive and one CTA per group, a 61-primitive frame with a clear of
// the whole frame took 47 us here and takes 4; a feedback frame's passes at 8x went from 15 to 4.6.
constexpr uint32_t BIN_GROUP_WARPS = 4;
// CTAs per SM that a launch aims at when its groups are fewer, up to 16 CTAs per group.
constexpr uint32_t BIN_CTAS_PER_SM = 4;

// One live primitive of a group, as the dealt-out tests read it.
struct BinItem
{
	PrimSetup s;
	uint32_t local;   // index in the dispatch's primitive range
	uint32_t ms_tri;
	uint32_t flags;   // what the primitive adds to a coarse tile's flags
	int32_t x0, y0, x1, y1; // its box inside the instance, relative to the instance's origin
};

// The items' candidate tiles of 2^shift pixels, dealt to the lanes: body(item,
// tile x, tile y) runs for every tile of every item's box.  All lanes of the
// calling warp take part.
template <typename F>
__device__ __forceinline__ void deal_tiles(const BinItem *items, uint32_t n, int shift, F &&body)
{
	const unsigned full = 0xffffffffu;
	const uint32_t lane = threadIdx.x & 31u;
	int32_t gx0 = 0, gy0 = 0, gw = 0;
	uint32_t count = 0;
	if (lane < n)
	{
		const BinItem &it = items[lane];
		gx0 = it.x0 >> shift;
		gy0 = it.y0 >> shift;
		gw = (it.x1 >> shift) - gx0 + 1;
		count = uint32_t(gw) * uint32_t((it.y1 >> shift) - gy0 + 1);
	}
	const uint32_t incl = warp_scan(count, lane), start = incl - count;
	const uint32_t total = __shfl_sync(full, incl, 31);
	const float inv = 1.0f / float(gw > 0 ? gw : 1);
	const uint32_t first = (blockIdx.y * BIN_GROUP_WARPS + (threadIdx.x >> 5)) * 32u;
	for (uint32_t base = first; base < total; base += 32u * BIN_GROUP_WARPS * gridDim.y)
	{
		// Every item has a candidate, so the starts are distinct: the owner of a
		// candidate is the last item that starts at or before it.
		const uint32_t before = __popc(__ballot_sync(full, count && start < base));
		const uint32_t here = __reduce_or_sync(full, count && start - base < 32u ? 1u << (start - base) : 0u);
		const uint32_t o = before + __popc(here & (2u << lane) - 1u) - 1u;
		const uint32_t k = base + lane - __shfl_sync(full, start, int(o & 31u));
		const int32_t o_gw = __shfl_sync(full, gw, int(o & 31u));
		const float o_inv = __shfl_sync(full, inv, int(o & 31u));
		const int32_t o_gx0 = __shfl_sync(full, gx0, int(o & 31u)), o_gy0 = __shfl_sync(full, gy0, int(o & 31u));
		if (base + lane >= total)
			continue;
		// k / gw for k below 2^17 and gw up to 512: half a unit away from the
		// next integer at k + 0.5, far more than the product's rounding.
		const int32_t row = int32_t((float(k) + 0.5f) * o_inv);
		body(items[o], o_gx0 + int32_t(k) - row * o_gw, o_gy0 + row);
	}
}

__global__ void __launch_bounds__(32 * BIN_GROUP_WARPS) bin_kernel(PassParams P, DevInstance I, uint32_t *sub_masks,
                                                                   uint32_t *tile_flags)
{
	__shared__ BinItem items[32];
	__shared__ uint32_t s_n;
	const uint32_t lane = threadIdx.x & 31u;
	const int ts = int(P.tile_size_log2);
	if (threadIdx.x < 32u)
	{
		const uint32_t local = blockIdx.x * 32u + lane, p = I.prim_lo + local;
		BinItem it;
		bool live = false;
		if (local < I.prim_count)
		{
			const pgs_primitive_attribute pa = P.prims[p];
			it.s = P.setup[p];
			it.local = local;
			it.ms_tri = ((pa.state >> STATE_BIT_MULTISAMPLE) & 1) && !((pa.state >> STATE_BIT_LINE) & 1);
			it.flags = TILE_NONEMPTY;
			if (I.rate_y_log2 != 0)
			{
				const uint32_t full_mask = (1u << STATE_BIT_SNAP_RASTER) | (1u << STATE_BIT_Z_TEST) | (1u << STATE_BIT_OPAQUE);
				const uint32_t color_mask = (1u << STATE_BIT_SNAP_RASTER) | (1u << STATE_BIT_OPAQUE);
				if ((pa.state & full_mask) != color_mask) it.flags |= TILE_REQ_SS_ZW;
				if ((pa.state & color_mask) != color_mask) it.flags |= TILE_REQ_SS;
				if (pa.state & (1u << STATE_BIT_Z_WRITE)) it.flags |= TILE_HAS_ZW;
				if (pa.tex & TEX_PER_SAMPLE_BIT) it.flags |= TILE_REQ_SS;
			}
			it.x0 = max(it.s.bb[0] - I.base_x, 0);
			it.y0 = max(it.s.bb[1] - I.base_y, 0);
			it.x1 = min(it.s.bb[2] - I.base_x, int32_t(I.tiles_w << ts) - 1);
			it.y1 = min(it.s.bb[3] - I.base_y, int32_t(I.tiles_h << ts) - 1);
			live = ((pa.state >> STATE_VERTEX_RENDER_PASS_INSTANCE_OFFSET) & 7u) == I.instance && it.s.bb[2] >= it.s.bb[0] &&
			       it.s.bb[3] >= it.s.bb[1] && it.x1 >= it.x0 && it.y1 >= it.y0;
		}
		const uint32_t alive = __ballot_sync(0xffffffffu, live);
		if (live)
			items[__popc(alive & ((1u << lane) - 1u))] = it;
		if (lane == 0)
			s_n = uint32_t(__popc(alive));
	}
	__syncthreads();
	const uint32_t n = s_n;
	if (!n)
		return;

	auto mark_tile = [&](const BinItem &it, uint32_t tile) {
		atomicOr(&tile_flags[tile], it.flags);
		// All of them counted for splitting as well take a launch of 20,000 primitives from 8.5 to 13 us.
		if (I.blend_demote)
			atomicAdd(&tile_flags[tile], 1u << TILE_COUNT_SHIFT);
		else if (I.split_count && !(it.local & 7u))
			atomicAdd(&tile_flags[tile], 8u << TILE_COUNT_SHIFT);
	};
	if (ts > 3)
		deal_tiles(items, n, ts, [&](const BinItem &it, int32_t tx, int32_t ty) {
			const int32_t lo0 = I.base_x + (tx << ts), lo1 = I.base_y + (ty << ts);
			if (intersects_tile(it.s, lo0, lo1, lo0 + (1 << ts) - 1, lo1 + (1 << ts) - 1, it.ms_tri))
				mark_tile(it, uint32_t(ty) * I.tiles_w + uint32_t(tx));
		});

	// A sub-tile that passes the test lies in a coarse tile that passes it
	// (the test is monotonic in the rectangle), so testing the sub-tiles of the
	// primitive's box inside the instance is the same as testing those of its
	// member coarse tiles.  Coarse tiles of 8x8 pixels are the sub-tiles.
	deal_tiles(items, n, 3, [&](const BinItem &it, int32_t gx, int32_t gy) {
		const int32_t sx = I.base_x + (gx << 3), sy = I.base_y + (gy << 3);
		if (!intersects_tile(it.s, sx, sy, sx + 7, sy + 7, it.ms_tri))
			return;
		// Result unused: a fire-and-forget reduction.
		const size_t sub = size_t(gy) * I.sub_w + size_t(gx);
		atomicOr(&sub_masks[sub * I.mask_words + (it.local >> 5)], 1u << (it.local & 31u));
		if (ts == 3)
			mark_tile(it, uint32_t(sub));
	});
}

// ---------------------------------------------------------------------------
// K5: texture decode.  One thread per four texels of a row of every texture of the pass.
__global__ void __launch_bounds__(256) texture_decode_kernel(PassParams P);

// ---------------------------------------------------------------------------
// K3: shading.
// A pending or candidate shade of one sample.  Only what changes per sample
// is kept; the state index, Z comparison, perspective and AA1 flags are
// read back from the primitive's state word when needed.
struct Request
{
	int coverage;
	bool z_test, z_write;
	uint32_t z;
	float i, j;
};

// unpackUnorm4x8 channel: float(c) / 255 correctly rounded.  The 256 values are
// computed on the host with IEEE division and read from a table.
__device__ __forceinline__ uint32_t pack_unorm(float r, float g, float b, float a)
{
	float v[4] = { r, g, b, a };
	uint32_t out = 0;
	#pragma unroll
	for (int k = 0; k < 4; k++)
	{
		float x = fminf(fmaxf(v[k], 0.0f), 1.0f);
		out |= uint32_t(rintf(fmul(x, 255.0f))) << (8 * k);
	}
	return out;
}

// An integral float clamped to 0..255 (the conversion to a byte saturates).
__device__ __forceinline__ uint32_t byte_clamp(float x)
{
	uint32_t r;
	asm("cvt.rni.sat.u8.f32 %0, %1;" : "=r"(r) : "f"(x));
	return r;
}

__device__ __forceinline__ uint32_t expand16(uint32_t c)
{
	uint32_t r = (c & 0x1fu) << 3, g = ((c >> 5) & 0x1fu) << 3, b = ((c >> 10) & 0x1fu) << 3;
	return r | (g << 8) | (b << 16) | ((c & 0x8000u) ? 0x80000000u : 0u);
}

struct ShadeCtx
{
	const PassParams *P;
	const DevInstance *I;
	bool ss;
	int dim;          // sampling rate y log2 when super-sampled, else 0
	int32_t snap_mask_x, snap_mask_y;
	bool zs;
	uint32_t fb_psm, zb_psm;
	uint32_t zmax;   // largest depth of the depth format
	uint32_t sample; // sample index of the thread in a super-sampled tile, else 0
};

__device__ __forceinline__ uint32_t clut_color(const PassParams &P, const pgs_texture_desc &t, uint32_t index)
{
	uint32_t bi = t.csa * 16u + index;
	bool c16 = t.cpsm == PSMCT16 || t.cpsm == PSMCT16S;
	if (t.psm == PSMT8 || t.psm == PSMT8H)
	{
		uint32_t bank = min(bi >> 4, c16 ? 31u : 15u);
		bi = bank * 16u + (bi & 15u);
	}
	bi = min(bi, c16 ? 511u : 255u);
	const uint16_t *cl = P.clut + size_t(t.clut_instance % PGS_CLUT_INSTANCES) * 512u;
	if (c16)
		return rgba16_to_rgba32(__ldg(cl + bi), t.aem, t.ta0, t.ta1);
	return uint32_t(__ldg(cl + bi)) | (uint32_t(__ldg(cl + bi + 256u)) << 16);
}

// The VRAM a texture of the pass decodes from: a snapshot taken before a
// transfer overwrote its source, or VRAM as the pass begins.
__device__ __forceinline__ const uint8_t *texture_source(const PassParams &P, uint32_t tex)
{
	for (uint32_t k = 0; k < P.num_snaps; k++)
		if (tex < P.snap_limit[k])
			return P.snap_vram[k];
	return P.vram;
}

// Address of pixel x + k of a row minus that of pixel x, x a multiple of 4: the
// four lie in one block, and their two low coordinate bits go to address bits of
// their own, clear in the first one's address.
__device__ __forceinline__ uint32_t quad_offset(uint32_t psm, uint32_t k)
{
	const uint32_t lo = k & 1u, hi = (k >> 1) & 1u;
	switch (psm)
	{
	case PSMCT16: case PSMCT16S: case PSMZ16: case PSMZ16S: return lo * 2u + hi * 8u; // halves
	case PSMT8: return lo * 4u + hi * 16u;                                              // bytes
	case PSMT4: return lo * 8u + hi * 32u;                                              // nibbles
	default: return lo + hi * 4u;                                                       // words
	}
}

// Texel at address a of the texture's format.
__device__ __forceinline__ uint32_t fetch_texel(const PassParams &P, const uint8_t *v, const pgs_texture_desc &t, uint32_t a)
{
	switch (t.psm)
	{
	case PSMCT24: case PSMZ24:
		return rgb24_to_rgba32(__ldg(reinterpret_cast<const uint32_t *>(v) + a), t.aem, t.ta0);
	case PSMCT16: case PSMCT16S: case PSMZ16: case PSMZ16S:
		return rgba16_to_rgba32(__ldg(reinterpret_cast<const uint16_t *>(v) + a), t.aem, t.ta0, t.ta1);
	case PSMT8: return clut_color(P, t, __ldg(v + a));
	case PSMT8H: return clut_color(P, t, __ldg(v + 4u * a + 3u));
	case PSMT4: return clut_color(P, t, (uint32_t(__ldg(v + (a >> 1))) >> ((a & 1u) * 4u)) & 15u);
	case PSMT4HL: return clut_color(P, t, (__ldg(reinterpret_cast<const uint32_t *>(v) + a) >> 24) & 15u);
	case PSMT4HH: return clut_color(P, t, __ldg(reinterpret_cast<const uint32_t *>(v) + a) >> 28);
	default: return __ldg(reinterpret_cast<const uint32_t *>(v) + a);
	}
}

// Texel of sample `s` of a super-sampled texture: the single-sampled texel
// unless the reference plane marks it super-sampled (upload.comp
// SUPER_SAMPLED, :131-220; 24-bit formats merge by the reference bits).
__device__ __forceinline__ uint32_t fetch_texel_sample(const PassParams &P, const uint8_t *v, const pgs_texture_desc &t,
                                                       int32_t x, int32_t y, uint32_t s)
{
	const uint32_t a = swizzle_address(uint32_t(x), uint32_t(y), t.tbp0, t.tbw, t.psm);
	const uint32_t *v32 = reinterpret_cast<const uint32_t *>(v);
	const uint16_t *v16 = reinterpret_cast<const uint16_t *>(v);
	const uint32_t V32 = VRAM_SIZE / 4, V16 = VRAM_SIZE / 2, V8 = VRAM_SIZE;
	switch (t.psm)
	{
	case PSMCT24: case PSMZ24:
	{
		uint32_t col = __ldg(v32 + a), ref = __ldg(v32 + a + V32);
		if (ref != 0u)
			col = (__ldg(v32 + a + (2u + s) * V32) & ref) | (col & ~ref);
		return rgb24_to_rgba32(col, t.aem, t.ta0);
	}
	case PSMCT16: case PSMCT16S: case PSMZ16: case PSMZ16S:
	{
		uint32_t col = __ldg(v16 + a);
		if (__ldg(v16 + a + V16) == 0xffffu)
			col = __ldg(v16 + a + (2u + s) * V16);
		return rgba16_to_rgba32(col, t.aem, t.ta0, t.ta1);
	}
	case PSMT8:
	{
		uint32_t idx = __ldg(v + a);
		if (__ldg(v + a + V8) == 0xffu)
			idx = __ldg(v + a + (2u + s) * V8);
		return clut_color(P, t, idx);
	}
	case PSMT8H:
	{
		const uint32_t a8 = 4u * a + 3u;
		uint32_t idx = __ldg(v + a8);
		if (__ldg(v + a8 + V8) == 0xffu)
			idx = __ldg(v + a8 + (2u + s) * V8);
		return clut_color(P, t, idx);
	}
	default:
	{
		uint32_t col = __ldg(v32 + a);
		if (__ldg(v32 + a + V32) == 0xffffffffu)
			col = __ldg(v32 + a + (2u + s) * V32);
		return col;
	}
	}
}

__device__ __forceinline__ void effective_wrap(pgs_texture_desc &t, uint32_t tex_word)
{
	if (t.wms < WRAP_REGION_CLAMP)
		t.wms = (tex_word & TEX_SAMPLER_CLAMP_S_BIT) ? WRAP_CLAMP : WRAP_REPEAT;
	if (t.wmt < WRAP_REGION_CLAMP)
		t.wmt = (tex_word & TEX_SAMPLER_CLAMP_T_BIT) ? WRAP_CLAMP : WRAP_REPEAT;
}

// A wrap mode as (v & and_mask | or_mask) clamped to [lo, hi]: REPEAT masks,
// CLAMP and REGION_CLAMP clamp, REGION_REPEAT masks with MINU and ors MAXU.
struct WrapAxis
{
	int32_t and_mask, or_mask, lo, hi;
};

__host__ __device__ __forceinline__ WrapAxis wrap_axis(uint32_t mode, uint32_t size_log2, uint32_t lo, uint32_t hi)
{
	const int32_t m = (1 << size_log2) - 1;
	switch (mode)
	{
	case WRAP_REPEAT: return { m, 0, INT32_MIN, INT32_MAX };
	case WRAP_CLAMP: return { -1, 0, 0, m };
	case WRAP_REGION_CLAMP: return { -1, 0, int32_t(lo), int32_t(hi) };
	default: return { m & int32_t(lo), int32_t(hi), INT32_MIN, INT32_MAX };
	}
}

__device__ __forceinline__ int32_t wrap_apply(int32_t v, const WrapAxis &w)
{
	return min(max((v & w.and_mask) | w.or_mask, w.lo), w.hi);
}

__device__ __forceinline__ int32_t wrap_coord(int32_t v, uint32_t mode, uint32_t size_log2, uint32_t lo, uint32_t hi)
{
	int32_t size = 1 << size_log2;
	switch (mode)
	{
	case WRAP_REPEAT: return v & (size - 1);
	case WRAP_CLAMP: return min(max(v, 0), size - 1);
	case WRAP_REGION_CLAMP: return min(max(v, int32_t(lo)), int32_t(hi));
	default: return int32_t(((uint32_t(v) & uint32_t(size - 1)) & lo) | hi);
	}
}

// Grid y = texture, z = slot (mip level, or sample layer of a super-sampled
// texture); level l reads from MIPTBP's base and stride (upload_texture's
// per-level loop, gs/gs_renderer.cpp:3543-3590).  A thread decodes four texels of
// a row, which share one address computation.
// Bound: issue of the address and palette arithmetic, not the few bytes per texel
// (eight 256x256 PSMT8 textures: a texel per thread 3.5 M warp instructions, so 1.9;
// a light frame that decodes and uploads them 25.6 -> 22.8 us per replay).
__global__ void __launch_bounds__(256) texture_decode_kernel(PassParams P)
{
	const uint32_t tex = blockIdx.y, level = blockIdx.z;
	if (tex >= P.num_textures)
		return;
	const pgs_texture_desc &t = P.textures[tex];
	if (level >= texture_slots(t))
		return;
	const TexImage im = P.tex_images[tex * TEX_SLOTS + level];
	const uint32_t quads = (im.ext_u + 3u) / 4u;
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= quads * im.ext_v)
		return;
	const uint32_t x = i % quads * 4u, y = i / quads;
	const uint8_t *src = texture_source(P, tex);
	uint32_t *dst = P.texels + im.offset + y * im.ext_u + x;
	const uint32_t n = min(im.ext_u - x, 4u);
	uint32_t c[4] = {};
	if (t.samples > 1 && level > 0)
	{
		#pragma unroll
		for (uint32_t k = 0; k < 4; k++)
			if (k < n)
				c[k] = fetch_texel_sample(P, src, t, int32_t(x + k), int32_t(y), level - 1u);
	}
	else
	{
		const uint32_t tbp = level ? t.mip[level - 1] & 0x3fffu : t.tbp0, tbw = level ? t.mip[level - 1] >> 16 : t.tbw;
		const uint32_t a = swizzle_address(x, y, tbp, tbw, t.psm);
		#pragma unroll
		for (uint32_t k = 0; k < 4; k++)
			if (k < n)
				c[k] = fetch_texel(P, src, t, a + quad_offset(t.psm, k));
	}
	if (!((im.offset | im.ext_u) & 3u))
		*reinterpret_cast<uint4 *>(dst) = make_uint4(c[0], c[1], c[2], c[3]);
	else
	{
		#pragma unroll
		for (uint32_t k = 0; k < 4; k++)
			if (k < n)
				dst[k] = c[k];
	}
}

// log2 of a positive normal float: ln m = 2 atanh(s), s = (m - 1) / (m + 1),
// by the series s + s^3/3 + ... + s^9/9 with m reduced to [sqrt(1/2), sqrt(2)]
// (|s| <= 0.172, truncation error below 2e-8).  Every operation is rounded on
// its own, so the CPU restatement computes the same bits.
__device__ __forceinline__ float lod_log2(float x)
{
	uint32_t b = f2u(x);
	int32_t e = int32_t((b >> 23) & 0xffu) - 127;
	float m = u2f((b & 0x7fffffu) | 0x3f800000u);
	if (m > 1.41421356f)
	{
		m = fmul(m, 0.5f);
		e++;
	}
	float s = __fdiv_rn(fsub(m, 1.0f), fadd(m, 1.0f));
	float s2 = fmul(s, s);
	float poly = fadd(fmul(s2, 1.0f / 9.0f), 1.0f / 7.0f);
	poly = fadd(fmul(s2, poly), 1.0f / 5.0f);
	poly = fadd(fmul(s2, poly), 1.0f / 3.0f);
	poly = fadd(fmul(s2, poly), 1.0f);
	float ln_m = fmul(fmul(2.0f, s), poly);
	return fadd(__int2float_rn(e), fmul(ln_m, 1.44269504f));
}

// Bilinear filter at (ku, kv) in 1/16 texels.
__device__ __forceinline__ void bilinear_texel(const uint32_t *img, uint32_t row, int32_t ku, int32_t kv, const WrapAxis &wu,
                                               const WrapAxis &wv, uint32_t rgba[4])
{
	int32_t bu = ku - 8, bv = kv - 8;
	int32_t x0 = bu >> 4, y0 = bv >> 4;
	uint32_t fx = uint32_t(bu) & 15u, fy = uint32_t(bv) & 15u;
	int32_t xs0 = wrap_apply(x0, wu);
	int32_t xs1 = wrap_apply(x0 + 1, wu);
	int32_t ys0 = wrap_apply(y0, wv);
	int32_t ys1 = wrap_apply(y0 + 1, wv);
	uint32_t w00 = (16u - fx) * (16u - fy), w10 = fx * (16u - fy), w01 = (16u - fx) * fy, w11 = fx * fy;
	const uint32_t *row0 = img + uint32_t(ys0) * row, *row1 = img + uint32_t(ys1) * row;
	uint32_t c00 = __ldg(row0 + xs0);
	uint32_t c10 = __ldg(row0 + xs1);
	uint32_t c01 = __ldg(row1 + xs0);
	uint32_t c11 = __ldg(row1 + xs1);
	// Two channels per 32-bit word (R and B, then G and A), 16 bits each:
	// the weights sum to 256, so a channel's sum stays below 2^16.
	const uint32_t m = 0x00ff00ffu;
	const uint32_t rb = w00 * (c00 & m) + w10 * (c10 & m) + w01 * (c01 & m) + w11 * (c11 & m);
	const uint32_t ga = w00 * ((c00 >> 8) & m) + w10 * ((c10 >> 8) & m) + w01 * ((c01 >> 8) & m) + w11 * ((c11 >> 8) & m);
	// acc / 256 rounded half to even, both halves of a word at once: an acc is
	// at most 255 * 256, so the rounding term stays in its half.
	auto round256 = [](uint32_t acc) { return ((acc + 0x007f007fu + ((acc >> 8) & 0x00010001u)) >> 8) & 0x00ff00ffu; };
	const uint32_t rb8 = round256(rb), ga8 = round256(ga);
	rgba[0] = rb8 & 0xffu;
	rgba[1] = ga8 & 0xffu;
	rgba[2] = rb8 >> 16;
	rgba[3] = ga8 >> 16;
}

// One filtered sample of mip level `level` (exact integer filtering; the
// level's coordinates follow sample_texture, ubershader.comp:1133-1151,
// 1214-1227, with region bounds and masks shifted down by the level as in
// texture_clamp, :947-953, and upload_texture, gs/gs_renderer.cpp:3578-3590).
__device__ void sample_level(const PassParams &P, uint32_t tex_index, const pgs_texture_desc &t, uint32_t level,
                             uint32_t slot, bool clamp_s, bool clamp_t, bool linear, float u, float v, bool perspective,
                             uint32_t rgba[4])
{
	const uint32_t twl = t.tw_log2 - level, thl = t.th_log2 - level;
	float uu, vv;
	if (perspective)
	{
		uu = fmul(u, float(1u << twl));
		vv = fmul(v, float(1u << thl));
	}
	else
	{
		float inv = u2f((127u - level) << 23);
		uu = fmul(u, inv);
		vv = fmul(v, inv);
	}
	const uint32_t minu = t.minu >> level, maxu = t.maxu >> level, minv = t.minv >> level, maxv = t.maxv >> level;
	if (clamp_s)
	{
		uint32_t lo = t.wms == WRAP_REGION_CLAMP ? minu : 0u;
		uint32_t hi = t.wms == WRAP_REGION_CLAMP ? maxu : (1u << twl) - 1u;
		uu = fminf(fmaxf(uu, fadd(float(lo), 0.5f)), fadd(float(hi), 0.5f));
	}
	if (clamp_t)
	{
		uint32_t lo = t.wmt == WRAP_REGION_CLAMP ? minv : 0u;
		uint32_t hi = t.wmt == WRAP_REGION_CLAMP ? maxv : (1u << thl) - 1u;
		vv = fminf(fmaxf(vv, fadd(float(lo), 0.5f)), fadd(float(hi), 0.5f));
	}
	int32_t ku = int32_t(floorf(fadd(fmul(uu, 16.0f), 1.0f / 64.0f)));
	int32_t kv = int32_t(floorf(fadd(fmul(vv, 16.0f), 1.0f / 64.0f)));
	const TexImage im = P.tex_images[tex_index * TEX_SLOTS + slot];
	const uint32_t *img = P.texels + im.offset;
	const WrapAxis wu = wrap_axis(t.wms, twl, minu, maxu), wv = wrap_axis(t.wmt, thl, minv, maxv);
	if (!linear)
	{
		int32_t x = wrap_apply(ku >> 4, wu);
		int32_t y = wrap_apply(kv >> 4, wv);
		uint32_t c = __ldg(img + uint32_t(y) * im.ext_u + uint32_t(x));
		#pragma unroll
		for (int k = 0; k < 4; k++)
			rgba[k] = (c >> (8 * k)) & 0xffu;
		return;
	}
	bilinear_texel(img, im.ext_u, ku, kv, wu, wv, rgba);
}

// Level 0 of a texture, from the constants of its sampler record: the same
// texels as sample_level with level 0 and coordinates clamped to +-2047 before
// (scaling by a power of two is exact, so the clamps commute with it).
__device__ __forceinline__ void sample_base(const PassParams &P, uint32_t tex_index, uint32_t tex_word, float u, float v,
                                            bool perspective, uint32_t rgba[4])
{
	const TexSampler &T = P.samplers[tex_index];
	const uint32_t way = perspective ? 2u : 0u;
	const TexAxis au = T.u[way + ((tex_word & TEX_SAMPLER_CLAMP_S_BIT) ? 1u : 0u)];
	const TexAxis av = T.v[way + ((tex_word & TEX_SAMPLER_CLAMP_T_BIT) ? 1u : 0u)];
	const float u16 = fminf(fmaxf(fmul(u, au.scale), au.clamp_lo), au.clamp_hi);
	const float v16 = fminf(fmaxf(fmul(v, av.scale), av.clamp_lo), av.clamp_hi);
	const int32_t ku = __float2int_rd(fadd(u16, 1.0f / 64.0f)), kv = __float2int_rd(fadd(v16, 1.0f / 64.0f));
	const uint32_t *img = P.texels + au.place;
	const WrapAxis wu = { au.and_mask, au.or_mask, au.lo, au.hi }, wv = { av.and_mask, av.or_mask, av.lo, av.hi };
	if (!(tex_word & TEX_SAMPLER_MAG_LINEAR_BIT))
	{
		const uint32_t c = __ldg(img + uint32_t(wrap_apply(kv >> 4, wv)) * av.place + uint32_t(wrap_apply(ku >> 4, wu)));
		#pragma unroll
		for (int k = 0; k < 4; k++)
			rgba[k] = (c >> (8 * k)) & 0xffu;
		return;
	}
	bilinear_texel(img, av.place, ku, kv, wu, wv, rgba);
}

// Level of detail and filter choice (sample_texture, ubershader.comp:1064-1131):
// LOD = ceil(-log2|Q| * 2^(L+4) + K) / 16 or the fixed K >> 4, clamped to
// [0, MXL]; MMIN applies when the LOD is positive; trilinear blends the next
// level by floor(fract * 16) / 16.  Levels beyond the texture's chain read its
// last level.  Returns level | next level << 4 | weight of the next level << 8
// | linear << 16.
__device__ __forceinline__ uint32_t select_lod(uint32_t levels, uint32_t tex_word, uint32_t tex2, float q)
{
	const bool mag_linear = (tex_word & TEX_SAMPLER_MAG_LINEAR_BIT) != 0;
	const bool min_linear = (tex_word & TEX_SAMPLER_MIN_LINEAR_BIT) != 0;
	const uint32_t max_mip = (tex_word >> TEX_MAX_MIP_LEVEL_OFFSET) & 7u;
	const int32_t K = int32_t(tex2 << 17) >> 20; // signed 12-bit field at bit 3
	float lod;
	bool linear;
	if ((tex2 & TEX2_FIXED_LOD_BIT) == 0)
	{
		const uint32_t L = (tex2 >> 1) & 3u;
		float aq = fabsf(q), formula = 0.0f;
		if (aq >= 1.17549435e-38f && aq <= 3.40282347e38f)
			formula = fadd(fmul(-lod_log2(aq), float(1u << (L + 4))), __int2float_rn(K));
		lod = fmul(ceilf(formula), 0.0625f);
		linear = formula > 0.0f ? min_linear : mag_linear;
	}
	else
	{
		lod = __int2float_rn(K >> 4);
		linear = lod > 0.0f ? min_linear : mag_linear;
	}
	lod = fminf(fmaxf(lod, 0.0f), float(max_mip));
	float l1 = floorf(lod), l2 = ceilf(lod);
	uint32_t weight = uint32_t(fmul(fsub(lod, l1), 16.0f));
	if ((tex_word & TEX_SAMPLER_MIPMAP_LINEAR_BIT) == 0)
	{
		weight = 0;
		l1 = float(int32_t(fadd(lod, 0.5f)));
	}
	const uint32_t last = max(levels, 1u) - 1u;
	return min(uint32_t(l1), last) | (min(uint32_t(l2), last) << 4) | (weight << 8) | (uint32_t(linear) << 16);
}

// MIP: the pass samples mip levels (some primitive has TEX1.MXL > 0 with a
// mipmapping MMIN) or super-sampled textures; without it every sample reads
// level 0 of a plain texture through MMAG.
// Super-sampled texture (ubershader.comp:1155-1212).  Sample mapping reads the
// layer of the shading sample, the resolved bit layer 0; otherwise the phase
// LUT picks up to four (layer, texel) taps around the texel below the
// sampling position, weighted in unorm8 (one tap when filtering is nearest or
// the texel is on a clamped region edge).  Taps wrap like the texture.
__device__ void sample_layered(const PassParams &P, uint32_t tex_index, const pgs_texture_desc &t, uint32_t tex_word,
                               float u, float v, bool perspective, uint32_t sample, uint32_t rx, uint32_t ry,
                               uint32_t rgba[4])
{
	const bool clamp_s = (tex_word & TEX_SAMPLER_CLAMP_S_BIT) != 0;
	const bool clamp_t = (tex_word & TEX_SAMPLER_CLAMP_T_BIT) != 0;
	const bool mag_linear = (tex_word & TEX_SAMPLER_MAG_LINEAR_BIT) != 0;
	if (tex_word & (TEX_SAMPLE_MAPPING_BIT | TEX_SAMPLE_RESOLVED_BIT))
	{
		const uint32_t layer = (tex_word & TEX_SAMPLE_MAPPING_BIT) ? min(sample + 1u, t.samples) : 0u;
		sample_level(P, tex_index, t, 0, layer, clamp_s, clamp_t, mag_linear, u, v, perspective, rgba);
		return;
	}
	const float w = float(1u << t.tw_log2), h = float(1u << t.th_log2);
	float uu = perspective ? fmul(u, w) : u;
	float vv = perspective ? fmul(v, h) : v;
	// Region of the reference's TexInfo (CLAMP: the image, REGION_CLAMP: MIN/MAX, else 0).
	const int32_t rx0 = t.wms == WRAP_REGION_CLAMP ? int32_t(t.minu) : 0;
	const int32_t rx1 = t.wms == WRAP_REGION_CLAMP ? int32_t(t.maxu) : (t.wms == WRAP_CLAMP ? int32_t(w) - 1 : 0);
	const int32_t ry0 = t.wmt == WRAP_REGION_CLAMP ? int32_t(t.minv) : 0;
	const int32_t ry1 = t.wmt == WRAP_REGION_CLAMP ? int32_t(t.maxv) : (t.wmt == WRAP_CLAMP ? int32_t(h) - 1 : 0);
	if (clamp_s)
		uu = fminf(fmaxf(uu, fadd(float(rx0), 0.5f)), fadd(float(rx1), 0.5f));
	if (clamp_t)
		vv = fminf(fmaxf(vv, fadd(float(ry0), 0.5f)), fadd(float(ry1), 0.5f));
	const float shift = fsub(0.5f, average_sampling_offset(rx, ry));
	const float su = fsub(fadd(uu, 1.0f / 1024.0f), shift), sv = fsub(fadd(vv, 1.0f / 1024.0f), shift);
	const float fu = floorf(su), fv = floorf(sv);
	const int32_t ix = int32_t(fu), iy = int32_t(fv);
	const float pu = fsub(su, fu), pv = fsub(sv, fv);
	uint32_t entry, weights = 0;
	if (mag_linear)
	{
		const uint32_t lx = min(uint32_t(fmul(pu, 64.0f)), 63u), ly = min(uint32_t(fmul(pv, 64.0f)), 63u);
		entry = __ldg(P.phase_lut + (ly * 64u + lx) * 2u);
		weights = __ldg(P.phase_lut + (ly * 64u + lx) * 2u + 1u);
	}
	else
	{
		const uint32_t lx = min(uint32_t(fmul(pu, 32.0f)), 31u), ly = min(uint32_t(fmul(pv, 32.0f)), 31u);
		entry = __ldg(P.phase_lut + 64u * 64u * 2u + ly * 32u + lx);
	}
	const bool force_nearest =
	    !mag_linear || ((clamp_s || clamp_t) && (ix == rx0 || iy == ry0 || ix == rx1 || iy == ry1));
	auto tap = [&](uint32_t layer, int32_t x, int32_t y) {
		layer = min(layer + 1u, t.samples);
		const TexImage im = P.tex_images[tex_index * TEX_SLOTS + layer];
		const int32_t wx = wrap_coord(x, t.wms, t.tw_log2, t.minu, t.maxu);
		const int32_t wy = wrap_coord(y, t.wmt, t.th_log2, t.minv, t.maxv);
		return __ldg(P.texels + im.offset + uint32_t(wy) * im.ext_u + uint32_t(wx));
	};
	const uint32_t c0 = tap(entry & 15u, ix, iy);
	if (force_nearest)
	{
		#pragma unroll
		for (int k = 0; k < 4; k++)
			rgba[k] = (c0 >> (8 * k)) & 0xffu;
		return;
	}
	uint32_t acc[4];
	const uint32_t w0 = weights & 0xffu;
	#pragma unroll
	for (int k = 0; k < 4; k++)
		acc[k] = w0 * ((c0 >> (8 * k)) & 0xffu);
	for (uint32_t i = 1; i < 4; i++)
	{
		const uint32_t wi = (weights >> (8 * i)) & 0xffu;
		if (!wi)
			continue;
		const int32_t ox = int32_t(entry << (14 - 4 * i)) >> 30, oy = int32_t(entry << (12 - 4 * i)) >> 30;
		const uint32_t c = tap((entry >> (4 * i)) & 15u, ix + ox, iy + oy);
		#pragma unroll
		for (int k = 0; k < 4; k++)
			acc[k] += wi * ((c >> (8 * k)) & 0xffu);
	}
	// round(acc / 255); a tie would need acc = 255 (2q + 1) / 2.
	#pragma unroll
	for (int k = 0; k < 4; k++)
	{
		const uint32_t q = acc[k] / 255u, r = acc[k] % 255u;
		rgba[k] = q + (2u * r > 255u ? 1u : 0u);
	}
}

template <bool MIP>
__device__ void sample_texture(const PassParams &P, uint32_t tex_word, uint32_t tex2, float u, float v, float q,
                               bool perspective, uint32_t sample, uint32_t rx, uint32_t ry, float out[4])
{
	const uint32_t tex_index = min(tex_word & TEX_TEXTURE_INDEX_MASK, P.num_textures - 1u);
	if (!MIP)
	{
		// Level 0 through MMAG: the level blend below is the identity.
		uint32_t c[4];
		sample_base(P, tex_index, tex_word, u, v, perspective, c);
		#pragma unroll
		for (int k = 0; k < 4; k++)
			out[k] = float(c[k]);
		return;
	}
	pgs_texture_desc t = P.textures[tex_index];
	// Descriptors keep only the region modes; plain REPEAT and CLAMP come from
	// the primitive's sampler bits, as the reference's shader takes them
	// (drawing_kick_update_texture, gs/gs_interface.cpp:1514-1528).
	effective_wrap(t, tex_word);
	if ((tex_word & TEX_PER_SAMPLE_BIT) && t.samples > 1)
	{
		uint32_t rgba[4];
		sample_layered(P, tex_index, t, tex_word, u, v, perspective, sample, rx, ry, rgba);
		#pragma unroll
		for (int k = 0; k < 4; k++)
			out[k] = float(rgba[k]);
		return;
	}
	const bool clamp_s = (tex_word & TEX_SAMPLER_CLAMP_S_BIT) != 0;
	const bool clamp_t = (tex_word & TEX_SAMPLER_CLAMP_T_BIT) != 0;
	uint32_t sel = (tex_word & TEX_SAMPLER_MAG_LINEAR_BIT) ? (1u << 16) : 0u;
	if ((tex_word >> TEX_MAX_MIP_LEVEL_OFFSET) & 7u)
		sel = select_lod(t.levels, tex_word, tex2, q);
	// One pass per sampled level: weight 16 - w on the first, w on the second,
	// then roundEven(sum / 16) (exact for a single level).
	const uint32_t weight = (sel >> 8) & 0xffu;
	uint32_t acc[4] = { 0, 0, 0, 0 };
	for (uint32_t pass = 0; pass < (weight ? 2u : 1u); pass++)
	{
		uint32_t c[4];
		const uint32_t lv = pass ? ((sel >> 4) & 15u) : (sel & 15u);
		sample_level(P, tex_index, t, lv, lv, clamp_s, clamp_t, (sel >> 16) != 0, u, v, perspective, c);
		const uint32_t w = pass ? weight : 16u - weight;
		#pragma unroll
		for (int k = 0; k < 4; k++)
			acc[k] += w * c[k];
	}
	#pragma unroll
	for (int k = 0; k < 4; k++)
	{
		uint32_t r = acc[k] >> 4, f = acc[k] & 15u;
		if (f > 8u || (f == 8u && (r & 1u)))
			r++;
		out[k] = float(r);
	}
}

__device__ __forceinline__ float interp(float c0, float d1, float d2, float i, float j)
{
	// c0 + d1 * i + d2 * j, left to right, one rounding per operation.
	return fadd(fadd(c0, fmul(d1, i)), fmul(d2, j));
}

template <bool MIP>
__device__ __forceinline__ void combined_color(const ShadeCtx &C, uint32_t pi, const Request &r, bool perspective,
                                               uint32_t combiner, uint32_t tex, uint32_t tex2, uint32_t fogcol, float cc[4])
{
	const PassParams &P = *C.P;
	const TransformedAttr a = P.tattr[pi];
	float col[4];
	#pragma unroll
	for (int k = 0; k < 4; k++)
	{
		float t = interp(a.rgba0[k], a.rgba1[k], a.rgba2[k], r.i, r.j);
		col[k] = floorf(fadd(fmul(255.0f, t), 1.0f / 256.0f));
	}
	bool fog = (combiner & COMBINER_FOG_BIT) != 0, tcc = (combiner & COMBINER_TCC_BIT) != 0;
	bool tme = (combiner & COMBINER_TME_BIT) != 0;
	uint32_t mode = combiner & COMBINER_MODE_MASK;
	if (tme)
	{
		float s = interp(a.stqf0[0], a.stqf1[0], a.stqf2[0], r.i, r.j);
		float t = interp(a.stqf0[1], a.stqf1[1], a.stqf2[1], r.i, r.j);
		float q = interp(a.stqf0[2], a.stqf1[2], a.stqf2[2], r.i, r.j);
		if (perspective && q != 1.0f)
		{
			s = __fdiv_rn(s, q);
			t = __fdiv_rn(t, q);
		}
		if (MIP)
		{
			// (sample_base's bounds include these.)
			s = fminf(fmaxf(s, -2047.0f), 2047.0f);
			t = fminf(fmaxf(t, -2047.0f), 2047.0f);
		}
		float tx[4];
		sample_texture<MIP>(P, tex, tex2, s, t, q, perspective, C.sample,
		                    C.ss ? C.I->rate_x_log2 : 0u, C.ss ? C.I->rate_y_log2 : 0u, tx);
		if (mode == COMBINER_DECAL)
		{
			cc[0] = tx[0]; cc[1] = tx[1]; cc[2] = tx[2]; cc[3] = tcc ? tx[3] : col[3];
		}
		else
		{
			#pragma unroll
			for (int k = 0; k < 4; k++)
				cc[k] = fminf(fmaxf(floorf(fmul(fmul(col[k], tx[k]), 1.0f / 128.0f)), 0.0f), 255.0f);
			if (mode == COMBINER_MODULATE)
			{
				if (!tcc) cc[3] = col[3];
			}
			else
			{
				cc[0] = fadd(cc[0], col[3]); cc[1] = fadd(cc[1], col[3]); cc[2] = fadd(cc[2], col[3]);
				if (mode == COMBINER_HIGHLIGHT)
					cc[3] = tcc ? fadd(tx[3], col[3]) : col[3];
				else
					cc[3] = tcc ? tx[3] : col[3];
				#pragma unroll
				for (int k = 0; k < 4; k++)
					cc[k] = fminf(fmaxf(cc[k], 0.0f), 255.0f);
			}
		}
	}
	else
	{
		cc[0] = col[0]; cc[1] = col[1]; cc[2] = col[2]; cc[3] = col[3];
	}
	if (fog)
	{
		float f = rintf(interp(a.stqf0[3], a.stqf1[3], a.stqf2[3], r.i, r.j));
		const uint32_t fc = fogcol;
		#pragma unroll
		for (int k = 0; k < 3; k++)
		{
			float fcol = fmul(unorm8_lut(P.unorm_lut, fc, k), 255.0f);
			float d = fmul(fmul(fsub(cc[k], fcol), f), 1.0f / 256.0f);
			cc[k] = floorf(fadd(fadd(fcol, d), 0.5f));
		}
	}
}

struct SampleState
{
	uint32_t color, depth;
	bool color_dirty, depth_dirty;
	int32_t hx, hy;
	Request pending;
	uint32_t pending_prim;
};

template <bool MIP, bool AA>
__device__ __forceinline__ void shade_resolve(const ShadeCtx &C, SampleState &S, uint32_t pi, const Request &r)
{
	const PassParams &P = *C.P;
	// The primitive's words in two loads: box, state, tex | tex2, alpha, fbmsk, fogcol.
	const uint4 *words = reinterpret_cast<const uint4 *>(P.prims + pi);
	const uint4 w0 = words[0], w1 = words[1];
	const uint32_t pst = w0.z, fbmsk = w1.z, alpha_word = w1.y;
	const uint4 sv = *reinterpret_cast<const uint4 *>(P.states + min(pst & STATE_INDEX_MASK, P.num_states - 1u));
	if (C.zs && r.z_test)
	{
		bool pass = ((pst >> STATE_BIT_Z_TEST_GREATER) & 1) ? r.z > S.depth : r.z >= S.depth;
		if (!pass)
			return;
	}
	float cc[4];
	combined_color<MIP>(C, pi, r, (pst >> STATE_BIT_PERSPECTIVE) & 1, sv.x, w0.w, w1.x, w1.w, cc);

	bool write_fb = true, write_zb = true, write_alpha = !psm_is_24bit(C.fb_psm);
	const uint32_t bm = sv.y;
	bool abe = (bm & BLEND_MODE_ABE_BIT) != 0;

	if (AA && P.has_aa1)
	{
		const bool multisample = (pst >> STATE_BIT_MULTISAMPLE) & 1;
		bool use_cov = (cc[3] == 128.0f || !abe) && multisample;
		if (use_cov)
			cc[3] = float(r.coverage);
		if (multisample)
			abe = true;
	}

	if (bm & BLEND_MODE_ATE_BIT)
	{
		const float aref = float(alpha_word & 0xffu);
		// Three bits per mode: passes when less, equal, greater.
		constexpr uint32_t modes = (0u << (3 * ATST_NEVER)) | (7u << (3 * ATST_ALWAYS)) | (1u << (3 * ATST_LESS)) |
		                           (3u << (3 * ATST_LEQUAL)) | (2u << (3 * ATST_EQUAL)) | (6u << (3 * ATST_GEQUAL)) |
		                           (4u << (3 * ATST_GREATER)) | (5u << (3 * ATST_NOTEQUAL));
		const uint32_t lge = modes >> (3u * ((bm >> BLEND_MODE_ATE_MODE_OFFSET) & 7u));
		if (!((lge >> (cc[3] < aref ? 0 : (cc[3] == aref ? 1 : 2))) & 1u))
		{
			switch ((bm >> BLEND_MODE_AFAIL_MODE_OFFSET) & 3u)
			{
			case AFAIL_KEEP: return;
			case AFAIL_FB_ONLY: write_zb = false; break;
			case AFAIL_ZB_ONLY: write_fb = false; write_alpha = false; break;
			default: if (psm_is_32bit(C.fb_psm)) write_alpha = false; write_zb = false; break;
			}
		}
	}

	if (!psm_is_24bit(C.fb_psm) && (bm & BLEND_MODE_DATE_BIT))
	{
		if (((bm & BLEND_MODE_DATM_BIT) ? 1u : 0u) != S.color >> 31)
			return;
	}

	if ((bm & BLEND_MODE_PABE_BIT) && cc[3] < 128.0f)
		abe = false;

	float bl[4] = { cc[0], cc[1], cc[2], cc[3] };
	if (abe)
	{
		const uint32_t cm = (bm >> BLEND_MODE_C_MODE_OFFSET) & 3u;
		float Cf = 0.0f;
		if (cm == BLEND_ALPHA_SOURCE) Cf = cc[3];
		else if (cm == BLEND_ALPHA_DEST) Cf = psm_is_24bit(C.fb_psm) ? 128.0f : float(S.color >> 24);
		else if (cm == BLEND_ALPHA_FIX) Cf = float((alpha_word >> ALPHA_AFIX_OFFSET) & 0xffu);
		// The destination colour as round(c / 255 * 255), which is the byte.
		const float fbc[3] = { float(S.color & 0xffu), float((S.color >> 8) & 0xffu), float((S.color >> 16) & 0xffu) };
		constexpr uint32_t abd = (3u << BLEND_MODE_A_MODE_OFFSET) | (3u << BLEND_MODE_B_MODE_OFFSET) | (3u << BLEND_MODE_D_MODE_OFFSET);
		constexpr uint32_t lerp = (uint32_t(BLEND_RGB_SOURCE) << BLEND_MODE_A_MODE_OFFSET) | (uint32_t(BLEND_RGB_DEST) << BLEND_MODE_B_MODE_OFFSET) |
		                          (uint32_t(BLEND_RGB_DEST) << BLEND_MODE_D_MODE_OFFSET);
		if ((bm & abd) == lerp)
		{
			// The usual (Cs - Cd) C + Cd without the operand selections.
			#pragma unroll
			for (int k = 0; k < 3; k++)
				bl[k] = fadd(floorf(fmul(fmul(fsub(cc[k], fbc[k]), Cf), 1.0f / 128.0f)), fbc[k]);
		}
		else
		{
			const uint32_t am = (bm >> BLEND_MODE_A_MODE_OFFSET) & 3u, bmo = (bm >> BLEND_MODE_B_MODE_OFFSET) & 3u;
			const uint32_t dm = (bm >> BLEND_MODE_D_MODE_OFFSET) & 3u;
			#pragma unroll
			for (int k = 0; k < 3; k++)
			{
				float A = am == 0 ? cc[k] : (am == 1 ? fbc[k] : 0.0f);
				float B = bmo == 0 ? cc[k] : (bmo == 1 ? fbc[k] : 0.0f);
				float D = dm == 0 ? cc[k] : (dm == 1 ? fbc[k] : 0.0f);
				bl[k] = fadd(floorf(fmul(fmul(fsub(A, B), Cf), 1.0f / 128.0f)), D);
			}
		}
	}

	if (bm & BLEND_MODE_DTHE_BIT)
	{
		const int px = (S.hx >> C.dim) & 3, py = (S.hy >> C.dim) & 3;
		const int bit = ((py * 4 + px) * 4) & 31;
		const uint32_t dimx = py < 2 ? sv.z : sv.w;
		const float fdv = float(int32_t(dimx << (29 - bit & 31)) >> 29);
		bl[0] = fadd(bl[0], fdv); bl[1] = fadd(bl[1], fdv); bl[2] = fadd(bl[2], fdv);
	}

	uint32_t packed;
	if (bm & BLEND_MODE_COLCLAMP_BIT)
	{
		// Every value here is integral (or far outside the byte's range), so
		// round(clamp(x / 255, 0, 1) * 255) is x clamped to a byte.
		packed = byte_clamp(bl[0]) | (byte_clamp(bl[1]) << 8) | (byte_clamp(bl[2]) << 16) | (byte_clamp(bl[3]) << 24);
	}
	else
	{
		float o[4];
		#pragma unroll
		for (int k = 0; k < 4; k++)
		{
			float x = fmul(bl[k], 1.0f / 256.0f);
			o[k] = fmul(fsub(x, floorf(x)), 256.0f / 255.0f);
		}
		packed = pack_unorm(o[0], o[1], o[2], o[3]);
	}
	if (bm & BLEND_MODE_FB_ALPHA_BIT)
		packed |= 0x80000000u;

	if (fbmsk != 0xffffffffu && (write_fb || write_alpha))
	{
		const uint32_t keep = fbmsk | (write_fb ? 0u : 0x00ffffffu) | (write_alpha ? 0u : 0xff000000u);
		S.color = (packed & ~keep) | (S.color & keep);
		if (psm_is_16bit(C.fb_psm))
			S.color &= 0x80f8f8f8u;
		S.color_dirty = true;
	}
	if (C.zs && write_zb && r.z_write)
	{
		S.depth = r.z;
		S.depth_dirty = true;
	}
}

__device__ __forceinline__ int evaluate_coverage(const PrimSetup &s, int32_t cx, int32_t cy, float &i, float &j, bool ms,
                                                 bool line, int dim)
{
	int32_t sx = cx >> dim, sy = cy >> dim;
	if (!(sx >= s.bb[0] && sy >= s.bb[1] && s.bb[2] >= sx && s.bb[3] >= sy))
		return 0;
	int32_t axw = s.a[0];
	bool par = (axw & 1) != 0;
	int32_t off_b = int32_t((uint32_t(axw) >> 2) & 3u) - 1;
	int32_t off_c = int32_t((uint32_t(axw) >> 4) & 3u) - 1;
	int32_t A[3] = { axw >> 6, s.a[1], s.a[2] };
	int32_t px = cx << (3 - dim), py = cy << (3 - dim);
	int32_t ea = idot3(A, px, py), eb = idot3(s.b, px, py), ec = idot3(s.c, px, py);
	i = fadd(fmul(__int2float_rn(eb), s.inv_area), s.error_i);
	j = fadd(fmul(__int2float_rn(ec), s.inv_area), s.error_j);
	bool ba = ea >= 0, bb = eb >= 0, bc = ec >= 0;
	if (par && ea < 0)
	{
		eb += ea + off_b;
		ec += ea + off_c;
		ea = 0;
	}
	bool center = ea >= 0 && eb >= 0 && ec >= 0;
	if (ms && line)
		return center ? int(fmaxf(0.0f, fsub(128.0f, fmul(256.0f, fabsf(fsub(0.5f, j)))))) : 0;
	if (center)
		return 0x80;
	if (ms && !par && (int(ba) + int(bb) + int(bc) == 2))
	{
		float neg;
		int32_t md;
		if (!ba)
		{
			md = max(abs(s.b[0] + s.c[0]), abs(s.b[1] + s.c[1]));
			neg = fsub(fadd(i, j), 1.0f);
		}
		else if (!bb)
		{
			md = max(abs(s.b[0]), abs(s.b[1]));
			neg = -i;
		}
		else
		{
			md = max(abs(s.c[0]), abs(s.c[1]));
			neg = -j;
		}
		float scaled = fmul(float(md), s.inv_area);
		float fc = fsub(8.0f, __fdiv_rn(neg, scaled));
		return int(fminf(fmaxf(fmul(16.0f, fc), 0.0f), 127.0f));
	}
	return 0;
}

// Must be called by all lanes of a warp; returns with warp_any == false (and no
// further work) when no lane of the warp is covered.  The AA1 variants' path
// (ubershader variant VARIANT_FLAG_HAS_AA1_BIT); the others go by coverage masks.
template <bool TEX_ARRAY>
__device__ __forceinline__ Request shade_early(const ShadeCtx &C, const PrimSetup &s, uint32_t pi, uint32_t st,
                                               const SampleState &S, bool &opaque, bool &warp_any)
{
	const PassParams &P = *C.P;
	Request r;
	opaque = (st >> STATE_BIT_OPAQUE) & 1;
	r.z_test = C.zs && ((st >> STATE_BIT_Z_TEST) & 1);
	r.z_write = C.zs && ((st >> STATE_BIT_Z_WRITE) & 1);
	const bool multisample = (st >> STATE_BIT_MULTISAMPLE) & 1;
	int32_t rx = S.hx, ry = S.hy;
	if (C.ss && (st & (1u << STATE_BIT_SNAP_RASTER)))
	{
		// Sample-mapped textures keep the full-rate row grid when rows are
		// snapped for field rendering (ubershader.comp:816-821).
		rx &= C.snap_mask_x;
		ry &= (TEX_ARRAY && (P.prims[pi].tex & TEX_SAMPLE_MAPPING_BIT)) ? C.snap_mask_x : C.snap_mask_y;
	}
	float i = 0.0f, j = 0.0f;
	r.coverage = evaluate_coverage(s, rx, ry, i, j, multisample, (st >> STATE_BIT_LINE) & 1, C.dim);
	if (P.has_scanmsk)
	{
		int32_t sy = S.hy;
		if (st & (1u << STATE_BIT_SPRITE))
			sy >>= C.dim;
		if ((sy & 1) == 0) { if ((st >> STATE_BIT_SCANMSK_EVEN) & 1) r.coverage = 0; }
		else if ((st >> STATE_BIT_SCANMSK_ODD) & 1) r.coverage = 0;
	}
	warp_any = __any_sync(0xffffffffu, r.coverage > 0);
	if (!warp_any)
		return r;
	if (C.zs && multisample && r.coverage < 0x80)
		r.z_write = false;
	uint32_t z = s.z[0];
	float zf = rintf(fadd(fmul(u2f(s.z[1]), i), fmul(u2f(s.z[2]), j)));
	zf = fminf(fmaxf(zf, 0.0f), 4294967040.0f);
	uint32_t dz = __float2uint_rz(zf);
	dz = min(dz, 0xffffffffu - z);
	z += dz;
	if (C.zs && psm_is_16bit(C.zb_psm)) z = min(z, 0xffffu);
	else if (C.zs && psm_is_24bit(C.zb_psm)) z = min(z, 0xffffffu);
	if (C.ss && r.coverage != 0)
	{
		uint32_t snap = st & ((1u << STATE_BIT_SNAP_RASTER) | (1u << STATE_BIT_SNAP_ATTRIBUTE));
		if (snap == (1u << STATE_BIT_SNAP_ATTRIBUTE))
		{
			int32_t qx = (S.hx & C.snap_mask_x) << (3 - C.dim), qy = (S.hy & C.snap_mask_y) << (3 - C.dim);
			i = fadd(fmul(__int2float_rn(idot3(s.b, qx, qy)), s.inv_area), s.error_i);
			j = fadd(fmul(__int2float_rn(idot3(s.c, qx, qy)), s.inv_area), s.error_j);
		}
		else if (TEX_ARRAY && snap == (1u << STATE_BIT_SNAP_RASTER))
		{
			// Per-sample textured sprite: coverage snapped, attributes
			// interpolated per sample (ubershader.comp:888-895).
			int32_t qx = S.hx << (3 - C.dim), qy = S.hy << (3 - C.dim);
			i = fadd(fmul(__int2float_rn(idot3(s.b, qx, qy)), s.inv_area), s.error_i);
			j = fadd(fmul(__int2float_rn(idot3(s.c, qx, qy)), s.inv_area), s.error_j);
		}
	}
	r.z = z;
	r.i = i;
	r.j = j;
	return r;
}

// Sample position within its pixel for sample s (32-wide subgroup layout of
// ubershader.comp get_tile_info, :253-340).  Ordered grids interleave x/y
// lane bits; a 2:1 grid is a checkerboard; a 4:1 grid puts one sample per
// high-res row at x offsets 0, 2, 3, 1 (the 0x78 pattern, :333-338).
__device__ __forceinline__ void sample_offset(uint32_t s, uint32_t xl, uint32_t yl, int32_t &ox, int32_t &oy)
{
	uint32_t b0 = s & 1u, b1 = (s >> 1) & 1u, b2 = (s >> 2) & 1u, b3 = (s >> 3) & 1u;
	if (xl == yl)
	{
		ox = int32_t(b1 | (b3 << 1));
		oy = int32_t(b0 | (b2 << 1));
	}
	else if (yl == xl + 2)
	{
		oy = int32_t(s & ((1u << yl) - 1u));
		ox = int32_t(((s >> yl) << 2) + ((0x78u >> ((oy & 3) * 2)) & 3u));
	}
	else
	{
		int32_t ly = int32_t(b0 | (xl >= 1 ? (b2 << 1) : 0u));
		int32_t lx = int32_t(xl >= 1 ? b1 : 0u);
		ox = (lx << 1) + (ly & 1);
		oy = ly;
	}
}

// Processes one primitive for the calling warp: coverage, early depth,
// deferred-shading bookkeeping (ubershader.comp:1694-1812).  Warp-uniform.
// A primitive that is not opaque (warp-uniform: a state bit) is shaded right
// away rather than left pending.  The result is the same as shading it at the
// next flush: leaving it pending only saves work when a later opaque primitive
// covers the sample, which blended primitives seldom meet, and shading now keeps
// every lane of the call on the same primitive.  What was pending is shaded first
// wherever this primitive covers a sample that has a pending one.  An opaque one
// replaces what was pending and writes its depth, so a pending primitive never
// has a depth test or write left to do.  With `flush` there is no primitive and
// all that is pending is shaded.
// With mip levels or layered textures the shading code is long: a copy of it for
// each call (five) had the warps wait 15 cycles per issue for instructions, so one
// call in a rolled loop serves both shadings and the flush (25,000 small mip-mapped
// triangles at 8x 652 -> 341 us, at 16x 1126 -> 572).  Without, two copies here and
// one behind the walk are faster: 10,000 mixed AA1 primitives at 4x 291 us, rolled 312.
template <bool MIP>
__device__ __forceinline__ void process_primitive(const ShadeCtx &C, uint32_t pi, bool flush, SampleState &S, uint32_t &covered)
{
	const PassParams &P = *C.P;
	const unsigned full = 0xffffffffu;
	Request q;
	q.coverage = 0;
	bool before = S.pending.coverage > 0;
	if (!flush)
	{
		const PrimSetup s = P.setup[pi];
		const uint32_t st = P.prims[pi].state;
		bool opaque, any_cov;
		q = shade_early<MIP>(C, s, pi, st, S, opaque, any_cov);
		if (!any_cov)
			return;
		covered += q.coverage > 0 ? 1u : 0u;
		if (q.z_test)
		{
			if (!(((st >> STATE_BIT_Z_TEST_GREATER) & 1) ? q.z > S.depth : q.z >= S.depth))
				q.coverage = 0;
			q.z_test = false;
		}
		if (opaque)
		{
			if (q.coverage > 0)
			{
				if (q.z_write)
				{
					S.depth = q.z;
					S.depth_dirty = true;
				}
				S.pending.coverage = q.coverage;
				S.pending.i = q.i;
				S.pending.j = q.j;
				S.pending_prim = pi;
			}
			return;
		}
		if (!__any_sync(full, q.coverage > 0))
			return;
		if (!__any_sync(full, q.coverage > 0 && before))
			before = false;
	}
	#pragma unroll (MIP ? 1 : 2)
	for (uint32_t step = __any_sync(full, before) ? 0u : 1u; step < (flush ? 1u : 2u); step++)
	{
		Request r = q;
		uint32_t rp = pi;
		if (!step)
		{
			r.coverage = before ? S.pending.coverage : 0;
			r.i = S.pending.i;
			r.j = S.pending.j;
			r.z_write = false;
			rp = S.pending_prim;
			S.pending.coverage = 0;
		}
		r.z_test = false;
		if (r.coverage > 0)
			shade_resolve<MIP, true>(C, S, rp, r);
	}
}

// ---------------------------------------------------------------------------
// Primitive culling per warp.  A warp's samples have raster positions (after
// any snapping of coverage) inside a rectangle; a primitive whose box misses
// it, or one of whose edges is negative at every point of it, covers none of
// the warp's samples and would be a no-op for that warp.  The edge test
// follows the coverage test's 32-bit wrapping arithmetic: the value at the
// rectangle's best corner is exact modulo 2^32, every other sample's value
// is that minus at most d, and a primitive is only dropped when no sample's
// value can wrap back to non-negative.

// Whether edge e can be non-negative somewhere in r (raster units, shift sh
// to the coverage test's sub-pixel units).
__device__ __forceinline__ bool edge_may_pass(const int32_t e[3], int4 r, int sh)
{
	const int32_t x = e[0] >= 0 ? r.z : r.x, y = e[1] >= 0 ? r.w : r.y;
	const int32_t v = idot3(e, x << sh, y << sh);
	if (v >= 0)
		return true;
	const int64_t d = llabs(int64_t(e[0])) * (int64_t(r.z - r.x) << sh) + llabs(int64_t(e[1])) * (int64_t(r.w - r.y) << sh);
	return int64_t(v) - d < -2147483648LL;
}

// Conservative: false only when the primitive covers no sample whose raster
// position lies in r = (x0, y0, x1, y1).  Parallelograms (sprites, lines,
// fused rectangles) shift edges past the diagonal and AA1 multisampled
// edges cover outside the triangle, so those keep to the box test.
__device__ __forceinline__ bool may_cover(const PrimSetup &s, uint32_t st, int4 r, int dim)
{
	if ((r.z >> dim) < s.bb[0] || (r.x >> dim) > s.bb[2] || (r.w >> dim) < s.bb[1] || (r.y >> dim) > s.bb[3])
		return false;
	if (((st >> STATE_BIT_PARALLELOGRAM) & 1u) || ((st >> STATE_BIT_MULTISAMPLE) & 1u))
		return true;
	const int sh = 3 - dim;
	const int32_t A[3] = { s.a[0] >> 6, s.a[1], s.a[2] };
	return edge_may_pass(A, r, sh) && edge_may_pass(s.b, r, sh) && edge_may_pass(s.c, r, sh);
}

// ---------------------------------------------------------------------------
// Coverage masks (variants without AA1).  A warp holds a block of PW x PH
// pixels with NS samples each; one lane takes one primitive and evaluates its
// coverage of all 32 samples by stepping the three edge values across the
// block, in the coverage test's wrapping 32-bit arithmetic, so a bit is set where
// evaluate_coverage without multisampling returns 0x80: inside the box, and all
// three edges not negative.
template <int NS>
struct WarpBlock
{
	static constexpr int PW = NS == 1 ? 8 : (NS <= 4 ? 4 : 2);
	static constexpr int PH = 32 / (NS * PW);
	static constexpr int P = PW * PH;
	// Mask bit of sample s of the pixel at (x, y) in the block.
	__device__ static constexpr uint32_t bit(uint32_t s, uint32_t x, uint32_t y) { return 31u - (s * P + y * PW + x); }
	// The bit of pixel 0 of each sample, in box_mask's order (ascending).
	static constexpr uint32_t sample_ones = NS == 1 ? 1u : NS == 2 ? 0x10001u : NS == 4 ? 0x01010101u : NS == 8 ? 0x11111111u : 0x55555555u;
};

// Where a warp's samples are: its first pixel and, in shared memory, the
// sub-pixel offset of each sample in coverage units (1/8 pixel).
struct WarpPlace
{
	int32_t px0, py0;
	const int2 *smp;
};

// Samples of the warp's block whose pixel lies in the primitive's box.
template <int NS>
__device__ __forceinline__ uint32_t box_mask(int4 bb, const WarpPlace &W)
{
	using B = WarpBlock<NS>;
	const int32_t xlo = max(bb.x - W.px0, 0), xhi = min(bb.z - W.px0, B::PW - 1);
	const int32_t ylo = max(bb.y - W.py0, 0), yhi = min(bb.w - W.py0, B::PH - 1);
	if (xlo > xhi || ylo > yhi)
		return 0u;
	// Bits in ascending order of (y, x), then reversed.
	const uint32_t cols = ((2u << xhi) - 1u) & (~0u << xlo);
	uint32_t m = 0;
	#pragma unroll
	for (int y = 0; y < B::PH; y++)
		if (y >= ylo && y <= yhi)
			m |= cols << (y * B::PW);
	return __brev(m * B::sample_ones);
}

// Bits of samples [s0, s1) in the low (s1 - s0) * P bits, set where the edges pass.
template <int NS, bool PAR>
__device__ __forceinline__ uint32_t edge_mask(const int32_t A[3], const int32_t Bc[3], const int32_t Cc[3], int32_t off_b,
                                              int32_t off_c, int32_t keep_x, int32_t keep_y, const WarpPlace &W, int s0, int s1)
{
	using B = WarpBlock<NS>;
	const int32_t x0 = W.px0 << 3, y0 = W.py0 << 3;
	const int32_t a0 = idot3(A, x0, y0), b0 = idot3(Bc, x0, y0), c0 = idot3(Cc, x0, y0);
	uint32_t outside = 0;
	#pragma unroll 1
	for (int s = s0; s < s1; s++)
	{
		int32_t as = a0, bs = b0, cs = c0;
		if (NS > 1)
		{
			const int2 o = W.smp[s];
			const int32_t ox = o.x & keep_x, oy = o.y & keep_y;
			as = int32_t(uint32_t(A[0]) * uint32_t(ox) + uint32_t(A[1]) * uint32_t(oy) + uint32_t(a0));
			bs = int32_t(uint32_t(Bc[0]) * uint32_t(ox) + uint32_t(Bc[1]) * uint32_t(oy) + uint32_t(b0));
			cs = int32_t(uint32_t(Cc[0]) * uint32_t(ox) + uint32_t(Cc[1]) * uint32_t(oy) + uint32_t(c0));
		}
		#pragma unroll
		for (int y = 0; y < B::PH; y++)
		{
			#pragma unroll
			for (int x = 0; x < B::PW; x++)
			{
				const int32_t ea = int32_t(uint32_t(as) + uint32_t(A[0]) * uint32_t(8 * x));
				const int32_t eb = int32_t(uint32_t(bs) + uint32_t(Bc[0]) * uint32_t(8 * x));
				const int32_t ec = int32_t(uint32_t(cs) + uint32_t(Cc[0]) * uint32_t(8 * x));
				int32_t neg = ea | eb | ec;
				if (PAR && ea < 0)
					neg = int32_t(uint32_t(eb) + uint32_t(ea) + uint32_t(off_b)) | int32_t(uint32_t(ec) + uint32_t(ea) + uint32_t(off_c));
				outside = __funnelshift_l(uint32_t(neg), outside, 1);
			}
			as = int32_t(uint32_t(as) + uint32_t(A[1]) * 8u);
			bs = int32_t(uint32_t(bs) + uint32_t(Bc[1]) * 8u);
			cs = int32_t(uint32_t(cs) + uint32_t(Cc[1]) * 8u);
		}
	}
	return ~outside;
}

// Whether the primitive fails its depth test on every sample it covers in the
// warp's block, given a lower bound `zmin` of the block's depths.  The bound of
// the primitive's depth is the interpolation plane at the block corner where it
// is largest, and for triangles no more than the largest vertex depth; both
// with a margin far above the rounding of the per-sample evaluation (each of
// its few operations is within 2^-24 of its operands' magnitude m, against a
// margin of 2^-17 m + 2).  Edges longer than 2048 pixels could wrap in 32 bits
// and are never dropped.
template <int NS>
__device__ __forceinline__ bool depth_hidden(const ShadeCtx &C, const PrimSetup &s, bool par, bool greater, int dim,
                                             const WarpPlace &W, uint32_t zmin)
{
	using B = WarpBlock<NS>;
	const int32_t a0 = s.a[0] >> 6;
	if ((abs(a0) | abs(s.a[1]) | abs(s.b[0]) | abs(s.b[1]) | abs(s.c[0]) | abs(s.c[1])) >= 1 << 15)
		return false;
	const float z1 = u2f(s.z[1]), z2 = u2f(s.z[2]);
	const float bx = float(s.b[0]), by = float(s.b[1]), cx = float(s.c[0]), cy = float(s.c[1]);
	// Last raster position of the block, in coverage units.
	const int32_t w = (B::PW << 3) - (8 >> dim), h = (B::PH << 3) - (8 >> dim);
	const int32_t x = (W.px0 << 3) + (z1 * bx + z2 * cx >= 0.0f ? w : 0), y = (W.py0 << 3) + (z1 * by + z2 * cy >= 0.0f ? h : 0);
	const float i = float(idot3(s.b, x, y)) * s.inv_area + s.error_i;
	const float j = float(idot3(s.c, x, y)) * s.inv_area + s.error_j;
	// A covered sample has i and j in [0, 1], so over the block they stay
	// within 1 plus their change across it.
	const float mag = z1 + z2 + (z1 * (fabsf(bx) * float(w) + fabsf(by) * float(h)) + z2 * (fabsf(cx) * float(w) + fabsf(cy) * float(h))) * s.inv_area;
	float top = z1 * i + z2 * j + mag * 0x1p-17f + 2.0f;
	if (!par)
		top = fminf(top, fmaxf(z1, z2) * (1.0f + 0x1p-18f) + 2.0f);
	uint32_t z = s.z[0];
	z = min(z + min(__float2uint_ru(top), 0xffffffffu - z), C.zmax);
	return greater ? z <= zmin : z < zmin;
}

// 32 primitives of the sub-tile's list, one per lane: coverage masks, the count
// of covered samples, the depth bound, then in order the primitives that are
// left.  zmin is taken once per call: depths only grow until a primitive writes
// depth without a test, so a lane behind such a primitive keeps its primitive.
// Bound: instruction issue (74 % of the issue slots, the integer pipe 62 % busy).
// A lane per primitive evaluates 32 samples of 32 primitives in about 250
// instructions where a lane per sample took about 70 per primitive, and on the
// textured 640x448 frame with 52,000 primitives at 4x the depth bound drops
// 3.2 M of the 4.4 M (primitive, warp) pairs that cover something; with the
// single shading call below, which keeps the loop in the instruction cache,
// the frame's shading went from 1.08 to 0.53 ms (1.12 G to 0.47 G warp
// instructions).  Plain 10,000-triangle frame at 1x: 70 to 47 us.
// With few primitives in the batch (NS >= 4), two or four lanes share one and
// take a part of its samples each.
template <int NS, bool SS>
__device__ __forceinline__ void walk_batch(const ShadeCtx &C, const uint32_t *ids, uint32_t n, const WarpPlace &W, uint32_t my_bit,
                                           uint32_t even_rows, uint32_t even_pixels, bool last, SampleState &S, uint32_t &covered)
{
	const PassParams &P = *C.P;
	const unsigned full = 0xffffffffu;
	const uint32_t lane = threadIdx.x & 31u;
	// log2 of the lanes per primitive, and this lane's primitive.
	const uint32_t share = NS >= 4 ? (n <= 8u ? 2u : n <= 16u ? 1u : 0u) : 0u;
	const uint32_t k = lane & (31u >> share);
	uint32_t pi = 0, st = 0, cov = 0;
	bool hidden = false;
	if (k < n)
	{
		pi = ids[k];
		st = P.prims[pi].state;
	}
	// Up to four parallelograms in a batch are evaluated by the whole warp, a sample
	// per lane (some 35 instructions each), so that the lanes of the triangles need
	// not wait for the parallelograms' loop (150): textured 4x frame, 4 % sprites,
	// 580 -> 562 us.  Not at one sample per pixel, where a plain frame lost 2 % to
	// the registers.
	constexpr bool TOGETHER = NS > 1;
	const uint32_t pars = TOGETHER ? __ballot_sync(full, k == lane && k < n && ((st >> STATE_BIT_PARALLELOGRAM) & 1u)) : 0u;
	const bool many = !TOGETHER || __popc(pars) > 4;
	if (k < n)
	{
		const PrimSetup s = P.setup[pi];
		cov = box_mask<NS>(make_int4(s.bb[0], s.bb[1], s.bb[2], s.bb[3]), W);
		const bool par = (s.a[0] & 1) != 0;
		uint32_t in = 0;
		if (cov)
		{
			const bool snap = SS && (st & (1u << STATE_BIT_SNAP_RASTER));
			const int32_t keep_x = snap ? int32_t(uint32_t(C.snap_mask_x) << (3 - C.dim)) : -1;
			const int32_t keep_y = snap ? int32_t(uint32_t(C.snap_mask_y) << (3 - C.dim)) : -1;
			const int32_t A[3] = { s.a[0] >> 6, s.a[1], s.a[2] };
			const int s0 = NS >= 4 ? int((lane >> (5u - share)) * (uint32_t(NS) >> share)) : 0;
			const int s1 = NS >= 4 ? s0 + int(uint32_t(NS) >> share) : NS;
			if (par)
			{
				if (many)
					in = edge_mask<NS, true>(A, s.b, s.c, int32_t((uint32_t(s.a[0]) >> 2) & 3u) - 1,
					                         int32_t((uint32_t(s.a[0]) >> 4) & 3u) - 1, keep_x, keep_y, W, s0, s1);
			}
			else
				in = edge_mask<NS, false>(A, s.b, s.c, 0, 0, keep_x, keep_y, W, s0, s1);
			in <<= (NS - s1) * WarpBlock<NS>::P;
		}
		if (NS < 4 || !share)
			cov &= in;
		else
		{
			// Only the lane's own samples are valid bits of `in`.
			const uint32_t part = 32u >> share, g = lane >> (5u - share);
			in &= (~0u << (32u - part)) >> (g * part);
			cov &= in;
		}
	}
	if constexpr (TOGETHER)
	for (uint32_t m = many ? 0u : pars; m; m &= m - 1u)
	{
		const int b = __ffs(m) - 1;
		const uint32_t bpi = __shfl_sync(full, pi, b), bst = __shfl_sync(full, st, b);
		const int4 *rec = reinterpret_cast<const int4 *>(P.setup + bpi);
		const int4 a4 = rec[0], b4 = rec[1], c4 = rec[2], bb = rec[3];
		int32_t x = S.hx, y = S.hy;
		if (SS && (bst & (1u << STATE_BIT_SNAP_RASTER)))
		{
			x &= C.snap_mask_x;
			y &= C.snap_mask_y;
		}
		const int sh = 3 - C.dim;
		const int32_t A[3] = { a4.x >> 6, a4.y, a4.z }, B3[3] = { b4.x, b4.y, b4.z }, C3[3] = { c4.x, c4.y, c4.z };
		const int32_t ea = idot3(A, x << sh, y << sh);
		int32_t eb = idot3(B3, x << sh, y << sh), ec = idot3(C3, x << sh, y << sh);
		if (ea < 0)
		{
			eb = int32_t(uint32_t(eb) + uint32_t(ea) + ((uint32_t(a4.x) >> 2) & 3u) - 1u);
			ec = int32_t(uint32_t(ec) + uint32_t(ea) + ((uint32_t(a4.x) >> 4) & 3u) - 1u);
		}
		const int32_t qx = x >> C.dim, qy = y >> C.dim;
		const uint32_t hit = __reduce_or_sync(full, qx >= bb.x && qy >= bb.y && qx <= bb.z && qy <= bb.w && (eb | ec) >= 0 ? 1u << my_bit : 0u);
		if (k == uint32_t(b))
			cov = hit;
	}
	if (NS >= 4 && share)
	{
		cov |= __shfl_xor_sync(full, cov, 16);
		if (share == 2u)
			cov |= __shfl_xor_sync(full, cov, 8);
	}
	// Not before it is needed: the first batch's records come while the depths do.
	const uint32_t zmin = C.zs ? __reduce_min_sync(full, S.depth) : 0u;
	if (cov)
	{
		if (P.has_scanmsk)
		{
			const uint32_t even = (st & (1u << STATE_BIT_SPRITE)) ? even_pixels : even_rows;
			if ((st >> STATE_BIT_SCANMSK_EVEN) & 1u) cov &= ~even;
			if ((st >> STATE_BIT_SCANMSK_ODD) & 1u) cov &= even;
		}
		if (lane != k)
			cov = 0;
		covered += uint32_t(__popc(cov));
		if (cov && C.zs && ((st >> STATE_BIT_Z_TEST) & 1u))
		{
			const PrimSetup &s = P.setup[pi];
			hidden = depth_hidden<NS>(C, s, (s.a[0] & 1) != 0, (st >> STATE_BIT_Z_TEST_GREATER) & 1u, C.dim, W, zmin);
		}
	}
	uint32_t bits = __ballot_sync(full, cov != 0u);
	uint32_t drop = __ballot_sync(full, hidden);
	if (drop)
	{
		const uint32_t lowers = __ballot_sync(full, cov != 0u && (st & ((1u << STATE_BIT_Z_TEST) | (1u << STATE_BIT_Z_WRITE))) ==
		                                                          (1u << STATE_BIT_Z_WRITE));
		// Primitives behind the first that may lower a depth stay.
		if (lowers)
			drop &= (lowers & (0u - lowers)) - 1u;
		bits &= ~drop;
	}
	// Early depth, then shading now or later (ubershader.comp:1694-1812).  A
	// primitive that is not opaque is shaded at once, after what was pending
	// under it; an opaque one replaces what was pending and writes its depth,
	// so a pending primitive never has a depth test or write left to do.  One
	// call shades what has to be: the pending ones under a primitive (which is
	// then taken again), the primitive itself, or, behind the sub-tile's last
	// one, all that is pending.
	for (;;)
	{
		Request r;
		uint32_t rp;
		bool act;
		r.coverage = 0x80;
		r.z_test = false;
		if (bits)
		{
			const int b = __ffs(bits) - 1;
			const uint32_t m = __shfl_sync(full, cov, b);
			const uint32_t bst = __shfl_sync(full, st, b);
			rp = __shfl_sync(full, pi, b);
			const int4 *rec = reinterpret_cast<const int4 *>(P.setup + rp);
			const int4 b4 = rec[1], c4 = rec[2], z4 = rec[4];
			const int32_t eb[3] = { b4.x, b4.y, b4.z }, ec[3] = { c4.x, c4.y, c4.z };
			const float inv_area = __int_as_float(z4.w), error_i = __int_as_float(b4.w), error_j = __int_as_float(c4.w);
			const int sh = 3 - C.dim;
			int32_t rx = S.hx, ry = S.hy;
			if (SS && (bst & (1u << STATE_BIT_SNAP_RASTER)))
			{
				rx &= C.snap_mask_x;
				ry &= C.snap_mask_y;
			}
			r.i = fadd(fmul(__int2float_rn(idot3(eb, rx << sh, ry << sh)), inv_area), error_i);
			r.j = fadd(fmul(__int2float_rn(idot3(ec, rx << sh, ry << sh)), inv_area), error_j);
			r.z = uint32_t(z4.x);
			act = (m >> my_bit) & 1u;
			if (C.zs)
			{
				// The conversion rounds to even and clamps at 0; the largest step is 4294967040.
				const uint32_t dz = __float2uint_rn(fadd(fmul(__int_as_float(z4.y), r.i), fmul(__int_as_float(z4.z), r.j)));
				r.z = min(r.z + min(min(dz, 4294967040u), 0xffffffffu - r.z), C.zmax);
				if ((bst >> STATE_BIT_Z_TEST) & 1u)
					act = act && (((bst >> STATE_BIT_Z_TEST_GREATER) & 1u) ? r.z > S.depth : r.z >= S.depth);
			}
			if (!__any_sync(full, act))
			{
				bits &= bits - 1u;
				continue;
			}
			r.z_write = C.zs && ((bst >> STATE_BIT_Z_WRITE) & 1u);
			if (SS && (bst & ((1u << STATE_BIT_SNAP_RASTER) | (1u << STATE_BIT_SNAP_ATTRIBUTE))) == (1u << STATE_BIT_SNAP_ATTRIBUTE))
			{
				const int32_t qx = (S.hx & C.snap_mask_x) << sh, qy = (S.hy & C.snap_mask_y) << sh;
				r.i = fadd(fmul(__int2float_rn(idot3(eb, qx, qy)), inv_area), error_i);
				r.j = fadd(fmul(__int2float_rn(idot3(ec, qx, qy)), inv_area), error_j);
			}
			if ((bst >> STATE_BIT_OPAQUE) & 1u)
			{
				if (act)
				{
					if (r.z_write)
					{
						S.depth = r.z;
						S.depth_dirty = true;
					}
					S.pending.coverage = 0x80;
					S.pending.i = r.i;
					S.pending.j = r.j;
					S.pending_prim = rp;
				}
				bits &= bits - 1u;
				continue;
			}
			const bool under = act && S.pending.coverage > 0;
			if (!__any_sync(full, under))
				bits &= bits - 1u;
			else
			{
				act = under;
				if (under)
				{
					r.i = S.pending.i;
					r.j = S.pending.j;
					rp = S.pending_prim;
					S.pending.coverage = 0;
				}
				r.z_write = false;
			}
		}
		else if (last)
		{
			last = false;
			act = S.pending.coverage > 0;
			if (!__any_sync(full, act))
				break;
			r.i = S.pending.i;
			r.j = S.pending.j;
			r.z = 0;
			r.z_write = false;
			rp = S.pending_prim;
			S.pending.coverage = 0;
		}
		else
			break;
		if (act)
			shade_resolve<false, false>(C, S, rp, r);
		__syncwarp();
	}
}

// Threads of a shading CTA: the 64 * NS samples of a sub-tile, 256 at most at a
// time; a CTA runs a sub-tile's parts one after the other on one expanded list.
// Whole sub-tiles in CTAs of 512 and 1024 threads at 8x and 16x leave two and one
// of them per SM, waiting for each other at every barrier; a CTA per part expands
// the list again and starts more CTAs (feedback frame of 100,000 primitives at 8x
// 2.48 ms whole, 1.93 a CTA per part, 1.72 so; at 16x 5.07, 3.51, 2.74).
// A long list is the launch's critical path, though, and the parts in turn make it
// as many times longer, so the sub-tiles of coarse tiles with many primitives are
// split.  Their parts are taken by CTAs in front of those of the sub-tiles, one per SM,
// so that a long list starts with the launch (3,000 primitives in 16x16 pixels next to
// 4,000 all over a 1024x900 frame at 8x: 440 us in turn, 441 split with all such CTAs
// behind, 291 so), and by more behind (2,000 blended triangles in one sub-tile at 16x
// 2.41 -> 0.77 ms, 36,000 AA1 triangles within 64x64 pixels 2.13 -> 0.68).  Which tiles:
// run_instance.
template <int NS>
struct ShadeCta
{
	static constexpr uint32_t THREADS = NS < PGS_SHADE_CTA_NS ? 64u * NS : 64u * PGS_SHADE_CTA_NS;
	static constexpr uint32_t PARTS = 64u * NS / THREADS;
	static constexpr uint32_t WARPS = THREADS / 32u;
};

// The sub-tile's primitive list, expanded by the T threads that shade it
// together into primitive indices in ascending order in shared memory (CAP at a
// time), then walked by each warp on its own, 32 primitives at a time.  Each
// thread takes LIST_WORDS mask words of a chunk of T * LIST_WORDS, all loads in
// flight at once, keeps them in registers, and writes the indices of their bits
// where a scan over the threads puts them.
// Bound: latency of the loads and barriers; most of a sub-tile's words are empty.
// A summary bitmask over the words, read first, saved reads of empty words but
// cost a round trip, and binning a second reduction per pair: plain frame of
// 10,000 primitives 48.6 us with it, 45.5 without; textured 4x frame of 52,000
// primitives 596 and 580 us (binning 45 and 37 of them).
constexpr uint32_t LIST_WORDS = 4;

template <uint32_t T, uint32_t CAP>
struct ListShared
{
	uint32_t ids[CAP];
	uint32_t count[LIST_WORDS * T / 32u]; // per word of the chunk and warp
	int2 smp[16];                         // sample offsets of WarpPlace
	uint32_t block[2];                    // colour and depth address of the sub-tile's first pixel
};

// The T threads that run a sub-tile together, thread 0 of them aligned to T: the CTA
// itself (GROUPS 0, barrier 0), or group k of GROUPS with barrier 1 + k of its own.
// The barrier's number is part of the instruction: with one in a register a kernel is
// taken to use all 16, and an SM has 64, for four CTAs, of 128 threads half of what its
// registers hold (64 small streams in rounds 2.83 ms, so 2.14).  Not with eight groups
// in 512 threads, where two CTAs fit anyway and choosing costs (AA1 streams 484 and 499 us).
template <uint32_t T, uint32_t GROUPS = 0>
struct ShadeGroup
{
	uint32_t k;
	__device__ __forceinline__ uint32_t thread() const { return threadIdx.x & (T - 1u); }
	template <uint32_t B = 1>
	__device__ __forceinline__ void sync() const
	{
		if constexpr (GROUPS == 0)
			asm volatile("bar.sync 0, %0;" ::"n"(T) : "memory");
		else if constexpr (T * GROUPS > 256u)
			asm volatile("bar.sync %0, %1;" ::"r"(1u + k), "n"(T) : "memory");
		else if (B == GROUPS || k + 1u == B)
			asm volatile("bar.sync %0, %1;" ::"n"(B), "n"(T) : "memory");
		else
			sync<(B < GROUPS ? B + 1 : B)>();
	}
};

template <uint32_t T, uint32_t CAP>
struct ListChunk
{
	static constexpr uint32_t WARPS = T / 32u;
	static_assert(LIST_WORDS == 4 && LIST_WORDS * WARPS <= 32, "two packed scans, one count per lane");
	uint32_t words[LIST_WORDS];
	uint32_t pos[LIST_WORDS]; // place of the thread's first index under each word
	uint32_t total;

	// Words [first, first + T * LIST_WORDS) of the `count` of the sub-tile.
	template <uint32_t GROUPS>
	__device__ __forceinline__ void load(const ShadeGroup<T, GROUPS> &G, const uint32_t *mask, uint32_t first, uint32_t count,
	                                     ListShared<T, CAP> &L)
	{
		const unsigned full = 0xffffffffu;
		const uint32_t t = G.thread(), lane = t & 31u, warp = t >> 5;
		#pragma unroll
		for (uint32_t k = 0; k < LIST_WORDS; k++)
			words[k] = first + k * T + t < count ? __ldg(mask + first + k * T + t) : 0u;
		// Two words' counts (1024 at most in a warp) per scan.
		const uint32_t c01 = uint32_t(__popc(words[0])) | (uint32_t(__popc(words[1])) << 16);
		const uint32_t c23 = uint32_t(__popc(words[2])) | (uint32_t(__popc(words[3])) << 16);
		const uint32_t x01 = warp_scan(c01, lane), x23 = first + 2u * T < count ? warp_scan(c23, lane) : 0u;
		if (lane == 31u)
		{
			L.count[warp] = x01 & 0xffffu;
			L.count[WARPS + warp] = x01 >> 16;
			L.count[2u * WARPS + warp] = x23 & 0xffffu;
			L.count[3u * WARPS + warp] = x23 >> 16;
		}
		G.sync();
		const uint32_t v = lane < LIST_WORDS * WARPS ? L.count[lane] : 0u, x = warp_scan(v, lane);
		total = __shfl_sync(full, x, 31);
		const uint32_t e01 = x01 - c01, e23 = x23 - c23;
		const uint32_t before[LIST_WORDS] = { e01 & 0xffffu, e01 >> 16, e23 & 0xffffu, e23 >> 16 };
		#pragma unroll
		for (uint32_t k = 0; k < LIST_WORDS; k++)
			pos[k] = __shfl_sync(full, x - v, int(k * WARPS + warp)) + before[k];
	}

	// Indices [round, round + CAP) of the chunk.
	template <uint32_t GROUPS>
	__device__ __forceinline__ void write(const ShadeGroup<T, GROUPS> &G, uint32_t prim_lo, uint32_t first, uint32_t round,
	                                      ListShared<T, CAP> &L) const
	{
		#pragma unroll
		for (uint32_t k = 0; k < LIST_WORDS; k++)
		{
			uint32_t p = pos[k] - round;
			for (uint32_t m = words[k]; m; m &= m - 1u, p++)
				if (p < CAP)
					L.ids[p] = prim_lo + (first + k * T + G.thread()) * 32u + uint32_t(__ffs(m) - 1);
		}
	}
};

// Walks the list: without AA1 through coverage masks (walk_batch); with AA1
// every lane tests one primitive against the warp's rectangle (may_cover) and
// the warp shades, in order, the primitives that can touch it, so that it sees
// the same sequence of covering primitives as walking the whole list.
// `chunk` is the list's first chunk, loaded by the caller; with `written`, it is
// the whole list and lies in L already.  RELOAD: of a list that is not, the caller
// kept only the length, and every part loads the first chunk again, the first part
// too: kept until then it cost registers in all of the walk (25,000 small mip-mapped
// triangles at 8x 341 -> 395 us, for 309 -> 307 us of 60,000 small triangles).
template <int NS, bool SS, bool AA, bool MIP, bool RELOAD, uint32_t T, uint32_t CAP, uint32_t GROUPS>
__device__ __forceinline__ void walk_list(const ShadeCtx &C, const DevInstance &I, const ShadeGroup<T, GROUPS> &G, const uint32_t *mask,
                                          ListChunk<T, CAP> &chunk, bool written, ListShared<T, CAP> &L, uint32_t t,
                                          SampleState &S, uint32_t &covered)
{
	const PassParams &P = *C.P;
	const uint32_t lane = threadIdx.x & 31u;
	const unsigned full = 0xffffffffu;
	WarpPlace W;
	uint32_t my_bit = 0, even_rows = 0, even_pixels = 0;
	int4 rect = {}; // of the warp's raster positions, the same in every lane
	if constexpr (!AA)
	{
		using B = WarpBlock<NS>;
		const int32_t px = S.hx >> C.dim, py = S.hy >> C.dim;
		W.px0 = __shfl_sync(full, px, 0);
		W.py0 = __shfl_sync(full, py, 0);
		W.smp = L.smp;
		my_bit = B::bit(t % NS, uint32_t(px - W.px0), uint32_t(py - W.py0));
		if (P.has_scanmsk)
		{
			even_rows = __reduce_or_sync(full, (S.hy & 1) ? 0u : 1u << my_bit);
			even_pixels = __reduce_or_sync(full, (py & 1) ? 0u : 1u << my_bit);
		}
	}
	else
	{
		const int32_t x0 = S.hx & C.snap_mask_x, y0 = S.hy & C.snap_mask_x & C.snap_mask_y;
		rect = make_int4(__reduce_min_sync(full, x0), __reduce_min_sync(full, y0), __reduce_max_sync(full, S.hx),
		                 __reduce_max_sync(full, S.hy));
	}
	if (RELOAD && !written)
	{
		G.sync();
		chunk.load(G, mask, 0, I.mask_words, L);
	}
	for (uint32_t first = 0;;)
	{
		const bool last_chunk = first + T * LIST_WORDS >= I.mask_words;
		for (uint32_t round = 0; round < chunk.total || (last_chunk && round == 0); round += CAP)
		{
			if (!written)
			{
				if (round)
					G.sync();
				chunk.write(G, I.prim_lo, first, round, L);
				G.sync();
			}
			const uint32_t n = min(chunk.total - round, CAP);
			const bool last_round = last_chunk && round + CAP >= chunk.total;
			if constexpr (!AA)
			{
				// The last batch, even an empty one, shades what is pending.
				for (uint32_t kb = 0; kb < n || (last_round && kb == 0); kb += 32u)
					walk_batch<NS, SS>(C, L.ids + kb, min(n - kb, 32u), W, my_bit, even_rows, even_pixels, last_round && kb + 32u >= n,
					                   S, covered);
			}
			else
			for (uint32_t kb = 0; kb < n || (last_round && kb == 0); kb += 32u)
			{
				const uint32_t k = kb + lane;
				uint32_t pi = 0;
				bool hit = false;
				if (k < n)
				{
					pi = L.ids[k];
					hit = may_cover(P.setup[pi], P.prims[pi].state, rect, C.dim);
				}
				uint32_t bits = __ballot_sync(full, hit);
				// Behind the sub-tile's last primitive, what is pending.
				const bool last = MIP && last_round && kb + 32u >= n;
				while (bits || last)
				{
					const bool flush = !bits;
					const int b = flush ? 0 : __ffs(bits) - 1;
					bits &= bits - 1u;
					process_primitive<MIP>(C, __shfl_sync(full, pi, b), flush, S, covered);
					if (flush)
						break;
				}
			}
		}
		if (last_chunk)
			break;
		first += T * LIST_WORDS;
		G.sync();
		chunk.load(G, mask, first, I.mask_words, L);
	}
}

// State of a coarse tile with these flags: 0 = empty, 1 = single-sampled,
// 2 = super-sampled (binning.comp:272-311 decision).
__device__ __forceinline__ uint32_t tile_mode(const DevInstance &I, uint32_t flags)
{
	if (!(flags & TILE_NONEMPTY))
		return 0;
	bool req = I.force_ss || (flags & TILE_REQ_SS);
	if (I.blend_demote && (flags >> TILE_COUNT_SHIFT) >= I.blend_demote && !(flags & TILE_HAS_ZW))
		req = false;
	req = req || ((flags & TILE_REQ_SS_ZW) && (flags & TILE_HAS_ZW));
	return (I.rate_y_log2 != 0 && req) ? 2u : 1u;
}

// Flags of the coarse tile of sub-tile `sub`.
__device__ __forceinline__ uint32_t subtile_flags(const PassParams &P, const DevInstance &I, const uint32_t *tile_flags,
                                                  uint32_t sub)
{
	const uint32_t gx = sub % I.sub_w, gy = sub / I.sub_w;
	const uint32_t sh = P.tile_size_log2 - 3u;
	return tile_flags[(gy >> sh) * I.tiles_w + (gx >> sh)];
}

// Whether the parts of the sub-tiles of a coarse tile go to CTAs of their own
// (ShadeCta).  Which CTA shades a part changes no result.
__device__ __forceinline__ bool split_tile(const DevInstance &I, uint32_t flags)
{
	return I.split_count && ((flags >> TILE_COUNT_SHIFT) >= I.split_count || I.split_count == SPLIT_ALL);
}

// Part number `item` of all parts of the sub-tiles of split super-sampled tiles:
// its sub-tile and part, or false behind the last.  All threads of the group.
template <uint32_t PARTS, uint32_t T, uint32_t CAP>
__device__ __forceinline__ bool split_part(const PassParams &P, const DevInstance &I, const uint32_t *tile_flags, uint32_t item,
                                           const ShadeGroup<T> &G, ListShared<T, CAP> &list, uint32_t &sub, uint32_t &part)
{
	constexpr uint32_t WARPS = T / 32u;
	static_assert(LIST_WORDS * WARPS == 32u, "one count per lane");
	const unsigned full = 0xffffffffu;
	const uint32_t sh = P.tile_size_log2 - 3u, per_tile = PARTS << (2u * sh);
	const uint32_t want = item / per_tile, k = item % per_tile; // tile by rank, part in it
	const uint32_t lane = G.thread() & 31u, warp = G.thread() >> 5, tiles = I.tiles_w * I.tiles_h;
	uint32_t seen = 0;
	for (uint32_t base = 0; base < tiles; base += T * LIST_WORDS)
	{
		uint32_t split[LIST_WORDS]; // of the warp's tiles
		#pragma unroll
		for (uint32_t q = 0; q < LIST_WORDS; q++)
		{
			const uint32_t tile = base + q * T + G.thread(), flags = tile < tiles ? tile_flags[tile] : 0u;
			split[q] = __ballot_sync(full, tile_mode(I, flags) == 2u && split_tile(I, flags));
			if (lane == 0)
				list.count[q * WARPS + warp] = uint32_t(__popc(split[q]));
		}
		G.sync();
		const uint32_t v = list.count[lane], x = warp_scan(v, lane), total = __shfl_sync(full, x, 31);
		if (want - seen < total)
		{
			#pragma unroll
			for (uint32_t q = 0; q < LIST_WORDS; q++)
			{
				const uint32_t before = seen + __shfl_sync(full, x - v, int(q * WARPS + warp));
				if (((split[q] >> lane) & 1u) && before + uint32_t(__popc(split[q] & ((1u << lane) - 1u))) == want)
					list.ids[0] = base + q * T + G.thread();
			}
			G.sync();
			const uint32_t t = list.ids[0], in = k / PARTS;
			sub = ((t / I.tiles_w << sh) + (in >> sh)) * I.sub_w + (t % I.tiles_w << sh) + (in & ((1u << sh) - 1u));
			part = k % PARTS;
			return true;
		}
		seen += total;
		G.sync();
	}
	return false;
}

// Samples t of the sub-tile at (sub_x, sub_y), one per thread of the group.
template <int NS, bool SS, bool AA, bool MIP, bool RELOAD, uint32_t T, uint32_t CAP, uint32_t GROUPS>
__device__ __forceinline__ void shade_part(const PassParams &P, const DevInstance &I, const ShadeGroup<T, GROUPS> &G, const uint32_t *mask,
                                           int32_t sub_x, int32_t sub_y, ListChunk<T, CAP> &chunk, bool written, uint32_t t,
                                           ListShared<T, CAP> &list)
{
	constexpr bool SHARE = T > 64u; // list.block is there
	ShadeCtx C;
	C.P = &P;
	C.I = &I;
	C.ss = SS;
	C.dim = SS ? int(I.rate_y_log2) : 0;
	C.snap_mask_x = -(1 << I.rate_y_log2);
	C.snap_mask_y = I.snap_mask_y;
	C.zs = I.zb_psm != 0xffffffffu;
	C.fb_psm = I.fb_psm;
	C.zb_psm = I.zb_psm;
	C.zmax = psm_is_16bit(I.zb_psm) ? 0xffffu : psm_is_24bit(I.zb_psm) ? 0xffffffu : 0xffffffffu;

	const uint32_t lane = t & 31u;
	const uint32_t sample = t % NS;
	C.sample = SS ? sample : 0u;
	const uint32_t pix = t / NS;
	// Pixel order inside the sub-tile: x from bits 0,2,4 and y from bits 1,3,5,
	// so that each warp covers a compact block.
	const int32_t lx = int32_t((pix & 1u) | ((pix >> 1) & 2u) | ((pix >> 2) & 4u));
	const int32_t ly = int32_t(((pix >> 1) & 1u) | ((pix >> 2) & 2u) | ((pix >> 3) & 4u));
	const int32_t px = sub_x + lx, py = sub_y + ly;

	SampleState S;
	S.hx = px << C.dim;
	S.hy = py << C.dim;
	if (SS)
	{
		const int2 o = list.smp[sample];
		S.hx += o.x >> (3 - C.dim);
		S.hy += o.y >> (3 - C.dim);
	}
	S.color_dirty = false;
	S.depth_dirty = false;
	S.pending.coverage = 0;
	S.pending.z_test = false;
	S.pending.z_write = false;
	S.pending.z = 0;
	S.pending_prim = 0;

	uint32_t fb_index, z_index;
	if (!SHARE || ((I.base_x | I.base_y) & 7))
	{
		fb_index = swizzle_address(uint32_t(px), uint32_t(py), I.fb_base, I.fb_stride, I.fb_psm);
		z_index = C.zs ? swizzle_address(uint32_t(px), uint32_t(py), I.zb_base, I.fb_stride, I.zb_psm) : 0u;
	}
	else
	{
		// On the 8-pixel grid a sub-tile is one block of a 32-bit format or half
		// of one of a 16-bit format: the pixel's place in it are its coordinates'
		// bits, 32-bit words x0 y0 x1 x2 y1 y2, 16-bit halves (x3) x0 y0 x1 x2 y1 y2.
		const uint32_t ux = uint32_t(lx), uy = uint32_t(ly);
		const uint32_t in_block = (ux & 1u) | ((uy & 1u) << 1) | ((ux & 6u) << 1) | ((uy & 6u) << 3);
		fb_index = list.block[0] + (psm_is_16bit(I.fb_psm) ? in_block << 1 : in_block);
		z_index = C.zs ? list.block[1] + (psm_is_16bit(I.zb_psm) ? in_block << 1 : in_block) : 0u;
	}
	const uint32_t V32 = VRAM_SIZE / 4, V16 = VRAM_SIZE / 2;
	uint32_t *vram32 = reinterpret_cast<uint32_t *>(P.vram);
	uint16_t *vram16 = reinterpret_cast<uint16_t *>(P.vram);

	// begin_tile.  Both buffers' pixels and reference flags are on their way before
	// the first is waited for, and so are both samples after them: two round trips
	// where colour's two and then depth's two were four (feedback frame of 100,000
	// primitives at 8x 1.64 -> 1.59 ms per replay, alone 2.15 -> 2.10, 16x 2.65 -> 2.61).
	const bool c16 = psm_is_16bit(I.fb_psm), z16 = psm_is_16bit(I.zb_psm);
	const uint8_t *zsrc = P.zcache ? P.zcache : P.vram;
	const uint32_t *zsrc32 = reinterpret_cast<const uint32_t *>(zsrc);
	const uint16_t *zsrc16 = reinterpret_cast<const uint16_t *>(zsrc);
	uint32_t col, col_ref = 0, dep = 0, dep_ref = 0;
	if (c16)
	{
		col = vram16[fb_index];
		if (SS)
			col_ref = vram16[fb_index + V16];
	}
	else
	{
		col = vram32[fb_index];
		if (SS)
			col_ref = vram32[fb_index + V32];
	}
	if (C.zs)
	{
		dep = z16 ? zsrc16[z_index] : zsrc32[z_index];
		if (SS)
			dep_ref = z16 ? zsrc16[z_index + V16] : zsrc32[z_index + V32];
	}
	if (SS)
	{
		const uint32_t cm = c16 ? 0xffffu : psm_is_24bit(I.fb_psm) ? 0xffffffu : 0xffffffffu;
		const bool cs = (col_ref & cm) == cm, ds = C.zs && (dep_ref & C.zmax) == C.zmax;
		uint32_t sc = col, sd = dep;
		if (cs)
			sc = c16 ? vram16[fb_index + (sample + 2u) * V16] : vram32[fb_index + (sample + 2u) * V32];
		if (ds)
			sd = z16 ? zsrc16[z_index + (sample + 2u) * V16] : zsrc32[z_index + (sample + 2u) * V32];
		col = psm_is_24bit(I.fb_psm) && col_ref != 0xffffffffu ? ((col & 0xff000000u) | (sc & 0xffffffu)) : sc;
		dep = sd;
	}
	S.color = c16 ? expand16(col) : col;
	S.depth = C.zs ? dep & C.zmax : 0u;

	uint32_t covered = 0;
	walk_list<NS, SS, AA, MIP, RELOAD, T, CAP>(C, I, G, mask, chunk, written, list, t, S, covered);

	// The other walks shade what is pending behind their last primitive.
	if (AA && !MIP && S.pending.coverage > 0)
		shade_resolve<MIP, AA>(C, S, S.pending_prim, S.pending);

	// Covered-sample counter: one atomic per warp.
	{
		const uint32_t c = __reduce_add_sync(0xffffffffu, covered);
		if (lane == 0 && c)
			atomicAdd(P.fragment_counter, (unsigned long long)c);
	}

	// end_tile
	const unsigned full = 0xffffffffu;
	if (!__any_sync(full, S.color_dirty || S.depth_dirty))
		return;
	uint32_t group_lane0 = (t & 31u) & ~uint32_t(NS - 1);
	bool req_color = false, req_depth = false;
	bool color_dirty = S.color_dirty, depth_dirty = S.depth_dirty;
	uint32_t color = S.color, depth = S.depth;
	uint32_t group_mask = (NS == 32) ? full : (((1u << NS) - 1u) << group_lane0);

	if (SS)
	{
		uint32_t first = __shfl_sync(full, S.color, int(group_lane0));
		req_color = I.preserve_samples ? true : ((__ballot_sync(full, first != S.color) & group_mask) != 0u);
		if (C.zs)
		{
			uint32_t zfirst = __shfl_sync(full, S.depth, int(group_lane0));
			req_depth = (__ballot_sync(full, zfirst != S.depth) & group_mask) != 0u;
		}
		color_dirty = (__ballot_sync(full, S.color_dirty) & group_mask) != 0u;
		// Butterfly sums in the order XOR NS/2 ... 1; every lane takes part.
		const float *lut = P.unorm_lut;
		float v0 = unorm8_lut(lut, S.color, 0), v1 = unorm8_lut(lut, S.color, 1), v2 = unorm8_lut(lut, S.color, 2), v3 = unorm8_lut(lut, S.color, 3);
		#pragma unroll
		for (int o = NS / 2; o >= 1; o >>= 1)
		{
			v0 = fadd(v0, __shfl_xor_sync(full, v0, o));
			v1 = fadd(v1, __shfl_xor_sync(full, v1, o));
			v2 = fadd(v2, __shfl_xor_sync(full, v2, o));
			v3 = fadd(v3, __shfl_xor_sync(full, v3, o));
		}
		const float n = 1.0f / float(NS); // a power of two: the product is the exact quotient
		uint32_t resolved = pack_unorm(fmul(v0, n), fmul(v1, n), fmul(v2, n), fmul(v3, n));
		uint32_t zmin = S.depth;
		#pragma unroll
		for (int o = NS / 2; o >= 1; o >>= 1)
			zmin = min(zmin, __shfl_xor_sync(full, zmin, o));
		if (C.zs)
			depth_dirty = (__ballot_sync(full, S.depth_dirty) & group_mask) != 0u;

		if (req_color)
		{
			if (color_dirty)
			{
				if (psm_is_16bit(I.fb_psm))
					vram16[fb_index + (sample + 2u) * V16] = uint16_t(rgba32_to_rgba16(S.color));
				else
					vram32[fb_index + (sample + 2u) * V32] = S.color;
			}
			color = I.preserve_samples ? first : resolved;
		}
		if (C.zs && req_depth)
		{
			if (depth_dirty)
			{
				if (psm_is_16bit(I.zb_psm))
					vram16[z_index + (sample + 2u) * V16] = uint16_t(S.depth);
				else
					vram32[z_index + (sample + 2u) * V32] = S.depth;
			}
			depth = zmin;
		}
	}

	bool first_sample = !SS || sample == 0;
	if (color_dirty && first_sample)
	{
		if (psm_is_16bit(I.fb_psm))
		{
			if (P.has_ss_reference)
				vram16[fb_index + V16] = req_color ? 0xffffu : 0u;
			vram16[fb_index] = uint16_t(rgba32_to_rgba16(color));
		}
		else
		{
			if (P.has_ss_reference)
				vram32[fb_index + V32] = req_color ? 0xffffffffu : 0u;
			vram32[fb_index] = color;
		}
	}
	if (C.zs && depth_dirty && first_sample)
	{
		if (psm_is_16bit(I.zb_psm))
		{
			if (P.has_ss_reference)
				vram16[z_index + V16] = req_depth ? 0xffffu : 0u;
			vram16[z_index] = uint16_t(depth);
		}
		else
		{
			if (P.has_ss_reference)
				vram32[z_index + V32] = req_depth ? (psm_is_24bit(I.zb_psm) ? 0xffffffu : 0xffffffffu) : 0u;
			if (psm_is_24bit(I.zb_psm))
			{
				uint8_t *b = P.vram + size_t(z_index) * 4u;
				*reinterpret_cast<uint16_t *>(b) = uint16_t(depth);
				b[2] = uint8_t(depth >> 16);
			}
			else
				vram32[z_index] = depth;
		}
	}
}

// Asks for the sub-tile's 256 bytes of every plane of the frame and depth buffers, a
// sector per thread, so that a sample's value is on its way while its reference flag is
// read, and a later part's while the first is shaded.
// Bound: latency (the loads of a part follow one another).  Feedback frame of 100,000
// primitives at 8x 1.72 -> 1.65 ms per replay of three in turn, 16x 2.74 -> 2.67, textured
// frame at 4x 559 -> 557 us; a lone replay at 8x, on planes that lie in memory, 2.16 ->
// 2.18 ms.  Planes 0 and 1 alone give 1.70 and 2.72 ms.
// fb and zb: swizzled index of the sub-tile's first pixel, which has to lie on the
// 8-pixel grid for the sub-tile to be (part of) one block; nothing is asked for otherwise.
template <int NS, uint32_t T, uint32_t GROUPS>
__device__ __forceinline__ void prefetch_planes(const PassParams &P, const DevInstance &I, const ShadeGroup<T, GROUPS> &G, uint32_t fb,
                                                uint32_t zb)
{
	if ((I.base_x | I.base_y) & 7)
		return;
	constexpr uint32_t SECTORS = (NS + 2u) * 8u;
	const bool zs = I.zb_psm != 0xffffffffu;
	for (uint32_t i = G.thread(); i < (zs ? 2u * SECTORS : SECTORS); i += T)
	{
		const bool z = i >= SECTORS;
		const uint32_t k = z ? i - SECTORS : i;
		const uint32_t block = ((z ? zb : fb) << (psm_is_16bit(z ? I.zb_psm : I.fb_psm) ? 1 : 2)) & ~255u;
		const uint8_t *base = z && P.zcache ? P.zcache : P.vram;
		asm volatile("prefetch.global.L1 [%0];" :: "l"(base + size_t(k / 8u) * VRAM_SIZE + block + (k & 7u) * 32u));
	}
}

// One sub-tile's pixel samples, NS per pixel, one thread per sample: the T
// threads of the group have samples t (of 64 * NS) and, with PARTS, the samples T,
// 2 T ... further on.  SS selects the super-sampled path.
template <int NS, bool SS, bool AA, bool MIP, uint32_t PARTS, uint32_t T, uint32_t CAP, uint32_t GROUPS>
__device__ __forceinline__ void shade_subtile(const PassParams &P, const DevInstance &I, const ShadeGroup<T, GROUPS> &G,
                                              const uint32_t *sub_masks, uint32_t sub, uint32_t t, ListShared<T, CAP> &list)
{
	const uint32_t gx = sub % I.sub_w, gy = sub / I.sub_w;
	const uint32_t *mask = sub_masks + size_t(sub) * I.mask_words;

	// What is the same for all warps is computed by one and waits for them at the
	// list's barrier: sample offsets by the first, block addresses by the last
	// (not for the two warps of a single-sampled sub-tile, where it costs more:
	// plain frame 45.6 us without, 46.2 with; feedback frame at 8x 1.97 and 1.96 ms).
	constexpr bool SHARE = T > 64u;
	const int32_t sub_x = I.base_x + int32_t(gx * 8u), sub_y = I.base_y + int32_t(gy * 8u);
	if (SS && G.thread() < NS)
	{
		int32_t x, y;
		sample_offset(G.thread(), I.rate_x_log2, I.rate_y_log2, x, y);
		list.smp[G.thread()] = make_int2(x << (3u - I.rate_y_log2), y << (3u - I.rate_y_log2));
	}
	if (SHARE && G.thread() >= T - 2u)
	{
		const bool z = G.thread() == T - 1u;
		list.block[z ? 1 : 0] = swizzle_address(uint32_t(sub_x), uint32_t(sub_y), z ? I.zb_base : I.fb_base, I.fb_stride,
		                                        z ? I.zb_psm : I.fb_psm);
	}

	// The list first: many sub-tiles of a pass of small primitives have none,
	// and the samples' loads overlap its expansion.
	ListChunk<T, CAP> chunk;
	chunk.load(G, mask, 0, I.mask_words, list);
	if (!chunk.total && I.mask_words <= T * LIST_WORDS)
		return;
	if constexpr (SS && SHARE)
		prefetch_planes<NS, T>(P, I, G, list.block[0], list.block[1]);
	if constexpr (PARTS == 1)
		shade_part<NS, SS, AA, MIP, false, T, CAP>(P, I, G, mask, sub_x, sub_y, chunk, false, t, list);
	else
	{
		// Nearly every list fits: written once, and no barrier from there on.
		const bool written = I.mask_words <= T * LIST_WORDS && chunk.total <= CAP;
		if (written)
		{
			chunk.write(G, I.prim_lo, 0, 0, list);
			G.sync();
		}
		#pragma unroll 1
		for (uint32_t part = 0; part < PARTS; part++)
			shade_part<NS, SS, AA, MIP, true, T, CAP>(P, I, G, mask, sub_x, sub_y, chunk, written, t + part * T, list);
	}
}

// Indices held in shared memory at a time.
constexpr uint32_t SHADE_LIST_CAP = 2048u, BATCH_LIST_CAP = 512u;

// Sub-tiles whose coarse tile selects the other path exit immediately.
template <int NS, bool SS, bool AA, bool MIP>
__global__ void __launch_bounds__(ShadeCta<NS>::THREADS, PGS_SHADE_MIN_BLOCKS(NS)) shade_kernel(PassParams P, DevInstance I, const uint32_t *sub_masks,
                                                        const uint32_t *tile_flags)
{
	constexpr uint32_t T = ShadeCta<NS>::THREADS, PARTS = ShadeCta<NS>::PARTS;
	__shared__ ListShared<T, SHADE_LIST_CAP> list;
	const ShadeGroup<T> G{ 0u };
	uint32_t sub = blockIdx.x - (PARTS > 1 ? I.split_first : 0u);
	// The usual case comes first: behind the other, each launch took 3 us longer.
	if (sub < I.sub_w * I.sub_h)
	{
		const uint32_t flags = subtile_flags(P, I, tile_flags, sub);
		if (tile_mode(I, flags) == (SS ? 2u : 1u) && !(PARTS > 1 && split_tile(I, flags)))
			shade_subtile<NS, SS, AA, MIP, PARTS, T, SHADE_LIST_CAP>(P, I, G, sub_masks, sub, threadIdx.x, list);
		return;
	}
	if constexpr (PARTS > 1)
	{
		// Every so many-th part of split sub-tiles.  (A counter that hands them out evened
		// the CTAs' loads a little, but the longer code cost all launches 4 us.)
		const uint32_t subs = I.sub_w * I.sub_h;
		uint32_t part, item = blockIdx.x < I.split_first ? blockIdx.x : blockIdx.x - subs;
		for (; split_part<PARTS>(P, I, tile_flags, item, G, list, sub, part); item += gridDim.x - subs)
		{
			shade_subtile<NS, SS, AA, MIP, 1, T, SHADE_LIST_CAP>(P, I, G, sub_masks, sub, threadIdx.x + part * T, list);
			__syncthreads();
		}
	}
}

// ---------------------------------------------------------------------------
// Batched shading: one launch shades the current instance segment of many
// independent command streams.  Each item is one (stream, pass, segment) with
// its own VRAM, records and bins; its samples, sub-tile after sub-tile, are cut
// into units of BLOCK that persistent CTAs take from a global counter, so
// streams of very different sizes share the GPU without a tail per stream.  In a
// unit the threads of each sub-tile form a group that expands and walks the
// sub-tile's list as a CTA of shade_kernel does (of a single-sampled sub-tile the
// first 64 threads do).
// Bound: issue of the shading itself, as in shade_kernel.  The five smallest of
// twelve mixed streams took 285 us in units of one warp, each of which walked its
// sub-tile's whole list on its own, and take 276 us.
struct ShadeItem
{
	PassParams P;
	DevInstance I;
	const uint32_t *masks, *flags;
	uint32_t ns_log2, aa;
	uint32_t unit_base, units;
};

// Sample counts the batched kernel shades itself (1x, 2x, 4x instances).
constexpr uint32_t BATCH_MAX_NS_LOG2 = 2;

// Separate functions per variant keep each variant's register allocation
// its own inside the batched kernel.
template <int NS, bool SS, bool AA, uint32_t T, uint32_t BLOCK>
__device__ __noinline__ void shade_subtile_call(const PassParams &P, const DevInstance &I, const uint32_t *sub_masks, uint32_t sub,
                                                uint32_t t, ListShared<T, BATCH_LIST_CAP> &list)
{
	shade_subtile<NS, SS, AA, false, 1, T, BATCH_LIST_CAP>(P, I, ShadeGroup<T, BLOCK / T>{ threadIdx.x / T }, sub_masks, sub, t, list);
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) batch_shade_kernel(const ShadeItem *items, uint32_t n_items,
                                                                         uint32_t total_units, uint32_t *counter)
{
	constexpr uint32_t T4 = BLOCK < 256 ? BLOCK : 256, T2 = 128, T1 = 64;
	// One list per 64 threads; a group of several uses the first of its own.
	struct Slot
	{
		ListShared<T1, BATCH_LIST_CAP> list;
	};
	static_assert(sizeof(ListShared<T4, BATCH_LIST_CAP>) <= (T4 / T1) * sizeof(Slot) &&
	                  sizeof(ListShared<T2, BATCH_LIST_CAP>) <= (T2 / T1) * sizeof(Slot),
	              "a group's list fits its slots");
	__shared__ PassParams P;
	__shared__ DevInstance I;
	__shared__ Slot slots[BLOCK / T1];
	__shared__ uint32_t s_unit[2];
	if (threadIdx.x == 0)
		s_unit[0] = atomicAdd(counter, 1u);
	__syncthreads();
	uint32_t loaded = 0xffffffffu;
	for (uint32_t step = 0;; step++)
	{
		const uint32_t unit = s_unit[step & 1u];
		if (unit >= total_units)
			break;
		// The next unit's number is on its way while this one is shaded.
		if (threadIdx.x == 0)
			s_unit[(step + 1u) & 1u] = atomicAdd(counter, 1u);
		uint32_t lo = 0, hi = n_items - 1;
		while (lo < hi)
		{
			uint32_t mid = (lo + hi + 1u) >> 1;
			if (items[mid].unit_base <= unit)
				lo = mid;
			else
				hi = mid - 1u;
		}
		const ShadeItem &it = items[lo];
		if (lo != loaded)
		{
			// Item parameters into shared memory (all are done with the last item's).
			const uint32_t *srcP = reinterpret_cast<const uint32_t *>(&it.P), *srcI = reinterpret_cast<const uint32_t *>(&it.I);
			for (uint32_t k = threadIdx.x; k < sizeof(PassParams) / 4; k += BLOCK)
				reinterpret_cast<uint32_t *>(&P)[k] = srcP[k];
			for (uint32_t k = threadIdx.x; k < sizeof(DevInstance) / 4; k += BLOCK)
				reinterpret_cast<uint32_t *>(&I)[k] = srcI[k];
			loaded = lo;
			__syncthreads();
		}
		const uint32_t sample = (unit - it.unit_base) * BLOCK + threadIdx.x;
		const uint32_t sub = sample >> (6u + it.ns_log2), t = sample & ((64u << it.ns_log2) - 1u);
		const uint32_t mode = sub < I.sub_w * I.sub_h ? tile_mode(I, subtile_flags(P, I, it.flags, sub)) : 0u;
		const uint32_t ns_log2 = mode == 2 ? it.ns_log2 : 0u;
		// A group's list lies in the slot of its first 64 threads.
		if (mode && t < (64u << ns_log2))
		{
			const bool aa = it.aa != 0;
			const uint32_t s4 = threadIdx.x / T4 * (T4 / T1), s2 = threadIdx.x / T2 * (T2 / T1), s1 = threadIdx.x / T1;
			switch (ns_log2)
			{
			case 0:
				if (aa) shade_subtile_call<1, false, true, T1, BLOCK>(P, I, it.masks, sub, t, slots[s1].list);
				else shade_subtile_call<1, false, false, T1, BLOCK>(P, I, it.masks, sub, t, slots[s1].list);
				break;
			case 1:
			{
				auto &list = reinterpret_cast<ListShared<T2, BATCH_LIST_CAP> &>(slots[s2]);
				if (aa) shade_subtile_call<2, true, true, T2, BLOCK>(P, I, it.masks, sub, t, list);
				else shade_subtile_call<2, true, false, T2, BLOCK>(P, I, it.masks, sub, t, list);
				break;
			}
			default:
			{
				auto &list = reinterpret_cast<ListShared<T4, BATCH_LIST_CAP> &>(slots[s4]);
				if (aa) shade_subtile_call<4, true, true, T4, BLOCK>(P, I, it.masks, sub, t, list);
				else shade_subtile_call<4, true, false, T4, BLOCK>(P, I, it.masks, sub, t, list);
				break;
			}
			}
		}
		__syncthreads();
	}
}

// ---------------------------------------------------------------------------
// CRTC circuit read-out (sample_circuit.frag:98-148).  One thread per output
// texel; a 2x2 high-resolution read-out averages the sample planes of the
// quad position in float, in plane order, then converts to unorm8.
__device__ __forceinline__ uint32_t circuit_payload(const uint8_t *vram, uint32_t psm, uint32_t addr, uint32_t plane)
{
	if (psm_is_16bit(psm))
	{
		uint16_t v = reinterpret_cast<const uint16_t *>(vram)[addr + plane * (VRAM_SIZE / 2)];
		return rgba16_to_rgba32(v, 0, 0x0, 0xff);
	}
	uint32_t v = reinterpret_cast<const uint32_t *>(vram)[addr + plane * (VRAM_SIZE / 4)];
	if (psm != PSMCT32)
		v = (v & ~0xff000000u) | 0x80000000u;
	return v;
}

__global__ void __launch_bounds__(256) circuit_kernel(pgs_circuit_params C, const uint8_t *vram, const float *unorm_lut,
                                                      uint32_t *dst)
{
	const uint32_t x = blockIdx.x * 32u + (threadIdx.x & 31u), y = blockIdx.y * 8u + (threadIdx.x >> 5);
	if (x >= C.width || y >= C.height)
		return;
	uint32_t out = 0;
	if (x < C.valid_width && y < C.valid_height)
	{
		const uint32_t sx = C.super_samples >= 4 ? x >> 1 : x, sy = C.super_samples >= 4 ? y >> 1 : y;
		const uint32_t cx = sx + C.dbx, cy = sy * C.phase_stride + C.dby + C.phase;
		const uint32_t addr = swizzle_address(cx, cy, C.fbp * BLOCKS_PER_PAGE, C.fbw, C.psm);
		bool resolve = false;
		if (C.super_samples >= 4)
		{
			if (psm_is_16bit(C.psm))
				resolve = reinterpret_cast<const uint16_t *>(vram)[addr + VRAM_SIZE / 2] == 0xffffu;
			else
			{
				uint32_t ref = reinterpret_cast<const uint32_t *>(vram)[addr + VRAM_SIZE / 4];
				resolve = C.psm != PSMCT32 ? (ref & 0xffffffu) == 0xffffffu : ref == 0xffffffffu;
			}
		}
		if (!resolve)
			out = circuit_payload(vram, C.psm, addr, 0);
		else
		{
			const uint32_t n = C.super_samples / 4;
			const uint32_t quad = C.super_samples != 8 ? (y & 1u) + (x & 1u) * 2u : (x & 1u) + (y & 1u) * 2u;
			const uint32_t base = 2u + n * quad;
			float v[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
			for (uint32_t i = 0; i < n; i++)
			{
				uint32_t c = circuit_payload(vram, C.psm, addr, base + i);
				#pragma unroll
				for (int k = 0; k < 4; k++)
					v[k] = fadd(v[k], unorm_lut[(c >> (8 * k)) & 0xffu]);
			}
			const float fn = float(n);
			out = pack_unorm(__fdiv_rn(v[0], fn), __fdiv_rn(v[1], fn), __fdiv_rn(v[2], fn), __fdiv_rn(v[3], fn));
		}
	}
	dst[size_t(y) * C.width + x] = out;
}

// ---------------------------------------------------------------------------
// vsync output merge (GSRenderer::vsync, gs/gs_renderer.cpp:4738-4866): the
// circuits are stretched into their CRTC viewports over a BGCOLOR clear.
// The stretch is bilinear with 8-bit sub-texel positions, clamped to the
// edge: texel coordinate = ((2 d + 1) * src / (2 * dst)) - 1/2 in 1/256 units,
// exact texels when source and viewport have the same size.  Blends are
// integer: (c * a + d * (255 - a)) / 255 rounded to nearest, alpha from the
// source (blend factors SRC/CONSTANT_ALPHA, ONE/ZERO on alpha).

__device__ __forceinline__ uint32_t stretch_sample(const uint32_t *img, uint32_t iw, uint32_t ih, int32_t dx, int32_t dy,
                                                   uint32_t vw, uint32_t vh)
{
	const int64_t fx = (int64_t(2 * dx + 1) * iw * 256) / (2 * int64_t(vw)) - 128;
	const int64_t fy = (int64_t(2 * dy + 1) * ih * 256) / (2 * int64_t(vh)) - 128;
	const int32_t x0 = int32_t(fx >> 8), y0 = int32_t(fy >> 8);
	const uint32_t wx = uint32_t(fx & 255), wy = uint32_t(fy & 255);
	const int32_t xa = min(max(x0, 0), int32_t(iw) - 1), xb = min(max(x0 + 1, 0), int32_t(iw) - 1);
	const int32_t ya = min(max(y0, 0), int32_t(ih) - 1), yb = min(max(y0 + 1, 0), int32_t(ih) - 1);
	const uint32_t c00 = img[size_t(ya) * iw + xa], c10 = img[size_t(ya) * iw + xb];
	const uint32_t c01 = img[size_t(yb) * iw + xa], c11 = img[size_t(yb) * iw + xb];
	const uint32_t w00 = (256u - wx) * (256u - wy), w10 = wx * (256u - wy), w01 = (256u - wx) * wy, w11 = wx * wy;
	uint32_t out = 0;
	#pragma unroll
	for (int k = 0; k < 4; k++)
	{
		const int sh = 8 * k;
		uint32_t acc = w00 * ((c00 >> sh) & 255u) + w10 * ((c10 >> sh) & 255u) + w01 * ((c01 >> sh) & 255u) +
		               w11 * ((c11 >> sh) & 255u);
		out |= ((acc + 32768u) >> 16) << sh;
	}
	return out;
}

__device__ __forceinline__ uint32_t blend255(uint32_t s, uint32_t d, uint32_t a)
{
	const uint32_t v = s * a + d * (255u - a);
	const uint32_t q = v / 255u, r = v % 255u;
	return q + (2u * r > 255u ? 1u : 0u);
}

__global__ void __launch_bounds__(256) merge_kernel(pgs_merge_params M, const uint32_t *c1, const uint32_t *c2, uint32_t *dst)
{
	const uint32_t x = blockIdx.x * 32u + (threadIdx.x & 31u), y = blockIdx.y * 8u + (threadIdx.x >> 5);
	if (x >= M.width || y >= M.height)
		return;
	uint32_t color = M.bgcolor & 0xffffffu;
	const int32_t ix = int32_t(x), iy = int32_t(y);
	if (M.draw_circuit2 && M.rect_w[1] && M.rect_h[1] && ix >= M.rect_x[1] && ix < M.rect_x[1] + int32_t(M.rect_w[1]) &&
	    iy >= M.rect_y[1] && iy < M.rect_y[1] + int32_t(M.rect_h[1]))
		color = stretch_sample(c2, M.circuit[1].width, M.circuit[1].height, ix - M.rect_x[1], iy - M.rect_y[1],
		                       M.rect_w[1], M.rect_h[1]);
	if (M.draw_circuit1 && M.rect_w[0] && M.rect_h[0] && ix >= M.rect_x[0] && ix < M.rect_x[0] + int32_t(M.rect_w[0]) &&
	    iy >= M.rect_y[0] && iy < M.rect_y[0] + int32_t(M.rect_h[0]))
	{
		const uint32_t s = stretch_sample(c1, M.circuit[0].width, M.circuit[0].height, ix - M.rect_x[0],
		                                  iy - M.rect_y[0], M.rect_w[0], M.rect_h[0]);
		if (M.blend == 0)
			color = s;
		else
		{
			const uint32_t a = M.blend == 1 ? M.alp : (s >> 24);
			uint32_t out = s & 0xff000000u;
			#pragma unroll
			for (int k = 0; k < 3; k++)
				out |= blend255((s >> (8 * k)) & 255u, (color >> (8 * k)) & 255u, a) << (8 * k);
			color = out;
		}
	}
	dst[size_t(y) * M.width + x] = color;
}

// EXTWRITE (extwrite.comp:37-98): the merged image or a circuit written back
// into VRAM as CT32 at (WDX, WDY) of EXBP / EXBW, nearest texel at
// uv = base + id * scale, optionally converted to Y / YCbCr / alpha.  Float
// expressions are evaluated left to right, one rounding per operation.
__global__ void __launch_bounds__(256) extwrite_kernel(pgs_merge_params M, const uint32_t *src, uint32_t sw, uint32_t sh,
                                                       const float *unorm_lut, uint8_t *vram, uint32_t invalidate_ss)
{
	const uint32_t gx = blockIdx.x * 32u + (threadIdx.x & 31u), gy = blockIdx.y * 8u + (threadIdx.x >> 5);
	if (gx >= M.ext_width || gy >= M.ext_height)
		return;
	const float u = fadd(M.ext_uv_base[0], fmul(__uint2float_rn(gx), M.ext_uv_scale[0]));
	const float v = fadd(M.ext_uv_base[1], fmul(__uint2float_rn(gy), M.ext_uv_scale[1]));
	const int32_t tx = min(max(int32_t(floorf(fmul(u, __uint2float_rn(sw)))), 0), int32_t(sw) - 1);
	const int32_t ty = min(max(int32_t(floorf(fmul(v, __uint2float_rn(sh)))), 0), int32_t(sh) - 1);
	const uint32_t c = src[size_t(ty) * sw + tx];
	const float r = unorm_lut[c & 255u], g = unorm_lut[(c >> 8) & 255u], b = unorm_lut[(c >> 16) & 255u];
	const float a = unorm_lut[c >> 24];
	const float ey = fadd(fadd(fmul(0.587f, g), fmul(0.114f, b)), fmul(0.299f, r));
	const float ecb = fsub(fadd(fmul(-0.311f, g), fmul(0.500f, b)), fmul(0.169f, r));
	const float ecr = fadd(fsub(fmul(-0.419f, g), fmul(0.081f, b)), fmul(0.500f, r));
	const float Y = __fdiv_rn(fadd(fmul(219.0f, ey), 16.0f), 255.0f);
	const float Cb = __fdiv_rn(fadd(fmul(224.0f, ecb), 128.0f), 255.0f);
	const float Cr = __fdiv_rn(fadd(fmul(224.0f, ecr), 128.0f), 255.0f);
	float o[4];
	switch (M.ext_emodc)
	{
	case 0: o[0] = r; o[1] = g; o[2] = b; break;
	case 1: o[0] = Y; o[1] = Y; o[2] = Y; break;
	case 2: o[0] = Y; o[1] = Cb; o[2] = Cr; break;
	default: o[0] = a; o[1] = a; o[2] = a; break;
	}
	switch (M.ext_emoda)
	{
	case 0: o[3] = a; break;
	case 1: o[3] = Y; break;
	case 2: o[3] = fmul(0.5f, Y); break;
	default: o[3] = 0.0f; break;
	}
	const uint32_t addr = swizzle_address(gx + M.ext_wdx, gy + M.ext_wdy, M.ext_exbp, M.ext_exbw, PSMCT32);
	reinterpret_cast<uint32_t *>(vram)[addr] = pack_unorm(o[0], o[1], o[2], o[3]);
	if (invalidate_ss)
		reinterpret_cast<uint32_t *>(vram)[addr + VRAM_SIZE / 4] = 0;
}

// FastMAD deinterlace (weave.frag): lines of the current field pass through;
// the others pick between the previous field (weave) and the average of the
// current field's neighbours (bob) by the local luma difference, with
// smoothstep(0.04, 0.06, diff) and mix() evaluated left to right.
__device__ __forceinline__ float luma_diff(const float *lut, uint32_t a, uint32_t b)
{
	const float dr = fsub(lut[a & 255u], lut[b & 255u]);
	const float dg = fsub(lut[(a >> 8) & 255u], lut[(b >> 8) & 255u]);
	const float db = fsub(lut[(a >> 16) & 255u], lut[(b >> 16) & 255u]);
	return fabsf(fadd(fadd(fmul(dr, 0.299f), fmul(dg, 0.587f)), fmul(db, 0.114f)));
}

__global__ void __launch_bounds__(256) weave_kernel(const uint32_t *f0, const uint32_t *f1, const uint32_t *f2,
                                                    const uint32_t *f3, uint32_t width, uint32_t field_height,
                                                    uint32_t phase, const float *lut, uint32_t *dst)
{
	const uint32_t x = blockIdx.x * 32u + (threadIdx.x & 31u), y = blockIdx.y * 8u + (threadIdx.x >> 5);
	const uint32_t height = 2u * field_height;
	if (x >= width || y >= height)
		return;
	uint32_t out;
	if ((y & 1u) == phase)
		out = f0[size_t(y >> 1) * width + x];
	else if (y == 0 || y == height - 1u)
		out = f1[size_t(y >> 1) * width + x];
	else
	{
		const uint32_t up = (y - 1u) >> 1;
		const uint32_t cur0 = f0[size_t(up) * width + x], cur1 = f0[size_t(up + 1u) * width + x];
		const uint32_t prev0 = f2[size_t(up) * width + x], prev1 = f2[size_t(up + 1u) * width + x];
		const uint32_t fld1 = f1[size_t(y >> 1) * width + x], fld3 = f3[size_t(y >> 1) * width + x];
		const float mh = luma_diff(lut, cur0, prev0), ml = luma_diff(lut, cur1, prev1), mc = luma_diff(lut, fld1, fld3);
		const float diff = fmaxf(fminf(mh, ml), mc);
		const float tt = fminf(fmaxf(__fdiv_rn(fsub(diff, 0.04f), fsub(0.06f, 0.04f)), 0.0f), 1.0f);
		const float bob = fmul(fmul(tt, tt), fsub(3.0f, fmul(2.0f, tt)));
		float o[3];
		#pragma unroll
		for (int k = 0; k < 3; k++)
		{
			const float avg = fmul(0.5f, fadd(lut[(cur0 >> (8 * k)) & 255u], lut[(cur1 >> (8 * k)) & 255u]));
			o[k] = fadd(fmul(lut[(fld1 >> (8 * k)) & 255u], fsub(1.0f, bob)), fmul(avg, bob));
		}
		out = pack_unorm(o[0], o[1], o[2], 1.0f);
	}
	dst[size_t(y) * width + x] = out;
}

// ---------------------------------------------------------------------------
// K4: VRAM transfers.
struct CopyParams
{
	uint32_t sbp, sbw, spsm, dbp, dbw, dpsm;
	uint32_t ssax, ssay, dsax, dsay, width, height;
	uint32_t xdir;
	uint64_t host_size, host_offset_qwords;
	const uint8_t *host;      // device copy of the HWREG payload
	const uint8_t *src_vram;  // snapshot for local->local
	uint32_t invalidate_ss;
};

__device__ __forceinline__ void write_pixel(uint8_t *vram, uint32_t psm, uint32_t addr, uint32_t data, bool inv)
{
	uint32_t *v32 = reinterpret_cast<uint32_t *>(vram);
	uint16_t *v16 = reinterpret_cast<uint16_t *>(vram);
	const uint32_t V32 = VRAM_SIZE / 4, V16 = VRAM_SIZE / 2;
	switch (psm)
	{
	case PSMCT24: case PSMZ24:
	{
		uint8_t *b = vram + size_t(addr) * 4u;
		b[0] = uint8_t(data); b[1] = uint8_t(data >> 8); b[2] = uint8_t(data >> 16);
		if (inv) { uint8_t *r = b + VRAM_SIZE; r[0] = 0; r[1] = 0; r[2] = 0; }
		break;
	}
	case PSMCT16: case PSMCT16S: case PSMZ16: case PSMZ16S:
		v16[addr] = uint16_t(data);
		if (inv) v16[addr + V16] = 0;
		break;
	case PSMT8:
		vram[addr] = uint8_t(data);
		if (inv) vram[addr + VRAM_SIZE] = 0;
		break;
	case PSMT8H:
		vram[addr * 4u + 3u] = uint8_t(data);
		if (inv) vram[addr * 4u + 3u + VRAM_SIZE] = 0;
		break;
	case PSMT4:
	{
		uint32_t word = addr >> 3, sh = 4u * (addr & 7u);
		atomicAnd(&v32[word], ~(0xfu << sh));
		atomicOr(&v32[word], (data & 0xfu) << sh);
		if (inv) atomicAnd(&v32[word + V32], ~(0xfu << sh));
		break;
	}
	case PSMT4HL: case PSMT4HH:
	{
		uint32_t sh = psm == PSMT4HL ? 24u : 28u;
		v32[addr] = (v32[addr] & ~(0xfu << sh)) | ((data & 0xfu) << sh);
		if (inv) v32[addr + V32] &= ~(0xfu << sh);
		break;
	}
	default:
		v32[addr] = data;
		if (inv) v32[addr + V32] = 0;
		break;
	}
}

__device__ __forceinline__ uint32_t read_pixel(const uint8_t *vram, uint32_t psm, uint32_t a)
{
	const uint32_t *v32 = reinterpret_cast<const uint32_t *>(vram);
	const uint16_t *v16 = reinterpret_cast<const uint16_t *>(vram);
	if (psm_is_16bit(psm)) return v16[a];
	if (psm == PSMT8) return vram[a];
	if (psm == PSMT8H) return vram[4u * a + 3u];
	if (psm == PSMT4) return (uint32_t(vram[a >> 1]) >> ((a & 1u) * 4u)) & 15u;
	if (psm == PSMT4HL) return (v32[a] >> 24) & 15u;
	if (psm == PSMT4HH) return v32[a] >> 28;
	return v32[a];
}

// One pixel of a transfer.  A single transfer's launch is its latency (eight 16x16
// uploads of one place, in turn: 20 us), so it takes the shortest code: four pixels
// per thread in all formats made them 25 to 29 us, and eight 256x256 local copies 45
// to 55 us instead of 35 to 41.
__device__ __forceinline__ void upload_pixel(const CopyParams &C, uint8_t *vram, uint32_t x, uint32_t y)
{
	if (x >= C.width || y >= C.height)
		return;
	uint32_t eff_stride = C.dbw;
	if (C.dpsm == PSMT4 || C.dpsm == PSMT8)
		eff_stride &= ~1u;
	if (x >= eff_stride * 64u)
	{
		Layout L = psm_layout(C.dpsm);
		uint32_t last = (C.dsay + C.height - 1u) >> L.ph, cur = (C.dsay + y) >> L.ph;
		if (last != cur)
			return;
	}
	uint32_t dx = (x + C.dsax) & 2047u, dy = (y + C.dsay) & 2047u;
	uint32_t data;
	if (C.xdir == HOST_TO_LOCAL)
	{
		uint64_t sa = uint64_t(y) * C.width + x;
		uint32_t b = psm_bits_per_pixel(C.dpsm);
		uint64_t factor = (b == 32 || b == 24) ? 2 : (b == 16 ? 4 : (b == 8 ? 8 : 16));
		uint64_t avail = b == 32 ? C.host_size / 4 : (b == 24 ? C.host_size / 3 : (b == 16 ? C.host_size / 2 : (b == 8 ? C.host_size : 2 * C.host_size)));
		if (sa * factor < C.host_offset_qwords || sa >= avail)
			return;
		// The payload starts 256-byte aligned: a warp's 32 consecutive pixels
		// read one contiguous span, with one load of the pixel's width each.
		const uint8_t *h = C.host;
		if (b == 24) data = uint32_t(h[3 * sa]) | (uint32_t(h[3 * sa + 1]) << 8) | (uint32_t(h[3 * sa + 2]) << 16);
		else if (b == 16) data = reinterpret_cast<const uint16_t *>(h)[sa];
		else if (b == 8) data = h[sa];
		else if (b == 4) data = (uint32_t(h[sa >> 1]) >> ((sa & 1) * 4)) & 15u;
		else data = reinterpret_cast<const uint32_t *>(h)[sa];
	}
	else
	{
		uint32_t sx = (x + C.ssax) & 2047u, sy = (y + C.ssay) & 2047u;
		data = read_pixel(C.src_vram, C.spsm, swizzle_address(sx, sy, C.sbp, C.sbw, C.spsm));
	}
	write_pixel(vram, C.dpsm, swizzle_address(dx, dy, C.dbp, C.dbw, C.dpsm), data, C.invalidate_ss != 0);
}

// Pixels of the 32 x 8 tile at (tx, ty), one per thread.
__host__ __device__ inline uint32_t pixel_tiles_x(const CopyParams &C) { return (C.width + 31u) / 32u; }
__host__ __device__ inline uint32_t pixel_tiles_y(const CopyParams &C) { return (C.height + 7u) / 8u; }

__device__ __forceinline__ void upload_tile(const CopyParams &C, uint8_t *vram, uint32_t tx, uint32_t ty)
{
	upload_pixel(C, vram, tx * 32u + (threadIdx.x & 31u), ty * 8u + (threadIdx.x >> 5));
}

__global__ void __launch_bounds__(256) upload_kernel(CopyParams C, uint8_t *vram)
{
	upload_tile(C, vram, blockIdx.x, blockIdx.y);
}

// Four pixels of the 32 x 32 tile at (tx, ty) of a PSMT8 upload per thread, from a
// multiple of 4 in the destination on: they share one address computation and, where
// they are aligned and all there, one payload load.  For the one format, the code is
// short.  Bound: issue of the address arithmetic and latency (four launches of sixteen
// 128x128 PSMT8 uploads 20.5 us with a pixel per thread, 16.1 so; light frame that
// uploads eight 256x256 textures 24.5 and 22.4).  With all formats the longer code
// made most batches slower (sixteen of PSMT4 22.6 -> 33, of PSMCT24 22.5 -> 28).
__host__ __device__ inline uint32_t quad_tiles_x(const CopyParams &C) { return ((C.dsax & 3u) + C.width + 31u) / 32u; }
__host__ __device__ inline uint32_t quad_tiles_y(const CopyParams &C) { return (C.height + 31u) / 32u; }

__device__ __forceinline__ void upload_quad_tile(const CopyParams &C, uint8_t *vram, uint32_t tx, uint32_t ty)
{
	// Pixel k of the quad is column x0 + k of the rectangle (x0 may be negative).
	const int32_t x0 = int32_t(tx * 32u + (threadIdx.x & 7u) * 4u) - int32_t(C.dsax & 3u);
	const uint32_t y = ty * 32u + (threadIdx.x >> 3);
	if (y >= C.height || x0 >= int32_t(C.width))
		return;
	uint32_t limit = C.width;
	// Columns past the buffer's stride are only written on the last page row.
	const Layout L = psm_layout(PSMT8);
	if ((C.dsay + C.height - 1u) >> L.ph != (C.dsay + y) >> L.ph)
		limit = min(limit, (C.dbw & ~1u) * 64u);
	uint32_t have = 0; // pixels to write
	const uint32_t row = y * C.width;
	#pragma unroll
	for (int k = 0; k < 4; k++)
	{
		const int32_t x = x0 + k;
		const uint64_t sa = uint64_t(row) + uint32_t(x);
		if (x >= 0 && uint32_t(x) < limit && sa * 8u >= C.host_offset_qwords && sa < C.host_size)
			have |= 1u << k;
	}
	if (!have)
		return;
	// The payload starts 256-byte aligned.
	const uint8_t *h = C.host;
	const uint32_t sa = row + uint32_t(x0); // of pixel 0, if it is there
	uint32_t data = 0;
	if (have == 15u && !(sa & 3u))
		data = *reinterpret_cast<const uint32_t *>(h + sa);
	else
	{
		#pragma unroll
		for (int k = 0; k < 4; k++)
			if ((have >> k) & 1u)
				data |= uint32_t(h[size_t(row) + uint32_t(x0 + k)]) << (8 * k);
	}
	const uint32_t a = swizzle_address(uint32_t(x0 + int32_t(C.dsax)) & 2047u, (y + C.dsay) & 2047u, C.dbp, C.dbw, PSMT8);
	#pragma unroll
	for (int k = 0; k < 4; k++)
		if ((have >> k) & 1u)
			write_pixel(vram, PSMT8, a + quad_offset(PSMT8, uint32_t(k)), data >> (8 * k), C.invalidate_ss != 0);
}

__host__ __device__ inline uint32_t upload_tiles(const CopyParams &C)
{
	return C.dpsm == PSMT8 ? quad_tiles_x(C) * quad_tiles_y(C) : pixel_tiles_x(C) * pixel_tiles_y(C);
}

// Consecutive host->local uploads whose destination blocks do not overlap, in
// one launch: the order among them cannot change VRAM.  Tiles are dealt out to the
// uploads by block_start.
constexpr uint32_t UPLOAD_BATCH_MAX = 16;
struct UploadBatch
{
	CopyParams c[UPLOAD_BATCH_MAX];
	uint32_t block_start[UPLOAD_BATCH_MAX + 1];
	uint32_t count;
};

__global__ void __launch_bounds__(256) upload_batch_kernel(UploadBatch B, uint8_t *vram)
{
	uint32_t i = 0;
	while (i + 1u < B.count && blockIdx.x >= B.block_start[i + 1])
		i++;
	const CopyParams &C = B.c[i];
	const uint32_t local = blockIdx.x - B.block_start[i];
	const uint32_t tiles_x = C.dpsm == PSMT8 ? quad_tiles_x(C) : pixel_tiles_x(C);
	if (C.dpsm == PSMT8)
		upload_quad_tile(C, vram, local % tiles_x, local / tiles_x);
	else
		upload_tile(C, vram, local % tiles_x, local / tiles_x);
}

// LOCAL->HOST read-out of a rectangle of plane 0 into linear bytes
// (vram_readback, gs/gs_util.hpp:50-110): pixels in row order at their host
// size (4, 3, 2 or 1 bytes).  Each thread packs 4 consecutive output bytes and
// writes them as one word where the output allows.  Bound: latency; 16 bytes a
// thread left a 64 KB rectangle on 16 CTAs (9.8 us, so 5.0).
struct ReadbackParams
{
	uint32_t sbp, sbw, spsm, ssax, ssay, width, height, bytes_per_pixel;
	uint64_t size; // output bytes
};

// Byte k of the pixel at word/halfword/byte address a.
__device__ __forceinline__ uint32_t readback_fetch(uint32_t spsm, const uint8_t *vram, uint32_t a, uint32_t k)
{
	switch (spsm)
	{
	case PSMCT16: case PSMCT16S: case PSMZ16: case PSMZ16S: return vram[2u * a + k];
	case PSMT8: return vram[a];
	case PSMT8H: return vram[4u * a + 3u];
	default: return vram[4u * a + k];
	}
}

__global__ void __launch_bounds__(256) readback_kernel(ReadbackParams R, const uint8_t *vram, uint8_t *out)
{
	const uint64_t first = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * 4u;
	if (first >= R.size)
		return;
	const uint32_t B = R.bytes_per_pixel;
	const uint64_t i = first / B;
	uint32_t k = uint32_t(first - i * B);
	uint32_t x = uint32_t(i % R.width), y = uint32_t(i / R.width);
	uint32_t a = swizzle_address((x + R.ssax) & 2047u, (y + R.ssay) & 2047u, R.sbp, R.sbw, R.spsm);
	auto next = [&]() {
		const uint32_t v = readback_fetch(R.spsm, vram, a, k);
		if (++k == B)
		{
			k = 0;
			if (++x == R.width)
			{
				x = 0;
				y++;
			}
			a = swizzle_address((x + R.ssax) & 2047u, (y + R.ssay) & 2047u, R.sbp, R.sbw, R.spsm);
		}
		return v;
	};
	if (first + 4u <= R.size)
	{
		uint32_t v = 0;
		#pragma unroll
		for (int b = 0; b < 4; b++)
			v |= next() << (8 * b);
		*reinterpret_cast<uint32_t *>(out + first) = v;
	}
	else
		for (uint64_t b = first; b < R.size; b++)
			out[b] = uint8_t(next());
}

// ---------------------------------------------------------------------------
// K6: CLUT load into a new ring instance.
struct ClutParams
{
	uint32_t psm, cbp, cpsm, csm, csa, cbw, cou, cov;
	float csm2_x_scale;
	uint32_t csm2_x_bias;
	uint32_t base_instance, instance;
};

// One CLUT load applied to the 512 entries in tmp (256 threads).
__device__ __forceinline__ void clut_apply(const ClutParams &C, const uint8_t *vram, uint16_t *tmp, uint32_t lane)
{
	bool index4 = C.psm == PSMT4 || C.psm == PSMT4HH || C.psm == PSMT4HL;
	bool active;
	uint32_t wc = lane + C.csa * 16u, rc = lane;
	if (index4)
		active = lane < 16u;
	else if (C.csm == 0)
	{
		uint32_t csa_count = C.cpsm == PSMCT32 ? 16u : 32u;
		active = lane < (csa_count - C.csa) * 16u;
		rc += C.csa * 16u;
	}
	else
		active = true;
	if (active)
	{
		uint32_t cx, cy;
		if (C.csm)
		{
			cx = uint32_t(fadd(fmul(float(rc), C.csm2_x_scale), 1.0f / 256.0f)) + C.csm2_x_bias + C.cou * 16u;
			cy = C.cov;
		}
		else
		{
			cx = (rc & 7u) | (((rc >> 4) & 1u) << 3);
			cy = ((rc >> 3) & 1u) | (((rc >> 5) & 7u) << 1);
		}
		if (C.cpsm == PSMCT32)
		{
			uint32_t v = reinterpret_cast<const uint32_t *>(vram)[swizzle_address(cx, cy, C.cbp, C.cbw, PSMCT32)];
			if (wc < 512u) tmp[wc] = uint16_t(v);
			if (wc + 256u < 512u) tmp[wc + 256u] = uint16_t(v >> 16);
		}
		else
		{
			uint32_t v = reinterpret_cast<const uint16_t *>(vram)[swizzle_address(cx, cy, C.cbp, C.cbw, C.cpsm)];
			if (wc < 512u) tmp[wc] = uint16_t(v);
		}
	}
}

__global__ void __launch_bounds__(256) clut_kernel(ClutParams C, const uint8_t *vram, uint16_t *clut)
{
	__shared__ uint16_t tmp[512];
	uint32_t lane = threadIdx.x;
	tmp[lane] = clut[size_t(C.base_instance) * 512u + lane];
	tmp[lane + 256u] = clut[size_t(C.base_instance) * 512u + lane + 256u];
	__syncthreads();
	clut_apply(C, vram, tmp, lane);
	__syncthreads();
	clut[size_t(C.instance) * 512u + lane] = tmp[lane];
	clut[size_t(C.instance) * 512u + lane + 256u] = tmp[lane + 256u];
}

// A chain of consecutive CLUT loads (each one's base is the previous one's
// instance) in one launch: block k starts from the first load's base and
// applies loads 0..k, so it writes the instance load k would have written.
// VRAM does not change between the loads, and no load of the chain writes
// the first load's base.
constexpr uint32_t CLUT_BATCH_MAX = 16;
struct ClutBatch
{
	ClutParams c[CLUT_BATCH_MAX];
	uint32_t count;
};

__global__ void __launch_bounds__(256) clut_batch_kernel(ClutBatch B, const uint8_t *vram, uint16_t *clut)
{
	__shared__ uint16_t tmp[512];
	const uint32_t lane = threadIdx.x, k = blockIdx.x;
	// An 8-bit CT32 load at CSA 0 rewrites all 512 entries: start from the
	// last one at or before k.
	uint32_t j0 = 0;
	for (uint32_t j = k + 1u; j-- > 0u;)
	{
		const ClutParams &c = B.c[j];
		if ((c.psm == PSMT8 || c.psm == PSMT8H) && c.csm == 0 && c.cpsm == PSMCT32 && c.csa == 0)
		{
			j0 = j;
			break;
		}
	}
	const uint32_t base = B.c[0].base_instance;
	tmp[lane] = clut[size_t(base) * 512u + lane];
	tmp[lane + 256u] = clut[size_t(base) * 512u + lane + 256u];
	__syncthreads();
	for (uint32_t j = j0; j <= k; j++)
	{
		clut_apply(B.c[j], vram, tmp, lane);
		__syncthreads();
	}
	clut[size_t(B.c[k].instance) * 512u + lane] = tmp[lane];
	clut[size_t(B.c[k].instance) * 512u + lane + 256u] = tmp[lane + 256u];
}
} // namespace pgs
