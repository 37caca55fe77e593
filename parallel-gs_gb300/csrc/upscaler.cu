// Learned anti-aliasing upscaler: 6 conv layers, 3x3, 32 channels, ReLU,
// residual over the input image.  BF16 activations and weights, FP32
// accumulation on the tensor cores; FP32 master weights trained with Adam.
//
// Layout: activations NHWC in BF16 with 16 (input, last-layer gradient) or 32
// channels.  A convolution is an implicit GEMM: M = pixels of a 16x16 tile,
// N = output channels, K = 9 taps x input channels.  Each CTA stages the
// 18x18 input halo and the layer's weights in shared memory; each warp owns
// two 16-pixel rows and all output channels.
//
//   layer 0: 4 (padded to 16) -> 32, ReLU
//   layers 1-4: 32 -> 32, ReLU
//   layer 5: 32 -> 4 (padded to 8), output = input + conv
//
// The 32 -> 32 layers run on tcgen05 (conv32_tc_kernel, further down) unless the
// tensor path is switched off.  The same kernels compute the data gradient
// (flipped, transposed weights; the epilogue multiplies by the ReLU mask of the
// layer below), and another the weight gradient (K = pixels).
#include "pgs.h"
#include "umma.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <utility>
#include <vector>

namespace pgs_up
{
constexpr int LAYERS = 6;
constexpr int TILE = 16;
constexpr int HALO = TILE + 2;
constexpr int REAL_IN[LAYERS] = { 4, 32, 32, 32, 32, 32 };
constexpr int REAL_OUT[LAYERS] = { 32, 32, 32, 32, 32, 4 };
constexpr int PAD_IN[LAYERS] = { 16, 32, 32, 32, 32, 32 };
constexpr int PAD_OUT[LAYERS] = { 32, 32, 32, 32, 32, 8 };
// Floats per layer of the padded weight and bias gradients.
constexpr size_t WGRAD_STRIDE = 9 * 32 * 32, BGRAD_STRIDE = 32;
// Device copies of the layer shapes.
__constant__ int d_real_in[LAYERS] = { 4, 32, 32, 32, 32, 32 };
__constant__ int d_real_out[LAYERS] = { 32, 32, 32, 32, 32, 4 };
__constant__ int d_pad_in[LAYERS] = { 16, 32, 32, 32, 32, 32 };
__constant__ int d_pad_out[LAYERS] = { 32, 32, 32, 32, 32, 8 };

#define UP_TRY(x)                                                                                                      \
	do                                                                                                                 \
	{                                                                                                                  \
		cudaError_t e_ = (x);                                                                                          \
		if (e_ != cudaSuccess)                                                                                         \
			return PGS_ERROR_CUDA;                                                                                     \
	} while (0)

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }

// 16 bytes from global to shared memory, or zeros.
__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool valid)
{
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3)
{
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
	             : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3)
{
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
	             : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}

__device__ __forceinline__ void ldsm_x2(uint32_t addr, uint32_t &r0, uint32_t &r1)
{
	asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(addr));
}

// D = A(16x16, row) * B(16x8, col) + D, BF16 in, FP32 accumulate.
__device__ __forceinline__ void mma_bf16(float *d, const uint32_t *a, uint32_t b0, uint32_t b1)
{
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
	             "{%0,%1,%2,%3};\n"
	             : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
{
	__nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
	return *reinterpret_cast<uint32_t *>(&v);
}

// A pixel of a caller's image, which may start at any byte.
__device__ __forceinline__ uint32_t load_pixel(const uint8_t *p)
{
	if (!(reinterpret_cast<uintptr_t>(p) & 3u))
		return *reinterpret_cast<const uint32_t *>(p);
	return uint32_t(p[0]) | (uint32_t(p[1]) << 8) | (uint32_t(p[2]) << 16) | (uint32_t(p[3]) << 24);
}

__device__ __forceinline__ void store_pixel(uint8_t *p, uint32_t c)
{
	if (!(reinterpret_cast<uintptr_t>(p) & 3u))
		*reinterpret_cast<uint32_t *>(p) = c;
	else
		for (int k = 0; k < 4; k++)
			p[k] = uint8_t(c >> (8 * k));
}

// The two BF16 values of v where those of m are positive, else 0.
__device__ __forceinline__ uint32_t mask_positive(uint32_t v, uint32_t m)
{
	const float lo = __uint_as_float(m << 16), hi = __uint_as_float(m & 0xffff0000u);
	return (lo > 0.0f ? v & 0xffffu : 0u) | (hi > 0.0f ? v & 0xffff0000u : 0u);
}

// One RGBA8 pixel as the network's first four input channels (x / 255 in
// BF16), two channels per word.
__device__ __forceinline__ void rgba8_to_bf16x4(uint32_t c, uint32_t &rg, uint32_t &ba)
{
	rg = pack_bf16x2(float(c & 0xffu) / 255.0f, float((c >> 8) & 0xffu) / 255.0f);
	ba = pack_bf16x2(float((c >> 16) & 0xffu) / 255.0f, float(c >> 24) / 255.0f);
}

// Programmatic dependent launch.  launch_dependents lets the next kernel of
// the stream start its CTAs (their set-up) once every CTA of this one has
// started; wait blocks until every kernel this one depends on has finished
// and its writes are visible.  Both do nothing when the launch did not ask
// for it.
__device__ __forceinline__ void griddep_launch_dependents()
{
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void griddep_wait()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Epilogue kinds of conv3x3_kernel.
enum : int
{
	EPI_RELU = 0,   // out = bf16(relu(acc + bias))
	EPI_LAST = 1,   // out_f32 = acc + bias + input image; optional RGBA8 copy
	EPI_MASK = 2,   // out = bf16(acc * (mask > 0))  (data gradient through ReLU)
};

struct ConvArgs
{
	const __nv_bfloat16 *in;     // N x H x W x CIN
	const uint8_t *in_rgba;      // CIN 16 only: N x H x W x 4 RGBA8 read in place of `in` (converted as by image_to_bf16_kernel)
	const __nv_bfloat16 *wt;     // 9 x COUT x CIN (tap, out channel, in channel)
	const float *bias;           // COUT (EPI_RELU / EPI_LAST)
	__nv_bfloat16 *out;          // N x H x W x COUT (EPI_RELU / EPI_MASK)
	const __nv_bfloat16 *mask;   // N x H x W x COUT (EPI_MASK)
	const uint8_t *image;        // N x H x W x 4 RGBA8 input image (EPI_LAST)
	float *out_f32;              // N x H x W x 4 (EPI_LAST)
	uint8_t *out_rgba;           // N x H x W x 4 (EPI_LAST, optional)
	int n, h, w;
};

// Grid: (ceil(W/16), ceil(H/16), N); 256 threads.
// Rows of 32 channels have their 16-byte chunks exchanged by bits of the row, rows
// of 16 are padded by 8 channels: either way eight rows read by ldmatrix lie in
// different banks.  Without padding eight CTAs of the last layer fit an SM, one
// wave of a 640x448 frame.
// Bound: latency (halo loads, barrier, fragment loads, one tile per CTA).  Network
// on one 640x448 frame: outputs staged for 16-byte stores and whole pixels 69.6 ->
// 69.1 us, halo by asynchronous copies and eight CTAs per SM -> 64.7.
template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(256, EPI == EPI_LAST ? 8 : 4) conv3x3_kernel(ConvArgs A)
{
	constexpr int PS = CIN == 32 ? 32 : CIN + 8; // row stride (elements)
	auto at = [](int row, int chunk) { return CIN == 32 ? row * PS + ((chunk ^ (row >> 1)) & 3) * 8 : row * PS + chunk * 8; };
	constexpr int NT = COUT / 8;       // n8 tiles
	constexpr int OS = COUT + 8;       // padded pixel stride of the staged output
	constexpr int IN = HALO * HALO * PS, OUT = EPI == EPI_LAST ? 0 : TILE * TILE * OS;
	// Input halo and weights; then, in their place, the tile's output.
	__shared__ __align__(16) __nv_bfloat16 s_buf[IN + 9 * COUT * PS > OUT ? IN + 9 * COUT * PS : OUT];
	__nv_bfloat16 *s_in = s_buf, *s_w = s_buf + IN;

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int x0 = blockIdx.x * TILE, y0 = blockIdx.y * TILE, img = blockIdx.z;
	griddep_launch_dependents();

	// Weights (not written by the kernels before this one), then the wait
	// for the previous layer, then its output.
	constexpr int CH = CIN / 8;
	for (int i = tid; i < 9 * COUT * CH; i += 256)
		*reinterpret_cast<uint4 *>(s_w + at(i / CH, i % CH)) = *reinterpret_cast<const uint4 *>(A.wt + size_t(i) * 8);
	griddep_wait();

	// Input halo, 16-byte chunks, zero outside the image.
	if (CIN == 16 && A.in_rgba)
	{
		// The RGBA8 image itself: channels 0-3 scaled by 1/255, 4-15 zero.
		for (int p = tid; p < HALO * HALO; p += 256)
		{
			int gx = x0 - 1 + p % HALO, gy = y0 - 1 + p / HALO;
			uint4 v = make_uint4(0, 0, 0, 0);
			if (gx >= 0 && gy >= 0 && gx < A.w && gy < A.h)
			{
				const uint32_t c = reinterpret_cast<const uint32_t *>(A.in_rgba)[(size_t(img) * A.h + gy) * A.w + gx];
				rgba8_to_bf16x4(c, v.x, v.y);
			}
			*reinterpret_cast<uint4 *>(s_in + p * PS) = v;
			*reinterpret_cast<uint4 *>(s_in + p * PS + 8) = make_uint4(0, 0, 0, 0);
		}
	}
	else
	for (int i = tid; i < HALO * HALO * CH; i += 256)
	{
		int p = i / CH, c = i % CH;
		int gx = x0 - 1 + p % HALO, gy = y0 - 1 + p / HALO;
		const bool in = gx >= 0 && gy >= 0 && gx < A.w && gy < A.h;
		const __nv_bfloat16 *src = A.in + ((size_t(img) * A.h + gy) * A.w + gx) * CIN + c * 8;
		if constexpr (CIN == 32)
			cp_async16(s_in + at(p, c), in ? src : A.in, in);
		else
			*reinterpret_cast<uint4 *>(s_in + at(p, c)) = in ? *reinterpret_cast<const uint4 *>(src) : make_uint4(0, 0, 0, 0);
	}
	if constexpr (CIN == 32)
		asm volatile("cp.async.wait_all;\n" ::: "memory");
	__syncthreads();

	float acc[2][NT][4];
	#pragma unroll
	for (int r = 0; r < 2; r++)
		#pragma unroll
		for (int j = 0; j < NT; j++)
			#pragma unroll
			for (int k = 0; k < 4; k++)
				acc[r][j][k] = 0.0f;

	#pragma unroll 1
	for (int tap = 0; tap < 9; tap++)
	{
		const int dy = tap / 3, dx = tap % 3;
		#pragma unroll
		for (int kc = 0; kc < CIN / 16; kc++)
		{
			uint32_t a[2][4];
			#pragma unroll
			for (int r = 0; r < 2; r++)
			{
				int py = warp * 2 + r + dy, px = (lane & 15) + dx;
				const __nv_bfloat16 *p = s_in + at(py * HALO + px, kc * 2 + (lane >> 4));
				ldsm_x4(smem_u32(p), a[r][0], a[r][1], a[r][2], a[r][3]);
			}
			#pragma unroll
			for (int j = 0; j < NT; j += 2)
			{
				if (j + 1 < NT)
				{
					// Two n-tiles: lanes 0-15 tile j (k 0-7, 8-15), 16-31 tile j+1.
					int nt = j + (lane >> 4), nrow = nt * 8 + (lane & 7), kh = (lane >> 3) & 1;
					const __nv_bfloat16 *p = s_w + at(tap * COUT + nrow, kc * 2 + kh);
					uint32_t b0, b1, b2, b3;
					ldsm_x4(smem_u32(p), b0, b1, b2, b3);
					#pragma unroll
					for (int r = 0; r < 2; r++)
					{
						mma_bf16(acc[r][j], a[r], b0, b1);
						mma_bf16(acc[r][j + 1], a[r], b2, b3);
					}
				}
				else
				{
					int nrow = j * 8 + (lane & 7), kh = (lane >> 3) & 1;
					const __nv_bfloat16 *p = s_w + at(tap * COUT + nrow, kc * 2 + kh);
					uint32_t b0, b1;
					ldsm_x2(smem_u32(p), b0, b1);
					#pragma unroll
					for (int r = 0; r < 2; r++)
						mma_bf16(acc[r][j], a[r], b0, b1);
				}
			}
		}
	}

	// Epilogue: thread holds rows g, g+8 and columns 2t, 2t+1 of each tile.
	const int g = lane >> 2, t = lane & 3;
	if constexpr (EPI == EPI_LAST)
	{
		// Residual over the input image in [0, 1]: the first lane of four has
		// channels 0 and 1, takes 2 and 3 from the next and stores the pixel.
		#pragma unroll
		for (int r = 0; r < 2; r++)
			#pragma unroll
			for (int half = 0; half < 2; half++)
			{
				float v[4] = { acc[r][0][half * 2], acc[r][0][half * 2 + 1] };
				v[2] = __shfl_down_sync(0xffffffffu, v[0], 1);
				v[3] = __shfl_down_sync(0xffffffffu, v[1], 1);
				const int gx = x0 + g + half * 8, gy = y0 + warp * 2 + r;
				if (t != 0 || gx >= A.w || gy >= A.h)
					continue;
				const size_t pix = (size_t(img) * A.h + gy) * A.w + gx;
				const uint32_t c = reinterpret_cast<const uint32_t *>(A.image)[pix];
				uint32_t packed = 0;
				#pragma unroll
				for (int k = 0; k < 4; k++)
				{
					v[k] = v[k] + A.bias[k] + float((c >> (8 * k)) & 0xffu) / 255.0f;
					packed |= uint32_t(rintf(fminf(fmaxf(v[k], 0.0f), 1.0f) * 255.0f)) << (8 * k);
				}
				if (A.out_f32)
					reinterpret_cast<float4 *>(A.out_f32)[pix] = make_float4(v[0], v[1], v[2], v[3]);
				if (A.out_rgba)
					store_pixel(A.out_rgba + pix * 4, packed);
			}
	}
	else
	{
		// Through shared memory, so that global memory sees 16 bytes a lane and
		// whole sectors (4 bytes a lane, 16 of each 32-byte sector, otherwise).
		__syncthreads();
		#pragma unroll
		for (int r = 0; r < 2; r++)
			#pragma unroll
			for (int half = 0; half < 2; half++)
				#pragma unroll
				for (int j = 0; j < NT; j++)
				{
					const int co = j * 8 + 2 * t;
					float v0 = acc[r][j][half * 2], v1 = acc[r][j][half * 2 + 1];
					if (EPI == EPI_RELU)
					{
						v0 = fmaxf(v0 + A.bias[co], 0.0f);
						v1 = fmaxf(v1 + A.bias[co + 1], 0.0f);
					}
					*reinterpret_cast<uint32_t *>(s_buf + ((warp * 2 + r) * TILE + g + half * 8) * OS + co) = pack_bf16x2(v0, v1);
				}
		__syncthreads();
		constexpr int CHUNKS = COUT / 8;
		#pragma unroll
		for (int i = tid; i < TILE * TILE * CHUNKS; i += 256)
		{
			const int p = i / CHUNKS, c = (i % CHUNKS) * 8;
			const int gx = x0 + p % TILE, gy = y0 + p / TILE;
			if (gx >= A.w || gy >= A.h)
				continue;
			const size_t at = ((size_t(img) * A.h + gy) * A.w + gx) * COUT + c;
			uint4 v = *reinterpret_cast<const uint4 *>(s_buf + p * OS + c);
			if (EPI == EPI_MASK)
			{
				const uint4 m = *reinterpret_cast<const uint4 *>(A.mask + at);
				v = make_uint4(mask_positive(v.x, m.x), mask_positive(v.y, m.y), mask_positive(v.z, m.z), mask_positive(v.w, m.w));
			}
			*reinterpret_cast<uint4 *>(A.out + at) = v;
		}
	}
}

// Weight gradient dW[tap][co][ci] += sum_p X[p + off(tap)][ci] * dY[p][co]
// (stored in the forward layout).  Each CTA walks 16x16 pixel tiles with a
// grid stride; one warp per tap keeps its tap's COUT x CIN sums in registers
// for the whole launch and adds them to global memory once.  A tile's halo of X
// and its dY are copied asynchronously into one of two buffers while the other
// is multiplied.  A tile's 16 k16 steps are summed by the tensor cores, the
// tiles' sums in FP32.
// Bound: latency, with the legacy MMA pipe at 42 % of its cycles: the warps wait on
// the fragments' shared-memory reads and on each tile's barriers, and the sums in
// registers (96 a thread) and the two buffers (93 KB) leave 18 warps per SM.  The version with a shared-memory sum that every warp
// added each tap of each tile to, and one thread per channel for the bias, took
// 138 us for a 32 -> 32 layer of 16 128x128 crops; this takes 23 us.  The bias
// goes to global memory once per CTA: once per warp and channel, on one cache
// line, took 64 us.  One CTA per SM: 27 us.
struct WgradArgs
{
	const __nv_bfloat16 *x;   // N x H x W x CIN (layer input)
	const __nv_bfloat16 *dy;  // N x H x W x COUT (gradient at the layer output, before bias)
	float *dw;                // 9 x COUT x CIN
	float *db;                // COUT
	int n, h, w;
};

constexpr int WGRAD_THREADS = 9 * 32;
constexpr int WGRAD_CTAS = 2; // per SM

// One buffer: the halo of X, then the tile of dY, rows padded by 16 bytes.
template <int CIN, int COUT>
__host__ __device__ constexpr size_t wgrad_buffer_bytes()
{
	return (HALO * HALO * (CIN + 8) + TILE * TILE * (COUT + 8)) * 2;
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(WGRAD_THREADS, 2) wgrad_kernel(WgradArgs A)
{
	constexpr int PS = CIN + 8;
	constexpr int PD = COUT + 8;
	constexpr int MT = COUT / 16;   // m16 tiles over output channels
	constexpr int NT = CIN / 8;     // n8 tiles over input channels
	constexpr int CHUNKS = COUT / 8;
	extern __shared__ __align__(16) uint8_t smem_raw[];

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int tiles_x = (A.w + TILE - 1) / TILE, tiles_y = (A.h + TILE - 1) / TILE;
	const int tiles = tiles_x * tiles_y * A.n;
	auto buffer_x = [&](int b) { return reinterpret_cast<__nv_bfloat16 *>(smem_raw + b * wgrad_buffer_bytes<CIN, COUT>()); };
	auto load = [&](int tile, int b) {
		const int img = tile / (tiles_x * tiles_y), rem = tile % (tiles_x * tiles_y);
		const int x0 = (rem % tiles_x) * TILE, y0 = (rem / tiles_x) * TILE;
		__nv_bfloat16 *s_x = buffer_x(b), *s_dy = s_x + HALO * HALO * PS;
		for (int i = tid; i < HALO * HALO * (CIN / 8); i += WGRAD_THREADS)
		{
			const int p = i / (CIN / 8), c = (i % (CIN / 8)) * 8;
			const int gx = x0 - 1 + p % HALO, gy = y0 - 1 + p / HALO;
			const bool in = gx >= 0 && gy >= 0 && gx < A.w && gy < A.h;
			cp_async16(s_x + p * PS + c, in ? A.x + ((size_t(img) * A.h + gy) * A.w + gx) * CIN + c : A.x, in);
		}
		for (int i = tid; i < TILE * TILE * CHUNKS; i += WGRAD_THREADS)
		{
			const int p = i / CHUNKS, c = (i % CHUNKS) * 8;
			const int gx = x0 + p % TILE, gy = y0 + p / TILE;
			const bool in = gx < A.w && gy < A.h;
			cp_async16(s_dy + p * PD + c, in ? A.dy + ((size_t(img) * A.h + gy) * A.w + gx) * COUT + c : A.dy, in);
		}
		asm volatile("cp.async.commit_group;\n" ::: "memory");
	};

	float sum[MT][NT][4] = {};
	// Bias gradient: column sums of dY (pixels outside the image are zero), 8
	// channels of every 256 / CHUNKS-th pixel per thread.
	float bias[8] = {};
	const int dy = warp / 3, dx = warp % 3;
	if (int(blockIdx.x) < tiles)
		load(blockIdx.x, 0);
	for (int tile = blockIdx.x, b = 0; tile < tiles; tile += gridDim.x, b ^= 1)
	{
		asm volatile("cp.async.wait_group 0;\n" ::: "memory");
		// This tile has arrived for all, and all are done with the other buffer.
		__syncthreads();
		if (tile + int(gridDim.x) < tiles)
			load(tile + gridDim.x, b ^ 1);
		const __nv_bfloat16 *s_x = buffer_x(b), *s_dy = s_x + HALO * HALO * PS;
		if (tid < 256)
		{
			const int c = tid % CHUNKS;
			#pragma unroll
			for (int p = tid / CHUNKS; p < TILE * TILE; p += 256 / CHUNKS)
			{
				const uint4 v = *reinterpret_cast<const uint4 *>(s_dy + p * PD + c * 8);
				const uint32_t q[4] = { v.x, v.y, v.z, v.w };
				#pragma unroll
				for (int k = 0; k < 4; k++)
				{
					bias[2 * k] += __uint_as_float(q[k] << 16);
					bias[2 * k + 1] += __uint_as_float(q[k] & 0xffff0000u);
				}
			}
		}
		float acc[MT][NT][4] = {};
		#pragma unroll 4
		for (int row = 0; row < TILE; row++)
		{
			// The 16 pixels of one tile row are one k16 step.
			// A (m = output channel, k = pixel): transposed 8x8 loads from
			// pixel-major memory.  Matrix q: pixels (q >> 1) * 8 + 0..7,
			// channels (q & 1) * 8 + 0..7.
			const int q = lane >> 3;
			uint32_t a[MT][4];
			#pragma unroll
			for (int m = 0; m < MT; m++)
				ldsm_x4_t(smem_u32(s_dy + (row * TILE + (q >> 1) * 8 + (lane & 7)) * PD + m * 16 + (q & 1) * 8), a[m][0], a[m][1],
				          a[m][2], a[m][3]);
			// B (k = pixel, n = input channel), two n8 tiles per load: matrix q
			// has pixels (q & 1) * 8 + 0..7 of channels (q >> 1) * 8 + 0..7.
			#pragma unroll
			for (int j = 0; j < NT; j += 2)
			{
				uint32_t b0, b1, b2, b3;
				ldsm_x4_t(smem_u32(s_x + ((row + dy) * HALO + dx + (q & 1) * 8 + (lane & 7)) * PS + (j + (q >> 1)) * 8), b0, b1, b2,
				          b3);
				#pragma unroll
				for (int m = 0; m < MT; m++)
				{
					mma_bf16(acc[m][j], a[m], b0, b1);
					mma_bf16(acc[m][j + 1], a[m], b2, b3);
				}
			}
		}
		#pragma unroll
		for (int m = 0; m < MT; m++)
			#pragma unroll
			for (int j = 0; j < NT; j++)
				#pragma unroll
				for (int k = 0; k < 4; k++)
					sum[m][j][k] += acc[m][j][k];
	}
	// sum[m][j]: rows (co) m*16 + g (+8), columns (ci) j*8 + 2t (+1).
	const int g = lane >> 2, t = lane & 3;
	#pragma unroll
	for (int m = 0; m < MT; m++)
		#pragma unroll
		for (int j = 0; j < NT; j++)
			#pragma unroll
			for (int half = 0; half < 2; half++)
			{
				float *dst = A.dw + (warp * COUT + m * 16 + g + half * 8) * CIN + j * 8 + 2 * t;
				asm volatile("red.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(dst), "f"(sum[m][j][2 * half]),
				             "f"(sum[m][j][2 * half + 1])
				             : "memory");
			}
	// Bias: lanes of a warp with the same chunk, then the warps, then one
	// addition per CTA and channel (all of them fall on one cache line).
	__shared__ float s_db[8][COUT];
	if (tid < 256)
	{
		#pragma unroll
		for (int k = 0; k < 8; k++)
		{
			#pragma unroll
			for (int o = CHUNKS; o < 32; o <<= 1)
				bias[k] += __shfl_xor_sync(0xffffffffu, bias[k], o);
			if (lane < CHUNKS)
				s_db[warp][lane * 8 + k] = bias[k];
		}
	}
	__syncthreads();
	if (tid < COUT)
	{
		float v = 0.0f;
		#pragma unroll
		for (int k = 0; k < 8; k++)
			v += s_db[k][tid];
		atomicAdd(&A.db[tid], v);
	}
}

// RGBA8 image -> BF16 16-channel input (channels 4..15 zero).
__global__ void __launch_bounds__(256) image_to_bf16_kernel(const uint8_t *img, __nv_bfloat16 *out, size_t pixels)
{
	size_t p = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
	if (p >= pixels)
		return;
	uint32_t c = reinterpret_cast<const uint32_t *>(img)[p];
	uint32_t w[8];
	rgba8_to_bf16x4(c, w[0], w[1]);
	for (int i = 2; i < 8; i++)
		w[i] = 0;
	uint4 *o = reinterpret_cast<uint4 *>(out + p * 16);
	o[0] = make_uint4(w[0], w[1], w[2], w[3]);
	o[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// MSE loss over the four channels against the target image, and its
// gradient 2 (out - target) / count as BF16 16-channel input of the last
// layer's backward pass.
// One addition to the sum per CTA: a CTA per 256 pixels with one per warp spent
// its time queueing 8192 additions at one address (16 crops of 128x128: 16.5 us
// against 9.5).
__global__ void __launch_bounds__(256) loss_kernel(const float *out, const uint8_t *target, size_t pixels, float scale,
                                                   __nv_bfloat16 *grad, double *loss_sum)
{
	__shared__ double s_part[8];
	double local = 0.0;
	for (size_t p = size_t(blockIdx.x) * 256 + threadIdx.x; p < pixels; p += size_t(gridDim.x) * 256)
	{
		const float4 v = reinterpret_cast<const float4 *>(out)[p];
		const uint32_t c = load_pixel(target + p * 4);
		const float d[4] = { v.x - float(c & 0xffu) / 255.0f, v.y - float((c >> 8) & 0xffu) / 255.0f,
		                     v.z - float((c >> 16) & 0xffu) / 255.0f, v.w - float(c >> 24) / 255.0f };
		#pragma unroll
		for (int k = 0; k < 4; k++)
			local += double(d[k]) * d[k];
		uint4 *o = reinterpret_cast<uint4 *>(grad + p * 16);
		o[0] = make_uint4(pack_bf16x2(scale * d[0], scale * d[1]), pack_bf16x2(scale * d[2], scale * d[3]), 0, 0);
		o[1] = make_uint4(0, 0, 0, 0);
	}
	for (int o = 16; o > 0; o >>= 1)
		local += __shfl_xor_sync(0xffffffffu, local, o);
	if ((threadIdx.x & 31) == 0)
		s_part[threadIdx.x >> 5] = local;
	__syncthreads();
	if (threadIdx.x == 0)
	{
		for (int k = 1; k < 8; k++)
			local += s_part[k];
		atomicAdd(loss_sum, local);
	}
}

// Parameter block of one layer inside the flat FP32 parameter vector:
// weights [tap][co][ci] (real sizes) then bias [co].
struct LayerOffsets
{
	int w[LAYERS], b[LAYERS];
	int total;
};

__constant__ LayerOffsets c_off;

// Adam step on the flat parameter vector, then the BF16 copies: the forward
// layout [tap][co_pad][ci_pad] and, for layers 1..5, the data-gradient layout
// [8 - tap][ci][co_pad_dgrad] (weights flipped and transposed).
__global__ void __launch_bounds__(256) adam_kernel(float *params, float *m, float *v, const float *grad, int count,
                                                   float lr, float b1, float b2, float eps, float c1, float c2)
{
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= count)
		return;
	float g = grad[i];
	float mi = b1 * m[i] + (1.0f - b1) * g;
	float vi = b2 * v[i] + (1.0f - b2) * g * g;
	m[i] = mi;
	v[i] = vi;
	params[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

struct BfLayout
{
	__nv_bfloat16 *fwd[LAYERS];
	__nv_bfloat16 *dgrad[LAYERS];
};

__global__ void __launch_bounds__(256) pack_weights_kernel(const float *params, BfLayout L)
{
	// One thread per forward-layout element of every layer.
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	for (int l = 0; l < LAYERS; l++)
	{
		int n = 9 * d_pad_out[l] * d_pad_in[l];
		if (i < n)
		{
			int tap = i / (d_pad_out[l] * d_pad_in[l]), co = (i / d_pad_in[l]) % d_pad_out[l], ci = i % d_pad_in[l];
			float w = (co < d_real_out[l] && ci < d_real_in[l])
			              ? params[c_off.w[l] + (tap * d_real_out[l] + co) * d_real_in[l] + ci] : 0.0f;
			L.fwd[l][i] = __float2bfloat16_rn(w);
		}
		if (l > 0)
		{
			// Data gradient of layer l: input channels = layer outputs padded to
			// 16 (layer 5) or 32, output channels = layer inputs (32).
			int din = l == LAYERS - 1 ? 16 : d_pad_out[l], dout = d_pad_in[l];
			int nd = 9 * dout * din;
			if (i < nd)
			{
				int tap = i / (dout * din), ci = (i / din) % dout, co = i % din;
				int src_tap = 8 - tap;
				float w = (co < d_real_out[l] && ci < d_real_in[l])
				              ? params[c_off.w[l] + (src_tap * d_real_out[l] + co) * d_real_in[l] + ci] : 0.0f;
				L.dgrad[l][i] = __float2bfloat16_rn(w);
			}
		}
	}
}

// The wgrad kernels write padded blocks of 32x32x9 weights and 32 biases per
// layer; this folds them into the flat gradient vector (grid y = layer).
__global__ void __launch_bounds__(256) gather_grad_kernel(const float *padded_w, const float *padded_b, float *grad)
{
	const int layer = blockIdx.y;
	padded_w += layer * WGRAD_STRIDE;
	padded_b += layer * BGRAD_STRIDE;
	// Gradients at the last layer's output are padded to 16 channels.
	const int cout_pad = layer == LAYERS - 1 ? 16 : 32, cin_pad = d_pad_in[layer];
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	int real_out = d_real_out[layer], real_in = d_real_in[layer];
	int nw = 9 * real_out * real_in;
	if (i < nw)
	{
		int tap = i / (real_out * real_in), co = (i / real_in) % real_out, ci = i % real_in;
		grad[c_off.w[layer] + i] = padded_w[(tap * cout_pad + co) * cin_pad + ci];
	}
	else if (i < nw + real_out)
		grad[c_off.b[layer] + (i - nw)] = padded_b[i - nw];
}


// ---------------------------------------------------------------------------
// Self-test of the tcgen05 building blocks: one CTA computes a 128x32 FP32
// tile D = A (128x32 BF16) x B (32x32 BF16)^T with two K=16 MMAs from shared
// memory in the given operand layout (0: no swizzle, 1: 64-byte swizzle) and
// writes D from tensor memory.  Inputs are small multiples of 1/8 so every
// product and sum is exact.
__device__ __forceinline__ float probe_a(uint32_t r, uint32_t k) { return float(int((r * 7u + k * 3u) % 17u) - 8) / 8.0f; }
__device__ __forceinline__ float probe_b(uint32_t n, uint32_t k) { return float(int((n * 5u + k * 11u) % 13u) - 6) / 4.0f; }

__global__ void __launch_bounds__(128) umma_probe_kernel(uint32_t mode, float *out, uint32_t *err)
{
	using namespace pgs_umma;
	extern __shared__ __align__(1024) uint8_t smem[];
	uint8_t *sa = smem;               // 128 rows x 64 B = 8 KiB
	uint8_t *sb = smem + 8192;        // 32 rows x 64 B = 2 KiB
	__shared__ uint64_t bar;
	__shared__ uint32_t tmem_slot;
	const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
	const uint32_t LBO = 128, SBO = 512;
	for (uint32_t i = tid; i < 128 * 32; i += 128)
	{
		uint32_t r = i / 32, k = i % 32;
		uint32_t off = mode == 1 ? swz64_offset(r, k) : canon_offset(r, k, LBO, SBO);
		*reinterpret_cast<__nv_bfloat16 *>(sa + off) = __float2bfloat16_rn(probe_a(r, k));
		// (mode 2 never reads these operands.)
	}
	for (uint32_t i = tid; i < 32 * 32; i += 128)
	{
		uint32_t n = i / 32, k = i % 32;
		uint32_t off = mode == 1 ? swz64_offset(n, k) : canon_offset(n, k, LBO, SBO);
		*reinterpret_cast<__nv_bfloat16 *>(sb + off) = __float2bfloat16_rn(probe_b(n, k));
	}
	if (warp == 0)
		tmem_alloc(&tmem_slot, 32);
	if (tid == 0)
	{
		mbar_init(&bar, 1);
		fence_barrier_init();
	}
	fence_proxy_async();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = tmem_slot;
	// Mode 2: nothing is issued, so nothing arrives on the barrier; the
	// bounded wait gives up, the error flag is set and TMEM is released.
	if (tid == 0 && mode != 2)
	{
		const uint32_t idesc = idesc_bf16_f32(128, 32);
		for (uint32_t ks = 0; ks < 2; ks++)
		{
			uint64_t ad, bd;
			if (mode == 1)
			{
				ad = smem_desc(smem_addr(sa) + ks * 32u, 16, SBO, LAYOUT_SWIZZLE_64B);
				bd = smem_desc(smem_addr(sb) + ks * 32u, 16, SBO, LAYOUT_SWIZZLE_64B);
			}
			else
			{
				ad = smem_desc(smem_addr(sa) + ks * 2u * LBO, LBO, SBO, LAYOUT_NONE);
				bd = smem_desc(smem_addr(sb) + ks * 2u * LBO, LBO, SBO, LAYOUT_NONE);
			}
			pgs_umma::mma_bf16(tmem, ad, bd, idesc, ks > 0);
		}
		mma_commit(&bar);
	}
	__syncwarp();
	bool ok = mode == 2 ? mbar_wait_limit(&bar, 0, 4096) : mbar_wait(&bar, 0);
	tc_fence_after();
	if (!ok)
	{
		if (lane == 0)
			atomicOr(err, 1u);
	}
	else
	{
		uint32_t v[32];
		tmem_ld32(tmem + ((warp * 32u) << 16), v);
		for (int c = 0; c < 32; c++)
			out[(warp * 32 + lane) * 32 + c] = __uint_as_float(v[c]);
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	if (warp == 0)
		tmem_dealloc(tmem, 32);
}

// ---------------------------------------------------------------------------
// 32 -> 32 convolution on the 5th-generation tensor cores (inference and the
// forward half of training).  Persistent CTAs own tiles of 16 rows x 8 columns
// = 128 output pixels.  Warp-specialised pipeline:
//  - warp 5, one lane: TMA loads of each tile's 18 x 10 x 32 input window (zero
//    fill outside the image, 64-byte swizzle), three or five stages.  It is not the lane
//    that issues the MMAs: refilling a stage waits for the MMAs that read it, and
//    one lane for both let the tensor cores run dry at every tile;
//  - warp 0, one lane: 9 taps x 2 K-steps of tcgen05.mma (M 128, N 32, K 16)
//    into one of four 32-column FP32 accumulators in tensor memory, committed to
//    the stage's "empty" and the accumulator's "full" barriers.  A
//    row group of A is the 8 pixels of one window row from the tap's column on:
//    groups lie one window row (640 bytes) apart, and since the swizzle is a
//    function of the shared-memory address, a group may start at any pixel;
//  - warps 1-4 (one per TMEM lane quarter) read the accumulator, release it,
//    add the bias, apply ReLU and hand their 8 x 4 pixels to a TMA store
//    (clipped at the image border), overlapping the MMAs of the next tile.
// The layer's weights sit in shared memory (9 x 32 x 32 BF16, 64-byte
// swizzled) for the whole launch.  Every wait is bounded and gives up when
// another warp has given up.
// Bound: shared-memory reads of A, 4 KiB per MMA of 16 tensor cycles (a layer of
// a 640x448 frame: 5.6 us), and the launch's start and end.  Measured on the
// network of one such frame, 83 us at first: one window per tile instead of three
// shifted by a column each (11.5 instead of 30 KB), boxes stored by TMA instead
// of 16 bytes a lane, and unrolled descriptors, together 81.6; loads from a warp
// of their own, 69.6.
namespace tc
{
constexpr int ROWS = 16, COLS = 8;
constexpr int WIN_ROWS = ROWS + 2, WIN_COLS = COLS + 2;
constexpr int ACCS = 4;
// Stages of input.  With five, two CTAs fill an SM's shared memory; with three, the
// next layer's CTAs (inference, programmatic dependent launch) get in beside them and
// are set up by the time this layer ends, which is what counts while a frame has few
// tiles.  Network on a frame of 192x256 (384 tiles) 42.2 us with five, 33.0 with
// three, 224x320 (560) 44.7 and 35.2, 256x384 (768) 48.4 and 46.4, 320x384 (960) 52.0
// and 51.1; then the five gain: 384x512 (1536) 63.2 and 66.6, 1080x1920 395 and 440.
constexpr int STAGES_MANY = 5, STAGES_FEW = 3, FEW_TILES = 6; // per SM
constexpr uint32_t ROW_BYTES = WIN_COLS * 64;               // 640
constexpr uint32_t WIN_BYTES = WIN_ROWS * ROW_BYTES;        // 11520
constexpr uint32_t STAGE_BYTES = 12288;                     // a window from a 1 KiB boundary
constexpr uint32_t W_BYTES = 9 * 32 * 64;                   // 18432
constexpr uint32_t OUT_BYTES = 32 * 64;                     // one warp's 8 x 4 pixels
constexpr int OUT_BUFS = 2;
constexpr uint32_t smem_bytes(int stages) { return 1024 + stages * STAGE_BYTES + W_BYTES + 4 * OUT_BUFS * OUT_BYTES; }
constexpr int THREADS = 192;
}

// EPI_RELU writes relu(acc + bias); EPI_MASK (the data gradient of a 32 -> 32
// layer through the ReLU before it) writes acc where mask > 0, else 0.
template <int EPI, int STAGES>
__global__ void __launch_bounds__(tc::THREADS, 2) conv32_tc_kernel(const __grid_constant__ CUtensorMap tmap,
                                                                    const __grid_constant__ CUtensorMap out_map,
                                                                    const __nv_bfloat16 *wt, const float *bias,
                                                                    const __nv_bfloat16 *mask, int n, int h, int w,
                                                                    uint32_t *err)
{
	using namespace pgs_umma;
	extern __shared__ uint8_t smem_dyn[];
	uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
	uint8_t *sw = base + STAGES * tc::STAGE_BYTES, *sout = sw + tc::W_BYTES;
	__shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[tc::ACCS], acc_empty[tc::ACCS];
	__shared__ uint32_t tmem_slot;
	__shared__ __align__(16) float s_bias[32];
	__shared__ volatile uint32_t s_abort;

	const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
	const int tiles_x = (w + tc::COLS - 1) / tc::COLS, tiles_y = (h + tc::ROWS - 1) / tc::ROWS;
	const int tiles = tiles_x * tiles_y * n;
	griddep_launch_dependents();

	// Weights: 16-byte chunks of 8 input channels into their swizzled slots.
	for (uint32_t i = tid; i < 9 * 32 * 4; i += tc::THREADS)
	{
		uint32_t tap = i / 128, co = (i / 4) % 32, ci = (i % 4) * 8;
		*reinterpret_cast<uint4 *>(sw + tap * 2048u + swz64_offset(co, ci)) =
		    *reinterpret_cast<const uint4 *>(wt + (tap * 32u + co) * 32u + ci);
	}
	if (tid < 32)
		s_bias[tid] = EPI == EPI_MASK ? 0.0f : bias[tid];
	if (warp == 0)
		tmem_alloc(&tmem_slot, tc::ACCS * 32);
	if (tid == 0)
	{
		for (int s = 0; s < STAGES; s++)
		{
			mbar_init(&full_bar[s], 1);
			mbar_init(&empty_bar[s], 1);
		}
		for (int a = 0; a < tc::ACCS; a++)
		{
			mbar_init(&acc_full[a], 1);
			mbar_init(&acc_empty[a], 4);
		}
		fence_barrier_init();
		s_abort = 0;
	}
	fence_proxy_async();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = tmem_slot;
	// Weights, barriers and tensor memory are set up; the input is the
	// previous layer's output.
	griddep_wait();

	auto tile_coords = [&](int tile, int &img, int &x0, int &y0) {
		img = tile / (tiles_x * tiles_y);
		int rem = tile % (tiles_x * tiles_y);
		x0 = (rem % tiles_x) * tc::COLS;
		y0 = (rem / tiles_x) * tc::ROWS;
	};
	const int first = blockIdx.x, step = gridDim.x;
	const int mine = first < tiles ? (tiles - 1 - first) / step + 1 : 0;

	if (warp == 0)
	{
		if (lane == 0)
		{
			const uint32_t idesc = idesc_bf16_f32(128, 32);
			const uint64_t bd = smem_desc(smem_addr(sw), 16, 512, LAYOUT_SWIZZLE_64B);
			for (int i = 0; i < mine && !s_abort; i++)
			{
				const int s = i % STAGES, a = i % tc::ACCS;
				if (!mbar_wait_or_abort(&full_bar[s], (i / STAGES) & 1, &s_abort) ||
				    (i >= tc::ACCS && !mbar_wait_or_abort(&acc_empty[a], ((i / tc::ACCS) - 1) & 1, &s_abort)))
				{
					atomicOr(err, 2u);
					s_abort = 1;
					break;
				}
				tc_fence_after();
				// Unrolled, with descriptors that differ from the first by constants
				// (addresses in 16-byte units in the low bits): this one thread's
				// instructions are what the tensor cores wait for otherwise.
				const uint64_t ad = smem_desc(smem_addr(base + s * tc::STAGE_BYTES), 16, tc::ROW_BYTES, LAYOUT_SWIZZLE_64B);
				const uint32_t d = tmem + uint32_t(a) * 32u;
				#pragma unroll
				for (int tap = 0; tap < 9; tap++)
				{
					const int dy = tap / 3, dx = tap % 3;
					#pragma unroll
					for (int ks = 0; ks < 2; ks++)
						pgs_umma::mma_bf16(d, ad + ((dy * tc::ROW_BYTES + dx * 64u + ks * 32u) >> 4), bd + ((tap * 2048u + ks * 32u) >> 4),
						                   idesc, tap + ks > 0);
				}
				mma_commit(&empty_bar[s]);
				mma_commit(&acc_full[a]);
			}
		}
		__syncwarp();
	}
	else if (warp == 5)
	{
		if (lane == 0)
		{
			int i = 0;
			for (; i < mine && !s_abort; i++)
			{
				const int s = i % STAGES;
				if (i >= STAGES && !mbar_wait_or_abort(&empty_bar[s], ((i / STAGES) - 1) & 1, &s_abort))
				{
					atomicOr(err, 1u);
					s_abort = 1;
					break;
				}
				int img, x0, y0;
				tile_coords(first + i * step, img, x0, y0);
				mbar_expect_tx(&full_bar[s], tc::WIN_BYTES);
				tma_load_4d(base + s * tc::STAGE_BYTES, &tmap, &full_bar[s], 0, x0 - 1, y0 - 1, img);
			}
			// Given up: the copies in flight still have to land.
			if (s_abort)
				for (int k = (i > STAGES ? i - STAGES : 0); k < i; k++)
					mbar_wait_limit(&full_bar[k % STAGES], (k / STAGES) & 1, 1u << 20);
		}
		__syncwarp();
	}
	else
	{
		// Epilogue warps: warp w reads TMEM lanes 32 * (w % 4) .. + 31.
		const uint32_t quarter = warp & 3u;
		for (int i = 0; i < mine; i++)
		{
			const int a = i % tc::ACCS;
			bool ok = mbar_wait_or_abort(&acc_full[a], (i / tc::ACCS) & 1, &s_abort);
			if (!__all_sync(0xffffffffu, ok))
			{
				if (lane == 0)
					atomicOr(err, 4u);
				s_abort = 1;
				break;
			}
			tc_fence_after();
			uint32_t v[32];
			tmem_ld32(tmem + uint32_t(a) * 32u + ((quarter * 32u) << 16), v);
			tc_fence_before();
			__syncwarp();
			if (lane == 0)
				mbar_arrive(&acc_empty[a]);
			int img, x0, y0;
			tile_coords(first + i * step, img, x0, y0);
			uint32_t m[16] = {};
			if (EPI == EPI_MASK)
			{
				const int gy = y0 + int(quarter * 4u + lane / 8u), gx = x0 + int(lane % 8u);
				if (gx < w && gy < h)
				{
					const uint4 *src = reinterpret_cast<const uint4 *>(mask + ((size_t(img) * h + gy) * w + gx) * 32);
					#pragma unroll
					for (int q = 0; q < 4; q++)
					{
						const uint4 t = src[q];
						m[4 * q] = t.x;
						m[4 * q + 1] = t.y;
						m[4 * q + 2] = t.z;
						m[4 * q + 3] = t.w;
					}
				}
			}
			uint32_t packed[16];
			#pragma unroll
			for (int c = 0; c < 16; c++)
			{
				float lo, hi;
				if (EPI == EPI_MASK)
				{
					// Data gradient through the ReLU: keep where the layer's output was positive.
					__nv_bfloat162 mk = *reinterpret_cast<const __nv_bfloat162 *>(&m[c]);
					lo = __bfloat162float(mk.x) > 0.0f ? __uint_as_float(v[2 * c]) : 0.0f;
					hi = __bfloat162float(mk.y) > 0.0f ? __uint_as_float(v[2 * c + 1]) : 0.0f;
				}
				else
				{
					lo = fmaxf(__uint_as_float(v[2 * c]) + s_bias[2 * c], 0.0f);
					hi = fmaxf(__uint_as_float(v[2 * c + 1]) + s_bias[2 * c + 1], 0.0f);
				}
				packed[c] = pack_bf16x2(lo, hi);
			}
			// The warp's other buffer may still be read by its last store, this
			// one by none (waited for by the lane that issues them).
			uint8_t *buf = sout + ((quarter * tc::OUT_BUFS + uint32_t(i) % tc::OUT_BUFS) * tc::OUT_BYTES);
			if (lane == 0)
				bulk_wait_read<tc::OUT_BUFS - 1>();
			__syncwarp();
			#pragma unroll
			for (int q = 0; q < 4; q++)
				*reinterpret_cast<uint4 *>(buf + swz64_offset(lane, uint32_t(q) * 8u)) =
				    make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
			fence_proxy_async();
			__syncwarp();
			if (lane == 0)
			{
				// A box that starts below the image is not stored.
				if (y0 + int(quarter * 4u) < h)
					tma_store_4d(&out_map, buf, 0, x0, y0 + int(quarter * 4u), img);
				bulk_commit();
			}
		}
		if (lane == 0)
			bulk_wait_all();
		__syncwarp();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	if (warp == 0)
		tmem_dealloc(tmem, tc::ACCS * 32);
}

// Tensor map of an N x H x W x 32 BF16 activation tensor for conv32_tc_kernel:
// boxes of 32 channels x cols x rows, 64-byte swizzle, zero fill.
static int make_act_tmap(CUtensorMap *m, const void *ptr, int n, int h, int w, int cols, int rows)
{
	using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
	                            const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
	                            CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
	static Encode encode = nullptr;
	if (!encode)
	{
		void *fn = nullptr;
		cudaDriverEntryPointQueryResult q;
		if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
		    q != cudaDriverEntryPointSuccess || !fn)
			return PGS_ERROR_UNSUPPORTED;
		encode = reinterpret_cast<Encode>(fn);
	}
	cuuint64_t dims[4] = { 32, cuuint64_t(w), cuuint64_t(h), cuuint64_t(n) };
	cuuint64_t strides[3] = { 64, cuuint64_t(w) * 64, cuuint64_t(h) * w * 64 };
	cuuint32_t box[4] = { 32, uint32_t(cols), uint32_t(rows), 1 };
	cuuint32_t estr[4] = { 1, 1, 1, 1 };
	CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(ptr), dims, strides, box, estr,
	                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
	                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	return r == CUDA_SUCCESS ? PGS_OK : PGS_ERROR_INVALID_ARGUMENT;
}

// ---------------------------------------------------------------------------
struct Upscaler
{
	int device = 0;
	cudaStream_t stream = nullptr;      // where the upscaler's work is queued
	cudaStream_t own_stream = nullptr;  // created with the upscaler
	LayerOffsets off = {};
	float *d_params = nullptr, *d_m = nullptr, *d_v = nullptr, *d_grad = nullptr;
	float *d_wgrad = nullptr, *d_bgrad = nullptr;   // padded scratch, per layer
	BfLayout bf = {};
	int adam_t = 0;
	// Activations for the current batch size.
	size_t cap_pixels = 0;
	__nv_bfloat16 *d_x0 = nullptr;              // input, 16 channels
	__nv_bfloat16 *d_act[LAYERS - 1] = {};      // outputs of layers 0..4, 32 channels
	__nv_bfloat16 *d_ga = nullptr, *d_gb = nullptr;   // gradient ping-pong, 32 channels
	__nv_bfloat16 *d_gout = nullptr;            // last-layer output gradient, 16 channels
	float *d_out = nullptr;                     // N x H x W x 4
	double *d_loss = nullptr;
	uint32_t *d_err = nullptr;
	int sm_count = 0;
	// 32 -> 32 layers: 0 = mma.sync, otherwise tcgen05 with this many
	// persistent CTAs per SM.
	int use_tc = 2;
	// Tensor maps of the activation buffers (encoded once per buffer and shape).
	struct TmapEntry
	{
		const void *ptr;
		int n, h, w;
		bool store;
		CUtensorMap map;
	};
	static constexpr int MAX_TMAPS = 24;
	TmapEntry tmaps[MAX_TMAPS] = {};
	int tmap_count = 0;

	// Map of the input windows, or of a warp's output boxes.
	int act_tmap(const void *ptr, int n, int h, int w, bool store, CUtensorMap &out)
	{
		for (int i = 0; i < tmap_count; i++)
			if (tmaps[i].ptr == ptr && tmaps[i].n == n && tmaps[i].h == h && tmaps[i].w == w && tmaps[i].store == store)
			{
				out = tmaps[i].map;
				return PGS_OK;
			}
		TmapEntry &e = tmaps[tmap_count < MAX_TMAPS ? tmap_count++ : MAX_TMAPS - 1];
		int r = store ? make_act_tmap(&e.map, ptr, n, h, w, tc::COLS, 4) : make_act_tmap(&e.map, ptr, n, h, w, tc::WIN_COLS, tc::WIN_ROWS);
		if (r)
		{
			e.ptr = nullptr;
			return r;
		}
		e.store = store;
		e.ptr = ptr;
		e.n = n;
		e.h = h;
		e.w = w;
		out = e.map;
		return PGS_OK;
	}

	int init(int dev)
	{
		device = dev;
		UP_TRY(cudaSetDevice(device));
		UP_TRY(cudaStreamCreateWithFlags(&own_stream, cudaStreamNonBlocking));
		stream = own_stream;
		UP_TRY(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
		int o = 0;
		for (int l = 0; l < LAYERS; l++)
		{
			off.w[l] = o;
			o += 9 * REAL_OUT[l] * REAL_IN[l];
			off.b[l] = o;
			o += REAL_OUT[l];
		}
		off.total = o;
		UP_TRY(cudaMemcpyToSymbol(c_off, &off, sizeof(off)));
		size_t n = size_t(off.total);
		UP_TRY(cudaMalloc(&d_params, n * 4));
		UP_TRY(cudaMalloc(&d_m, n * 4));
		UP_TRY(cudaMalloc(&d_v, n * 4));
		UP_TRY(cudaMalloc(&d_grad, n * 4));
		UP_TRY(cudaMemset(d_params, 0, n * 4));
		UP_TRY(cudaMemset(d_m, 0, n * 4));
		UP_TRY(cudaMemset(d_v, 0, n * 4));
		UP_TRY(cudaMalloc(&d_wgrad, LAYERS * WGRAD_STRIDE * 4));
		UP_TRY(cudaMalloc(&d_bgrad, LAYERS * BGRAD_STRIDE * 4));
		for (int l = 0; l < LAYERS; l++)
		{
			UP_TRY(cudaMalloc(&bf.fwd[l], size_t(9) * PAD_OUT[l] * PAD_IN[l] * 2));
			UP_TRY(cudaMalloc(&bf.dgrad[l], size_t(9) * 32 * 32 * 2));
		}
		UP_TRY(cudaMalloc(&d_loss, sizeof(double)));
		UP_TRY(cudaMalloc(&d_err, sizeof(uint32_t)));
		UP_TRY(cudaMemset(d_err, 0, sizeof(uint32_t)));
		const int few = int(tc::smem_bytes(tc::STAGES_FEW)), many = int(tc::smem_bytes(tc::STAGES_MANY));
		const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
		UP_TRY(cudaFuncSetAttribute(conv32_tc_kernel<EPI_RELU, tc::STAGES_FEW>, attr, few));
		UP_TRY(cudaFuncSetAttribute(conv32_tc_kernel<EPI_RELU, tc::STAGES_MANY>, attr, many));
		UP_TRY(cudaFuncSetAttribute(conv32_tc_kernel<EPI_MASK, tc::STAGES_MANY>, attr, many));
		return PGS_OK;
	}

	void destroy()
	{
		cudaSetDevice(device);
		if (stream)
			cudaStreamSynchronize(stream);
		cudaFree(d_params);
		cudaFree(d_m);
		cudaFree(d_v);
		cudaFree(d_grad);
		cudaFree(d_wgrad);
		cudaFree(d_bgrad);
		for (int l = 0; l < LAYERS; l++)
		{
			cudaFree(bf.fwd[l]);
			cudaFree(bf.dgrad[l]);
		}
		free_acts();
		cudaFree(d_loss);
		cudaFree(d_err);
		if (own_stream)
			cudaStreamDestroy(own_stream);
	}

	// Later work goes to `s` (the upscaler's own stream when null), after
	// what is queued on the current one.
	int set_stream(cudaStream_t s)
	{
		UP_TRY(cudaSetDevice(device));
		UP_TRY(cudaStreamSynchronize(stream));
		stream = s ? s : own_stream;
		return PGS_OK;
	}

	void free_acts()
	{
		cudaFree(d_x0);
		for (auto &a : d_act)
			cudaFree(a);
		cudaFree(d_ga);
		cudaFree(d_gb);
		cudaFree(d_gout);
		cudaFree(d_out);
		d_x0 = d_ga = d_gb = d_gout = nullptr;
		for (auto &a : d_act)
			a = nullptr;
		d_out = nullptr;
		cap_pixels = 0;
	}

	int ensure(size_t pixels)
	{
		if (pixels <= cap_pixels)
			return PGS_OK;
		UP_TRY(cudaStreamSynchronize(stream));
		free_acts();
		tmap_count = 0;
		UP_TRY(cudaMalloc(&d_x0, pixels * 16 * 2));
		for (auto &a : d_act)
			UP_TRY(cudaMalloc(&a, pixels * 32 * 2));
		UP_TRY(cudaMalloc(&d_ga, pixels * 32 * 2));
		UP_TRY(cudaMalloc(&d_gb, pixels * 32 * 2));
		UP_TRY(cudaMalloc(&d_gout, pixels * 16 * 2));
		UP_TRY(cudaMalloc(&d_out, pixels * 4 * 4));
		cap_pixels = pixels;
		return PGS_OK;
	}

	int pack()
	{
		int n = 9 * 32 * 32;
		pack_weights_kernel<<<(n + 255) / 256, 256, 0, stream>>>(d_params, bf);
		UP_TRY(cudaGetLastError());
		return PGS_OK;
	}

	int set_params(const float *host, size_t count)
	{
		if (count != size_t(off.total))
			return PGS_ERROR_INVALID_ARGUMENT;
		UP_TRY(cudaMemcpyAsync(d_params, host, count * 4, cudaMemcpyHostToDevice, stream));
		UP_TRY(cudaMemsetAsync(d_m, 0, count * 4, stream));
		UP_TRY(cudaMemsetAsync(d_v, 0, count * 4, stream));
		adam_t = 0;
		int r = pack();
		if (r)
			return r;
		UP_TRY(cudaStreamSynchronize(stream));
		return PGS_OK;
	}

	int get(const float *src, float *host, size_t count)
	{
		if (count != size_t(off.total))
			return PGS_ERROR_INVALID_ARGUMENT;
		UP_TRY(cudaMemcpyAsync(host, src, count * 4, cudaMemcpyDeviceToHost, stream));
		UP_TRY(cudaStreamSynchronize(stream));
		return PGS_OK;
	}

	// 3x3 convolution of a 32-channel tensor into 32 accumulator channels on
	// tcgen05 (conv32_tc_kernel) with the given epilogue.
	template <int EPI>
	int conv_tc(const ConvArgs &a, bool pdl = false)
	{
		CUtensorMap in, out;
		int r = act_tmap(a.in, a.n, a.h, a.w, false, in);
		if (!r)
			r = act_tmap(a.out, a.n, a.h, a.w, true, out);
		if (r)
			return r;
		int tiles = ((a.w + tc::COLS - 1) / tc::COLS) * ((a.h + tc::ROWS - 1) / tc::ROWS) * a.n;
		int grid = std::min(tiles, sm_count * use_tc);
		if constexpr (EPI == EPI_RELU)
			if (pdl && tiles <= tc::FEW_TILES * sm_count)
				return launch(conv32_tc_kernel<EPI, tc::STAGES_FEW>, dim3(grid), dim3(tc::THREADS),
				              tc::smem_bytes(tc::STAGES_FEW), pdl, in, out, a.wt, a.bias, a.mask, a.n, a.h, a.w, d_err);
		return launch(conv32_tc_kernel<EPI, tc::STAGES_MANY>, dim3(grid), dim3(tc::THREADS), tc::smem_bytes(tc::STAGES_MANY),
		              pdl, in, out, a.wt, a.bias, a.mask, a.n, a.h, a.w, d_err);
	}

	template <int CIN, int COUT, int EPI>
	int conv(const ConvArgs &a, bool pdl = false)
	{
		dim3 grid((a.w + TILE - 1) / TILE, (a.h + TILE - 1) / TILE, a.n);
		return launch(conv3x3_kernel<CIN, COUT, EPI>, grid, dim3(256), 0, pdl, a);
	}

	// Launch on the upscaler's stream; pdl: the kernel may start while the
	// one before it in the stream runs (it waits for it in griddep_wait).
	template <typename... KArgs, typename... Args>
	int launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, bool pdl, Args &&...args)
	{
		cudaLaunchConfig_t cfg = {};
		cfg.gridDim = grid;
		cfg.blockDim = block;
		cfg.dynamicSmemBytes = smem;
		cfg.stream = stream;
		cudaLaunchAttribute attr[1];
		attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
		attr[0].val.programmaticStreamSerializationAllowed = 1;
		cfg.attrs = attr;
		cfg.numAttrs = pdl ? 1 : 0;
		UP_TRY(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
		return PGS_OK;
	}

	// Forward pass of `n` images of h x w RGBA8 (device memory).  out_rgba
	// (device, optional) gets the result clamped and rounded to RGBA8.
	// keep_input (training): the 16-channel BF16 input is kept in d_x0, for the
	// first layer's weight gradient; otherwise the first layer reads the RGBA8
	// image directly.  The FP32 result goes to d_out with keep_input or without
	// out_rgba; else d_out keeps what it held.
	int forward(const uint8_t *d_img, int n, int h, int w, uint8_t *out_rgba, bool keep_input)
	{
		size_t pixels = size_t(n) * h * w;
		int r = ensure(pixels);
		if (r)
			return r;
		if (keep_input)
		{
			image_to_bf16_kernel<<<unsigned((pixels + 255) / 256), 256, 0, stream>>>(d_img, d_x0, pixels);
			UP_TRY(cudaGetLastError());
		}
		ConvArgs k = {};
		k.n = n;
		k.h = h;
		k.w = w;
		for (int l = 0; l < LAYERS; l++)
		{
			k.in = l == 0 ? d_x0 : d_act[l - 1];
			k.in_rgba = l == 0 && !keep_input ? d_img : nullptr;
			k.wt = bf.fwd[l];
			k.bias = d_params + off.b[l];
			if (l < LAYERS - 1)
			{
				k.out = d_act[l];
				// The 4 -> 32 layer stays on mma.sync: on tcgen05 it would be a
				// 32 -> 32 layer with 28 zero input channels, which measured slower.
				// Inference launches every layer after the first with
				// programmatic dependent launch: its set-up overlaps the
				// previous layer's last wave.
				const bool pdl = !keep_input && l > 0;
				if (l == 0)
					r = conv<16, 32, EPI_RELU>(k);
				else if (use_tc)
					r = conv_tc<EPI_RELU>(k, pdl);
				else
					r = conv<32, 32, EPI_RELU>(k, pdl);
			}
			else
			{
				// 32 -> 4 likewise (N = 32 with 28 zero output channels).
				k.out = nullptr;
				k.image = d_img;
				k.out_f32 = keep_input || !out_rgba ? d_out : nullptr; // training reads it
				k.out_rgba = out_rgba;
				r = conv<32, 8, EPI_LAST>(k, !keep_input);
			}
			if (r)
				return r;
		}
		return PGS_OK;
	}

	template <int CIN, int COUT>
	int wgrad(const __nv_bfloat16 *x, const __nv_bfloat16 *dy, int layer, int n, int h, int w)
	{
		WgradArgs a = { x, dy, d_wgrad + layer * WGRAD_STRIDE, d_bgrad + layer * BGRAD_STRIDE, n, h, w };
		int tiles = ((w + TILE - 1) / TILE) * ((h + TILE - 1) / TILE) * n;
		int grid = std::min(tiles, sm_count * WGRAD_CTAS);
		constexpr size_t smem = 2 * wgrad_buffer_bytes<CIN, COUT>();
		UP_TRY(cudaFuncSetAttribute(wgrad_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
		wgrad_kernel<CIN, COUT><<<grid, WGRAD_THREADS, smem, stream>>>(a);
		UP_TRY(cudaGetLastError());
		return PGS_OK;
	}

	// Loss and parameter gradient (into d_grad) for a batch; *loss = mean
	// squared error over all four channels.
	int backward(const uint8_t *d_img, const uint8_t *d_target, int n, int h, int w, double *loss)
	{
		int r = forward(d_img, n, h, w, nullptr, true);
		if (r)
			return r;
		size_t pixels = size_t(n) * h * w;
		UP_TRY(cudaMemsetAsync(d_loss, 0, sizeof(double), stream));
		UP_TRY(cudaMemsetAsync(d_wgrad, 0, LAYERS * WGRAD_STRIDE * 4, stream));
		UP_TRY(cudaMemsetAsync(d_bgrad, 0, LAYERS * BGRAD_STRIDE * 4, stream));
		float scale = 2.0f / float(pixels * 4);
		loss_kernel<<<unsigned(std::min((pixels + 255) / 256, size_t(sm_count) * 4)), 256, 0, stream>>>(d_out, d_target, pixels, scale, d_gout, d_loss);
		UP_TRY(cudaGetLastError());
		// Layer 5: weight gradient from the 16-channel output gradient, data
		// gradient into layer 4's output through its ReLU.
		if ((r = wgrad<32, 16>(d_act[4], d_gout, 5, n, h, w)))
			return r;
		ConvArgs k = {};
		k.n = n;
		k.h = h;
		k.w = w;
		k.in = d_gout;
		k.wt = bf.dgrad[5];
		k.mask = d_act[4];
		k.out = d_ga;
		if ((r = conv<16, 32, EPI_MASK>(k)))
			return r;
		__nv_bfloat16 *g = d_ga, *g2 = d_gb;
		for (int l = 4; l >= 1; l--)
		{
			if ((r = wgrad<32, 32>(d_act[l - 1], g, l, n, h, w)))
				return r;
			k.in = g;
			k.wt = bf.dgrad[l];
			k.mask = d_act[l - 1];
			k.out = g2;
			if ((r = use_tc ? conv_tc<EPI_MASK>(k) : conv<32, 32, EPI_MASK>(k)))
				return r;
			std::swap(g, g2);
		}
		if ((r = wgrad<16, 32>(d_x0, g, 0, n, h, w)))
			return r;
		gather_grad_kernel<<<dim3((9 * 32 * 32 + 32 + 255) / 256, LAYERS), 256, 0, stream>>>(d_wgrad, d_bgrad, d_grad);
		UP_TRY(cudaGetLastError());
		if (loss)
		{
			double s = 0.0;
			UP_TRY(cudaMemcpyAsync(&s, d_loss, sizeof(double), cudaMemcpyDeviceToHost, stream));
			UP_TRY(cudaStreamSynchronize(stream));
			*loss = s / double(pixels * 4);
		}
		return PGS_OK;
	}

	int step(float lr)
	{
		adam_t++;
		const float b1 = 0.9f, b2 = 0.999f;
		float c1 = 1.0f - std::pow(b1, float(adam_t)), c2 = 1.0f - std::pow(b2, float(adam_t));
		adam_kernel<<<(off.total + 255) / 256, 256, 0, stream>>>(d_params, d_m, d_v, d_grad, off.total, lr, b1, b2, 1e-8f,
		                                                         c1, c2);
		UP_TRY(cudaGetLastError());
		return pack();
	}
};
} // namespace pgs_up

using pgs_up::Upscaler;

extern "C" {
void *pgs_upscaler_create(int device, int *status)
{
	int dummy;
	if (!status)
		status = &dummy;
	int count = 0;
	if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0)
	{
		*status = PGS_ERROR_NO_DEVICE;
		return nullptr;
	}
	auto *u = new (std::nothrow) Upscaler();
	if (!u)
	{
		*status = PGS_ERROR_OUT_OF_MEMORY;
		return nullptr;
	}
	int r = u->init(device);
	if (r)
	{
		u->destroy();
		delete u;
		*status = r;
		return nullptr;
	}
	*status = PGS_OK;
	return u;
}

void pgs_upscaler_destroy(void *up)
{
	if (!up)
		return;
	static_cast<Upscaler *>(up)->destroy();
	delete static_cast<Upscaler *>(up);
}

uint32_t pgs_upscaler_param_count(void *up) { return up ? uint32_t(static_cast<Upscaler *>(up)->off.total) : 0; }

int pgs_upscaler_set_params(void *up, const float *params, uint32_t count)
{
	return up && params ? static_cast<Upscaler *>(up)->set_params(params, count) : PGS_ERROR_INVALID_ARGUMENT;
}

int pgs_upscaler_get_params(void *up, float *params, uint32_t count)
{
	if (!up || !params)
		return PGS_ERROR_INVALID_ARGUMENT;
	Upscaler *u = static_cast<Upscaler *>(up);
	return u->get(u->d_params, params, count);
}

int pgs_upscaler_get_gradient(void *up, float *grad, uint32_t count)
{
	if (!up || !grad)
		return PGS_ERROR_INVALID_ARGUMENT;
	Upscaler *u = static_cast<Upscaler *>(up);
	return u->get(u->d_grad, grad, count);
}

int pgs_upscaler_forward(void *up, const void *d_images, uint32_t n, uint32_t h, uint32_t w, void *d_out_rgba)
{
	if (!up || !d_images || !n || !h || !w)
		return PGS_ERROR_INVALID_ARGUMENT;
	Upscaler *u = static_cast<Upscaler *>(up);
	cudaSetDevice(u->device);
	return u->forward(static_cast<const uint8_t *>(d_images), int(n), int(h), int(w), static_cast<uint8_t *>(d_out_rgba),
	                  false);
}

int pgs_upscaler_backward(void *up, const void *d_images, const void *d_targets, uint32_t n, uint32_t h, uint32_t w,
                          double *loss)
{
	if (!up || !d_images || !d_targets || !n || !h || !w)
		return PGS_ERROR_INVALID_ARGUMENT;
	Upscaler *u = static_cast<Upscaler *>(up);
	cudaSetDevice(u->device);
	return u->backward(static_cast<const uint8_t *>(d_images), static_cast<const uint8_t *>(d_targets), int(n), int(h),
	                   int(w), loss);
}

int pgs_upscaler_adam_step(void *up, float lr)
{
	if (!up)
		return PGS_ERROR_INVALID_ARGUMENT;
	Upscaler *u = static_cast<Upscaler *>(up);
	cudaSetDevice(u->device);
	return u->step(lr);
}

int pgs_umma_selftest(int device, uint32_t mode, float *out_host)
{
	if (!out_host || mode > 2)
		return PGS_ERROR_INVALID_ARGUMENT;
	UP_TRY(cudaSetDevice(device));
	float *d_out = nullptr;
	uint32_t *d_err = nullptr;
	UP_TRY(cudaMalloc(&d_out, 128 * 32 * 4));
	UP_TRY(cudaMalloc(&d_err, 4));
	UP_TRY(cudaMemset(d_out, 0, 128 * 32 * 4));
	UP_TRY(cudaMemset(d_err, 0, 4));
	// Generous allocation: every address the descriptors can form stays inside.
	const int smem = 96 * 1024;
	UP_TRY(cudaFuncSetAttribute(pgs_up::umma_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
	pgs_up::umma_probe_kernel<<<1, 128, smem>>>(mode, d_out, d_err);
	cudaError_t e = cudaDeviceSynchronize();
	uint32_t err = 0;
	if (e == cudaSuccess)
		e = cudaMemcpy(out_host, d_out, 128 * 32 * 4, cudaMemcpyDeviceToHost);
	if (e == cudaSuccess)
		e = cudaMemcpy(&err, d_err, 4, cudaMemcpyDeviceToHost);
	cudaFree(d_out);
	cudaFree(d_err);
	if (e != cudaSuccess)
		return PGS_ERROR_CUDA;
	return err ? PGS_ERROR_DEVICE_FLAG : PGS_OK;
}

int pgs_upscaler_set_tensor_path(void *up, int tcgen05)
{
	if (!up)
		return PGS_ERROR_INVALID_ARGUMENT;
	if (tcgen05 < 0 || tcgen05 > 2)
		return PGS_ERROR_INVALID_ARGUMENT;
	static_cast<Upscaler *>(up)->use_tc = tcgen05;
	return PGS_OK;
}

int pgs_upscaler_get_error(void *up, uint32_t *flags)
{
	if (!up || !flags)
		return PGS_ERROR_INVALID_ARGUMENT;
	Upscaler *u = static_cast<Upscaler *>(up);
	UP_TRY(cudaMemcpyAsync(flags, u->d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, u->stream));
	UP_TRY(cudaStreamSynchronize(u->stream));
	return *flags ? PGS_ERROR_DEVICE_FLAG : PGS_OK;
}

void *pgs_upscaler_stream(void *up) { return up ? static_cast<void *>(static_cast<Upscaler *>(up)->stream) : nullptr; }

int pgs_upscaler_set_stream(void *up, void *stream)
{
	if (!up)
		return PGS_ERROR_INVALID_ARGUMENT;
	return static_cast<Upscaler *>(up)->set_stream(static_cast<cudaStream_t>(stream));
}

int pgs_upscaler_synchronize(void *up)
{
	if (!up)
		return PGS_ERROR_INVALID_ARGUMENT;
	return cudaStreamSynchronize(static_cast<Upscaler *>(up)->stream) == cudaSuccess ? PGS_OK : PGS_ERROR_CUDA;
}
}
