// Learned preconditioner for flexible CG: a 6-layer 3x3 convolutional
// network on one complex image (real and imaginary parts as 2 channels),
// 2 -> 32 -> 32 -> 32 -> 32 -> 32 -> 2 channels, ReLU after layers 1-5,
// zero padding. Weights are bfloat16, accumulation float32.
//
// Activations are bfloat16 in NHWC order, 32 channels per pixel
// (act[((img * Y + y) * X + x) * 32 + c]), pixel (x, y) of a BART image
// [X, Y] (x fastest). Layers 2-5 run on the tensor cores (mma.sync
// m16n8k16 bf16 -> f32): a block computes a 32 x 8 pixel tile of all 32
// output channels as a GEMM of the tile's im2col rows (K = 9 taps x 32
// channels) with the weight matrix, both staged in shared memory. Layers 1
// and 6 (2 input / 2 output channels) are thin and run on the FP32 pipes.
//
// Training uses the same kernels plus the backward passes: the data
// gradient of a 32 -> 32 layer is the forward kernel with the weights
// transposed and the taps flipped, masked by the ReLU of the layer below;
// weight gradients are FP32 sums over pixels, per block (layers 2-5 on the
// tensor cores), then reduced in a fixed order (bit-reproducible).
//
// Parameter vector (float32), per layer l = 1..6: W_l[cout][tap][cin]
// (tap = 3 ky + kx), then b_l[cout].
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "nufft_kernels.cuh"

namespace bn {

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

enum { NET_C = 32, NET_TILE_X = 32, NET_TILE_Y = 8, NET_THREADS = 256 };

constexpr int NET_SA_STRIDE = 40;	// bf16 per pixel in the halo tile (32 + 8 pad: conflict-free fragments)
constexpr int NET_SW_STRIDE = 296;	// bf16 per output channel in the weight tile (288 + 8 pad)
constexpr int NET_HALO_X = NET_TILE_X + 2, NET_HALO_Y = NET_TILE_Y + 2;
constexpr size_t NET_CONV_SMEM = sizeof(bf16) * (NET_HALO_X * NET_HALO_Y * NET_SA_STRIDE + NET_C * NET_SW_STRIDE);

struct NetLayout {

	// parameter offsets of W_l and b_l, l = 0..5
	__host__ __device__ static constexpr int cin(int l) { return (0 == l) ? 2 : NET_C; }
	__host__ __device__ static constexpr int cout(int l) { return (5 == l) ? 2 : NET_C; }
	__host__ __device__ static constexpr int wsize(int l) { return cout(l) * 9 * cin(l); }
	__host__ __device__ static constexpr int size(int l) { return wsize(l) + cout(l); }
	__host__ __device__ static constexpr int woff(int l) { return (0 == l) ? 0 : woff(l - 1) + size(l - 1); }
	__host__ __device__ static constexpr int boff(int l) { return woff(l) + wsize(l); }
	__host__ __device__ static constexpr int total() { return woff(5) + size(5); }
};

static_assert(NetLayout::total() == 38178, "parameter count");

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
		uint32_t b0, uint32_t b1)
{
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
		"{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
		: "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
		: "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t lds32(const bf16* p) { return *(const uint32_t*)p; }

// 32 -> 32 channel 3x3 convolution on the tensor cores.
//   MODE 0 (forward):  out = bf16(relu(conv(in, w) + bias))
//   MODE 1 (backward): out = bf16(conv(in, w) * (mask > 0)), with in = the
//                      gradient of the layer above and w its transposed,
//                      tap-flipped weights.
// w: bf16 [32 cout][9 tap][32 cin]. grid (ceil(X/32), ceil(Y/8), nimg).
template <int MODE>
__global__ void __launch_bounds__(NET_THREADS) k_conv32(const bf16* __restrict__ in, const bf16* __restrict__ w,
		const float* __restrict__ bias, const bf16* __restrict__ mask, bf16* __restrict__ out, int X, int Y,
		const int* done, const int* skip = nullptr)
{
	extern __shared__ __align__(16) unsigned char net_smem[];
	bf16* sA = (bf16*)net_smem;
	bf16* sW = sA + NET_HALO_X * NET_HALO_Y * NET_SA_STRIDE;

	if ((done && *done) || (skip && *skip))
		return;

	const int x0 = blockIdx.x * NET_TILE_X;
	const int y0 = blockIdx.y * NET_TILE_Y;
	const long ibase = (long)blockIdx.z * X * Y;

	// weights: 32 rows of 288 bf16 = 36 x 16 B
	for (int i = threadIdx.x; i < NET_C * 36; i += NET_THREADS) {

		int co = i / 36;
		int j = i % 36;
		*(uint4*)(sW + co * NET_SW_STRIDE + j * 8) = ((const uint4*)(w + co * 288))[j];
	}

	// halo tile: 10 x 34 pixels, 64 B each (4 x 16 B), zero outside the image
	for (int i = threadIdx.x; i < NET_HALO_X * NET_HALO_Y * 4; i += NET_THREADS) {

		int q = i & 3;
		int pix = i >> 2;
		int gy = y0 + pix / NET_HALO_X - 1;
		int gx = x0 + pix % NET_HALO_X - 1;
		uint4 v = make_uint4(0u, 0u, 0u, 0u);

		if ((gy >= 0) && (gy < Y) && (gx >= 0) && (gx < X))
			v = ((const uint4*)(in + (ibase + (long)gy * X + gx) * NET_C))[q];

		*(uint4*)(sA + pix * NET_SA_STRIDE + q * 8) = v;
	}

	__syncthreads();

	const int warp = threadIdx.x >> 5;	// tile row
	const int lane = threadIdx.x & 31;
	const int g = lane >> 2;
	const int t = lane & 3;

	float acc[2][4][4];
#pragma unroll
	for (int mt = 0; mt < 2; mt++)
#pragma unroll
		for (int nt = 0; nt < 4; nt++)
#pragma unroll
			for (int e = 0; e < 4; e++)
				acc[mt][nt][e] = 0.f;

#pragma unroll 1
	for (int tap = 0; tap < 9; tap++) {

		const int ky = tap / 3;
		const int kx = tap % 3;
#pragma unroll
		for (int h = 0; h < 2; h++) {	// input channels 16 h .. 16 h + 15

			uint32_t b[4][2];
#pragma unroll
			for (int nt = 0; nt < 4; nt++) {

				const bf16* wp = sW + (nt * 8 + g) * NET_SW_STRIDE + tap * NET_C + h * 16 + 2 * t;
				b[nt][0] = lds32(wp);
				b[nt][1] = lds32(wp + 8);
			}
#pragma unroll
			for (int mt = 0; mt < 2; mt++) {

				const bf16* ap = sA + ((warp + ky) * NET_HALO_X + mt * 16 + g + kx) * NET_SA_STRIDE + h * 16 + 2 * t;
				uint32_t a0 = lds32(ap);
				uint32_t a1 = lds32(ap + 8 * NET_SA_STRIDE);
				uint32_t a2 = lds32(ap + 8);
				uint32_t a3 = lds32(ap + 8 * NET_SA_STRIDE + 8);
#pragma unroll
				for (int nt = 0; nt < 4; nt++)
					mma_bf16(acc[mt][nt], a0, a1, a2, a3, b[nt][0], b[nt][1]);
			}
		}
	}

	const int gy = y0 + warp;

	if (gy >= Y)
		return;

#pragma unroll
	for (int mt = 0; mt < 2; mt++) {
#pragma unroll
		for (int hh = 0; hh < 2; hh++) {

			const int gx = x0 + mt * 16 + g + 8 * hh;

			if (gx >= X)
				continue;

			const long o = (ibase + (long)gy * X + gx) * NET_C;
#pragma unroll
			for (int nt = 0; nt < 4; nt++) {

				const int co = nt * 8 + 2 * t;
				float v0 = acc[mt][nt][2 * hh];
				float v1 = acc[mt][nt][2 * hh + 1];

				if (0 == MODE) {

					v0 = fmaxf(v0 + bias[co], 0.f);
					v1 = fmaxf(v1 + bias[co + 1], 0.f);

				} else {

					bf162 m = *(const bf162*)(mask + o + co);
					v0 = (__bfloat162float(m.x) > 0.f) ? v0 : 0.f;
					v1 = (__bfloat162float(m.y) > 0.f) ? v1 : 0.f;
				}

				*(bf162*)(out + o + co) = __floats2bfloat162_rn(v0, v1);
			}
		}
	}
}

// The thin layers (2 channels on one side) take a quad of lanes per four
// consecutive pixels: lane q holds channels 8 q .. 8 q + 7 of all four, so the
// 64 bytes of a pixel's activation are one access of the quad and a weight
// vector read from shared memory serves four pixels. (One thread per pixel
// read or wrote sixteen lines per warp access and reloaded the weights for
// every pixel: seven 256^2 images took 34 us in layer 1, 54 us in layer 6 and
// 52 us in its backward pass; 25, 37 and 33 us so.) Blocks cover 256 pixels.
struct NetPix {

	long p0;		// first of the quad's pixels
	int q;			// lane in the quad
	unsigned in[4];		// bit per tap: the neighbour is inside the image

	__device__ __forceinline__ NetPix(int X, int Y, long P)
	{
		q = threadIdx.x & 3;
		p0 = ((long)blockIdx.x * NET_THREADS + threadIdx.x) / 4 * 4;
		const long XY = (long)X * Y;
		const int rest = (int)(min(p0, P - 1) % XY);
		int y = rest / X, x = rest - y * X;
#pragma unroll
		for (int i = 0; i < 4; i++) {

			// columns x - 1, x, x + 1 of a row, the three rows
			const unsigned row = ((x > 0) ? 1u : 0u) | 2u | ((x + 1 < X) ? 4u : 0u);
			in[i] = (p0 + i < P) ? (((y > 0) ? row : 0u) | (row << 3) | ((y + 1 < Y) ? row << 6 : 0u)) : 0u;

			if (++x == X) {

				x = 0;
				y = (y + 1 == Y) ? 0 : y + 1;
			}
		}
	}

	// pixel i has a neighbour at this tap
	__device__ __forceinline__ bool has(int i, int tap) const { return 0 != ((in[i] >> tap) & 1u); }

	// first pixel plus the tap's offset
	__device__ __forceinline__ long base(int tap, int X) const { return p0 + (long)(tap / 3 - 1) * X + tap % 3 - 1; }
};

// Position of a work item among nx x ny per image, advanced by a fixed step
// without a division per item.
struct NetWalk {

	int x, y, z, nx, ny, sx, sy, sz;	// z: image

	__device__ __forceinline__ NetWalk(long first, long step, int nx_, int ny_) : nx(nx_), ny(ny_)
	{
		x = (int)(first % nx);
		y = (int)((first / nx) % ny);
		z = (int)(first / nx / ny);
		sx = (int)(step % nx);
		sy = (int)((step / nx) % ny);
		sz = (int)(step / nx / ny);
	}

	__device__ __forceinline__ void next()
	{
		x += sx;
		y += sy;
		z += sz;

		if (x >= nx) {

			x -= nx;
			y++;
		}

		if (y >= ny) {

			y -= ny;
			z++;
		}
	}
};

__device__ __forceinline__ void net_bf16x8(const uint4& u, float (&f)[8])
{
	const bf162* h = (const bf162*)&u;
#pragma unroll
	for (int j = 0; j < 4; j++) {

		const float2 v = __bfloat1622float2(h[j]);
		f[2 * j] = v.x;
		f[2 * j + 1] = v.y;
	}
}

// eight floats as pairs (two-wide arithmetic)
__device__ __forceinline__ void net_lds8(const float* s, float2 (&f)[4])
{
	const float4 a = *(const float4*)s, b = *(const float4*)(s + 4);
	f[0] = make_float2(a.x, a.y), f[1] = make_float2(a.z, a.w);
	f[2] = make_float2(b.x, b.y), f[3] = make_float2(b.z, b.w);
}

// Layer 1 (2 -> 32): act = bf16(relu(conv(s * in) + b)),
// in complex [nimg][Y][X], s = *scale, or 1 / sqrt(sum of norm_part) (the
// input's norm from the partials of the pass that wrote it), or 1. w: float
// [32][9][2] (values already rounded to bf16), b: [32]. Nothing is done when
// *done or *skip (the learned term switched off).
__global__ void __launch_bounds__(NET_THREADS) k_net_in(const float2* __restrict__ in, int X, int Y, long P,
		const float* __restrict__ w, const float* __restrict__ b, const float* scale, const double* norm_part,
		int nnorm, bf16* __restrict__ out, const int* done, const int* skip)
{
	__shared__ __align__(16) float sw[19 * NET_C];	// [2 tap + channel][cout], then the biases
	__shared__ double red[32];

	if ((done && *done) || (skip && *skip))
		return;

	for (int i = threadIdx.x; i < 19 * NET_C; i += NET_THREADS)
		sw[i] = (i < 18 * NET_C) ? w[(i % NET_C) * 18 + i / NET_C] : b[i - 18 * NET_C];

	float s = 1.f;

	if (scale) {

		s = *scale;

	} else if (norm_part) {

		const double n2 = sum_partials_d(norm_part, nnorm, red);
		s = (n2 > 0.) ? (float)(1. / sqrt(n2)) : 0.f;
	}

	__syncthreads();

	const NetPix px(X, Y, P);
	float2 acc[4][4], wv[4];	// pixel, channel pair
	net_lds8(sw + 18 * NET_C + 8 * px.q, wv);
#pragma unroll
	for (int i = 0; i < 4; i++)
#pragma unroll
		for (int c = 0; c < 4; c++)
			acc[i][c] = wv[c];

#pragma unroll 3
	for (int tap = 0; tap < 9; tap++) {

		const float2* nb = in + px.base(tap, X);
		float2 v[4];
#pragma unroll
		for (int i = 0; i < 4; i++) {

			v[i] = px.has(i, tap) ? nb[i] : make_float2(0.f, 0.f);
			v[i].x *= s;
			v[i].y *= s;
		}

		net_lds8(sw + 2 * tap * NET_C + 8 * px.q, wv);
#pragma unroll
		for (int i = 0; i < 4; i++)
#pragma unroll
			for (int c = 0; c < 4; c++)
				acc[i][c] = cfma(wv[c], make_float2(v[i].x, v[i].x), acc[i][c]);

		net_lds8(sw + (2 * tap + 1) * NET_C + 8 * px.q, wv);
#pragma unroll
		for (int i = 0; i < 4; i++)
#pragma unroll
			for (int c = 0; c < 4; c++)
				acc[i][c] = cfma(wv[c], make_float2(v[i].y, v[i].y), acc[i][c]);
	}

#pragma unroll
	for (int i = 0; i < 4; i++) {

		uint4 o;
		uint32_t* pk = (uint32_t*)&o;
#pragma unroll
		for (int j = 0; j < 4; j++) {

			const bf162 h = __floats2bfloat162_rn(fmaxf(acc[i][j].x, 0.f), fmaxf(acc[i][j].y, 0.f));
			pk[j] = *(const uint32_t*)&h;
		}

		if (px.p0 + i < P)
			*(uint4*)(out + (px.p0 + i) * NET_C + 8 * px.q) = o;
	}
}

// Layer 6 (32 -> 2):
//   out = zc + s * (conv(act, w) + b)   (zc = 0 if null),
// s = *scale, or sqrt(sum of norm_part) (the norm of zc, from the partials
// of the pass that wrote it), or 1; out = zc when *net_off (the stall
// fallback of the flexible CG). With pdot: per-block partials Re<pdot, out>.
__global__ void __launch_bounds__(NET_THREADS) k_net_out(const bf16* __restrict__ act, int X, int Y, long P,
		const float* __restrict__ w, const float* __restrict__ b, const float* scale, const double* norm_part,
		int nnorm, const float2* zc, float2* out, const float2* __restrict__ pdot, double* __restrict__ dot_part,
		const int* done, const int* net_off)
{
	__shared__ __align__(16) float sw[2 * 9 * NET_C + 2];
	__shared__ double red[32];

	if (done && *done)
		return;

	for (int i = threadIdx.x; i < 2 * 9 * NET_C + 2; i += NET_THREADS)
		sw[i] = (i < 2 * 9 * NET_C) ? w[i] : b[i - 2 * 9 * NET_C];

	const float s = scale ? *scale : (norm_part ? (float)sqrt(sum_partials_d(norm_part, nnorm, red)) : 1.f);
	__syncthreads();

	const bool off = net_off && *net_off;
	const NetPix px(X, Y, P);
	const long p = px.p0 + px.q;		// the pixel this lane writes
	float2 o = make_float2(0.f, 0.f);

	if (!off) {	// block-uniform

		float2 acc[4];
#pragma unroll
		for (int i = 0; i < 4; i++)
			acc[i] = make_float2(0.f, 0.f);
#pragma unroll 3
		for (int tap = 0; tap < 9; tap++) {

			const bf16* nb = act + px.base(tap, X) * NET_C + 8 * px.q;
			uint4 u[4];
#pragma unroll
			for (int i = 0; i < 4; i++) {

				u[i] = px.has(i, tap) ? *(const uint4*)(nb + i * NET_C) : make_uint4(0u, 0u, 0u, 0u);
			}

			// (pairs of outputs in two-wide sums would spend the instructions
			// saved on doubling the activations: 42 against 37 us)
			float2 w0[4], w1[4];
			net_lds8(sw + tap * NET_C + 8 * px.q, w0);
			net_lds8(sw + 9 * NET_C + tap * NET_C + 8 * px.q, w1);
#pragma unroll
			for (int i = 0; i < 4; i++) {

				float f[8];
				net_bf16x8(u[i], f);
#pragma unroll
				for (int c = 0; c < 4; c++) {

					acc[i].x = fmaf(w0[c].x, f[2 * c], acc[i].x);
					acc[i].y = fmaf(w1[c].x, f[2 * c], acc[i].y);
					acc[i].x = fmaf(w0[c].y, f[2 * c + 1], acc[i].x);
					acc[i].y = fmaf(w1[c].y, f[2 * c + 1], acc[i].y);
				}
			}
		}

		// sums over the quad's channels; lane q keeps pixel q
		auto shfl = [](float2 v, int m) {
			return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
		};
		float2 k0 = (px.q & 2) ? acc[2] : acc[0], k1 = (px.q & 2) ? acc[3] : acc[1];
		k0 = cadd(k0, shfl((px.q & 2) ? acc[0] : acc[2], 2));
		k1 = cadd(k1, shfl((px.q & 2) ? acc[1] : acc[3], 2));
		o = cadd((px.q & 1) ? k1 : k0, shfl((px.q & 1) ? k0 : k1, 1));
	}

	double dot = 0.;

	if (p < P) {

		float2 v = zc ? zc[p] : make_float2(0.f, 0.f);

		if (!off) {

			v.x = fmaf(s, o.x + sw[2 * 9 * NET_C], v.x);
			v.y = fmaf(s, o.y + sw[2 * 9 * NET_C + 1], v.y);
		}

		out[p] = v;

		if (pdot) {

			float2 q = pdot[p];
			dot = (double)q.x * (double)v.x + (double)q.y * (double)v.y;
		}
	}

	if (pdot) {

		double t = block_sum_d(dot, red);

		if (0 == threadIdx.x)
			dot_part[blockIdx.x] = t;
	}
}

// Backward of layer 6 to its input, masked by the ReLU of layer 5:
//   gu5[q][ci] = bf16((act5[q][ci] > 0) * sum_{co, tap} w[co][8 - tap][ci] gout[q + off(tap)][co])
__global__ void __launch_bounds__(NET_THREADS) k_net_out_bwd(const float2* __restrict__ gout, const bf16* __restrict__ act5,
		int X, int Y, long P, const float* __restrict__ w, bf16* __restrict__ gu5)
{
	__shared__ __align__(16) float sw[2 * 9 * NET_C];

	for (int i = threadIdx.x; i < 2 * 9 * NET_C; i += NET_THREADS)
		sw[i] = w[i];

	__syncthreads();

	const NetPix px(X, Y, P);
	float2 acc[4][4];	// pixel, channel pair
#pragma unroll
	for (int i = 0; i < 4; i++)
#pragma unroll
		for (int c = 0; c < 4; c++)
			acc[i][c] = make_float2(0.f, 0.f);

#pragma unroll 3
	for (int tap = 0; tap < 9; tap++) {

		const float2* nb = gout + px.base(tap, X);
		float2 g[4];
#pragma unroll
		for (int i = 0; i < 4; i++) {

			g[i] = px.has(i, tap) ? nb[i] : make_float2(0.f, 0.f);
		}

		float2 w0[4], w1[4];
		net_lds8(sw + (8 - tap) * NET_C + 8 * px.q, w0);
		net_lds8(sw + 9 * NET_C + (8 - tap) * NET_C + 8 * px.q, w1);
#pragma unroll
		for (int i = 0; i < 4; i++)
#pragma unroll
			for (int c = 0; c < 4; c++) {

				acc[i][c] = cfma(w0[c], make_float2(g[i].x, g[i].x), acc[i][c]);
				acc[i][c] = cfma(w1[c], make_float2(g[i].y, g[i].y), acc[i][c]);
			}
	}

#pragma unroll
	for (int i = 0; i < 4; i++) {

		if (px.p0 + i >= P)
			break;

		float m[8];
		net_bf16x8(*(const uint4*)(act5 + (px.p0 + i) * NET_C + 8 * px.q), m);
		uint4 o;
		uint32_t* pk = (uint32_t*)&o;
#pragma unroll
		for (int j = 0; j < 4; j++) {

			const bf162 h = __floats2bfloat162_rn((m[2 * j] > 0.f) ? acc[i][j].x : 0.f,
					(m[2 * j + 1] > 0.f) ? acc[i][j].y : 0.f);
			pk[j] = *(const uint32_t*)&h;
		}

		*(uint4*)(gu5 + (px.p0 + i) * NET_C + 8 * px.q) = o;
	}
}

// Weight and bias gradients -----------------------------------------------------
//
// Both kernels are persistent: a block takes units of 256 pixels (image tiles, or
// rows of its warps) blockIdx.x, blockIdx.x + gridDim.x, ..., sums each in float32
// as before and leaves a partial vector of the layer's parameters after every
// WG_RUN units, which k_wgrad_reduce adds in float64. So no float32 sum grows with
// the number of images, there are a few hundred vectors to reduce instead of one
// per tile, and the order is fixed: the gradients are the same bits every run.
// Partial f of block b is vector b + f gridDim.x (slots):
//   part[slot][(co * 9 + tap) * CIN + ci] = sum_p g[p][co] a[p + off(tap)][ci]
//   part[slot][COUT * 9 * CIN + co]       = sum_p g[p][co]
enum { WG_RUN = 8 };

// partial vectors of nblk <= units blocks
inline long wg_slots(long units, long nblk)
{
	const long most = (units + nblk - 1) / nblk;			// units of the first blocks; the others one less
	const long full = (most - 1) / WG_RUN;				// partials before the first blocks' last
	const bool all = (most - 1 > full * WG_RUN);			// the other blocks have one more too
	return nblk * full + (all ? nblk : units - nblk * (most - 1));
}

// 32 -> 32 channels on the tensor cores (mma.sync, bf16 in, float32 sums).
// Per tile of 32 x 8 pixels the gradient rows and the activations' halo lie
// in shared memory pixel by pixel; ldmatrix.trans reads both as MMA operands
// with the pixels as K. Warp w owns tap w: its 32 x 32 sums are 32 registers, and
// 32 more for the run's (one set over a whole block's tiles took 39 us a layer of
// seven 256^2 images instead of 42, but its error grew with the images: equal terms
// of 128 of 250^2 were off by 2.9e-4, now by 6e-8).
// The next tile arrives by cp.async while this one is summed, one barrier per
// tile. Bound by the mma.sync rate (half of the tensor cycles); the FP32-pipe kernel it replaced took two shared-memory
// loads per FMA (1019 us a layer; the whole forward and gradient pass 5.37 ms
// then, 0.65 ms now).
constexpr int WG_WARPS = 9;
constexpr int WG_THREADS = 32 * WG_WARPS;
constexpr int WG_STAGE = (NET_HALO_X * NET_HALO_Y + NET_TILE_X * NET_TILE_Y) * NET_SA_STRIDE;	// bf16 per buffer
constexpr size_t WG_SMEM = 2 * sizeof(bf16) * WG_STAGE;

__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr)
{
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
		: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// 16 bytes global -> shared, zeros where !ok (nothing is read there)
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool ok)
{
	const int n = ok ? 16 : 0;
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(dst), "l"(src), "r"(n));
}

__global__ void __launch_bounds__(WG_THREADS, 2) k_wgrad32(const bf16* __restrict__ a, const bf16* __restrict__ g,
		int X, int Y, int tx, int ty, long ntiles, float* __restrict__ part)
{
	extern __shared__ __align__(16) unsigned char wg_smem[];
	const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(wg_smem);
	constexpr int HALO = NET_HALO_X * NET_HALO_Y;
	constexpr uint32_t PIX = NET_SA_STRIDE * 2;		// bytes per pixel
	constexpr uint32_t STAGE = WG_STAGE * 2;
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	const int ky = warp / 3, kx = warp % 3;

	NetWalk pos(blockIdx.x, gridDim.x, tx, ty);	// the tile to load next

	auto load = [&](int buf) {
		const int x0 = pos.x * NET_TILE_X, y0 = pos.y * NET_TILE_Y;
		const long ibase = pos.z * ((long)X * Y);
		const uint32_t sa = s0 + buf * STAGE, sg = sa + HALO * PIX;
		pos.next();
#pragma unroll
		for (int i = threadIdx.x; i < HALO * 4; i += WG_THREADS) {

			const int q = i & 3, pix = i >> 2;
			const int gy = y0 + pix / NET_HALO_X - 1, gx = x0 + pix % NET_HALO_X - 1;
			const bool ok = (gy >= 0) && (gy < Y) && (gx >= 0) && (gx < X);
			cp_async16_zfill(sa + pix * PIX + q * 16, ok ? a + (ibase + (long)gy * X + gx) * NET_C + q * 8 : a, ok);
		}

#pragma unroll
		for (int i = threadIdx.x; i < NET_TILE_X * NET_TILE_Y * 4; i += WG_THREADS) {

			const int q = i & 3, pix = i >> 2;
			const int gy = y0 + pix / NET_TILE_X, gx = x0 + pix % NET_TILE_X;
			const bool ok = (gy < Y) && (gx < X);
			cp_async16_zfill(sg + pix * PIX + q * 16, ok ? g + (ibase + (long)gy * X + gx) * NET_C + q * 8 : g, ok);
		}

		asm volatile("cp.async.commit_group;\n" ::: "memory");
	};

	float sum[2][4][4], bsum[2][2];		// over the run's tiles

	auto clear = [&]() {
#pragma unroll
		for (int mt = 0; mt < 2; mt++) {

			bsum[mt][0] = bsum[mt][1] = 0.f;
#pragma unroll
			for (int nt = 0; nt < 4; nt++)
#pragma unroll
				for (int e = 0; e < 4; e++)
					sum[mt][nt][e] = 0.f;
		}
	};

	clear();

	// lane's row of the 8x8 matrices of one ldmatrix: gradient matrices are
	// (pixels 0-7, co 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15) of a 16 x 16
	// block, activation ones (0-7, ci 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
	const int mrow = lane & 7, msel = lane >> 3;
	const uint32_t goff = ((msel >> 1) * 8 + mrow) * PIX + (msel & 1) * 16;
	const uint32_t aoff = ((msel & 1) * 8 + mrow + ky * NET_HALO_X + kx) * PIX + (msel >> 1) * 16;
	int buf = 0, run = 0, slot = blockIdx.x;
	int left = (int)((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);	// the block's tiles

	if (left > 0)
		load(0);

	for (; left > 0; left--) {

		// this tile has arrived and the other buffer has been read by all
		asm volatile("cp.async.wait_group 0;\n" ::: "memory");
		__syncthreads();

		if (left > 1)
			load(buf ^ 1);

		float acc[2][4][4], bacc[2][4];		// over this tile
#pragma unroll
		for (int mt = 0; mt < 2; mt++) {
#pragma unroll
			for (int e = 0; e < 4; e++) {

				bacc[mt][e] = 0.f;
#pragma unroll
				for (int nt = 0; nt < 4; nt++)
					acc[mt][nt][e] = 0.f;
			}
		}

		const uint32_t sa = s0 + buf * STAGE + aoff, sg = s0 + buf * STAGE + HALO * PIX + goff;
#pragma unroll 2
		for (int k = 0; k < NET_TILE_X * NET_TILE_Y / 16; k++) {

			const int py = k / 2, px = (k % 2) * 16;
			uint32_t fa[2][4], fb[2][4];
			ldsm_x4_t(fa[0], sg + (py * NET_TILE_X + px) * PIX);
			ldsm_x4_t(fa[1], sg + (py * NET_TILE_X + px) * PIX + 32);
			ldsm_x4_t(fb[0], sa + (py * NET_HALO_X + px) * PIX);
			ldsm_x4_t(fb[1], sa + (py * NET_HALO_X + px) * PIX + 32);
#pragma unroll
			for (int mt = 0; mt < 2; mt++) {
#pragma unroll
				for (int nt = 0; nt < 4; nt++)
					mma_bf16(acc[mt][nt], fa[mt][0], fa[mt][1], fa[mt][2], fa[mt][3], fb[nt / 2][2 * (nt & 1)],
							fb[nt / 2][2 * (nt & 1) + 1]);

				if (4 == warp)	// the bias gradient: a column of ones
					mma_bf16(bacc[mt], fa[mt][0], fa[mt][1], fa[mt][2], fa[mt][3], 0x3f803f80u, 0x3f803f80u);
			}
		}

		buf ^= 1;
#pragma unroll
		for (int mt = 0; mt < 2; mt++) {

			bsum[mt][0] += bacc[mt][0];
			bsum[mt][1] += bacc[mt][2];
#pragma unroll
			for (int nt = 0; nt < 4; nt++)
#pragma unroll
				for (int e = 0; e < 4; e++)
					sum[mt][nt][e] += acc[mt][nt][e];
		}

		if ((++run < WG_RUN) && (left > 1))
			continue;

		float* dst = part + (long)slot * (NET_C * 9 * NET_C + NET_C);
		const int r = lane >> 2, t = lane & 3;
#pragma unroll
		for (int mt = 0; mt < 2; mt++) {
#pragma unroll
			for (int hh = 0; hh < 2; hh++) {

				const int co = mt * 16 + hh * 8 + r;
#pragma unroll
				for (int nt = 0; nt < 4; nt++)
					*(float2*)(dst + (co * 9 + warp) * NET_C + nt * 8 + 2 * t)
						= make_float2(sum[mt][nt][2 * hh], sum[mt][nt][2 * hh + 1]);

				if ((4 == warp) && (0 == t))
					dst[NET_C * 9 * NET_C + co] = bsum[mt][hh];
			}
		}

		slot += gridDim.x;
		run = 0;
		clear();
	}
}

// Layers 1 and 6 (2 channels on one side) on the FP32 pipes: lane = channel of
// the 32-channel tensor w, whose pixels are read once each; the 3 x 3 window
// of the complex (2-channel) image t around a pixel slides along x in
// registers, so a pixel costs one 2-byte load and three broadcast 8-byte
// loads for 36 FMAs. A warp takes rows of 32 pixels.
//   OUT6 (layer 6): w = activations at q, t = output gradient: tap k of pixel q
//          meets t at q - off(k); outputs [co 2][tap][ci = lane], bias from t
//   else (layer 1): w = output gradient at p, t = input: tap k meets t at
//          p + off(k); outputs [co = lane][tap][ci 2], bias from w
constexpr int WT_WARPS = 8;

template <bool OUT6>
__global__ void __launch_bounds__(32 * WT_WARPS, 4) k_wgrad_thin(const bf16* __restrict__ w, const float2* __restrict__ t,
		int X, int Y, int tx, long nrows, float* __restrict__ part)
{
	constexpr int O = 2 * 9 * NET_C;
	constexpr int OB = OUT6 ? 2 : NET_C;		// bias gradients
	__shared__ float red[WT_WARPS][O + NET_C];
	__shared__ float2 win[WT_WARPS][3][NET_TILE_X + 2];
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	float* dst = part + (long)blockIdx.x * (O + OB);

	// work rows: 32 pixels of one image row; tx of them per image row
	NetWalk pos((long)blockIdx.x * WT_WARPS + warp, (long)gridDim.x * WT_WARPS, tx, Y);

	// units of the block (a row per warp) and rows of this warp
	int units = (int)(((nrows + WT_WARPS - 1) / WT_WARPS - blockIdx.x + gridDim.x - 1) / gridDim.x);
	int rows = (int)((nrows - (long)blockIdx.x * WT_WARPS - warp + (long)gridDim.x * WT_WARPS - 1) / ((long)gridDim.x * WT_WARPS));

	for (; units > 0; units -= WG_RUN, rows -= WG_RUN) {	// a run

		float2 acc[9];
		float2 bsum = make_float2(0.f, 0.f);
#pragma unroll
		for (int k = 0; k < 9; k++)
			acc[k] = make_float2(0.f, 0.f);

		for (int u = 0; u < min(rows, (int)WG_RUN); u++, pos.next()) {

			const int x0 = pos.x * NET_TILE_X, y = pos.y;
			const long base = pos.z * ((long)X * Y);
			__syncwarp();

			for (int i = lane; i < 3 * (NET_TILE_X + 2); i += 32) {

				const int dy = i / (NET_TILE_X + 2), dx = i % (NET_TILE_X + 2);
				const int yy = y + dy - 1, xx = x0 + dx - 1;
				win[warp][dy][dx] = ((yy >= 0) && (yy < Y) && (xx >= 0) && (xx < X)) ? t[base + (long)yy * X + xx]
						: make_float2(0.f, 0.f);
			}

			__syncwarp();
			const bf16* wp = w + (base + (long)y * X + x0) * NET_C + lane;
			const int n = min(NET_TILE_X, X - x0);
			float2 c0[3], c1[3], c2[3];			// window columns x - 1, x, x + 1
#pragma unroll
			for (int d = 0; d < 3; d++) {

				c0[d] = win[warp][d][0];
				c1[d] = win[warp][d][1];
			}
#pragma unroll 8
			for (int px = 0; px < NET_TILE_X; px++) {

				const float v = (px < n) ? __bfloat162float(wp[(long)px * NET_C]) : 0.f;
#pragma unroll
				for (int d = 0; d < 3; d++)
					c2[d] = win[warp][d][px + 2];
#pragma unroll
				for (int d = 0; d < 3; d++) {

					const int r0 = OUT6 ? 3 * (2 - d) + 2 : 3 * d;		// the tap that meets row d, column x - 1
					const int r1 = OUT6 ? 3 * (2 - d) + 1 : 3 * d + 1;
					const int r2 = OUT6 ? 3 * (2 - d) : 3 * d + 2;
					acc[r0] = cfma(make_float2(v, v), c0[d], acc[r0]);
					acc[r1] = cfma(make_float2(v, v), c1[d], acc[r1]);
					acc[r2] = cfma(make_float2(v, v), c2[d], acc[r2]);
				}

				if (!OUT6)
					bsum.x += v;
#pragma unroll
				for (int d = 0; d < 3; d++) {

					c0[d] = c1[d];
					c1[d] = c2[d];
				}
			}

			if (OUT6) {	// lane's pixel of the row: the bias gradient (summed over lanes below)

				const float2 v = win[warp][1][lane + 1];

				if (lane < n) {

					bsum.x += v.x;
					bsum.y += v.y;
				}
			}
		}

#pragma unroll
		for (int k = 0; k < 9; k++) {

			red[warp][OUT6 ? k * NET_C + lane : (lane * 9 + k) * 2] = acc[k].x;
			red[warp][OUT6 ? (9 + k) * NET_C + lane : (lane * 9 + k) * 2 + 1] = acc[k].y;
		}

		if (OUT6) {

			for (int o = 16; o > 0; o >>= 1) {

				bsum.x += __shfl_xor_sync(0xffffffffu, bsum.x, o);
				bsum.y += __shfl_xor_sync(0xffffffffu, bsum.y, o);
			}

			if (0 == lane) {

				red[warp][O] = bsum.x;
				red[warp][O + 1] = bsum.y;
			}

		} else {

			red[warp][O + lane] = bsum.x;
		}

		__syncthreads();

		for (int o = threadIdx.x; o < O + OB; o += 32 * WT_WARPS) {

			float s = 0.f;
#pragma unroll
			for (int k = 0; k < WT_WARPS; k++)
				s += red[k][o];

			dst[o] = s;
		}

		__syncthreads();	// before the next run's sums
		dst += (long)gridDim.x * (O + OB);
	}
}

// grad[o] = sum over the partial vectors part[slot][o] in float64: 32 outputs per block,
// WR_SLICES slices of the partials, combined in a fixed order
enum { WR_SLICES = 32 };

__global__ void __launch_bounds__(32 * WR_SLICES) k_wgrad_reduce(const float* __restrict__ part, int nblk, int O,
		float* __restrict__ grad)
{
	__shared__ double sh[WR_SLICES][32];
	const int o = blockIdx.x * 32 + threadIdx.x % 32, sl = threadIdx.x / 32;
	double acc = 0.;

	if (o < O) {
#pragma unroll 4
		for (int k = sl; k < nblk; k += WR_SLICES)
			acc += part[(long)k * O + o];
	}

	sh[sl][threadIdx.x % 32] = acc;
	__syncthreads();

	if ((0 == sl) && (o < O)) {
#pragma unroll
		for (int k = 1; k < WR_SLICES; k++)
			acc += sh[k][threadIdx.x];

		grad[o] = (float)acc;
	}
}

// gout = c (out - target), loss partials sum |out - target|^2 per block
__global__ void k_net_loss(const float2* __restrict__ out, const float2* __restrict__ target, long P, float c,
		float2* __restrict__ gout, double* __restrict__ loss_part)
{
	__shared__ double red[32];
	double acc = 0.;

	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < P; i += (long)gridDim.x * blockDim.x) {

		float2 d = make_float2(out[i].x - target[i].x, out[i].y - target[i].y);
		gout[i] = make_float2(c * d.x, c * d.y);
		acc += (double)d.x * d.x + (double)d.y * d.y;
	}

	double t = block_sum_d(acc, red);

	if (0 == threadIdx.x)
		loss_part[blockIdx.x] = t;
}

// Adam (Kingma & Ba, ICLR 2015) on the float32 master parameters
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ gr, float* __restrict__ m, float* __restrict__ v,
		int n, float lr, float b1, float b2, float eps, float c1, float c2)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {

		float gi = gr[i];
		float mi = b1 * m[i] + (1.f - b1) * gi;
		float vi = b2 * v[i] + (1.f - b2) * gi * gi;
		m[i] = mi;
		v[i] = vi;
		p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
	}
}

// Working copies of the parameters: float values rounded to bf16 (all
// weights; biases stay float) and, for layers 2-5, bf16 forward weights
// [co][tap][ci] and transposed tap-flipped weights [ci][8 - tap][co].
__global__ void k_net_pack(const float* __restrict__ p, float* __restrict__ pr, bf16* __restrict__ wf, bf16* __restrict__ wt)
{
	const int n = NetLayout::total();

	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {

		int l = 0;

		while ((l < 5) && (i >= NetLayout::woff(l + 1)))
			l++;

		const int r = i - NetLayout::woff(l);
		const bool weight = (r < NetLayout::wsize(l));
		bf16 h = __float2bfloat16_rn(p[i]);
		pr[i] = weight ? __bfloat162float(h) : p[i];

		if (weight && (l >= 1) && (l <= 4)) {

			const int co = r / 288;
			const int tap = (r / 32) % 9;
			const int ci = r % 32;
			wf[(l - 1) * 9216 + r] = h;
			wt[(l - 1) * 9216 + (ci * 9 + (8 - tap)) * 32 + co] = h;
		}
	}
}

} // namespace bn
