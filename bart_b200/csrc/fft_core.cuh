// Shared-memory Stockham FFT core for sm_100a.
//
// A thread block transforms B sequences of length L (power of two, 16..4096,
// or one of the mixed lengths further down).
// Each sequence is served by T = L/8 threads (index jt). Between stages the
// data lives in shared memory in one of two layouts (ColLayout for column
// passes, RowLayout for row passes; see below), chosen so that both the
// global accesses and the shared-memory stages stay conflict-free. Stages are
// radix 8 with a final radix 4 or 2 (Stockham autosort, so the result is in
// natural order without a bit-reversal pass).
//
// Register ownership: before the first stage and after the last stage a
// thread holds the eight elements at positions jt + T*m (m = 0..7) in
// v[m]. The first stage reads exactly these positions and the last stage
// writes them, so the caller loads stage-1 input straight from global memory
// and consumes the last-stage output in registers (e.g. the Toeplitz PSF
// product between a forward and an inverse transform needs no shared-memory
// pass at all).
//
// Forward = exp(-2 pi i jk / L), inverse = exp(+2 pi i jk / L), unnormalised,
// as FFTW's / the reference's FFT (src/num/fft_plan.c:227). Twiddles come
// from a table tw[m] = exp(-2 pi i m / L) computed on the host in float64.
#pragma once

#include <cuda_runtime.h>

namespace bn {

// In a chain of kernels of which each may start while the one before drains
// (launch_chained): wait until all earlier kernels are complete and their writes
// visible. The first thing such a kernel does on every path; what earlier
// kernels of the chain write it reads through pointers that are not
// __restrict__, so that no load is moved ahead. Nothing in an ordinary launch.
// Hides the launch latency between the five short kernels of a CG iteration
// (256^2, 16 coils, 30 iterations: 1804 -> 1759 us); telling the next kernel to
// start earlier (griddepcontrol.launch_dependents) was slower, 1778 us: its
// waiting blocks take the running ones' places.
__device__ __forceinline__ void pdl_wait()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Complex sums as one packed instruction each (the same two IEEE operations):
// the transforms are bound by instruction issue, not by the FP32 pipes.
__device__ __forceinline__ float2 cadd(float2 a, float2 b)
{
	float2 r;
	asm("{\n\t.reg .b64 a, b, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
		"add.rn.f32x2 r, a, b;\n\tmov.b64 {%0, %1}, r;\n\t}"
		: "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
	return r;
}

__device__ __forceinline__ float2 csub(float2 a, float2 b)
{
	float2 r;
	asm("{\n\t.reg .b64 a, b, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
		"sub.rn.f32x2 r, a, b;\n\tmov.b64 {%0, %1}, r;\n\t}"
		: "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
	return r;
}

// (a.x b.x + c.x, a.y b.y + c.y)
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c)
{
	float2 r;
	asm("{\n\t.reg .b64 a, b, c, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
		"fma.rn.f32x2 r, a, b, c;\n\tmov.b64 {%0, %1}, r;\n\t}"
		: "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
	return r;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
	return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b)
{
	return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// multiply by -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 rot90(float2 a)
{
	return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft2(float2* v)
{
	float2 a = v[0];
	v[0] = cadd(a, v[1]);
	v[1] = csub(a, v[1]);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2& v0, float2& v1, float2& v2, float2& v3)
{
	float2 a0 = cadd(v0, v2), a1 = csub(v0, v2);
	float2 a2 = cadd(v1, v3), a3 = rot90<INV>(csub(v1, v3));
	v0 = cadd(a0, a2);
	v2 = csub(a0, a2);
	v1 = cadd(a1, a3);
	v3 = csub(a1, a3);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2* v) { dft4<INV>(v[0], v[1], v[2], v[3]); }

template <bool INV>
__device__ __forceinline__ void dft8(float2* v)
{
	// decimation in time: two length-4 DFTs, then W8^k twiddles and a radix-2 combine
	float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
	float2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
	dft4<INV>(e0, e1, e2, e3);
	dft4<INV>(o0, o1, o2, o3);
	const float c = 0.70710678118654752440f;
	// W8^1 = (c, -+c), W8^2 = -+i, W8^3 = (-c, -+c)
	float2 t1 = INV ? make_float2(c * (o1.x - o1.y), c * (o1.x + o1.y))
			: make_float2(c * (o1.x + o1.y), c * (o1.y - o1.x));
	float2 t2 = rot90<INV>(o2);
	float2 t3 = INV ? make_float2(-c * (o3.x + o3.y), c * (o3.x - o3.y))
			: make_float2(c * (o3.y - o3.x), -c * (o3.x + o3.y));
	v[0] = cadd(e0, o0);
	v[4] = csub(e0, o0);
	v[1] = cadd(e1, t1);
	v[5] = csub(e1, t1);
	v[2] = cadd(e2, t2);
	v[6] = csub(e2, t2);
	v[3] = cadd(e3, t3);
	v[7] = csub(e3, t3);
}

// dft8 of (v0, v1, 0, 0, 0, 0, v6, v7): the first stage of a transform whose
// input is zero-padded to twice its length with the centred placement (the
// nonzero half at positions < L/4 and >= 3L/4, i.e. registers 0, 1, 6, 7).
// The same operations as dft8 minus those on the known zeros, so the same
// results (up to the sign of exact zeros).
template <bool INV>
__device__ __forceinline__ void dft8_half(float2* v)
{
	// dft4 of (a, 0, 0, b): (a + b, a + rot(-b), a - b, a - rot(-b))
	const float2 e0 = cadd(v[0], v[6]), e2 = csub(v[0], v[6]);
	const float2 eb = rot90<INV>(make_float2(-v[6].x, -v[6].y));
	const float2 e1 = cadd(v[0], eb), e3 = csub(v[0], eb);
	const float2 o0 = cadd(v[1], v[7]), o2 = csub(v[1], v[7]);
	const float2 ob = rot90<INV>(make_float2(-v[7].x, -v[7].y));
	const float2 o1 = cadd(v[1], ob), o3 = csub(v[1], ob);
	const float c = 0.70710678118654752440f;
	float2 t1 = INV ? make_float2(c * (o1.x - o1.y), c * (o1.x + o1.y))
			: make_float2(c * (o1.x + o1.y), c * (o1.y - o1.x));
	float2 t2 = rot90<INV>(o2);
	float2 t3 = INV ? make_float2(-c * (o3.x + o3.y), c * (o3.x - o3.y))
			: make_float2(c * (o3.y - o3.x), -c * (o3.x + o3.y));
	v[0] = cadd(e0, o0);
	v[4] = csub(e0, o0);
	v[1] = cadd(e1, t1);
	v[5] = csub(e1, t1);
	v[2] = cadd(e2, t2);
	v[6] = csub(e2, t2);
	v[3] = cadd(e3, t3);
	v[7] = csub(e3, t3);
}

template <int R, bool INV>
__device__ __forceinline__ void butterfly(float2* v)
{
	if constexpr (R == 8)
		dft8<INV>(v);
	else if constexpr (R == 4)
		dft4<INV>(v);
	else
		dft2<INV>(v);
}

// twiddle v[i] *= w^(i*k), w = exp(-+2 pi i / (Ns*R)): w^k from the table
// tw[m] = exp(-2 pi i m / L), its powers by complex multiplication (one
// shared-memory load per stage instead of R - 1; the products add a few
// float32 roundings, well below the transforms' own error)
template <int L, int Ns, int R, bool INV>
__device__ __forceinline__ void twiddle(float2* v, int k, const float2* tw)
{
	if constexpr (Ns > 1) {

		float2 w1 = tw[k * (L / (Ns * R))];

		if (INV)
			w1.y = -w1.y;

		float2 w = w1;
#pragma unroll
		for (int i = 1; i < R; i++) {

			v[i] = cmul(v[i], w);

			if (i + 1 < R)
				w = cmul(w, w1);
		}
	}
}

// The same with the powers 1 and 4 of w^k from the table and the others by one to
// three products of them. The mixed lengths use it: seven powers multiplied up
// one after the other left their transforms with 1.2 to 1.3 times the rounding
// error (Toeplitz normal on 192 and 640 points a side: 4.5e-7 and 5.4e-7 so, 3.5e-7
// and 4.5e-7 with these; three entries, 1, 2 and 4, give 3.2e-7 and 4.4e-7 but cost
// the 24 uneven slices 2.1 % instead of 1.0 %).
template <int L, int Ns, int R, bool INV>
__device__ __forceinline__ void twiddle_short(float2* v, int k, const float2* tw)
{
	static_assert(Ns > 1, "the first stage has no twiddles");
	const int t = k * (L / (Ns * R));
	float2 w[R];
#pragma unroll
	for (int i = 1; i < R; i++) {

		if ((1 == i) || (4 == i)) {

			w[i] = tw[i * t];

			if (INV)
				w[i].y = -w[i].y;

		} else {

			w[i] = cmul((i > 4) ? w[4] : w[i - 1], (i > 4) ? w[i - 4] : w[1]);
		}

		v[i] = cmul(v[i], w[i]);
	}
}

// Shared-memory layouts of B sequences of length L (element indices).
//
// ColLayout: sequences interleaved, element p of sequence b at p*SB + b
// (SB = B|1 odd, so a half-warp's 8-byte accesses hit distinct banks);
// thread t serves sequence t % B with index t / B. A warp covers the same
// element of consecutive sequences: coalesced for columns of an x-fastest
// array.
template <int L, int B>
struct ColLayout {

	static constexpr int SB = B | 1;
	static constexpr int SMEM = L * SB;

	__device__ static __forceinline__ int idx(int p, int b) { return p * SB + b; }
	__device__ static __forceinline__ int seq() { return threadIdx.x % B; }
	__device__ static __forceinline__ int jt() { return threadIdx.x / B; }
};

// RowLayout: each sequence contiguous with one pad element after every 8
// (p + p/8 breaks the stride-8 bank pattern of the first stage's stores);
// thread t serves sequence t / (L/8) with index t % (L/8). A warp covers
// consecutive elements of one sequence: coalesced for contiguous rows.
template <int L, int B>
struct RowLayout {

	static constexpr int SL = L + L / 8;
	static constexpr int SMEM = B * SL;

	__device__ static __forceinline__ int idx(int p, int b) { return b * SL + p + (p >> 3); }
	__device__ static __forceinline__ int seq() { return threadIdx.x / (L / 8); }
	__device__ static __forceinline__ int jt() { return threadIdx.x % (L / 8); }
};

// Stage with Ns = product of earlier radices, Ns > 1: smem -> smem (middle
// stages) or smem -> registers (the last stage).
template <int L, typename LAY, int Ns, bool INV, bool SHORT>
__device__ __forceinline__ void fft_tail(float2 (&v)[8], float2* s, int b, int jt, const float2* tw)
{
	constexpr int REM = L / Ns;
	constexpr int R = (REM >= 8) ? 8 : REM;
	constexpr int NB = L / R;
	constexpr int T = L / 8;
	constexpr int PER = NB / T;
	constexpr bool LAST = (Ns * R == L);

	float2 u[PER][R];

#pragma unroll
	for (int q = 0; q < PER; q++) {
#pragma unroll
		for (int i = 0; i < R; i++)
			u[q][i] = s[LAY::idx(jt + q * T + i * NB, b)];
	}

	if constexpr (!LAST)
		__syncthreads();

#pragma unroll
	for (int q = 0; q < PER; q++) {

		int j = jt + q * T;
		int k = j % Ns;

		if constexpr (SHORT)
			twiddle_short<L, Ns, R, INV>(u[q], k, tw);
		else
			twiddle<L, Ns, R, INV>(u[q], k, tw);

		butterfly<R, INV>(u[q]);

		if constexpr (LAST) {
			// outputs at j + NB*i = jt + T*(q + PER*i)
#pragma unroll
			for (int i = 0; i < R; i++)
				v[q + PER * i] = u[q][i];

		} else {

			int idxD = (j / Ns) * Ns * R + k;
#pragma unroll
			for (int i = 0; i < R; i++)
				s[LAY::idx(idxD + i * Ns, b)] = u[q][i];
		}
	}

	if constexpr (!LAST) {

		__syncthreads();
		fft_tail<L, LAY, Ns * R, INV, SHORT>(v, s, b, jt, tw);
	}
}

// Full transform of the register set v (positions jt + (L/8)*m in, same
// out). Begins with a barrier, so the caller may have been reading s just
// before; the caller must barrier before writing s after it returns.
// half_in: registers 2..5 are known zeros (input of length L/2, centred).
// SHORT: with twiddle_short.
template <int L, typename LAY, bool INV, bool SHORT = false>
__device__ __forceinline__ void fft_regs(float2 (&v)[8], float2* s, const float2* tw, bool half_in = false)
{
	static_assert(L >= 16 && L <= 4096 && (L & (L - 1)) == 0, "power-of-two length 16..4096");
	const int b = LAY::seq();
	const int jt = LAY::jt();

	// stage 1 (Ns = 1, radix 8, no twiddles): registers -> smem at 8*jt + i
	if (half_in)
		dft8_half<INV>(v);
	else
		butterfly<8, INV>(v);
	__syncthreads();
#pragma unroll
	for (int i = 0; i < 8; i++)
		s[LAY::idx(8 * jt + i, b)] = v[i];
	__syncthreads();

	fft_tail<L, LAY, 8, INV, SHORT>(v, s, b, jt, tw);
}

// Double-buffered form for transforms of three stages (L = 128, 256, 512):
// stage 1 writes s, stage 2 reads s and writes s2, stage 3 reads s2. Each
// stage writes a buffer that no thread reads any more (the other one was
// read in the stage before, which every thread finished before the last
// barrier), so one barrier per exchange suffices and the transform needs no
// barrier on entry: two transforms in a row (forward, then inverse) are
// safe, since the second one's stage 1 writes s, last read in the first
// one's stage 2. Same arithmetic as fft_regs, so the same results.
template <int L, typename LAY, int Ns, bool INV>
__device__ __forceinline__ void fft_tail_db(float2 (&v)[8], const float2* sr, float2* sw, int b, int jt,
		const float2* tw)
{
	constexpr int REM = L / Ns;
	constexpr int R = (REM >= 8) ? 8 : REM;
	constexpr int NB = L / R;
	constexpr int T = L / 8;
	constexpr int PER = NB / T;
	constexpr bool LAST = (Ns * R == L);

	float2 u[PER][R];

#pragma unroll
	for (int q = 0; q < PER; q++) {
#pragma unroll
		for (int i = 0; i < R; i++)
			u[q][i] = sr[LAY::idx(jt + q * T + i * NB, b)];
	}

#pragma unroll
	for (int q = 0; q < PER; q++) {

		int j = jt + q * T;
		int k = j % Ns;
		twiddle<L, Ns, R, INV>(u[q], k, tw);
		butterfly<R, INV>(u[q]);

		if constexpr (LAST) {
#pragma unroll
			for (int i = 0; i < R; i++)
				v[q + PER * i] = u[q][i];

		} else {

			int idxD = (j / Ns) * Ns * R + k;
#pragma unroll
			for (int i = 0; i < R; i++)
				sw[LAY::idx(idxD + i * Ns, b)] = u[q][i];
		}
	}

	if constexpr (!LAST) {

		__syncthreads();
		fft_tail_db<L, LAY, Ns * R, INV>(v, sw, const_cast<float2*>(sr), b, jt, tw);
	}
}

template <int L, typename LAY, bool INV>
__device__ __forceinline__ void fft_regs_db(float2 (&v)[8], float2* s, float2* s2, const float2* tw,
		bool half_in = false)
{
	static_assert((L >= 128) && (L <= 512), "three-stage lengths only");
	const int b = LAY::seq();
	const int jt = LAY::jt();

	if (half_in)
		dft8_half<INV>(v);
	else
		butterfly<8, INV>(v);
#pragma unroll
	for (int i = 0; i < 8; i++)
		s[LAY::idx(8 * jt + i, b)] = v[i];
	__syncthreads();

	fft_tail_db<L, LAY, 8, INV>(v, s, s2, b, jt, tw);
}

// Mixed lengths L = 64 R, R in {3, 5, 6, 7, 9, 10, 12} ------------------------
//
// They fill the gaps between the powers of two (192, 320, 384, 448, 576, 640,
// 768), so that a transform of a given minimum length costs at most 1.3 times
// the points it needs per axis instead of 2. Three stages with the same
// L / 8 threads per sequence and the same shared-memory layouts:
//   forward: radix 8, 8, then R (64 butterflies): the input is held as in the
//            power-of-two transforms (positions jt + (L/8) m in v[m]), the
//            spectrum as spec_pos says: butterfly j = jt + q L/8 (< 64) leaves
//            positions j + 64 i in w[q R + i];
//   inverse: the mirror image, radix R, 8, 8, from that spectrum order back to
//            positions jt + (L/8) m.
// So forward, product with a spectrum, inverse still chain in registers. The
// powers of the last forward twiddle come from four table entries and at most
// two products each.
__host__ __device__ constexpr bool is_mix(int L) { return 0 != (L & (L - 1)); }

// registers of the spectrum-side set of a thread
__host__ __device__ constexpr int spec_regs(int L) { return is_mix(L) ? ((64 + L / 8 - 1) / (L / 8)) * (L / 64) : 8; }

// position of register m of the spectrum-side set (>= L: none)
template <int L, typename LAY>
__device__ __forceinline__ int spec_pos(int m)
{
	if constexpr (is_mix(L)) {

		const int j = LAY::jt() + (m / (L / 64)) * (L / 8);
		return (j < 64) ? j + 64 * (m % (L / 64)) : L;

	} else {

		return LAY::jt() + (L / 8) * m;
	}
}

template <bool INV>
__device__ __forceinline__ void dft3(float2& x0, float2& x1, float2& x2)
{
	const float s = 0.86602540378443864676f;	// sin(pi / 3)
	const float2 t = cadd(x1, x2), d = rot90<INV>(cscale(csub(x1, x2), s));
	const float2 m = make_float2(fmaf(-0.5f, t.x, x0.x), fmaf(-0.5f, t.y, x0.y));
	x0 = cadd(x0, t);
	x1 = cadd(m, d);
	x2 = csub(m, d);
}

// odd length n from the sums and differences of the pairs x[k], x[n - k]:
// X[k] = x0 + sum_j cos(2 pi jk / n) t_j -+ i sum_j sin(2 pi jk / n) d_j
template <int N, bool INV>
__device__ __forceinline__ void dft_odd(float2 (&x)[N], const float (&c)[N], const float (&s)[N])
{
	constexpr int H = (N - 1) / 2;
	float2 t[H + 1], d[H + 1];
	float2 sum = x[0];
#pragma unroll
	for (int j = 1; j <= H; j++) {

		t[j] = cadd(x[j], x[N - j]);
		d[j] = csub(x[j], x[N - j]);
		sum = cadd(sum, t[j]);
	}

	const float2 x0 = x[0];
	x[0] = sum;
#pragma unroll
	for (int k = 1; k <= H; k++) {

		float2 a = x0, b = make_float2(0.f, 0.f);
#pragma unroll
		for (int j = 1; j <= H; j++) {

			a.x = fmaf(c[(j * k) % N], t[j].x, a.x);
			a.y = fmaf(c[(j * k) % N], t[j].y, a.y);
			b.x = fmaf(s[(j * k) % N], d[j].x, b.x);
			b.y = fmaf(s[(j * k) % N], d[j].y, b.y);
		}

		b = rot90<INV>(b);
		x[k] = cadd(a, b);
		x[N - k] = csub(a, b);
	}
}

// cos and sin of 2 pi k / 5, 2 pi k / 7 and 2 pi k / 9
template <bool INV>
__device__ __forceinline__ void dft5(float2 (&x)[5])
{
	constexpr float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;
	constexpr float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;
	const float c[5] = { 1.f, c1, c2, c2, c1 };
	const float s[5] = { 0.f, s1, s2, -s2, -s1 };
	dft_odd<5, INV>(x, c, s);
}

template <bool INV>
__device__ __forceinline__ void dft7(float2 (&x)[7])
{
	constexpr float c1 = 0.62348980185873353053f, c2 = -0.22252093395631440429f, c3 = -0.90096886790241912624f;
	constexpr float s1 = 0.78183148246802980871f, s2 = 0.97492791218182360702f, s3 = 0.43388373911755812048f;
	const float c[7] = { 1.f, c1, c2, c3, c3, c2, c1 };
	const float s[7] = { 0.f, s1, s2, s3, -s3, -s2, -s1 };
	dft_odd<7, INV>(x, c, s);
}

// 3 x 3: columns x[a], x[a + 3], x[a + 6], twiddles W9^(a b), rows
template <bool INV>
__device__ __forceinline__ void dft9(float2 (&x)[9])
{
	const float sg = INV ? 1.f : -1.f;
	const float2 w1 = make_float2(0.76604444311897803520f, sg * 0.64278760968653932632f);
	const float2 w2 = make_float2(0.17364817766693034885f, sg * 0.98480775301220805937f);
	const float2 w4 = make_float2(-0.93969262078590838405f, sg * 0.34202014332566873304f);
#pragma unroll
	for (int a = 0; a < 3; a++)
		dft3<INV>(x[a], x[a + 3], x[a + 6]);

	x[4] = cmul(x[4], w1);		// column 1, frequency 1
	x[7] = cmul(x[7], w2);		// column 1, frequency 2
	x[5] = cmul(x[5], w2);		// column 2, frequency 1
	x[8] = cmul(x[8], w4);		// column 2, frequency 2
	float2 y[9];
#pragma unroll
	for (int b = 0; b < 3; b++) {

		float2 p = x[3 * b], q = x[3 * b + 1], r = x[3 * b + 2];
		dft3<INV>(p, q, r);
		y[b] = p;
		y[b + 3] = q;
		y[b + 6] = r;
	}
#pragma unroll
	for (int k = 0; k < 9; k++)
		x[k] = y[k];
}

// R = A B with coprime factors (prime-factor algorithm, no twiddles): input
// index (B a + A b) mod R, output k from (k mod A, k mod B)
template <int A, int B, bool INV>
__device__ __forceinline__ void dft_pfa(float2 (&x)[A * B])
{
	float2 y[A][B];
#pragma unroll
	for (int b = 0; b < B; b++) {

		float2 u[A];
#pragma unroll
		for (int a = 0; a < A; a++)
			u[a] = x[(B * a + A * b) % (A * B)];

		if constexpr (2 == A)
			dft2<INV>(u);
		else
			dft4<INV>(u);
#pragma unroll
		for (int a = 0; a < A; a++)
			y[a][b] = u[a];
	}
#pragma unroll
	for (int a = 0; a < A; a++) {

		if constexpr (3 == B)
			dft3<INV>(y[a][0], y[a][1], y[a][2]);
		else
			dft5<INV>(y[a]);
	}
#pragma unroll
	for (int k = 0; k < A * B; k++)
		x[k] = y[k % A][k % B];
}

template <int R, bool INV>
__device__ __forceinline__ void dft_mix(float2 (&x)[R])
{
	static_assert((3 == R) || (5 == R) || (6 == R) || (7 == R) || (9 == R) || (10 == R) || (12 == R), "built radices");

	if constexpr (3 == R)
		dft3<INV>(x[0], x[1], x[2]);
	else if constexpr (5 == R)
		dft5<INV>(x);
	else if constexpr (7 == R)
		dft7<INV>(x);
	else if constexpr (9 == R)
		dft9<INV>(x);
	else if constexpr (6 == R)
		dft_pfa<2, 3, INV>(x);
	else if constexpr (10 == R)
		dft_pfa<2, 5, INV>(x);
	else
		dft_pfa<4, 3, INV>(x);
}

// Forward transform of v (positions jt + (L/8) m) into the spectrum-side set
// w. DB: two exchange buffers, one barrier per exchange (see fft_regs_db);
// else s2 == s and a barrier on entry.
template <int L, typename LAY, bool DB>
__device__ __forceinline__ void mix_fwd(float2 (&v)[8], float2 (&w)[spec_regs(L)], float2* s, float2* s2,
		const float2* tw, bool half_in)
{
	constexpr int R = L / 64, T = L / 8;
	const int b = LAY::seq(), jt = LAY::jt();

	if (half_in)
		dft8_half<false>(v);
	else
		dft8<false>(v);

	if (!DB)
		__syncthreads();
#pragma unroll
	for (int i = 0; i < 8; i++)
		s[LAY::idx(8 * jt + i, b)] = v[i];

	__syncthreads();
#pragma unroll
	for (int i = 0; i < 8; i++)
		v[i] = s[LAY::idx(jt + i * T, b)];

	if (!DB)
		__syncthreads();

	const int k = jt % 8;
	twiddle_short<L, 8, 8, false>(v, k, tw);
	dft8<false>(v);
#pragma unroll
	for (int i = 0; i < 8; i++)
		s2[LAY::idx((jt - k) * 8 + k + 8 * i, b)] = v[i];

	__syncthreads();
#pragma unroll
	for (int q = 0; q < spec_regs(L) / R; q++) {

		const int j = min(jt + q * T, 63);	// surplus threads repeat the last butterfly
		float2 u[R];
#pragma unroll
		for (int i = 0; i < R; i++)
			u[i] = s2[LAY::idx(j + 64 * i, b)];

		// W_L^(i j): entries j, 2j, 4j, 8j and products
		const float2 w1 = tw[j], w2 = tw[2 * j], w3 = cmul(w2, w1);
		u[1] = cmul(u[1], w1);
		u[2] = cmul(u[2], w2);

		if constexpr (R > 3) {

			const float2 w4 = tw[4 * j];
			u[3] = cmul(u[3], w3);
			u[4] = cmul(u[4], w4);

			if constexpr (R > 5)
				u[5] = cmul(u[5], cmul(w4, w1));

			if constexpr (R > 6)
				u[6] = cmul(u[6], cmul(w4, w2));

			if constexpr (R > 7)
				u[7] = cmul(u[7], cmul(w4, w3));
		}

		if constexpr (R > 8) {

			const float2 w8 = tw[8 * j];
			u[8] = cmul(u[8], w8);

			if constexpr (R > 9)
				u[9] = cmul(u[9], cmul(w8, w1));

			if constexpr (R > 11) {

				u[10] = cmul(u[10], cmul(w8, w2));
				u[11] = cmul(u[11], cmul(w8, w3));
			}
		}

		dft_mix<R, false>(u);
#pragma unroll
		for (int i = 0; i < R; i++)
			w[q * R + i] = u[i];
	}
}

// Inverse transform of the spectrum-side set w into v.
template <int L, typename LAY, bool DB>
__device__ __forceinline__ void mix_inv(float2 (&w)[spec_regs(L)], float2 (&v)[8], float2* s, float2* s2,
		const float2* tw)
{
	constexpr int R = L / 64, T = L / 8;
	const int b = LAY::seq(), jt = LAY::jt();

	if (!DB)
		__syncthreads();
#pragma unroll
	for (int q = 0; q < spec_regs(L) / R; q++) {

		const int j = jt + q * T;
		float2 u[R];
#pragma unroll
		for (int i = 0; i < R; i++)
			u[i] = w[q * R + i];

		dft_mix<R, true>(u);

		if (j < 64) {
#pragma unroll
			for (int i = 0; i < R; i++)
				s[LAY::idx(R * j + i, b)] = u[i];
		}
	}

	__syncthreads();
#pragma unroll
	for (int i = 0; i < 8; i++)
		v[i] = s[LAY::idx(jt + i * T, b)];

	if (!DB)
		__syncthreads();

	const int k = jt % R;
	twiddle_short<L, R, 8, true>(v, k, tw);
	dft8<true>(v);
#pragma unroll
	for (int i = 0; i < 8; i++)
		s2[LAY::idx((jt - k) * 8 + k + R * i, b)] = v[i];

	__syncthreads();
#pragma unroll
	for (int i = 0; i < 8; i++)
		v[i] = s2[LAY::idx(jt + i * T, b)];

	twiddle_short<L, 8 * R, 8, true>(v, jt, tw);
	dft8<true>(v);
}

// Forward and inverse transforms of any built length between the input-side
// set v and the spectrum-side set w (the same registers for powers of two);
// single exchange buffer, barrier on entry.
template <int L, typename LAY, bool SHORT = false>
__device__ __forceinline__ void fft_fwd(float2 (&v)[8], float2 (&w)[spec_regs(L)], float2* s, const float2* tw,
		bool half_in = false)
{
	if constexpr (is_mix(L)) {

		mix_fwd<L, LAY, false>(v, w, s, s, tw, half_in);

	} else {

		fft_regs<L, LAY, false, SHORT>(v, s, tw, half_in);
#pragma unroll
		for (int m = 0; m < 8; m++)
			w[m] = v[m];
	}
}

template <int L, typename LAY, bool SHORT = false>
__device__ __forceinline__ void fft_inv(float2 (&w)[spec_regs(L)], float2 (&v)[8], float2* s, const float2* tw)
{
	if constexpr (is_mix(L)) {

		mix_inv<L, LAY, false>(w, v, s, s, tw);

	} else {
#pragma unroll
		for (int m = 0; m < 8; m++)
			v[m] = w[m];

		fft_regs<L, LAY, true, SHORT>(v, s, tw);
	}
}

// stage-1 position of register m for this thread
template <int L, typename LAY>
__device__ __forceinline__ int reg_pos(int m) { return LAY::jt() + (L / 8) * m; }

} // namespace bn
