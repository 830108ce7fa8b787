// jms_nn.cu -- kernels of the control-variate surrogate network (BF16
// storage, FP32 accumulation), training and inference.
//
// The surrogate maps a local projected-potential patch around the probe
// (one channel per depth bin) to the integrated detector signals at the
// readout thicknesses.  Layers: 3x3 convolutions of stride 2 and padding 1,
// with or without ReLU (BF16 activations and weights), a global average pool,
// and a linear layer (FP32).  The host side (jmultislicelib_b200/surrogate.py)
// owns the buffers and the training loop; these kernels are the building
// blocks: forward, both backward products, loss, Adam.
//
// Layouts: activations [B][C][H][W]; conv weights [Co][Ci][3][3]; linear
// weights [O][C].  The ReLU mask of a layer is its stored output (y > 0).
#include "../../include/jms_b200.h"
#include "jms_kernels.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace {

__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }

// The convolutions are small (at most a few tens of MMAC): what bounds them is
// latency, so each kernel spreads its outputs over the SMs, stages its operands
// in shared memory in one pass of independent loads per chunk of channels, and
// keeps the reuse of a value in registers.  Batch 256, ten 16 x 16 channels, all
// layers of a training step, against one thread per output (or per sum) reading
// every operand from global memory: forward 92 -> 53 us, weight gradients
// 152 -> 80, data gradients 102 -> 51; still mostly waiting on global loads.
// Every sum has one order of its FP32 additions, given at its kernel, that no
// tile, chunk or grid changes: Adam divides a gradient by its own magnitude, so
// in a few training steps another rounding of a gradient near zero becomes 1e-4
// of a bias.

// y[b][co][oy][ox] = relu(bias[co] + sum_ci,ky,kx w[co][ci][ky][kx] x[b][ci][2oy-1+ky][2ox-1+kx])
// A CTA makes PT output pixels (flattened b, oy, ox) of 16 output channels; 4 PT
// threads compute, one pixel and four channels each, in the order bias, channel,
// tap (the sum is rounded to BF16: another order would move values that lie next
// to a tie); all threads stage.  A chunk of input channels costs one memory
// latency, so the small tile takes 32 of them at once.
constexpr int kNnThr = 256;
template <int PT, class I>
__global__ void __launch_bounds__(kNnThr) k_conv_fwd(const __nv_bfloat16* __restrict__ x,
	const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias, __nv_bfloat16* __restrict__ y, int B, int Ci,
	int H, int W, int Co, int relu)
{
	constexpr int CI = PT == 16 ? 32 : 8, K = 9 * CI;
	constexpr int WROW = 20;                           // 16 channels; rows of 20 spread the stores over the banks
	__shared__ float xs[K][PT];                        // taps of the CTA's pixels
	__shared__ __align__(16) float ws[K][WROW];        // weights of its channels
	const int Ho = H / 2, Wo = W / 2, hw = Ho * Wo;
	const I npix = (I)B * hw, pix0 = (I)blockIdx.x * PT;
	const int co0 = blockIdx.y * 16, px = threadIdx.x % PT, cg = threadIdx.x / PT;
	const I pix = pix0 + px;
	const int b = (int)(pix / hw), p = (int)(pix - (I)b * hw), oy = p / Wo, ox = p - oy * Wo;
	float acc[4];
	#pragma unroll
	for (int c = 0; c < 4; c++) acc[c] = cg < 4 && co0 + 4 * cg + c < Co ? bias[co0 + 4 * cg + c] : 0.f;
	for (int c0 = 0; c0 < Ci; c0 += CI) {
		const int nc = min(CI, Ci - c0);
		__syncthreads();
		// a thread stages taps of its own pixel: k = cg, cg + 256 / PT, ...
		#pragma unroll 6
		for (int k = cg; k < 9 * nc; k += kNnThr / PT) {
			const int ci = k / 9, t = k - 9 * ci;
			const int iy = 2 * oy - 1 + t / 3, ix = 2 * ox - 1 + t % 3;
			xs[k][px] = (pix < npix && iy >= 0 && ix >= 0)
				? bf(x[(((long long)b * Ci + c0 + ci) * H + iy) * W + ix]) : 0.f;
		}
		#pragma unroll 6
		for (int i = threadIdx.x; i < 16 * K; i += kNnThr) {
			const int co = i / K, k = i - co * K;
			if (k < 9 * nc) ws[k][co] = co0 + co < Co ? bf(w[((long long)(co0 + co) * Ci + c0) * 9 + k]) : 0.f;
		}
		__syncthreads();
		if (cg < 4) {
			for (int ci = 0; ci < nc; ci++) {
				#pragma unroll
				for (int t = 0; t < 9; t++) {
					if ((t < 3 && oy == 0) || (t % 3 == 0 && ox == 0)) continue;   // outside the image
					const float v = xs[9 * ci + t][px];
					const float4 q = *reinterpret_cast<const float4*>(&ws[9 * ci + t][4 * cg]);
					acc[0] = fmaf(q.x, v, acc[0]);
					acc[1] = fmaf(q.y, v, acc[1]);
					acc[2] = fmaf(q.z, v, acc[2]);
					acc[3] = fmaf(q.w, v, acc[3]);
				}
			}
		}
	}
	if (cg >= 4 || pix >= npix) return;
	#pragma unroll
	for (int c = 0; c < 4; c++) {
		const int co = co0 + 4 * cg + c;
		if (co >= Co) continue;
		y[((long long)b * Co + co) * hw + p] = __float2bfloat16(relu && acc[c] < 0.f ? 0.f : acc[c]);
	}
}

// dx[b][ci][iy][ix] = sum_co,ky,kx g[b][co][oy][ox] w[co][ci][ky][kx], iy = 2oy-1+ky,
// with g = dy * (y > 0) when relu.  A thread makes the 2 x 2 block of input
// pixels at (2a, 2b') of one channel, which sees the four outputs (a, b'),
// (a, b'+1), (a+1, b'), (a+1, b'+1): nine products per output channel and no
// masked taps.  A CTA takes 16 blocks x 16 input channels and output channels in
// chunks of kBwdCo.  A sum runs tap by tap (ky, kx ascending), over the output
// channels within a tap: four sweeps over the channels, one per tap of the
// pixel that has four.  Up to kBwdCo output channels are staged once for all
// four.
constexpr int kBwdCo = 64;
template <class I>
__global__ void __launch_bounds__(kNnThr) k_conv_bwd_data(const float* __restrict__ dy,
	const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ w, float* __restrict__ dx, int B, int Ci,
	int H, int W, int Co, int relu)
{
	__shared__ __align__(16) float gs[kBwdCo][16][4];
	__shared__ __nv_bfloat16 ws[kBwdCo][9][16];
	const int Ho = H / 2, Wo = W / 2, hw = Ho * Wo;
	const I npix = (I)B * hw, pix0 = (I)blockIdx.x * 16;
	const int ci0 = blockIdx.y * 16, c = threadIdx.x % 16, q = threadIdx.x / 16;
	const I pix = pix0 + q;
	const int b = (int)(pix / hw), p = (int)(pix - (I)b * hw), a = p / Wo, d = p - a * Wo;
	const bool right = d + 1 < Wo, down = a + 1 < Ho;
	float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
	for (int sweep = 0; sweep < 4; sweep++) {
		for (int k0 = 0; k0 < Co; k0 += kBwdCo) {
			const int nk = min(kBwdCo, Co - k0);
			if (sweep == 0 || Co > kBwdCo) {
				__syncthreads();
				#pragma unroll 8
				for (int i = threadIdx.x; i < nk * 64; i += kNnThr) {
					const int k = i / 64, h = i % 4;
					const I pi = pix0 + (i / 4) % 16;
					const int bi = (int)(pi / hw), ri = (int)(pi - (I)bi * hw), ai = ri / Wo + (h >> 1), di = ri % Wo + (h & 1);
					const bool in = pi < npix && ai < Ho && di < Wo;
					const long long o = (((long long)bi * Co + k0 + k) * Ho + ai) * Wo + di;
					const float g = in ? dy[o] : 0.f;
					const __nv_bfloat16 yv = in && relu ? y[o] : __nv_bfloat16(1.f);
					gs[k][(i / 4) % 16][h] = bf(yv) > 0.f ? g : 0.f;
				}
				#pragma unroll 12
				for (int i = threadIdx.x; i < nk * 144; i += kNnThr) {
					const int k = i / 144, r = i - 144 * k;
					if (ci0 + r / 9 < Ci) ws[k][r % 9][r / 9] = w[((long long)(k0 + k) * Ci + ci0) * 9 + r];
				}
				__syncthreads();
			}
			auto tap = [&](int k, int t) { return bf(ws[k][t][c]); };
			auto grad = [&](int k) { return *reinterpret_cast<const float4*>(gs[k][q]); };   // (a,b'), (a,b'+1), (a+1,b'), (a+1,b'+1)
			if (sweep == 0) {
				#pragma unroll 4
				for (int k = 0; k < nk; k++) {
					const float4 g = grad(k);
					o0 = fmaf(g.x, tap(k, 4), o0);
					if (right) o1 = fmaf(g.y, tap(k, 3), o1);
					if (down) o2 = fmaf(g.z, tap(k, 1), o2);
					if (right && down) o3 = fmaf(g.w, tap(k, 0), o3);
				}
			}
			else if (sweep == 1) {
				#pragma unroll 4
				for (int k = 0; k < nk; k++) {
					const float4 g = grad(k);
					o1 = fmaf(g.x, tap(k, 5), o1);
					o2 = fmaf(g.x, tap(k, 7), o2);
					if (down) o3 = fmaf(g.z, tap(k, 2), o3);
				}
			}
			else if (sweep == 2) {
				#pragma unroll 8
				for (int k = 0; k < nk; k++)
					if (right) o3 = fmaf(gs[k][q][1], tap(k, 6), o3);
			}
			else {
				#pragma unroll 8
				for (int k = 0; k < nk; k++) o3 = fmaf(gs[k][q][0], tap(k, 8), o3);
			}
		}
	}
	if (pix >= npix || ci0 + c >= Ci) return;
	float* out = dx + (((long long)b * Ci + ci0 + c) * H + 2 * a) * W + 2 * d;
	out[0] = o0;
	out[1] = o1;
	out[W] = o2;
	out[W + 1] = o3;
}

// dw[co][ci][ky][kx] = sum_b,oy,ox g[b][co][oy][ox] x[b][ci][iy][ix]; db[co] = sum g.
// A CTA takes NCO output channels, one input channel and one row ky of taps: a
// thread reads an output pixel's three taps once for its channels.  Four channels
// where that gives every SM two CTAs, else one: the first layers have the most
// pixels and the fewest channels (1024 images of 3 x 64 x 64: 8.1 -> 1.1 ms for
// the first layer with the next).  U pixels' loads are in flight at once, the
// ReLU's outputs among them: loaded under a test of their own, each would be
// waited for.  A sum runs over a thread's pixels (t, t + 256, ...),
// then over the lanes of a warp in halves, then over the warps.  The CTAs of
// ci = 0, ky = 1 also make db.
template <class I, bool RELU, int NCO, int U>
__global__ void __launch_bounds__(kNnThr) k_conv_bwd_weight(const __nv_bfloat16* __restrict__ x,
	const float* __restrict__ dy, const __nv_bfloat16* __restrict__ y, float* __restrict__ dw, float* __restrict__ db,
	int B, int Ci, int H, int W, int Co)
{
	constexpr int K = 4 * NCO;
	__shared__ float red[kNnThr / 32][K];
	const int ci = blockIdx.x, co0 = blockIdx.y * NCO, ky = blockIdx.z;
	const int Ho = H / 2, Wo = W / 2, hw = Ho * Wo;
	const I n = (I)B * hw;
	float a[K];              // sum 4 c + kx of channel c, and 4 c + 3 its sum of g
	#pragma unroll
	for (int k = 0; k < K; k++) a[k] = 0.f;
	// pixel (b, oy, ox) of i and its step of 256 pixels, carried instead of divided
	int b = (int)threadIdx.x / hw, oy = (int)threadIdx.x % hw / Wo, ox = (int)threadIdx.x % hw % Wo;
	const int sb = kNnThr / hw, sy = kNnThr % hw / Wo, sx = kNnThr % hw % Wo;
	for (I i = threadIdx.x; i < n; i += U * kNnThr) {
		float v[U][3], g[U][NCO];
		__nv_bfloat16 yv[RELU ? U : 1][NCO];
		bool top[U], left[U], live[U];
		#pragma unroll
		for (int u = 0; u < U; u++) {
			const int p = oy * Wo + ox, iy = 2 * oy - 1 + ky, ix = 2 * ox - 1;
			live[u] = u == 0 || n - i > u * kNnThr;
			top[u] = live[u] && iy >= 0;
			left[u] = top[u] && ix >= 0;
			const __nv_bfloat16* xp = x + (((long long)b * Ci + ci) * H + iy) * W + ix;
			v[u][0] = left[u] ? bf(xp[0]) : 0.f;
			v[u][1] = top[u] ? bf(xp[1]) : 0.f;
			v[u][2] = top[u] ? bf(xp[2]) : 0.f;
			const long long o = ((long long)b * Co + co0) * hw + p;
			#pragma unroll
			for (int c = 0; c < NCO; c++) {
				const bool in = live[u] && co0 + c < Co;
				g[u][c] = in ? dy[o + (long long)c * hw] : 0.f;
				if constexpr (RELU) yv[u][c] = in ? y[o + (long long)c * hw] : __nv_bfloat16(0.f);
			}
			ox += sx;
			oy += sy + (ox >= Wo);
			ox -= ox >= Wo ? Wo : 0;
			b += sb + (oy >= Ho);
			oy -= oy >= Ho ? Ho : 0;
		}
		#pragma unroll
		for (int u = 0; u < U; u++) {
			#pragma unroll
			for (int c = 0; c < NCO; c++) {
				const float gc = !RELU || bf(yv[RELU ? u : 0][c]) > 0.f ? g[u][c] : 0.f;
				if (left[u]) a[4 * c] = fmaf(gc, v[u][0], a[4 * c]);
				if (top[u]) a[4 * c + 1] = fmaf(gc, v[u][1], a[4 * c + 1]);
				if (top[u]) a[4 * c + 2] = fmaf(gc, v[u][2], a[4 * c + 2]);
				if (live[u]) a[4 * c + 3] += gc;
			}
		}
	}
	// all K sums at once: each step halves the sums a lane holds, until lane
	// 32 / K k holds sum k
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	#pragma unroll
	for (int h = 16, m = K / 2; h > 0; h >>= 1, m >>= 1) {
		const bool up = lane & h;
		#pragma unroll
		for (int k = 0; k < m; k++) {
			const float keep = up ? a[k + m] : a[k], send = up ? a[k] : a[k + m];
			a[k] = keep + __shfl_xor_sync(0xffffffffu, send, h);
		}
		if (m == 0) a[0] += __shfl_xor_sync(0xffffffffu, a[0], h);
	}
	if (lane % (32 / K) == 0) red[warp][lane / (32 / K)] = a[0];
	__syncthreads();
	const int k = threadIdx.x;
	if (k >= K || co0 + k / 4 >= Co) return;
	float s = 0.f;
	#pragma unroll
	for (int q = 0; q < kNnThr / 32; q++) s += red[q][k];
	if (k % 4 < 3) dw[((long long)(co0 + k / 4) * Ci + ci) * 9 + 3 * ky + k % 4] = s;
	else if (ci == 0 && ky == 1) db[co0 + k / 4] = s;
}

// out[b][o] = bl[o] + sum_c wl[o][c] mean_hw h[b][c][hw], summed in that order
__global__ void k_pool_linear_fwd(const __nv_bfloat16* __restrict__ h, const float* __restrict__ wl,
	const float* __restrict__ bl, float* __restrict__ out, int B, int C, int HW, int O)
{
	extern __shared__ float pooled[];   // [C]
	const int b = blockIdx.x;
	for (int c = threadIdx.x; c < C; c += blockDim.x) {
		const __nv_bfloat16* hp = h + ((long long)b * C + c) * HW;
		float s = 0.f;
		for (int k = 0; k < HW; k++) s += bf(hp[k]);
		pooled[c] = s / (float)HW;
	}
	__syncthreads();
	for (int o = threadIdx.x; o < O; o += blockDim.x) {
		float s = bl[o];
		#pragma unroll 16
		for (int c = 0; c < C; c++) s = fmaf(__ldg(wl + (long long)o * C + c), pooled[c], s);
		out[(long long)b * O + o] = s;
	}
}

// dh[b][c][hw] = sum_o dout[b][o] wl[o][c] / HW; dwl, dbl by a second kernel
__global__ void k_pool_linear_bwd_data(const float* __restrict__ wl, const float* __restrict__ dout,
	float* __restrict__ dh, int B, int C, int HW, int O)
{
	const long long n = (long long)B * C * HW;
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const int c = (int)((i / HW) % C), b = (int)(i / ((long long)HW * C));
	float s = 0.f;
	for (int o = 0; o < O; o++) s = fmaf(dout[(long long)b * O + o], wl[(long long)o * C + c], s);
	dh[i] = s / (float)HW;
}

// dwl[o][c] = sum_b dout[b][o] pooled[b][c]; dbl[o] = sum_b dout[b][o], summed
// in the order of b.  A CTA makes 16 x 16 sums (the bias is column C, whose
// factor is 1) and stages their factors for kPlB images at once, so a sum waits
// for memory once per chunk (256 x 64 x 30: 8 us; reading both factors in its
// loop, 101 us).
constexpr int kPlB = 256;
__global__ void __launch_bounds__(kNnThr) k_pool_linear_bwd_weight(const __nv_bfloat16* __restrict__ h,
	const float* __restrict__ dout, float* __restrict__ dwl, float* __restrict__ dbl, int B, int C, int HW, int O)
{
	__shared__ float ps[kPlB][16], gs[kPlB][16];
	const int nct = C / 16 + 1, c0 = blockIdx.x % nct * 16, o0 = blockIdx.x / nct * 16;   // C + 1 columns
	const int tc = threadIdx.x % 16, to = threadIdx.x / 16, c = c0 + tc, o = o0 + to;
	float s = 0.f;
	for (int b0 = 0; b0 < B; b0 += kPlB) {
		const int nb = min(kPlB, B - b0);
		__syncthreads();
		#pragma unroll 8
		for (int k = to; k < nb; k += kNnThr / 16) gs[k][tc] = o0 + tc < O ? dout[(long long)(b0 + k) * O + o0 + tc] : 0.f;
		const __nv_bfloat16* hp = h + ((long long)b0 * C + c) * HW;
		if (c >= C || HW == 1) {   // independent loads
			#pragma unroll 8
			for (int k = to; k < nb; k += kNnThr / 16) ps[k][tc] = c < C ? bf(hp[(long long)k * C]) : 1.f;
		}
		else {
			for (int k = to; k < nb; k += kNnThr / 16) {
				float p = 0.f;
				#pragma unroll 4
				for (int i = 0; i < HW; i++) p += bf(hp[(long long)k * C * HW + i]);
				ps[k][tc] = p / (float)HW;
			}
		}
		__syncthreads();
		#pragma unroll 16
		for (int k = 0; k < nb; k++) s = fmaf(gs[k][to], ps[k][tc], s);
	}
	if (o >= O || c > C) return;
	if (c == C) dbl[o] = s;
	else dwl[(long long)o * C + c] = s;
}

// dout = 2 (out - t) / n; loss partial sums of (out - t)^2 / n (atomic into *loss)
__global__ void k_mse(const float* __restrict__ out, const float* __restrict__ t, float* __restrict__ dout,
	float* __restrict__ loss, int n)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	float e = 0.f;
	if (i < n) {
		const float d = out[i] - t[i];
		dout[i] = 2.f * d / (float)n;
		e = d * d / (float)n;
	}
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
	if ((threadIdx.x & 31) == 0 && loss) atomicAdd(loss, e);
}

// Adam (Kingma & Ba 2015) on FP32 master weights, optional BF16 copy.
__device__ __forceinline__ void adam_one(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
	float* __restrict__ v, __nv_bfloat16* __restrict__ pb, int i, float lr, float b1, float b2, float eps, float c1,
	float c2)
{
	const float gi = g[i];
	const float mi = b1 * m[i] + (1.f - b1) * gi;
	const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
	m[i] = mi;
	v[i] = vi;
	const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
	p[i] = pi;
	if (pb) pb[i] = __float2bfloat16(pi);
}
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
	float* __restrict__ v, __nv_bfloat16* __restrict__ pb, int n, float lr, float b1, float b2, float eps,
	float c1, float c2)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) adam_one(p, g, m, v, pb, i, lr, b1, b2, eps, c1, c2);
}

// The same step on several parameter tensors in one launch: blockIdx.y is the tensor.
constexpr int kAdamMax = 32;
struct AdamSet {
	float* p[kAdamMax];
	const float* g[kAdamMax];
	float* m[kAdamMax];
	float* v[kAdamMax];
	__nv_bfloat16* pb[kAdamMax];
	int n[kAdamMax];
};
__global__ void k_adam_set(const AdamSet a, float lr, float b1, float b2, float eps, float c1, float c2)
{
	const int t = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < a.n[t]) adam_one(a.p[t], a.g[t], a.m[t], a.v[t], a.pb[t], i, lr, b1, b2, eps, c1, c2);
}

__global__ void k_cast_bf16(const float* __restrict__ s, __nv_bfloat16* __restrict__ d, long long n)
{
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) d[i] = __float2bfloat16(s[i]);
}

constexpr long long kMaxPix32 = 1LL << 30;   // output pixels up to which pixel indices are 32-bit
inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// Surrogate inputs: thread per output value out[c][p][b][u][v], the mean over
// the object slices of depth bin b (bins of nobj / nbins slices, the first
// nobj % nbins one slice longer) and over a pool x pool pixel block of the
// projected potential of configuration c, in the win x win window centred on
// pixel (px, py) of position p (periodic).
__global__ void k_patches(const float* __restrict__ pot, int nvar, int nx, int ny, const int* __restrict__ objslc,
	int nobj, const int* __restrict__ var, int nconf, const int* __restrict__ pix, int npos, int nbins, int win,
	int pool, float* __restrict__ out)
{
	const int m = win / pool;
	const long long n = (long long)nconf * npos * nbins * m * m;
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const int v = (int)(i % m), u = (int)((i / m) % m);
	const int b = (int)((i / ((long long)m * m)) % nbins);
	const int p = (int)((i / ((long long)m * m * nbins)) % npos);
	const int c = (int)(i / ((long long)m * m * nbins * npos));
	const int q = nobj / nbins, r = nobj % nbins;
	const int s0 = b * q + min(b, r), s1 = s0 + q + (b < r ? 1 : 0);
	const int x0 = pix[2 * p] - win / 2 + v * pool, y0 = pix[2 * p + 1] - win / 2 + u * pool;
	const long long N = (long long)nx * ny;
	float acc = 0.f;
	for (int s = s0; s < s1; s++) {
		const float* map = pot + ((long long)objslc[s] * nvar + var[(long long)c * nobj + s]) * N;
		for (int dy = 0; dy < pool; dy++) {
			int y = (y0 + dy) % ny;
			if (y < 0) y += ny;
			for (int dx = 0; dx < pool; dx++) {
				int x = (x0 + dx) % nx;
				if (x < 0) x += nx;
				acc += __ldg(map + (long long)y * nx + x);
			}
		}
	}
	out[i] = acc / (float)((s1 - s0) * pool * pool);
}
inline int ok(cudaStream_t) { return cudaGetLastError() == cudaSuccess ? 0 : 1; }

} // namespace

extern "C" {

int JMS_NnConvForward(const void* x, const void* w, const float* bias, void* y, int B, int Ci, int H, int W, int Co,
	int relu, void* stream)
{
	if (!x || !w || !bias || !y || B < 1 || Ci < 1 || Co < 1 || H < 2 || W < 2 || (H & 1) || (W & 1)) return 2;
	cudaStream_t s = (cudaStream_t)stream;
	// 64-pixel tiles (four channels a thread) where they give every SM a CTA,
	// else 16-pixel tiles
	const long long npix = (long long)B * (H / 2) * (W / 2);
	const unsigned ncg = (unsigned)((Co + 15) / 16);
	const bool wide = (npix + 63) / 64 * ncg >= jms::kSMs;
	const long long tile = wide ? 64 : 16;
	auto kern = npix > kMaxPix32 ? k_conv_fwd<64, long long> : wide ? k_conv_fwd<64, int> : k_conv_fwd<16, int>;
	kern<<<dim3((unsigned)((npix + tile - 1) / tile), ncg), kNnThr, 0, s>>>((const __nv_bfloat16*)x,
		(const __nv_bfloat16*)w, bias, (__nv_bfloat16*)y, B, Ci, H, W, Co, relu);
	return ok(s);
}

int JMS_NnConvBackward(const void* x, const void* w, const void* y, const float* dy, float* dx, float* dw, float* db,
	int B, int Ci, int H, int W, int Co, int relu, void* stream)
{
	if (!x || !w || !y || !dy || !dw || !db || B < 1 || Ci < 1 || Co < 1 || (H & 1) || (W & 1)) return 2;
	cudaStream_t s = (cudaStream_t)stream;
	const long long npix = (long long)B * (H / 2) * (W / 2);
	const bool big = npix > kMaxPix32;
	if (dx)
		(big ? k_conv_bwd_data<long long> : k_conv_bwd_data<int>)<<<dim3((unsigned)((npix + 15) / 16), (unsigned)((Ci + 15) / 16)), kNnThr, 0, s>>>(dy,
			(const __nv_bfloat16*)y, (const __nv_bfloat16*)w, dx, B, Ci, H, W, Co, relu);
	const bool many = 3LL * Ci * ((Co + 3) / 4) >= 2 * jms::kSMs;
	auto pick = [&](auto i) {
		using I = decltype(i);
		return relu ? (many ? k_conv_bwd_weight<I, true, 4, 4> : k_conv_bwd_weight<I, true, 1, 8>)
			: (many ? k_conv_bwd_weight<I, false, 4, 4> : k_conv_bwd_weight<I, false, 1, 8>);
	};
	auto kern = big ? pick(0LL) : pick(0);
	const unsigned nq = (unsigned)(many ? (Co + 3) / 4 : Co);
	kern<<<dim3((unsigned)Ci, nq, 3), kNnThr, 0, s>>>((const __nv_bfloat16*)x, dy, (const __nv_bfloat16*)y, dw, db, B, Ci, H,
		W, Co);
	return ok(s);
}

int JMS_NnPoolLinearForward(const void* h, const float* wl, const float* bl, float* out, int B, int C, int HW, int O,
	void* stream)
{
	if (!h || !wl || !bl || !out || B < 1 || C < 1 || HW < 1 || O < 1 || C > 8192) return 2;
	cudaStream_t s = (cudaStream_t)stream;
	k_pool_linear_fwd<<<(unsigned)B, 128, sizeof(float) * C, s>>>((const __nv_bfloat16*)h, wl, bl, out, B, C, HW, O);
	return ok(s);
}

int JMS_NnPoolLinearBackward(const void* h, const float* wl, const float* dout, float* dh, float* dwl, float* dbl,
	int B, int C, int HW, int O, void* stream)
{
	if (!h || !wl || !dout || !dwl || !dbl || B < 1 || C < 1 || HW < 1 || O < 1) return 2;
	cudaStream_t s = (cudaStream_t)stream;
	if (dh) {
		const long long n = (long long)B * C * HW;
		k_pool_linear_bwd_data<<<nblk(n, 256), 256, 0, s>>>(wl, dout, dh, B, C, HW, O);
	}
	k_pool_linear_bwd_weight<<<(unsigned)(C / 16 + 1) * (unsigned)((O + 15) / 16), kNnThr, 0, s>>>((const __nv_bfloat16*)h,
		dout, dwl, dbl, B, C, HW, O);
	return ok(s);
}

int JMS_NnMseLoss(const float* out, const float* target, float* dout, float* loss, int n, void* stream)
{
	if (!out || !target || !dout || n < 1) return 2;
	cudaStream_t s = (cudaStream_t)stream;
	if (loss) cudaMemsetAsync(loss, 0, sizeof(float), s);
	k_mse<<<nblk(n, 256), 256, 0, s>>>(out, target, dout, loss, n);
	return ok(s);
}

int JMS_NnAdam(float* p, const float* g, float* m, float* v, void* p_bf16, int n, float lr, float b1, float b2,
	float eps, int step, void* stream)
{
	if (!p || !g || !m || !v || n < 1 || step < 1) return 2;
	cudaStream_t s = (cudaStream_t)stream;
	const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
	k_adam<<<nblk(n, 256), 256, 0, s>>>(p, g, m, v, (__nv_bfloat16*)p_bf16, n, lr, b1, b2, eps, c1, c2);
	return ok(s);
}

int JMS_NnAdamSet(int nset, float* const* p, const float* const* g, float* const* m, float* const* v,
	void* const* p_bf16, const int* n, float lr, float b1, float b2, float eps, int step, void* stream)
{
	if (nset < 1 || nset > kAdamMax || !p || !g || !m || !v || !n || step < 1) return 2;
	AdamSet a = {};
	int most = 0;
	for (int t = 0; t < nset; t++) {
		if (!p[t] || !g[t] || !m[t] || !v[t] || n[t] < 1) return 2;
		a.p[t] = p[t];
		a.g[t] = g[t];
		a.m[t] = m[t];
		a.v[t] = v[t];
		a.pb[t] = p_bf16 ? (__nv_bfloat16*)p_bf16[t] : nullptr;
		a.n[t] = n[t];
		most = n[t] > most ? n[t] : most;
	}
	cudaStream_t s = (cudaStream_t)stream;
	const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
	k_adam_set<<<dim3(nblk(most, 256), nset), 256, 0, s>>>(a, lr, b1, b2, eps, c1, c2);
	return ok(s);
}

int JMS_NnPatches(const float* pot, int ntype, int nvar, int nx, int ny, const int* objslc, int nobj, const int* var,
	int nconf, const int* pix, int npos, int nbins, int win, int pool, float* out, void* stream)
{
	if (!pot || !objslc || !var || !pix || !out || ntype < 1 || nvar < 1 || nx < 1 || ny < 1 || nobj < 1 ||
		nconf < 1 || npos < 1 || nbins < 1 || nbins > nobj || win < 1 || pool < 1 || win % pool)
		return 2;
	cudaStream_t s = (cudaStream_t)stream;
	const long long m = win / pool, n = (long long)nconf * npos * nbins * m * m;
	k_patches<<<nblk(n, 256), 256, 0, s>>>(pot, nvar, nx, ny, objslc, nobj, var, nconf, pix, npos, nbins, win, pool,
		out);
	return ok(s);
}

int JMS_NnCastBf16(const float* src, void* dst, long long n, void* stream)
{
	if (!src || !dst || n < 1) return 2;
	cudaStream_t s = (cudaStream_t)stream;
	k_cast_bf16<<<nblk(n, 256), 256, 0, s>>>(src, (__nv_bfloat16*)dst, n);
	return ok(s);
}

} // extern "C"
