// jms_passes.cuh -- fused FP32 multislice pass kernels (templates) for sm_100a.
//
// Included by the jms_inst_*.cu files, which instantiate the launchers for
// their share of the supported line lengths; jms_kernels.cu dispatches on the
// grid size.  See jms_kernels.h for the pass structure and jms_fft.cuh for the
// in-register DFTs.  Reference semantics followed here:
//   slice loop order          src/JMultiSlice.cpp:4590-4651 (GPUMultislice)
//   Fourier-space readout     src/JMultiSlice.cpp:4218-4367 (ReadoutDifDet_d)
//   real-space readout        src/JMultiSlice.cpp:4369-4465 (ReadoutImgDet_d)
//   grating multiply          src/cu/ArrayOps.cu:202-234 (MulKernel / sub-frame)
//   probe offset              src/JMultiSlice.cpp:1961-2084, src/cu/ArrayOps.cu:340-421
//
// Line transforms.  A line of N = A*B points is held by B threads, thread j
// owning x[j + B m] (m < A): loads and stores of that layout are coalesced.
// A transform runs in two register stages around one shared-memory exchange
// and leaves the line in a "middle" layout, where the pass applies its
// elementwise work (x P and Fourier readout, or real-space readout and x t);
// the opposite-direction transform then returns the line to the load layout.
//   split 1 (A, B any):  the middle layout has A threads per line, thread k1
//       holding X[k1 + A k2] (k2 < B); threads k1 >= A idle in the middle.
//   split 2 (B = 2A):   the B-point stage is shared by a thread pair with a
//       radix-2 step over warp shuffles, so every thread keeps A values in all
//       stages: thread (k1, h) = 2 k1 + h holds X[k1 + A (k + A h)], k < A.
// In the row passes a line whose threads fit in one warp in every stage
// (split 2, split 1 with A = B, and split 1 with B > A on a row tile of B
// threads per line) exchanges under warp barriers only, so the warps of a CTA
// run their lines independently; column lines span the CTA's warps and take
// CTA barriers.  Stage twiddles come from a shared copy (TwShared).
//
// A launch of many waves holds two of them per thread (cpair, jms_fft.cuh) in
// packed arithmetic: 61 thread instructions per element of the column pass
// against 84 with one wave.  Per 512-wave launch at 512^2 the column pass takes
// 424 us against 505, the row pass 278 against 311 (16 warps of 128 registers
// per SM against 32 of 64).  No pipe is full: of a 256-wave launch (ncu) the
// column pass keeps issue 44 %, FMA 46 %, shared memory 59 % and DRAM 31 % busy,
// the row pass 45, 53, 74 and 53 %, and the longest stall of both is for global
// loads.  The form before the early gratings took 377 of its 449 us without any
// wave loads and stores.  Measured slower: 8 x 8 x 8 lines (589 / 510 us),
// 4 or 16 columns of pairs per tile (476, 604), fewer registers with spills
// (513, 649), and the halves of one line as a pair in place of two waves
// (440 / 328).
#pragma once
#include "jms_fft.cuh"
#include "jms_kernels.h"
#include "jms_sizes.h"

namespace jms {

// ---------------------------------------------------------------------------
// tiles: thread <-> (line, position) maps and exchange-buffer layouts
// ---------------------------------------------------------------------------
// Row tile: LINES rows per CTA; thread t -> (line t / P, position t % P) for a
// role of P threads per line, or (line t / W, position t % W) in every role
// when the tile has a fixed line width W (positions P ... W - 1 then idle).
template <int LINES, int W = 0>
struct RowTile {
	static constexpr int kLines = LINES;
	static constexpr int kWidth = W;
	static constexpr int kPartner = 1;   // lane distance of positions 2k and 2k+1
	template <int P>
	__device__ __forceinline__ static void role(int tid, int& line, int& pos)
	{
		static_assert(W == 0 || P <= W, "a role wider than the tile's lines");
		constexpr int Q = W > 0 ? W : P;
		line = tid / Q;
		pos = tid % Q;
	}
	// Lines of P threads (P dividing 32) lie inside one warp, and so do their
	// exchange regions: a transform whose stages keep that role needs only
	// warp barriers, and the warps of a CTA run their lines independently.
	template <int P>
	__host__ __device__ static constexpr bool warp_lines() { return 32 % (W > 0 ? W : P) == 0; }
	// Lines of two or more whole warps synchronise by themselves (barriers 1 to 15).
	template <int P>
	__host__ __device__ static constexpr bool own_barrier() { return W == 0 && P > 32 && P % 32 == 0 && LINES <= 15; }
	// split 1 exchange S(line, k1, j), k1 < A, j < B, rows of odd length.  A
	// line's region has the same size for <A, B> and <B, A> (the forward and
	// inverse exchanges), so with warp-local lines one line's inverse exchange
	// never writes into another line's forward exchange.
	template <int A, int B>
	__host__ __device__ static constexpr int pad_line() { return A * (B | 1) > B * (A | 1) ? A * (B | 1) : B * (A | 1); }
	template <int A, int B>
	__device__ __forceinline__ static int s_pad(int line, int k1, int j) { return line * pad_line<A, B>() + k1 * (B | 1) + j; }
	template <int A, int B>
	static constexpr int sm_pad() { return LINES * pad_line<A, B>(); }
	// split 2 exchanges S(line, a, b), a < A, b < B, rows padded to B+2: the
	// pair reads of a half warp (a = 0..7, b = 2i + h) land on 16 distinct
	// bank pairs, and every per-thread loop has a constant address stride
	//   forward: a = k1, b = j (written by j, read by the pair (k1, h) at j = 2i + h)
	//   inverse: a = n1, b = q2 (written by the pair (n1, h) at q2 = 2m + h, read by q2)
	template <int A, int B>
	__device__ __forceinline__ static int s_fwd(int line, int a, int b) { return (line * A + a) * (B + 2) + b; }
	template <int A, int B>
	__device__ __forceinline__ static int s_inv(int line, int q2, int n1) { return (line * A + n1) * (B + 2) + q2; }
	template <int A, int B>
	static constexpr int sm_split() { return LINES * A * (B + 2); }
	// 3-stage exchanges for N = R^3 (see fft3): S1(line, k1, t) and
	// S2(line, k1, k2, j) in separate regions; the strides make the 16 lanes
	// of a half warp (k1 = t mod R fastest) hit distinct bank pairs
	template <int R>
	__host__ __device__ static constexpr int s3a_row() { return R * R + ((16 / R - R * R) % 16 + 16) % 16; }   // = 16/R mod 16
	template <int R>
	__host__ __device__ static constexpr int s3b_j() { return R + ((1 - R) % 16 + 16) % 16; }                    // = 1 mod 16
	template <int R>
	__host__ __device__ static constexpr int s3b_k1()
	{
		constexpr int base = R * s3b_j<R>();
		return base + ((16 / R - base) % 16 + 16) % 16;                                          // = 16/R mod 16
	}
	template <int R>
	__host__ __device__ static constexpr int s3_line() { return R * s3a_row<R>() + R * s3b_k1<R>(); }
	template <int R>
	__device__ __forceinline__ static int s3a(int line, int k1, int t) { return line * s3_line<R>() + k1 * s3a_row<R>() + t; }
	template <int R>
	__device__ __forceinline__ static int s3b(int line, int k1, int k2, int j)
	{
		return line * s3_line<R>() + R * s3a_row<R>() + k1 * s3b_k1<R>() + k2 * s3b_j<R>() + j;
	}
	template <int R>
	static constexpr int sm3() { return LINES * s3_line<R>(); }
};

// Column tile: C columns per CTA; thread t -> (column t % C, position t / C),
// so a warp touches C consecutive complex values of a few rows.  Exchange
// buffers keep the column index fastest; a pad of C complex per k1 block keeps
// the k1 groups of a half warp on distinct banks when C < 16.
template <int C>
struct ColTile {
	static constexpr int kLines = C;
	static constexpr int kPartner = C;
	static constexpr int PAD = (C < 16) ? C : 0;
	static constexpr int kWidth = 0;
	template <int P>
	__device__ __forceinline__ static void role(int tid, int& line, int& pos) { line = tid % C; pos = tid / C; }
	template <int P>
	__host__ __device__ static constexpr bool warp_lines() { return false; }   // a column's positions span warps
	template <int P>
	__host__ __device__ static constexpr bool own_barrier() { return false; }
	template <int A, int B>
	__device__ __forceinline__ static int s_pad(int line, int k1, int j) { return k1 * (B * C + PAD) + j * C + line; }
	template <int A, int B>
	static constexpr int sm_pad() { return A * (B * C + PAD); }
	template <int A, int B>
	__device__ __forceinline__ static int s_fwd(int line, int k1, int j) { return k1 * (B * C + PAD) + j * C + line; }
	template <int A, int B>
	__device__ __forceinline__ static int s_inv(int line, int q2, int n1) { return n1 * (B * C + PAD) + q2 * C + line; }
	template <int A, int B>
	static constexpr int sm_split() { return A * (B * C + PAD); }
	// 3-stage exchanges: S1(c, k1, t) then S2(c, k1, k2, j), column fastest
	template <int R>
	__device__ __forceinline__ static int s3a(int line, int k1, int t) { return k1 * (R * R * C + PAD) + t * C + line; }
	template <int R>
	__device__ __forceinline__ static int s3b(int line, int k1, int k2, int j)
	{
		return R * (R * R * C + PAD) + k1 * (R * R * C + PAD) + (k2 * R + j) * C + line;
	}
	template <int R>
	static constexpr int sm3() { return 2 * R * (R * R * C + PAD); }
};

// Barrier around an exchange of lines of P threads: a warp barrier (which also
// orders the warp's shared-memory accesses) when every line and its exchange
// region lie inside one warp, a named barrier of the line's own where it is a
// few whole warps, else a CTA barrier.
template <class Tile, int P>
__device__ __forceinline__ void line_sync()
{
	if constexpr (Tile::template warp_lines<P>()) __syncwarp();
	else if constexpr (Tile::template own_barrier<P>())
		asm volatile("bar.sync %0, %1;\n" ::"r"(1 + (int)threadIdx.x / P), "n"(P) : "memory");
	else __syncthreads();
}

// twiddle by table value w = exp(-2 pi i k / N) (conjugated for the inverse)
template <bool INV, class V>
__device__ __forceinline__ V tw_mul(V v, float2 w) { return INV ? cmulc(v, w) : cmul(v, w); }

// Stage twiddles W_N^(a b), a on the A-point side of a plan and b on the
// B-point side: from the N-entry table in global memory (read-only path), or
// from a CTA's shared copy laid out [a][b] with rows of ROW.  A 64-bit shared
// access is served per half warp, whose 16 lanes need distinct bank pairs.
// Split 2 reads W^(k1 j) over consecutive j and W^(n1 q2) over the pairs
// (n1 < 8, h; q2 = 2m + h) at ROW n1 + h + 2m: ROW = B + 2 = 2 mod 16 keeps
// both distinct (with rows of B+1 the lanes (n1, 1) and (n1 + 1, 0) collided).
// Split 1 reads along either index, so its rows are odd.
struct TwGlobal {
	const float2* p;
	__device__ __forceinline__ float2 operator()(int a, int b) const { return __ldg(p + a * b); }
};
template <int ROW>
struct TwShared {
	const float2* s;
	__device__ __forceinline__ float2 operator()(int a, int b) const { return s[a * ROW + b]; }
};
template <class TW>
struct TwSwapped {   // the same table with its indices exchanged
	TW t;
	__device__ __forceinline__ float2 operator()(int a, int b) const { return t(b, a); }
};
// Fills a shared [A][ROW] twiddle copy from the global table; the caller
// places a CTA barrier before its first use.
template <int A, int B, int ROW, int NT>
__device__ __forceinline__ void fill_tw_shared(float2* tws, const float2* __restrict__ tw, int tid)
{
	for (int i = tid; i < A * ROW; i += NT) {
		const int a = i / ROW, b = i - a * ROW;
		tws[i] = b < B ? __ldg(tw + a * b) : make_float2(0.f, 0.f);
	}
}
struct NoPrefetch {
	__device__ __forceinline__ void operator()() const {}
};

// ---- split 1 -----------------------------------------------------------------
// in: B threads/line, thread j holds x[j + B m] (m < A)
// out: A threads/line, thread k1 holds X[k1 + A k2] (k2 < B)
// LAST: no further exchange follows, so the reads need no barrier after them.
// prefetch() runs once the exchange is read: loads it issues overlap the
// second DFT.
template <int A, int B, bool INV, bool LAST, class Tile, class V, int RM, class TW, class PF>
__device__ __forceinline__ void fft_s1(V (&v)[RM], V* sm, const TW& tw, int tid, const PF& prefetch)
{
	int line, j;
	Tile::template role<B>(tid, line, j);
	const bool in_role = line < Tile::kLines && j < B;
	if (in_role) {
		dft_reg<A, 1, 0, INV>(v);
		#pragma unroll
		for (int k1 = 1; k1 < A; k1++) v[k1] = tw_mul<INV>(v[k1], tw(k1, j));
		#pragma unroll
		for (int k1 = 0; k1 < A; k1++) sm[Tile::template s_pad<A, B>(line, k1, j)] = v[k1];
	}
	// with A = B, or a tile whose lines keep max(A, B) threads in every role,
	// both stages give a line the same threads, so a line inside a warp
	// exchanges under a warp barrier
	constexpr int P = A > B ? A : B;
	constexpr bool same = A == B || Tile::kWidth >= P;
	auto sync = [] {
		if constexpr (same) line_sync<Tile, P>();
		else __syncthreads();
	};
	sync();
	Tile::template role<A>(tid, line, j);
	const bool out_role = line < Tile::kLines && j < A;
	if (out_role) {
		#pragma unroll
		for (int jj = 0; jj < B; jj++) v[jj] = sm[Tile::template s_pad<A, B>(line, j, jj)];
	}
	if constexpr (!LAST) sync();
	prefetch();
	if (out_role) dft_reg<B, 1, 0, INV>(v);
}

// ---- split 2 (B = 2A) ------------------------------------------------------------
// in: B threads/line, thread j holds x[j + B m] (m < A)
// out: B threads/line, thread (k1, h) = 2 k1 + h holds X[k1 + A (k + A h)] (k < A)
template <int A, bool INV, class Tile, class V, int RM, class TW, class PF>
__device__ __forceinline__ void fft_s2_fwd(V (&v)[RM], V* sm, const TW& tw, int tid, const PF& prefetch)
{
	constexpr int B = 2 * A;
	int line, j;
	Tile::template role<B>(tid, line, j);
	dft_reg<A, 1, 0, INV>(v);
	#pragma unroll
	for (int k1 = 1; k1 < A; k1++) v[k1] = tw_mul<INV>(v[k1], tw(k1, j));
	#pragma unroll
	for (int k1 = 0; k1 < A; k1++) sm[Tile::template s_fwd<A, B>(line, k1, j)] = v[k1];
	line_sync<Tile, B>();
	const int k1 = j >> 1, h = j & 1;
	#pragma unroll
	for (int i = 0; i < A; i++) v[i] = sm[Tile::template s_fwd<A, B>(line, k1, 2 * i + h)];
	line_sync<Tile, B>();
	prefetch();
	dft_reg<A, 1, 0, INV>(v);
	// radix-2 across the pair: Y[k] = E[k] + W_B^k O[k], Y[k + A] = E[k] - W_B^k O[k].
	// The odd thread twiddles its own value before the exchange, so both
	// threads finish with one sign-weighted add: u + o (h = 0), o - u (h = 1).
	const float sgn = h ? -1.f : 1.f;
	static_for<A>([&](auto K) {
		constexpr int k = K.value;
		const V u = h ? twiddle_ct<k, B, INV>(v[k]) : v[k];
		v[k] = cfma(sgn, u, cshfl_xor(u, Tile::kPartner));
	});
}

// in: B threads/line, thread (n1, h) = 2 n1 + h holds x[n1 + A (k + A h)] (k < A)
// out: B threads/line, thread j holds y[j + B m] (m < A)
template <int A, bool INV, class Tile, class V, int RM, class TW>
__device__ __forceinline__ void fft_s2_inv(V (&v)[RM], V* sm, const TW& tw, int tid)
{
	constexpr int B = 2 * A;
	int line, j;
	Tile::template role<B>(tid, line, j);
	const int n1 = j >> 1, h = j & 1;
	// radix-2 decimation in frequency over n2 = k + A h across the pair:
	// v + o (h = 0), W_B^k (o - v) (h = 1)
	const float sgn = h ? -1.f : 1.f;
	static_for<A>([&](auto K) {
		constexpr int k = K.value;
		const V d = cfma(sgn, v[k], cshfl_xor(v[k], Tile::kPartner));
		v[k] = h ? twiddle_ct<k, B, INV>(d) : d;
	});
	dft_reg<A, 1, 0, INV>(v);   // output q2 = 2 m + h
	#pragma unroll
	for (int m = 0; m < A; m++) {
		const int q2 = 2 * m + h;
		if (n1 > 0) v[m] = tw_mul<INV>(v[m], tw(n1, q2));
		sm[Tile::template s_inv<A, B>(line, q2, n1)] = v[m];
	}
	line_sync<Tile, B>();
	#pragma unroll
	for (int i = 0; i < A; i++) v[i] = sm[Tile::template s_inv<A, B>(line, j, i)];
	dft_reg<A, 1, 0, INV>(v);
}

// ---- 3 stages, N = R^3 ---------------------------------------------------------
// T = R^2 threads per line; thread t holds x[t + T m] (m < R) on entry and
// X[t + T k3] (k3 < R) on exit, so the transform maps its layout onto itself.
//   stage A: R-point DFT over m, twiddle W_N^(t k1), exchange S1;
//   stage B: thread (k1 = t mod R, j = t / R) takes Y[k1][j + R m'], R-point
//            DFT over m', twiddle W_N^(R j k2), exchange S2;
//   stage C: thread (k1, k2 = t / R) takes the R values over j, R-point DFT.
// S1 and S2 are separate regions, so two barriers per transform suffice.
template <int R, bool INV, class Tile, class V, int RM, class TW>
__device__ __forceinline__ void fft3(V (&v)[RM], V* sm, const TW& tw, int tid)
{
	constexpr int T = R * R;
	int line, t;
	Tile::template role<T>(tid, line, t);
	dft_reg<R, 1, 0, INV>(v);
	#pragma unroll
	for (int k1 = 1; k1 < R; k1++) v[k1] = tw_mul<INV>(v[k1], tw(t, k1));
	#pragma unroll
	for (int k1 = 0; k1 < R; k1++) sm[Tile::template s3a<R>(line, k1, t)] = v[k1];
	line_sync<Tile, T>();
	const int k1 = t % R, jj = t / R;
	#pragma unroll
	for (int m = 0; m < R; m++) v[m] = sm[Tile::template s3a<R>(line, k1, jj + R * m)];
	dft_reg<R, 1, 0, INV>(v);
	#pragma unroll
	for (int k2 = 1; k2 < R; k2++) v[k2] = tw_mul<INV>(v[k2], tw(R * jj, k2));
	#pragma unroll
	for (int k2 = 0; k2 < R; k2++) sm[Tile::template s3b<R>(line, k1, k2, jj)] = v[k2];
	line_sync<Tile, T>();
	#pragma unroll
	for (int j = 0; j < R; j++) v[j] = sm[Tile::template s3b<R>(line, k1, jj, j)];
	dft_reg<R, 1, 0, INV>(v);
}

// ---- plans -------------------------------------------------------------------------
template <int A_, int B_, int CC_>
struct Plan {
	static constexpr int A = A_, B = B_, N = A_ * B_;
	static constexpr int S = (B_ == 2 * A_ && A_ >= 4) ? 2 : 1;
	static constexpr int RM = (S == 2) ? A_ : (A_ > B_ ? A_ : B_);   // registers per thread (complex)
	static constexpr int T = B_;                                       // threads per line (load layout)
	static constexpr int TMID = (S == 2) ? B_ : A_;                    // threads per line (middle layout)
	static constexpr int EMID = (S == 2) ? A_ : B_;                    // values per thread (middle layout)
	static constexpr int TMAX = (T > TMID) ? T : TMID;
	static constexpr int CC = CC_;                                     // columns per column-pass CTA
	// the passes keep a shared [A][ROW] copy of the stage twiddles
	static constexpr bool SMEM_TW = true;
	static constexpr int ROW = S == 2 ? B_ + 2 : (B_ | 1);
	static constexpr int TWS = A_ * ROW;
	// line index of the e-th middle value of position pos
	__device__ __forceinline__ static int mid(int pos, int e)
	{
		if constexpr (S == 2) return (pos >> 1) + A * (e + A * (pos & 1));
		else return pos + A * e;
	}
	template <bool INV, class Tile, class V, class TW, class PF = NoPrefetch>
	__device__ __forceinline__ static void to_mid(V (&v)[RM], V* sm, const TW& tw, int tid, const PF& prefetch = PF{})
	{
		if constexpr (S == 2) fft_s2_fwd<A, INV, Tile>(v, sm, tw, tid, prefetch);
		else fft_s1<A, B, INV, false, Tile>(v, sm, tw, tid, prefetch);
	}
	// the last exchange of a pass
	template <bool INV, class Tile, class V, class TW>
	__device__ __forceinline__ static void from_mid(V (&v)[RM], V* sm, const TW& tw, int tid)
	{
		if constexpr (S == 2) fft_s2_inv<A, INV, Tile>(v, sm, tw, tid);
		else fft_s1<B, A, INV, true, Tile>(v, sm, TwSwapped<TW>{tw}, tid, NoPrefetch{});
	}
	// Threads per line of the row tile in every role: a split-1 plan with
	// B > A gives its middle role (A threads) the load role's B threads, A of
	// them active, so a line keeps its threads through both stages; 15, 24 and
	// 30 threads are rounded up to 16 and 32, so the line stays inside a warp
	// too; 0 (the role's own count) otherwise.
	static constexpr int ROWW = (S == 1 && B_ > A_) ? (B_ == 15 ? 16 : B_ == 30 || B_ == 24 ? 32 : B_) : 0;
	static constexpr int ROWT = ROWW > 0 ? ROWW : TMAX;               // row-tile threads per line
	// every exchange of to_mid / from_mid takes only warp barriers (a split-1
	// plan with A > B changes the threads of a line between its stages and
	// keeps CTA barriers)
	template <class Tile>
	__host__ __device__ static constexpr bool warp_local()
	{
		if constexpr (S == 2 || A_ == B_) return Tile::template warp_lines<B>();
		else return Tile::kWidth >= B_ && B_ > A_ && Tile::template warp_lines<B>();
	}
	template <class Tile>
	static constexpr int smem_elems()
	{
		if constexpr (S == 2) return Tile::template sm_split<A, B>();
		else {
			constexpr int a = Tile::template sm_pad<A, B>(), b = Tile::template sm_pad<B, A>();
			return a > b ? a : b;
		}
	}
};

// Three equal radices: N = R^3, R^2 threads per line with R values each; the
// middle layout equals the load layout.
template <int R_, int CC_ = 8>
struct Plan3 {
	static constexpr int R = R_, N = R_ * R_ * R_;
	static constexpr int A = R_, B = R_ * R_;            // load layout: thread j holds x[j + B m], m < A
	static constexpr int RM = R_, T = B, TMID = B, EMID = R_, TMAX = B;
	static constexpr int CC = CC_;
	static constexpr int ROWW = 0, ROWT = TMAX;
	static constexpr bool SMEM_TW = false;
	static constexpr int TWS = 1, ROW = 1;
	__device__ __forceinline__ static int mid(int pos, int e) { return pos + B * e; }
	template <bool INV, class Tile, class V, class TW, class PF = NoPrefetch>
	__device__ __forceinline__ static void to_mid(V (&v)[RM], V* sm, const TW& tw, int tid, const PF& prefetch = PF{})
	{
		fft3<R_, INV, Tile>(v, sm, tw, tid);
		prefetch();
	}
	template <bool INV, class Tile, class V, class TW>
	__device__ __forceinline__ static void from_mid(V (&v)[RM], V* sm, const TW& tw, int tid)
	{
		// the second transform writes S1 before its first barrier; the barriers
		// of the first transform already ordered all reads of S1 before it
		fft3<R_, INV, Tile>(v, sm, tw, tid);
	}
	template <class Tile>
	__host__ __device__ static constexpr bool warp_local() { return Tile::template warp_lines<B>(); }
	template <class Tile>
	static constexpr int smem_elems() { return Tile::template sm3<R_>(); }
};

__host__ __device__ constexpr int gcd_ct(int a, int b) { return b == 0 ? a : gcd_ct(b, a % b); }
// rows per row-pass CTA: about 256 threads, a whole number of warps
template <class PL>
__host__ __device__ constexpr int row_lines()
{
	constexpr int T = PL::ROWT;
	constexpr int m = 32 / gcd_ct(T, 32);
	constexpr int l = (256 / T) / m * m;
	return l < m ? m : l;
}
template <class PL>
__host__ __device__ constexpr int row_threads() { return row_lines<PL>() * PL::ROWT; }
// the row tile of a plan
template <class PL>
using RowTileOf = RowTile<row_lines<PL>(), PL::ROWW>;
// rows of a narrow CTA of about 64 threads, for launches that would leave SMs
// idle (one wave of 512^2: 43 CTAs with live rows, 171 narrow ones)
template <class PL>
__host__ __device__ constexpr int narrow_lines()
{
	constexpr int m = 32 / gcd_ct(PL::ROWT, 32);
	constexpr int l = (64 / PL::ROWT) / m * m;
	return l < m ? m : l;
}

// ---------------------------------------------------------------------------
// one wave or two waves per element
// ---------------------------------------------------------------------------
// A pass runs on single waves (V = float2, work buffer [nwave][ny][nx]) or on
// pairs of consecutive waves (V = cpair, work buffer [ceil(nwave / 2)][ny][nx]
// of cpair; with an odd count the last pair's second place repeats its first
// wave and is not read out).
template <class V> struct Waves;
template <> struct Waves<float2> { static constexpr int kN = 1; };
template <> struct Waves<cpair> { static constexpr int kN = 2; };

template <class V> __device__ __forceinline__ V join(float2 a, float2 b);
template <> __device__ __forceinline__ float2 join<float2>(float2 a, float2) { return a; }
template <> __device__ __forceinline__ cpair join<cpair>(float2 a, float2 b)
{
	return {make_float2(a.x, b.x), make_float2(a.y, b.y)};
}
__device__ __forceinline__ float2 load_v(const float2* p) { return *p; }
__device__ __forceinline__ cpair load_v(const cpair* p)
{
	const float4 q = *reinterpret_cast<const float4*>(p);
	return {make_float2(q.x, q.y), make_float2(q.z, q.w)};
}
__device__ __forceinline__ void store_v(float2* p, float2 v) { *p = v; }
__device__ __forceinline__ void store_v(cpair* p, cpair v)
{
	*reinterpret_cast<float4*>(p) = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}
// Programmatic launches: a pass lets the next one start once all its CTAs run
// (its twiddles, and single waves' gratings and propagators, are then loaded
// while this one finishes), and waits for the previous one's results before it
// touches the waves.  Every CTA waits, also one with nothing to do, so a pass
// never ends before the one ahead of it.
__device__ __forceinline__ void pass_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pass_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// the exchange buffer of a pass
template <class V>
__device__ __forceinline__ V* pass_smem()
{
	extern __shared__ float4 sm_pass[];
	return reinterpret_cast<V*>(sm_pass);
}

// ---------------------------------------------------------------------------
// readouts
// ---------------------------------------------------------------------------
// Detector sums: a thread adds its elements of a row in FP32, everything beyond
// is added in FP64, so the result does not depend on how rows and lanes are
// grouped (to 1e-16).
__device__ __forceinline__ double warp_sum(double v)
{
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}
__device__ __forceinline__ float fma_w(float pw, float w, float s) { return fmaf(pw, w, s); }
__device__ __forceinline__ float2 fma_w(float2 pw, float w, float2 s) { return __ffma2_rn(pw, bcast(w), s); }

// Scrambled pixel index at which psi(ky = y, kx) is read out, after the
// integer-pixel diffraction descan (DescanDifN, src/JMultiSlice.cpp:2184-2273:
// psi(kx, ky) is read out at pixel (kx - dnx, ky - dny), periodic)
__device__ __forceinline__ void readout_pixel(const PassArgs& p, int& y, int& kx)
{
	if (p.descan_x | p.descan_y) {
		kx -= p.descan_x; kx %= p.nx; if (kx < 0) kx += p.nx;
		y -= p.descan_y; y %= p.ny; if (y < 0) y += p.ny;
	}
}

// Adds w * f(e), e < E, to the elements idx(e) of a channel: all loads, then all
// stores (one element after the other, each load would wait for the store
// before it).
template <int E, class F, class IX>
__device__ __forceinline__ void add_channel(float* ch, float w, const F& f, const IX& idx)
{
	float old[E];
	#pragma unroll
	for (int e = 0; e < E; e++) old[e] = ch[idx(e)];
	#pragma unroll
	for (int e = 0; e < E; e++) ch[idx(e)] = old[e] + w * f(e);
}
template <int E, class F, class IX>
__device__ __forceinline__ void add_channel(float2* ch, float w, const F& f, const IX& idx)
{
	float2 old[E];
	#pragma unroll
	for (int e = 0; e < E; e++) old[e] = ch[idx(e)];
	#pragma unroll
	for (int e = 0; e < E; e++) ch[idx(e)] = __ffma2_rn(f(e), make_float2(w, w), old[e]);
}

// Adds weight * pw of pixel (y, kx) to the binned pattern of wave b's position.
__device__ __forceinline__ void readout_bin(const PassArgs& p, int b, int y, int kx, float pw)
{
	readout_pixel(p, y, kx);
	// unscrambled position (zero beam at nx/2, ny/2 as GetUnscrambleHash,
	// src/JMultiSlice.cpp:1932-1958), then bin x bin pixel blocks
	int ux = kx + (p.nx >> 1); if (ux >= p.nx) ux -= p.nx;
	int uy = y + (p.ny >> 1); if (uy >= p.ny) uy -= p.ny;
	int bx = ux / p.bin, by = uy / p.bin;
	const int bp = p.wave_pos > 0 ? b % p.wave_pos : b;   // the wave's probe position
	if (bx < p.nbx && by < p.nby)
		atomicAdd(p.bin_out + ((long long)bp * p.nby + by) * p.nbx + bx, p.weight * pw);
}

// Fourier-space readout of a row tile: thread (y, live) holds the E values v of
// row y at columns kx_of(e); b0 is the (first) wave.  Called by every thread
// of the CTA.  CHAN: with the channels of a single wave, whose loads in flight
// take 114 registers at 512 points (without them it is 64, and none spills).
template <bool CHAN, int NT, int E, class V, int RM, class KX>
__device__ __forceinline__ void readout_rows(const PassArgs& p, int b0, int y, bool live, const V (&v)[RM], const KX& kx_of)
{
	constexpr int NW = Waves<V>::kN;
	// channels in loops of their own (uniform tests)
	if constexpr (CHAN && NW == 1) {
		if ((p.dif || p.dif_avg || p.wff || p.wff_avg) && live) {
			// diffraction and wave channels (ReadoutDifDet_d, src/JMultiSlice.cpp:4277-4359)
			const long long c = (long long)b0 * p.chan_wstride + (long long)p.plane * p.nx * p.ny;
			auto idx = [&](int e) {
				int yd = y, kx = kx_of(e);
				readout_pixel(p, yd, kx);
				return yd * p.nx + kx;
			};
			auto pw = [&](int e) { return cnorm(v[e]); };
			auto psi = [&](int e) { return v[e]; };
			if (p.dif) add_channel<E>(p.dif + c, p.weight, pw, idx);
			if (p.dif_avg) add_channel<E>(p.dif_avg + c, p.weight, pw, idx);
			if (p.wff) add_channel<E>(p.wff + c, p.weight, psi, idx);
			if (p.wff_avg) add_channel<E>(p.wff_avg + c, p.weight, psi, idx);
		}
	}
	const bool two = NW == 2 && b0 + 1 < p.nwave;
	if (p.bin_out && p.plane == p.bin_plane && live) {
		#pragma unroll
		for (int e = 0; e < E; e++) {
			if constexpr (NW == 1) readout_bin(p, b0, y, kx_of(e), cnorm(v[e]));
			else {
				const float2 pw = cnorm(v[e]);
				readout_bin(p, b0, y, kx_of(e), pw.x);
				if (two) readout_bin(p, b0 + 1, y, kx_of(e), pw.y);
			}
		}
	}
	// integrating detectors one at a time (a rolled loop): unrolled over the
	// detectors, the compiler kept every element's detector loads in flight
	// (128 registers, half the plain pass's occupancy).  Each warp's sums wait
	// in shared memory for one CTA barrier after the last detector.
	__shared__ double red[NT / 32][kMaxDet * NW];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	#pragma unroll 1
	for (int d = 0; d < p.ndet; d++) {
		const float* det = p.det + (long long)d * p.nx * p.ny;   // detector d: [ny][nx]
		if constexpr (NW == 1) {
			float s = 0.f;
			if (live) {
				#pragma unroll
				for (int e = 0; e < E; e++) {
					int yd = y, kx = kx_of(e);
					readout_pixel(p, yd, kx);
					s = fma_w(cnorm(v[e]), __ldg(det + yd * p.nx + kx), s);
				}
			}
			const double t = warp_sum((double)s);
			if (lane == 0) red[warp][d] = t;
		}
		else {
			float2 s = make_float2(0.f, 0.f);
			if (live) {
				#pragma unroll
				for (int e = 0; e < E; e++) {
					int yd = y, kx = kx_of(e);
					readout_pixel(p, yd, kx);
					s = fma_w(cnorm(v[e]), __ldg(det + yd * p.nx + kx), s);
				}
			}
			const double t0 = warp_sum((double)s.x), t1 = warp_sum((double)s.y);
			if (lane == 0) { red[warp][2 * d] = t0; red[warp][2 * d + 1] = t1; }
		}
	}
	if (p.ndet > 0) {
		__syncthreads();
		const int d = threadIdx.x / NW, w = threadIdx.x % NW;
		if (d < p.ndet && (w == 0 || two)) {
			double t = 0.0;
			#pragma unroll
			for (int k = 0; k < NT / 32; k++) t += red[k][threadIdx.x];
			p.partial[(((long long)(b0 + w) * p.ndetslc + p.plane) * p.ndet + d) * p.nblk + blockIdx.x] = t;
		}
	}
}

// Real-space readout of the E values v of column x at rows y_of(e) of wave b
// (ReadoutImgDet_d, src/JMultiSlice.cpp:4392-4459).
template <int E, int RM, class YY>
__device__ __forceinline__ void readout_cols(const PassArgs& p, int b, int x, const float2 (&v)[RM], const YY& y_of)
{
	const long long c = (long long)b * p.chan_wstride + (long long)p.plane * p.nx * p.ny + x;
	auto idx = [&](int e) { return y_of(e) * p.nx; };
	auto pw = [&](int e) { return cnorm(v[e]); };
	auto psi = [&](int e) { return v[e]; };
	if (p.img) add_channel<E>(p.img + c, p.weight, pw, idx);
	if (p.img_avg) add_channel<E>(p.img_avg + c, p.weight, pw, idx);
	if (p.wfr) add_channel<E>(p.wfr + c, p.weight, psi, idx);
	if (p.wfr_avg) add_channel<E>(p.wfr_avg + c, p.weight, psi, idx);
}

// offset phase plate exp(-i (2 pi turns + cppl)) at scrambled pixel (i, j);
// turns = fi dx/a + fj dy/b + fz (fi^2/a^2 + fj^2/b^2) is formed in FP64 and
// reduced mod 1 before the FP32 sincos (large k.dx phases keep full accuracy).
__device__ __forceinline__ float2 offset_factor(const double* sh, int i, int j, int nx, int ny, float cp)
{
	// signed frequency index (i + n/2) mod n - n/2 of bin i < n, without a division
	const int fi = i < nx - (nx >> 1) ? i : i - nx;
	const int fj = j < ny - (ny >> 1) ? j : j - ny;
	const double di = (double)fi, dj = (double)fj;
	double t = di * sh[0] + dj * sh[1] + di * di * sh[2] + dj * dj * sh[3];
	t -= floor(t);
	float s, c;
	if (cp != 0.f) {
		sincosf(6.283185307179586f * (float)t + cp, &s, &c);
	}
	else {
		sincospif(2.f * (float)t, &s, &c);
	}
	return make_float2(c, -s);
}

// Element kx of row y of wave b at the entry: the incident wave with the probe
// offset (phase only where the probe is nonzero, inside its aperture), the wave
// at wav0, or the work buffer's.
template <int N>
__device__ __forceinline__ float2 entry_source(const PassArgs& p, int b, int y, int kx)
{
	if (p.shift) {
		int sx = kx, sy = y;
		if (p.ibtx | p.ibty) {   // beam tilt: a periodic shift of the incident wave (uniform branch)
			sx -= p.ibtx; sx %= N; if (sx < 0) sx += N;
			sy -= p.ibty; sy %= p.ny; if (sy < 0) sy += p.ny;
		}
		const float2 a = __ldg(p.wav0 + (long long)sy * N + sx);
		if (a.x == 0.f && a.y == 0.f) return a;
		const float cp = p.cppl ? __ldg(p.cppl + (long long)y * N + kx) : 0.f;
		return cmul(a, offset_factor(p.shift + 4 * b, kx, y, N, p.ny, cp));
	}
	return p.wav0 ? __ldg(p.wav0 + (long long)y * N + kx) : p.work[(long long)b * p.wstride + (long long)y * N + kx];
}

// ---------------------------------------------------------------------------
// pass kernels (template parameters: the line plan of the transformed axis and
// the element type V)
// ---------------------------------------------------------------------------
// Entry row pass: [offset] -> Fourier readout (plane) -> IFT_x.
template <class PL, class V>
__global__ void __launch_bounds__(row_threads<PL>())
k_entry_rows(const PassArgs p)
{
	constexpr int N = PL::N, L = row_lines<PL>(), NT = L * PL::ROWT, NW = Waves<V>::kN;
	using T = RowTileOf<PL>;
	V* sm = pass_smem<V>();
	const int tid = threadIdx.x, b = blockIdx.y * NW, row0 = blockIdx.x * L;
	const int b1 = min(b + 1, p.nwave - 1);
	const int nval = min(L, p.ny - row0);
	// Rows outside the source's band of live rows (row_k1 / row_k2: the
	// incident wave's all-zero rows, for scans without beam tilt) are zero: a
	// CTA of such rows does nothing, and they are neither read, read out nor
	// stored (the first column pass reads them as zero).
	if (row0 > p.row_k1 && row0 + nval - 1 < p.row_k2) return;
	V* W = reinterpret_cast<V*>(p.work) + (long long)blockIdx.y * p.wstride;
	V v[PL::RM];
	#pragma unroll
	for (int m = 0; m < PL::RM; m++) v[m] = czero<V>();
	int line, j;
	T::template role<PL::T>(tid, line, j);
	const bool live = line < nval && j < PL::T && (row0 + line <= p.row_k1 || row0 + line >= p.row_k2);
	const int y = row0 + line;
	if (live) {
		#pragma unroll
		for (int m = 0; m < PL::A; m++) {
			const int kx = j + PL::B * m;
			if constexpr (NW == 1) v[m] = entry_source<N>(p, b, y, kx);
			else if (p.shift || p.wav0) v[m] = join<V>(entry_source<N>(p, b, y, kx), entry_source<N>(p, b1, y, kx));
			else v[m] = load_v(W + (long long)y * N + kx);
		}
	}
	if (p.plane >= 0) readout_rows<true, NT, PL::A>(p, b, y, live, v, [&](int m) { return j + PL::B * m; });
	PL::template to_mid<true, T>(v, sm, TwGlobal{p.twx}, tid);
	int pos;
	T::template role<PL::TMID>(tid, line, pos);
	if (line < nval && pos < PL::TMID && (row0 + line <= p.row_k1 || row0 + line >= p.row_k2)) {
		V* dst = W + (long long)(row0 + line) * N;
		#pragma unroll
		for (int e = 0; e < PL::EMID; e++) store_v(dst + PL::mid(pos, e), v[e]);
	}
}

// Row pass: FT_x -> x P -> Fourier readout (plane) -> IFT_x.  READ selects
// the variant with the readout code (used at readout planes only, as the
// kernel k_row_pass_read with launch bounds of its own), so the steps without
// readout do not carry its registers.
// L rows per CTA.  FEW: single waves that are all resident at once (few_waves).
// CHAN: the readout adds to channels too.
template <class PL, bool READ, class V, int L, bool FEW, bool CHAN>
__device__ __forceinline__ void row_pass_body(const PassArgs& p)
{
	constexpr int N = PL::N, NT = L * PL::ROWT;
	using T = RowTile<L, PL::ROWW>;
	V* sm = pass_smem<V>();
	const int tid = threadIdx.x, row0 = blockIdx.x * L;
	const int nval = min(L, p.ny - row0);
	// rows outside the propagator's band end up exactly zero: a CTA whose rows
	// are all outside does nothing, and such rows are neither read nor stored
	// (the column pass reads them as zero)
	pass_trigger();
	if (row0 > p.row_k1 && row0 + nval - 1 < p.row_k2) {
		pass_wait();
		return;
	}
	__shared__ float2 tws[PL::TWS];
	const auto tw = [&] {
		if constexpr (PL::SMEM_TW) return TwShared<PL::ROW>{tws};
		else return TwGlobal{p.twx};
	}();
	V* W = reinterpret_cast<V*>(p.work) + (long long)blockIdx.y * p.wstride;
	V v[PL::RM];
	#pragma unroll
	for (int m = 0; m < PL::RM; m++) v[m] = czero<V>();
	int line, j;
	T::template role<PL::T>(tid, line, j);
	const int yl = row0 + line;
	const bool live = line < nval && j < PL::T && (yl <= p.row_k1 || yl >= p.row_k2);
	// a launch of few single waves is a chain of latencies: the propagator is
	// loaded ahead of the wait
	constexpr bool EARLY = FEW && !READ && PL::EMID <= 16;
	float2 w[EARLY ? PL::EMID : 1];
	if constexpr (EARLY) {
		int l2, pos;
		T::template role<PL::TMID>(tid, l2, pos);
		if (l2 < nval && pos < PL::TMID) {
			const float2* P = p.mul + (long long)(row0 + l2) * N;
			#pragma unroll
			for (int e = 0; e < PL::EMID; e++) w[e] = __ldg(P + PL::mid(pos, e));
		}
	}
	if constexpr (EARLY && PL::SMEM_TW) fill_tw_shared<PL::A, PL::B, PL::ROW, NT>(tws, p.twx, tid);
	pass_wait();
	if (live) {
		const V* src = W + (long long)yl * N;
		#pragma unroll
		for (int m = 0; m < PL::A; m++) v[m] = load_v(src + j + PL::B * m);
	}
	// the twiddle copy is filled while the row loads are in flight, so the
	// barrier waits for both latencies at once
	if constexpr (PL::SMEM_TW) {
		if constexpr (!EARLY) fill_tw_shared<PL::A, PL::B, PL::ROW, NT>(tws, p.twx, tid);
		__syncthreads();
	}
	// with warp-local lines and no CTA-wide readout, a warp whose lines are
	// all dead (band gap, past the last row) has nothing more to do
	if constexpr (!READ && PL::template warp_local<T>())
		if (__all_sync(0xffffffffu, !live)) return;
	PL::template to_mid<false, T>(v, sm, tw, tid);
	{
		int pos;
		T::template role<PL::TMID>(tid, line, pos);
		const bool mid_live = line < nval && pos < PL::TMID;
		const int y = row0 + line;
		if (mid_live) {
			const float2* P = p.mul + (long long)y * N;
			#pragma unroll
			for (int e = 0; e < PL::EMID; e++) {
				if constexpr (EARLY) v[e] = cmul(v[e], w[e]);
				else v[e] = cmul(v[e], __ldg(P + PL::mid(pos, e)));
			}
		}
		if constexpr (READ)
			readout_rows<CHAN, NT, PL::EMID>(p, blockIdx.y * Waves<V>::kN, y, mid_live, v,
				[&](int e) { return PL::mid(pos, e); });
	}
	if (!p.store) return;
	PL::template from_mid<true, T>(v, sm, tw, tid);
	if (live) {
		V* dst = W + (long long)yl * N;
		#pragma unroll
		for (int m = 0; m < PL::A; m++) store_v(dst + j + PL::B * m, v[m]);
	}
}

// Resident CTAs asked of the readout kernel: for plans of at most 16 values
// a thread (whose plain pass takes 64 registers) the plain pass's count, so
// the readout code spills a few bytes instead of halving the occupancy;
// larger plans are held to about 112 registers.
template <class PL>
__host__ __device__ constexpr int read_min_blocks()
{
	return 65536 / (row_threads<PL>() * (PL::RM <= 16 ? 64 : 112)) > 0
		? 65536 / (row_threads<PL>() * (PL::RM <= 16 ? 64 : 112)) : 1;
}
// Resident CTAs asked of a plain pass of NT threads: the count at 64
// registers for plans of at most 16 values a thread, at 128 for larger ones.
// Left free, the compiler took 70 (512 rows), 142 (1024 rows) and 140 (1024
// columns) once the lines ran warp by warp and the twiddles came from shared
// memory, each dropping a resident CTA.
template <class PL, int NT>
__host__ __device__ constexpr int pass_min_blocks()
{
	return 65536 / (NT * (PL::RM <= 16 ? 64 : 128)) > 0 ? 65536 / (NT * (PL::RM <= 16 ? 64 : 128)) : 1;
}
template <class PL>
__host__ __device__ constexpr int row_min_blocks() { return pass_min_blocks<PL, row_threads<PL>()>(); }
// resident CTAs asked of a pass over wave pairs: at most 128 registers
template <int NT>
__host__ __device__ constexpr int pair_min_blocks() { return 65536 / (NT * 128) > 0 ? 65536 / (NT * 128) : 1; }
template <class PL, class V>
__host__ __device__ constexpr int row_blocks_sm(bool read)
{
	if (Waves<V>::kN == 2) return pair_min_blocks<row_threads<PL>()>();
	return read ? read_min_blocks<PL>() : row_min_blocks<PL>();
}
// Single waves of plans of at most 16 values a thread have two forms.  Where all
// waves of a launch are resident at once (kResidentPoints) it is a chain of
// latencies, and the propagators or gratings are loaded ahead of the wait, which
// takes 80 to 100 registers; a larger launch keeps to 64, since it needs the
// CTAs.  Us a slice, early loads against 64 registers: 64^2, 73 waves 5.0
// against 7.5, 192^2, 32 waves 10.8 / 14.1, 240^2, 27 waves 12.9 / 17.2, 256^2,
// 18 waves 9.5 / 13.8, 36 waves 16.8 / 17.2; 1024 x 512, 64 waves (512-point
// columns, one CTA per SM in place of two) 300 / 240.
inline bool few_waves(const PassArgs& p) { return (long long)p.nwave * p.nx * p.ny < kResidentPoints; }
// Narrow tiles (4 columns, or rows for about 64 threads) in place of ctas full
// ones: for lines of 256 or more up to 16 values a thread where the full tiles
// do not reach every SM (512^2, us a slice with full rows and columns, narrow
// rows, both narrow: one wave 12.6, 14.0, 11.0; four 19.7, 17.5, 16.6), for
// longer ones from 480 on where they leave a third of the SMs idle (480^2, one
// wave 12.9 / 12.1, 768^2 18.6 / 17.5; but 320^2 8.3 / 9.4, 384^2, two waves
// 10.1 / 13.2, 1024^2 22.1 / 23.1).
template <class PL>
constexpr bool has_narrow() { return PL::N >= (PL::RM <= 16 ? 256 : 480); }
template <class PL>
constexpr bool use_narrow(long long ctas) { return PL::RM <= 16 ? ctas < kSMs : 3 * ctas <= 2 * kSMs; }
constexpr int kNarrow = 4;
// plain row pass; the readout planes use k_row_pass_read
template <class PL, class V, int L, bool FEW>
__global__ void __launch_bounds__(L * PL::ROWT, FEW ? 0 : row_blocks_sm<PL, V>(false))
k_row_pass(const PassArgs p)
{
	row_pass_body<PL, false, V, L, FEW, false>(p);
}
template <class PL, class V, bool CHAN>
__global__ void __launch_bounds__(row_threads<PL>(), CHAN ? 0 : row_blocks_sm<PL, V>(true))
k_row_pass_read(const PassArgs p)
{
	row_pass_body<PL, true, V, row_lines<PL>(), false, CHAN>(p);
}

// Live rows of a column-pass thread as a bit mask: bit m is set when row
// y = j + B m (m < A) lies outside the band gap (k1, k2), i.e. y <= k1 or
// y >= k2.  One mask per thread replaces a comparison per element.
template <int A, int B>
__device__ __forceinline__ unsigned live_rows(int j, int k1, int k2)
{
	static_assert(A <= 32, "one bit per value");
	const int lo = k1 >= j ? min((k1 - j) / B, A - 1) : -1;          // last m with y <= k1
	const int hi = k2 > j ? min((k2 - j + B - 1) / B, 32) : 0;       // first m with y >= k2
	const unsigned low = lo < 0 ? 0u : (lo >= 31 ? 0xffffffffu : ((2u << lo) - 1u));
	const unsigned high = hi >= 32 ? 0u : (0xffffffffu << hi);
	return low | high;
}

// exp(2 pi i (sx x / nx + sy y / ny)): the real-space ramp of a plasmon shift
__device__ __forceinline__ float2 plasmon_ramp(int sx, int sy, int x, int y, int nx, int ny)
{
	const float tx = (float)(int)(((long long)sx * x) % nx) / (float)nx;
	const float ty = (float)(int)(((long long)sy * y) % ny) / (float)ny;
	float sn, cs;
	sincospif(2.f * (tx + ty), &sn, &cs);
	return make_float2(cs, sn);
}

// Columns per column-pass CTA: of single waves the plan's own, of wave pairs
// half of it, so a CTA holds the same shared memory and half the threads; a
// narrow tile where a launch would leave SMs idle.
template <class PL, class V>
__host__ __device__ constexpr int col_width(bool narrow)
{
	return narrow && PL::CC / Waves<V>::kN > kNarrow ? kNarrow : PL::CC / Waves<V>::kN;
}

// Column pass: IFT_y -> real-space readout (plane) -> x t -> FT_y.  NXC is the
// row stride when it is known at compile time (square grids, nx = N), so the
// element offsets of the wave and grating accesses are constants; 0 reads it
// from the arguments.
// The pass on one tile (grid row blockIdx.y, columns col0 ... col0 + C - 1).
// SYNC places a CTA barrier between the wave loads and the first transform
// (which makes a shared twiddle copy filled just before visible).
// Up to 16 grating values a thread are loaded into registers early: for wave
// pairs and plans of more values before the second DFT, whose arithmetic hides
// the loads' latency (512^2 pairs, 512 waves: 449 -> 424 us; 1024^2, 128 waves:
// 533 -> 503 us), for other single waves in launches of few (FEW) ahead of
// everything else.
template <class PL, class V, int C, bool READ, int NXC, bool FEW, bool SYNC, class TW>
__device__ __forceinline__ void col_pass_tile(const PassArgs& p, int col0, const TW& tw, V* sm)
{
	constexpr int NW = Waves<V>::kN;
	// values loaded early
	constexpr int PRE = READ || (NW == 1 && PL::EMID <= 16 && !FEW) ? 0 : PL::EMID <= 16 ? PL::EMID : 16;
	constexpr bool EARLY = PRE > 0;
	static_assert(!(READ && NW == 2), "images are read out of single waves only");
	using T = ColTile<C>;
	const int tid = threadIdx.x, b = blockIdx.y * NW;
	const int b1 = min(b + 1, p.nwave - 1);
	const int nx = NXC > 0 ? NXC : p.nx;
	const int nval = min(C, nx - col0);
	V* W = reinterpret_cast<V*>(p.work) + (long long)blockIdx.y * p.wstride + col0;
	V v[PL::RM];
	#pragma unroll
	for (int m = 0; m < PL::RM; m++) v[m] = czero<V>();
	int c, j;
	T::template role<PL::T>(tid, c, j);
	// element offsets of the waves' gratings
	const int o0 = p.mul_w ? __ldg(p.mul_w + b) : 0, o1 = NW == 2 && p.mul_w ? __ldg(p.mul_w + b1) : o0;
	const bool full = p.npgx == nx && p.npgy == p.ny;   // grating of the grid size
	const bool early = EARLY && full && o0 == o1;
	int cm, pos;
	T::template role<PL::TMID>(tid, cm, pos);
	const bool mid_live = cm < nval && pos < PL::TMID;
	const int x = col0 + cm;
	float2 t[EARLY ? PRE : 1];
	auto load_t = [&] {
		if constexpr (EARLY) {
			if (early && mid_live) {
				const float2* g = p.mul + o0 + x;
				#pragma unroll
				for (int e = 0; e < PRE; e++) t[e] = __ldg(g + PL::mid(pos, e) * nx);
			}
		}
	};
	if constexpr (NW == 1 && PL::EMID <= 16) load_t();   // few single waves: ahead of the wait
	pass_wait();
	// 32-bit offsets within a wave (nx * ny < 2^31): one base pointer per
	// thread and a row stride, instead of a 64-bit product per element
	const int stride = PL::B * nx;
	if (c < nval && j < PL::T) {
		const V* src = W + j * nx + c;
		const unsigned lin = live_rows<PL::A, PL::B>(j, p.in_k1, p.in_k2);
		#pragma unroll
		for (int m = 0; m < PL::A; m++)
			if (lin & (1u << m)) v[m] = load_v(src + m * stride);
	}
	if constexpr (SYNC) __syncthreads();
	PL::template to_mid<true, T>(v, sm, tw, tid, [&] {
		if constexpr (NW == 2 || PL::EMID > 16) load_t();
	});
	if (mid_live) {
		if constexpr (READ) readout_cols<PL::EMID>(p, b, x, v, [&](int e) { return PL::mid(pos, e); });
		const float2* mul = p.mul + o0;
		if (early) {
			if constexpr (EARLY) {
				#pragma unroll
				for (int e = 0; e < PL::EMID; e++)
					v[e] = e < PRE ? cmul(v[e], t[e < PRE ? e : 0]) : cmul(v[e], __ldg(mul + x + PL::mid(pos, e) * nx));
			}
		}
		else if (NW == 1 || o0 == o1) {
			if (full) {
				#pragma unroll
				for (int e = 0; e < PL::EMID; e++) v[e] = cmul(v[e], __ldg(mul + x + PL::mid(pos, e) * nx));
			}
			else { // sub-frame grating repeated periodically
				const int xs = x % p.npgx;
				#pragma unroll
				for (int e = 0; e < PL::EMID; e++)
					v[e] = cmul(v[e], __ldg(mul + (long long)(PL::mid(pos, e) % p.npgy) * p.npgx + xs));
			}
		}
		else if constexpr (NW == 2) { // the two waves are of different configurations
			const float2* mul1 = p.mul + o1;
			const int xs = full ? x : x % p.npgx;
			#pragma unroll
			for (int e = 0; e < PL::EMID; e++) {
				const int y = PL::mid(pos, e);
				const int q = (full ? y : y % p.npgy) * p.npgx + xs;
				v[e] = cmul(v[e], __ldg(mul + q), __ldg(mul1 + q));
			}
		}
		int sx = p.plas_x, sy = p.plas_y, sx1 = NW == 2 ? sx : 0, sy1 = NW == 2 ? sy : 0;
		if (p.plas_w) {
			sx = __ldg(p.plas_w + 2 * b); sy = __ldg(p.plas_w + 2 * b + 1);
			if constexpr (NW == 2) { sx1 = __ldg(p.plas_w + 2 * b1); sy1 = __ldg(p.plas_w + 2 * b1 + 1); }
		}
		if (sx | sy | sx1 | sy1) { // plasmon shift of the spectrum (uniform branch)
			#pragma unroll
			for (int e = 0; e < PL::EMID; e++) {
				const int y = PL::mid(pos, e);
				const float2 r = plasmon_ramp(sx, sy, x, y, nx, p.ny);
				if constexpr (NW == 1) v[e] = cmul(v[e], r);
				else v[e] = cmul(v[e], r, plasmon_ramp(sx1, sy1, x, y, nx, p.ny));
			}
		}
	}
	PL::template from_mid<false, T>(v, sm, tw, tid);
	T::template role<PL::T>(tid, c, j);
	if (c < nval && j < PL::T) {
		V* dst = W + j * nx + c;
		const unsigned lout = live_rows<PL::A, PL::B>(j, p.out_k1, p.out_k2);
		#pragma unroll
		for (int m = 0; m < PL::A; m++)
			if (lout & (1u << m)) store_v(dst + m * stride, v[m]);
	}
}

// Resident CTAs asked of a column pass: wave pairs at most 128 registers; many
// single waves as the row pass; few are free.
template <class PL, class V, int C>
__host__ __device__ constexpr int col_blocks_sm(bool read, bool few)
{
	constexpr int NT = C * PL::TMAX;
	if (Waves<V>::kN == 2) return pair_min_blocks<NT>();
	return read || (few && PL::RM <= 16) ? 0 : pass_min_blocks<PL, NT>();
}
template <class PL, class V, int C, bool READ, int NXC, bool FEW>
__global__ void __launch_bounds__(C * PL::TMAX, col_blocks_sm<PL, V, C>(READ, FEW))
k_col_pass(const PassArgs p)
{
	pass_trigger();
	V* sm = pass_smem<V>();
	__shared__ float2 tws[PL::TWS];
	if constexpr (PL::SMEM_TW) {
		fill_tw_shared<PL::A, PL::B, PL::ROW, C * PL::TMAX>(tws, p.twy, threadIdx.x);   // barrier after the wave loads
		col_pass_tile<PL, V, C, READ, NXC, FEW, true>(p, blockIdx.x * C, TwShared<PL::ROW>{tws}, sm);
	}
	else col_pass_tile<PL, V, C, READ, NXC, FEW, false>(p, blockIdx.x * C, TwGlobal{p.twy}, sm);
}

// Exit column pass: IFT_y -> real-space readout (plane), no store.
template <class PL>
__global__ void __launch_bounds__(PL::CC * PL::TMAX)
k_exit_cols(const PassArgs p)
{
	constexpr int C = PL::CC;
	using T = ColTile<C>;
	float2* sm = pass_smem<float2>();
	const int tid = threadIdx.x, b = blockIdx.y, col0 = blockIdx.x * C;
	const int nval = min(C, p.nx - col0);
	const int nx = p.nx;
	const float2* W = p.work + (long long)b * p.wstride + col0;
	float2 v[PL::RM];
	#pragma unroll
	for (int m = 0; m < PL::RM; m++) v[m] = make_float2(0.f, 0.f);
	int c, j;
	T::template role<PL::T>(tid, c, j);
	if (c < nval && j < PL::T) {
		#pragma unroll
		for (int m = 0; m < PL::A; m++) {
			const int y = j + PL::B * m;
			if (y <= p.in_k1 || y >= p.in_k2) v[m] = W[(long long)y * nx + c];
		}
	}
	PL::template to_mid<true, T>(v, sm, TwGlobal{p.twy}, tid);
	int pos;
	T::template role<PL::TMID>(tid, c, pos);
	if (c < nval && pos < PL::TMID) readout_cols<PL::EMID>(p, b, col0 + c, v, [&](int e) { return PL::mid(pos, e); });
}

// ---------------------------------------------------------------------------
// launchers (explicitly instantiated per size in jms_inst_*.cu)
// ---------------------------------------------------------------------------
// closes a group of cp.async copies (the phase-grating synthesis stages its
// atom chunks with them)
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

// chained: a pass kernel that waits for the one ahead of it itself (pass_wait)
template <class PL, class K>
cudaError_t launch_k(K kern, dim3 grid, int threads, int smem, const PassArgs& p, cudaStream_t s, bool chained = false)
{
	static_assert(sizeof(PassArgs) < 4000, "kernel parameter block too large");
	// the limit of 48 KB without this call includes a kernel's static part: at
	// most the twiddle copy and the detector sums of 16 warps
	constexpr int fixed = PL::TWS * (int)sizeof(float2) + 16 * 2 * kMaxDet * (int)sizeof(double);
	if (smem + fixed > 48 * 1024) {
		cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
		if (e != cudaSuccess) return e;
	}
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = dim3(threads);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cudaLaunchAttribute at;
	at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at.val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = &at;
	cfg.numAttrs = chained ? 1 : 0;
	return cudaLaunchKernelEx(&cfg, kern, p);
}

template <class PL>
int row_blocks_t(int ny) { return (ny + row_lines<PL>() - 1) / row_lines<PL>(); }

// grid rows: waves, or pairs of waves
template <class V>
unsigned wave_rows(const PassArgs& p) { return (unsigned)((p.nwave + Waves<V>::kN - 1) / Waves<V>::kN); }

template <class PL, class V>
cudaError_t launch_entry_t(const PassArgs& p, cudaStream_t s)
{
	constexpr int L = row_lines<PL>();
	constexpr int smem = PL::template smem_elems<RowTileOf<PL>>() * (int)sizeof(V);
	return launch_k<PL>(k_entry_rows<PL, V>, dim3((p.ny + L - 1) / L, wave_rows<V>(p)), L * PL::ROWT, smem, p, s);
}
template <class PL, class V>
cudaError_t launch_row_t(const PassArgs& p, cudaStream_t s)
{
	constexpr int L = row_lines<PL>();
	constexpr int smem = PL::template smem_elems<RowTileOf<PL>>() * (int)sizeof(V);
	const dim3 grid((p.ny + L - 1) / L, wave_rows<V>(p));
	if (p.plane >= 0) {
		// Channels come with runs of one wave.  Plans of at most 16 values take
		// that form for few waves too: its registers keep all of a detector's
		// loads in flight, and two CTAs are resident on an SM.  Us a slice with a
		// readout in each, against the form without channels: 512^2, four waves
		// (170 CTAs of live rows) 19.6 / 25.2, six (255) 21.6 / 26.2, eight (341)
		// 28.1 / 26.7; 256^2, 24 waves (256) 18.1 / 22.0, 32 (341) 25.7 / 23.4.
		if constexpr (Waves<V>::kN == 1) {
			const int gap = p.row_k2 - p.row_k1 - 1;      // rows of the propagator's band gap
			const long long live = gap > 0 && gap < p.ny ? p.ny - gap : p.ny;
			if (p.dif || p.dif_avg || p.wff || p.wff_avg ||
				(PL::RM <= 16 && (long long)grid.x * p.nwave * live <= 2LL * kSMs * p.ny))
				return launch_k<PL>(k_row_pass_read<PL, V, true>, grid, L * PL::ROWT, smem, p, s, true);
		}
		return launch_k<PL>(k_row_pass_read<PL, V, false>, grid, L * PL::ROWT, smem, p, s, true);
	}
	if constexpr (Waves<V>::kN == 1) {
		if constexpr (has_narrow<PL>()) {
			constexpr int LN = narrow_lines<PL>();
			constexpr int smem_n = PL::template smem_elems<RowTile<LN, PL::ROWW>>() * (int)sizeof(V);
			if (use_narrow<PL>((long long)grid.x * p.nwave))
				return launch_k<PL>(k_row_pass<PL, V, LN, true>, dim3((p.ny + LN - 1) / LN, p.nwave), LN * PL::ROWT, smem_n, p, s, true);
		}
		if constexpr (PL::RM <= 16)
			if (few_waves(p)) return launch_k<PL>(k_row_pass<PL, V, L, true>, grid, L * PL::ROWT, smem, p, s, true);
	}
	return launch_k<PL>(k_row_pass<PL, V, L, false>, grid, L * PL::ROWT, smem, p, s, true);
}
template <class PL, class V, int C, bool READ, int NXC, bool FEW>
cudaError_t launch_col_c(const PassArgs& p, cudaStream_t s)
{
	constexpr int smem = PL::template smem_elems<ColTile<C>>() * (int)sizeof(V);
	return launch_k<PL>(k_col_pass<PL, V, C, READ, NXC, FEW>, dim3((p.nx + C - 1) / C, wave_rows<V>(p)), C * PL::TMAX, smem, p, s,
		true);
}
template <class PL, class V>
cudaError_t launch_col_t(const PassArgs& p, cudaStream_t s)
{
	constexpr int C = col_width<PL, V>(false), CN = col_width<PL, V>(true), N = PL::N;
	const bool square = p.nx == N;
	if constexpr (Waves<V>::kN == 1) {
		if (p.plane >= 0)
			return square ? launch_col_c<PL, V, C, true, N, false>(p, s) : launch_col_c<PL, V, C, true, 0, false>(p, s);
		// 256-point columns gain nothing by narrow tiles (4.5 us either way)
		if constexpr (has_narrow<PL>() && N >= 320) {
			if (use_narrow<PL>((long long)((p.nx + C - 1) / C) * p.nwave)) return launch_col_c<PL, V, CN, false, 0, true>(p, s);
		}
		else if constexpr (PL::RM <= 16) {
			if (few_waves(p))
				return square ? launch_col_c<PL, V, C, false, N, true>(p, s) : launch_col_c<PL, V, C, false, 0, true>(p, s);
		}
	}
	return square ? launch_col_c<PL, V, C, false, N, false>(p, s) : launch_col_c<PL, V, C, false, 0, false>(p, s);
}
template <class PL>
cudaError_t launch_exit_t(const PassArgs& p, cudaStream_t s)
{
	constexpr int C = PL::CC;
	constexpr int smem = PL::template smem_elems<ColTile<C>>() * (int)sizeof(float2);
	return launch_k<PL>(k_exit_cols<PL>, dim3((p.nx + C - 1) / C, p.nwave), C * PL::TMAX, smem, p, s);
}

// The passes of a plan.  Wave pairs need the plan's values twice in registers:
// plans of at most 16 values a thread have them.
template <class PL>
PlanOps plan_ops_t(int n, const char* name)
{
	PlanOps o = {n, name, &row_blocks_t<PL>, &launch_entry_t<PL, float2>, &launch_row_t<PL, float2>,
		&launch_col_t<PL, float2>, &launch_exit_t<PL>, nullptr, nullptr, nullptr};
	if constexpr (PL::RM <= 16) {
		o.entry2 = &launch_entry_t<PL, cpair>;
		o.row2 = &launch_row_t<PL, cpair>;
		o.col2 = &launch_col_t<PL, cpair>;
	}
	return o;
}

#define JMS_INSTANTIATE(PL) template PlanOps plan_ops_t<PL>(int, const char*);

} // namespace jms
