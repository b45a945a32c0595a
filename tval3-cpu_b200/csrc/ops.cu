// Measurement operators (sm_100a); see ops.cuh.
//
//   dense     y = A x: four warps per row, float4 loads (2d/mat_mult.h:18-21)
//             y = A^T x: blocks of (1024 columns x row chunk) write partial
//             column sums, a second pass adds the chunks in order
//   CSR       forward: sub-warp per row gather (mkl_csrmv, 2d/mat_mult.h:58-61);
//             adjoint: gather over the device-built CSC (mkl_cscmv, :63-66)
//   rays      forward: one thread per ray, or a few lanes per ray where there
//             are few rays, taking Bresenham steps in closed form
//             (2d/mat_mult.h:145-181, 3d/mat_mult.h:241-359);
//             adjoint: pixel-major gather over the ray->pixel index transposed
//             once on the device (deterministic, no atomics in the solve); in
//             2D per pixel tile, through shared memory
#include "ops.cuh"

#include <algorithm>
#include <vector>

#include "async.cuh"

TG_BEGIN

#define OPROLOGUE()                                                                   \
	pdl_launch_next();                                                                \
	if (launches && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(launches, 1ull);   \
	const int2 tl_ = map.tiles[blockIdx.x];                                           \
	const Inst &I = tab[tl_.x];                                                       \
	const long long local = tl_.y;                                                    \
	pdl_wait_prev();                                                                  \
	if (!pred_ok(*I.ctrl, pred)) return;

// ---------------------------------------------------------------------------
// dense
// ---------------------------------------------------------------------------
// y = A x, every product formed and added in FP64, WPR warps per row (which of
// the forms a launch takes: dense_form).  k_dense_fwd reads A and x straight
// from global memory; k_dense_fwd_smem, for long rows that are not float4
// aligned, has x converted once per block, chunk by chunk into shared memory.
// The segments of 32 elements (float4s) that a row is read in go to CLASSES
// classes in turn - four, fewer for long rows; lane l adds the l-th products of
// a class in order, then its classes' sums, then the lanes are added by halves:
// the same bits in a launch of few rows and of many.
// Bound: the float-to-double conversions (two a product; with x in shared memory
// one), A from memory where it is larger than L2; for few rows the loads in
// flight.  Measured, us (one warp a row in one class, straight from memory -> this):
//   few rows, aligned: 1229 x 4096 11.0 -> 5.8 (this with one warp a row 10.0),
//   4915 x 16384 116 -> 57 (77); not aligned: 1116 x 3721 9.4 -> 5.1 (9.7), 1968 x
//   6561 17.5 -> 10.9 (15.8), 3060 x 10201 35.8 -> 33 (34), 4839 x 16129 86 -> 66 (80)
//   many rows: 8 layers of 1228 x 4096 24.0 -> 23.6 (this with four warps a row
//   31), 16 of 188 x 625 5.3 -> 4.5 (8.1), of 1968 x 6561 103 -> 91 (two warps:
//   116), of 4836 x 16129 832 -> 767 (824)
//   FP64 build, an iteration of a solve: 1116 x 3721 33.0 with four warps, 34.6
//   with one; 1968 x 6561 67.1 with four classes, 64.6 with one; 2764 x 9216 103
//   and 100
// acc += the row's products, by class (XA: x is float4 aligned too)
template <int WPR, int CLASSES, bool XA>
__device__ __forceinline__ void dense_row4(const float4 *__restrict__ a, const float *__restrict__ x, int n4, int sub,
                                           double (&acc)[CLASSES / WPR]) {
	constexpr int STEP = 32 * WPR, U = 4, NC = CLASSES / WPR;
	auto load = [&](int j) {
		if (XA) return ld_vec(reinterpret_cast<const float4 *>(x) + j);
		const float *p = x + 4LL * j;
		return make_float4(ld_vec(p), ld_vec(p + 1), ld_vec(p + 2), ld_vec(p + 3));
	};
	auto add = [&](double &s, const float4 &av, const float4 &xv) {
		s = fma((double)av.x, (double)xv.x, s);
		s = fma((double)av.y, (double)xv.y, s);
		s = fma((double)av.z, (double)xv.z, s);
		s = fma((double)av.w, (double)xv.w, s);
	};
	int j = sub * 32 + (threadIdx.x & 31);
	for (; j + (U - 1) * STEP < n4; j += U * STEP) {   // U segments of the row in flight per lane
		float4 av[U], xv[U];
#pragma unroll
		for (int u = 0; u < U; u++) {
			av[u] = __ldg(a + j + u * STEP);
			xv[u] = load(j + u * STEP);
		}
#pragma unroll
		for (int u = 0; u < U; u++) add(acc[u % NC], av[u], xv[u]);
	}
#pragma unroll
	for (int u = 0; u < U - 1; u++)
		if (j + u * STEP < n4) add(acc[u % NC], __ldg(a + j + u * STEP), load(j + u * STEP));
}

// rows that are not float4 aligned and too short for shared memory (in the FP64
// build: all): element by element, U in flight per lane
template <int WPR, int CLASSES>
__device__ __forceinline__ void dense_row1d(const real *__restrict__ a, const real *__restrict__ x, int n, int sub,
                                            double (&acc)[CLASSES / WPR]) {
	constexpr int STEP = 32 * WPR, U = 8, NC = CLASSES / WPR;
	int j = sub * 32 + (threadIdx.x & 31);
	for (; j + (U - 1) * STEP < n; j += U * STEP) {
		real av[U], xv[U];
#pragma unroll
		for (int u = 0; u < U; u++) {
			av[u] = __ldg(a + j + u * STEP);
			xv[u] = ld_vec(x + j + u * STEP);
		}
#pragma unroll
		for (int u = 0; u < U; u++) acc[u % NC] = fma((double)av[u], (double)xv[u], acc[u % NC]);
	}
#pragma unroll
	for (int u = 0; u < U - 1; u++)
		if (j + u * STEP < n) acc[u % NC] = fma((double)__ldg(a + j + u * STEP), (double)ld_vec(x + j + u * STEP), acc[u % NC]);
}

#ifndef TVAL3G_FP64
// the same with x in shared memory.  CLASSES 4: segment by segment in turn, as
// above; 2: eight segments by eight, so that one warp a row adds each batch of
// loads in one chain (segment by segment, three layers of 4836 x 16129 took 196
// us instead of 167)
template <int WPR, int CLASSES>
__device__ __forceinline__ void dense_row1(const real *__restrict__ a, const real *__restrict__ x, int n, int sub,
                                           double *sx, double (&acc)[CLASSES / WPR]) {
	constexpr int CHUNK = DENSE_CHUNK, G = 8, GROUPS = CHUNK / (32 * WPR * G), NC = CLASSES / WPR;   // (CHUNK doubles: one buffer)
	constexpr bool TURN = CLASSES == 4;
	const int lane = threadIdx.x & 31;
	auto at = [&](int g, int u) { return (TURN ? (g * G + u) * WPR + sub : (g * WPR + sub) * G + u) * 32 + lane; };
	auto sum = [&](int g, int u) -> double & { return acc[(TURN ? u : g) % NC]; };
	real xv[CHUNK / 256];
	auto load_x = [&](int c) {
#pragma unroll
		for (int u = 0; u < CHUNK / 256; u++) {
			const int j = c * CHUNK + u * 256 + threadIdx.x;
			xv[u] = j < n ? ld_vec(x + j) : (real)0;
		}
	};
	load_x(0);
	const int nc = (int)((n + (CHUNK - 1LL)) / CHUNK);   // (the last chunk's end may lie beyond the largest int)
	for (int c = 0, buf = 0; c < nc; c++, buf ^= 1) {
		double *bx = sx + buf * CHUNK;
#pragma unroll
		for (int u = 0; u < CHUNK / 256; u++) bx[u * 256 + threadIdx.x] = (double)xv[u];
		if (c + 1 < nc) load_x(c + 1);
		const real *ac = a + (long long)c * CHUNK;
		const int len = n - c * CHUNK;
		if (len >= CHUNK) {
			real av[2][G];
#pragma unroll
			for (int u = 0; u < G; u++) av[0][u] = __ldg(ac + at(0, u));
			__syncthreads();
#pragma unroll
			for (int g = 0; g < GROUPS; g++) {
				if (g + 1 < GROUPS)
#pragma unroll
					for (int u = 0; u < G; u++) av[(g + 1) & 1][u] = __ldg(ac + at(g + 1, u));
#pragma unroll
				for (int u = 0; u < G; u++) sum(g, u) = fma((double)av[g & 1][u], bx[at(g, u)], sum(g, u));
			}
		} else {
			__syncthreads();
			constexpr int GS = TURN ? 1 : NC;   // groups until the classes repeat
			for (int g0 = 0; at(g0, 0) < len; g0 += GS)
#pragma unroll
				for (int g = 0; g < GS; g++)
#pragma unroll
					for (int u = 0; u < G; u++)
						if (at(g0 + g, u) < len)
							sum(g, u) = fma((double)__ldg(ac + at(g0 + g, u)), bx[at(g0 + g, u)], sum(g, u));
		}
	}
}
#endif

// the row of this thread's warp, one of WPR on it
template <int WPR, int CLASSES>
struct DenseRow {
	static constexpr int NC = CLASSES / WPR;   // classes of a warp: sub, sub + WPR, ...
	int n, sub;   // this warp: part sub of the row
	int out;             // its element of y; -1: beyond the last row (which is read again, not stored)
	const real *a, *x;
	double acc[NC] = {};
	__device__ __forceinline__ DenseRow(const Inst &I, const VecSel &xs, int local) {
		constexpr unsigned ROWS = WARPS / WPR;
		const unsigned m = (unsigned)I.op.m, rt = (m + ROWS - 1) / ROWS, warp = threadIdx.x >> 5;
		n = (int)I.op.n;
		sub = (int)(warp % WPR);
		const unsigned layer = (unsigned)local / rt, row = ((unsigned)local - layer * rt) * ROWS + warp / WPR;
		out = row < m ? (int)(layer * m + row) : -1;
		a = I.op.A + (long long)min(row, m - 1) * n;
		x = vsel(I, xs) + (long long)layer * n;
	}
	// y = the lanes' sums of the classes, in order, then the lanes by halves; the
	// warps of a row meet in shared memory before that
	__device__ __forceinline__ void store(const Inst &I, const VecSel &ys) {
		const int lane = threadIdx.x & 31;
		double t = acc[0];
		if (WPR == 1) {
#pragma unroll
			for (int k = 1; k < CLASSES; k++) t += acc[k < NC ? k : 0];
		} else {
			__shared__ double ws[WARPS / WPR][CLASSES][32];
			double(*w)[32] = ws[(threadIdx.x >> 5) / WPR];
#pragma unroll
			for (int k = 0; k < NC; k++) w[k * WPR + sub][lane] = acc[k];
			__syncthreads();
			if (sub) return;
			t = w[0][lane];
#pragma unroll
			for (int k = 1; k < CLASSES; k++) t += w[k][lane];
		}
		t = warp_sum(t);
		if (lane == 0 && out >= 0) vselw(I, ys)[out] = (real)t;
	}
};

template <int WPR, int CLASSES>
__global__ void __launch_bounds__(256, 4) k_dense_fwd(const Inst *tab, TileMap map, int pred, VecSel xs, VecSel ys,
                                                      unsigned long long *launches) {
	OPROLOGUE();
	DenseRow<WPR, CLASSES> r(I, xs, local);
#ifndef TVAL3G_FP64
	// the same choice in every thread of the block
	if ((r.n & 3) == 0 && (reinterpret_cast<uintptr_t>(I.op.A) & 15) == 0) {
		const float4 *a4 = reinterpret_cast<const float4 *>(r.a);
		if ((reinterpret_cast<uintptr_t>(r.x) & 15) == 0) dense_row4<WPR, CLASSES, true>(a4, r.x, r.n >> 2, r.sub, r.acc);
		else dense_row4<WPR, CLASSES, false>(a4, r.x, r.n >> 2, r.sub, r.acc);
	} else
#endif
		dense_row1d<WPR, CLASSES>(r.a, r.x, r.n, r.sub, r.acc);
	r.store(I, ys);
}

#ifndef TVAL3G_FP64
template <int WPR, int CLASSES>
__global__ void __launch_bounds__(256, 4) k_dense_fwd_smem(const Inst *tab, TileMap map, int pred, VecSel xs, VecSel ys,
                                                           unsigned long long *launches) {
	OPROLOGUE();
	__shared__ double sx[2 * DENSE_CHUNK];
	DenseRow<WPR, CLASSES> r(I, xs, local);
	dense_row1<WPR, CLASSES>(r.a, r.x, r.n, r.sub, sx, r.acc);
	r.store(I, ys);
}
#endif

// partial column sums of A^T x over one row chunk
__global__ void __launch_bounds__(256) k_dense_adj(const Inst *tab, TileMap map, int pred, VecSel xs,
                                                   VecSel ys, real *part, unsigned long long *launches) {
	OPROLOGUE();
	const OpDev &op = I.op;
	const long long m = op.m, n = op.n;
	const int K = op.dense_kchunks;
	const long long ct_n = (n + 1023) / 1024;
	const long long layer = local / (ct_n * K);
	const long long rem = local - layer * ct_n * K;
	const long long ct = rem / K, kc = rem - ct * K;
	const long long rows_per = (m + K - 1) / K;
	const long long r0 = kc * rows_per, r1 = min(m, r0 + rows_per);
	const long long c0 = ct * 1024 + threadIdx.x * 4;
	const real *x = vsel(I, xs) + layer * m;
	double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0, acc3 = 0.0;   // FP64 accumulation
	if (!FP64_BUILD && (n & 3) == 0 && (reinterpret_cast<uintptr_t>(op.A) & 15) == 0) {
		if (c0 < n) {
			long long r = r0;
			// four rows in flight per thread; the FMA order is the plain loop's
			for (; r + 3 < r1; r += 4) {
				real xv[4];
				float4 av[4];
#pragma unroll
				for (int u = 0; u < 4; u++) {
					xv[u] = ld_vec(x + r + u);
					av[u] = __ldg(reinterpret_cast<const float4 *>(op.A + (r + u) * n + c0));
				}
#pragma unroll
				for (int u = 0; u < 4; u++) {
					acc0 = fma((double)av[u].x, (double)xv[u], acc0);
					acc1 = fma((double)av[u].y, (double)xv[u], acc1);
					acc2 = fma((double)av[u].z, (double)xv[u], acc2);
					acc3 = fma((double)av[u].w, (double)xv[u], acc3);
				}
			}
			for (; r < r1; r++) {
				real xv = ld_vec(x + r);
				float4 av = __ldg(reinterpret_cast<const float4 *>(op.A + r * n + c0));
				acc0 = fma((double)av.x, (double)xv, acc0);
				acc1 = fma((double)av.y, (double)xv, acc1);
				acc2 = fma((double)av.z, (double)xv, acc2);
				acc3 = fma((double)av.w, (double)xv, acc3);
			}
		}
	} else {
		for (long long r = r0; r < r1; r++) {
			real xv = ld_vec(x + r);
			const real *ar = op.A + r * n;
			if (c0 + 0 < n) acc0 = fma((double)__ldg(ar + c0 + 0), (double)xv, acc0);
			if (c0 + 1 < n) acc1 = fma((double)__ldg(ar + c0 + 1), (double)xv, acc1);
			if (c0 + 2 < n) acc2 = fma((double)__ldg(ar + c0 + 2), (double)xv, acc2);
			if (c0 + 3 < n) acc3 = fma((double)__ldg(ar + c0 + 3), (double)xv, acc3);
		}
	}
	real *p = part + op.dense_part + (layer * K + kc) * n;
	if (c0 + 0 < n) p[c0 + 0] = (real)acc0;
	if (c0 + 1 < n) p[c0 + 1] = (real)acc1;
	if (c0 + 2 < n) p[c0 + 2] = (real)acc2;
	if (c0 + 3 < n) p[c0 + 3] = (real)acc3;
}

// y = sum of the K row-chunk partials, 32 columns per block: warp w adds the
// partials k = w, w + 8, ... of its lane's column, then warp 0 adds the eight
// warp sums in a fixed order (deterministic)
__global__ void __launch_bounds__(256) k_dense_red(const Inst *tab, TileMap map, int pred, VecSel xs, VecSel ys,
                                                   const real *part, unsigned long long *launches) {
	OPROLOGUE();
	__shared__ double ws[8][32];
	const OpDev &op = I.op;
	const long long n = op.n;
	const int K = op.dense_kchunks;
	const long long ct_n = (n + 31) / 32;
	const long long layer = local / ct_n, ct = local - layer * ct_n;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const long long c = ct * 32 + lane;
	const real *p = part + op.dense_part + layer * K * n;
	double s = 0.0;
	if (c < n)
		for (int k = warp; k < K; k += 8) s += p[(long long)k * n + c];
	ws[warp][lane] = s;
	__syncthreads();
	if (warp == 0 && c < n) {
		double t = ws[0][lane];
		for (int w = 1; w < 8; w++) t += ws[w][lane];
		vselw(I, ys)[layer * n + c] = (real)t;
	}
}

#ifndef TVAL3G_FP64   // one-pass dense normal product: FP32 data only
// ---------------------------------------------------------------------------
// dense normal product, A read once (get_g_mult's cache-blocked dense path,
// 2d/tval3_cpu_2d.cpp:361-394): Au = A u and g = A^T Au in one pass over A.
// A is cut into bands of R = grid x rpc rows; CTA c owns rows c rpc ..
// c rpc + rpc - 1 of every band and the column slab [c S, c S + S) of g.
// Each CTA's warps take three roles that run concurrently:
//   producer (warp 0): streams the CTA's rows, chunk by chunk, with the
//     matching chunk of u, into a ring of shared-memory stages by bulk
//     asynchronous copies (full / empty barriers per stage);
//   consumers (warps 1-7): the rows' dot products from the stages; thread 0
//     of the role writes each row of Au and, after the band's rows, publishes
//     them with a release increment of flags[band];
//   reducers (warps 8-15): band after band, once all rows of the band are
//     published, the slab of A_band^T Au_band added into FP64 accumulators
//     kept for the whole launch - the band is read again from L2, where the
//     producer just brought it.
// The producer starts band b only when its CTA's reducers have finished band
// b - 2, so two bands at most are in L2.  All CTAs must be co-resident
// (cooperative launch).  Every wait is bounded: one that gives up sets *err
// and the CTA's abort flag, after which no role waits again (every named
// barrier is still passed the same number of times) and the producer lets
// its copies in flight land before the CTA exits.  Products are summed in
// FP32 over short runs (a thread's share of one chunk of a row; eight rows of
// a column) and those sums in FP64, in a fixed order: deterministic.
// ---------------------------------------------------------------------------
constexpr int FUSED_THREADS = 512;
constexpr int FUSED_ROLE = 256;                     // reducer threads
constexpr int FUSED_CONS = 224;                     // consumer threads (warps 1-7)
constexpr int FUSED_RPC_MAX = 16;                   // rows per CTA per band
constexpr int FUSED_GRID_MAX = 160;
constexpr int FUSED_NS = 4;                         // ring stages
constexpr int FUSED_CH = 4096;                      // floats per chunk (16 KB of A, 16 KB of u)
constexpr int FUSED_STAGE_BYTES = 2 * FUSED_CH * 4;
constexpr int FUSED_DYN_BYTES = FUSED_NS * FUSED_STAGE_BYTES + 2 * FUSED_NS * 8;
constexpr long long FUSED_BAND_BYTES = 24LL << 20;  // target band size
constexpr long long FUSED_L2_BYTES = 96LL << 20;    // two bands must stay in L2
constexpr unsigned FUSED_SPIN_MAX = 1u << 21;       // bounded waits (~0.2 s)

__device__ __forceinline__ int ld_acquire(const int *p) {
	int v;
	asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void named_sync(int id, int threads) {   // barrier of one role's threads
	asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// one thread polls a stage barrier; false (err raised) if it gives up
__device__ __forceinline__ bool mbar_wait1(unsigned bar, unsigned parity, int *err) {
	for (unsigned i = 0; i < ASYNC_WAIT_LIMIT; i++)
		if (mbar_try(bar, parity)) return true;
	atomicExch(err, 1);
	return false;
}

__global__ void __launch_bounds__(FUSED_THREADS, 1) k_dense_normal(const Inst *tab, int inst, int pred, VecSel us,
                                                                   VecSel aus, VecSel gs, int *flags, int *err,
                                                                   unsigned long long *launches) {
	if (launches && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(launches, 1ull);
	const Inst &I = tab[inst];
	if (!pred_ok(*I.ctrl, pred)) return;   // the same in every CTA: ctrl is not written here
	extern __shared__ __align__(128) unsigned char dsm[];
	__shared__ float sauf[FUSED_GRID_MAX * FUSED_RPC_MAX];   // the band's Au (reducers)
	__shared__ double sau[FUSED_GRID_MAX * FUSED_RPC_MAX];   // the row groups' column sums
	__shared__ double spart[2][8];                           // consumer warps' row partials
	__shared__ volatile int s_done, s_abort;                 // bands reduced; a wait gave up
	const OpDev &op = I.op;
	const int m = (int)op.m, n = (int)op.n;
	const int G = gridDim.x, c = blockIdx.x, rpc = op.fused_rpc, R = G * rpc;
	const int nb = (m + R - 1) / R, nch = (n + FUSED_CH - 1) / FUSED_CH;
	const float *A = op.A;
	const int S = op.fused_slab;   // slab width, a multiple of 4
	const int c0 = min(n, c * S), c1 = min(n, c0 + S);
	const unsigned full0 = smem_u32(dsm + FUSED_NS * FUSED_STAGE_BYTES), empty0 = full0 + 8u * FUSED_NS;
	auto stage_a = [&](int st) { return reinterpret_cast<float4 *>(dsm + st * FUSED_STAGE_BYTES); };
	auto stage_u = [&](int st) { return reinterpret_cast<float4 *>(dsm + st * FUSED_STAGE_BYTES + FUSED_CH * 4); };
	if (threadIdx.x == 0) {
		s_done = 0;
		s_abort = 0;
		for (int st = 0; st < FUSED_NS; st++) {
			mbar_init(full0 + 8u * st, 1);
			mbar_init(empty0 + 8u * st, FUSED_CONS / 32);
		}
		fence_mbar_init();
	}
	__syncthreads();
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	if (warp == 0) {
		// ---- producer ----
		if (lane == 0) {
			const float *u = vsel(I, us);
			// A's lines are read again by the reducers of other CTAs (from L2):
			// kept there until then; u is read for every row
			const unsigned long long keep = l2_policy_evict_last();
			long long it = 0;
			for (int b = 0; b < nb && !s_abort; b++) {
				for (unsigned sp = 0; s_done < b - 1 && !s_abort; sp++) {
					if (sp > FUSED_SPIN_MAX) { atomicExch(err, 1); s_abort = 1; }
					__nanosleep(32);
				}
				const int r0 = b * R + c * rpc;
				for (int j = 0; j < rpc && r0 + j < m && !s_abort; j++)
					for (int ch = 0; ch < nch && !s_abort; ch++, it++) {
						const int st = (int)(it % FUSED_NS);
						const long long ph = it / FUSED_NS;
						if (ph > 0 && !mbar_wait1(empty0 + 8u * st, (unsigned)(ph - 1) & 1u, err)) {
							s_abort = 1;
							break;
						}
						const int cnt = min(FUSED_CH, n - ch * FUSED_CH);
						mbar_expect_tx(full0 + 8u * st, 8u * cnt);
						bulk_g2s_hint(smem_u32(stage_a(st)), A + (long long)(r0 + j) * n + (long long)ch * FUSED_CH,
						              4u * cnt, full0 + 8u * st, keep);
						bulk_g2s_hint(smem_u32(stage_u(st)), u + (long long)ch * FUSED_CH, 4u * cnt, full0 + 8u * st,
						              keep);
					}
			}
			if (s_abort)   // let the copies in flight land before the CTA exits (bounded)
				for (long long k = it > FUSED_NS ? it - FUSED_NS : 0; k < it; k++)
					mbar_wait1(full0 + 8u * (int)(k % FUSED_NS), (unsigned)(k / FUSED_NS) & 1u, err);
		}
	} else if (warp < 8) {
		// ---- consumers ----
		const int ct = threadIdx.x - 32, cw = warp - 1;
		float *au = vselw(I, aus);
		long long it = 0;
		int rowc = 0;
		for (int b = 0; b < nb; b++) {
			const int r0 = b * R + c * rpc;
			for (int j = 0; j < rpc && r0 + j < m; j++, rowc++) {
				double acc = 0.0;
				for (int ch = 0; ch < nch; ch++, it++) {
					const int st = (int)(it % FUSED_NS);
					if (!s_abort && !mbar_wait_warp(full0 + 8u * st, (unsigned)(it / FUSED_NS) & 1u, err))
						if (lane == 0) s_abort = 1;
					if (!s_abort) {
						// the thread's few products of this chunk (at most 19
						// float4) summed in FP32, the chunk sums in FP64: one
						// conversion per chunk instead of two per element
						const int cnt4 = min(FUSED_CH, n - ch * FUSED_CH) >> 2;
						const float4 *sa = stage_a(st), *su = stage_u(st);
						float pf = 0.f;
						for (int k = ct; k < cnt4; k += FUSED_CONS) {
							const float4 av = sa[k], uv = su[k];
							pf = fmaf(av.x, uv.x, pf);
							pf = fmaf(av.y, uv.y, pf);
							pf = fmaf(av.z, uv.z, pf);
							pf = fmaf(av.w, uv.w, pf);
						}
						acc += (double)pf;
					}
					__syncwarp();
					if (lane == 0) mbar_arrive(empty0 + 8u * st);
				}
				acc = warp_sum(acc);
				if (lane == 0) spart[rowc & 1][cw] = acc;
				named_sync(1, FUSED_CONS);
				if (ct == 0) {
					double t = 0.0;
					for (int w = 0; w < FUSED_CONS / 32; w++) t += spart[rowc & 1][w];
					au[r0 + j] = (float)t;
				}
			}
			if (ct == 0 && r0 < m) {
				__threadfence();
				atomicAdd(&flags[b], 1);
			}
		}
	} else {
		// ---- reducers ----
		const int t = threadIdx.x - FUSED_ROLE;
		const float *au = vsel(I, aus);
		const int SV = S / 4;                                   // float4 per slab row
		const int Q = SV >= FUSED_ROLE ? 1 : FUSED_ROLE / SV;   // row groups
		const int j = t % SV, q = t / SV;
		const bool act = q < Q && c0 + 4 * j < c1;
		const unsigned long long last_use = l2_policy_evict_first();   // the second and last read of A's lines
		double acc[4] = {0.0, 0.0, 0.0, 0.0};
		for (int b = 0; b < nb; b++) {
			const int r0 = b * R, rows = min(R, m - r0);
			const int expect = min(G, (rows + rpc - 1) / rpc);
			if (t == 0 && !s_abort) {
				unsigned sp = 0;
				while (ld_acquire(flags + b) < expect) {
					if (++sp > FUSED_SPIN_MAX) { atomicExch(err, 1); s_abort = 1; break; }
					__nanosleep(32);
				}
			}
			named_sync(2, FUSED_ROLE);
			for (int k = t; k < rows; k += FUSED_ROLE) sauf[k] = __ldcg(au + r0 + k);
			named_sync(2, FUSED_ROLE);
			if (act && !s_abort) {
				// eight rows' products summed in FP32, those sums in FP64
				const float *a = A + (long long)r0 * n + c0 + 4 * j;
				int r = q;
				for (; r + 7 * Q < rows; r += 8 * Q) {
					float4 v[8];
#pragma unroll
					for (int e = 0; e < 8; e++) v[e] = ld_f4_hint(a + (long long)(r + e * Q) * n, last_use);
					float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
					for (int e = 0; e < 8; e++) {
						const float w = sauf[r + e * Q];
						p0 = fmaf(v[e].x, w, p0);
						p1 = fmaf(v[e].y, w, p1);
						p2 = fmaf(v[e].z, w, p2);
						p3 = fmaf(v[e].w, w, p3);
					}
					acc[0] += (double)p0;
					acc[1] += (double)p1;
					acc[2] += (double)p2;
					acc[3] += (double)p3;
				}
				for (; r < rows; r += Q) {
					const float w = sauf[r];
					const float4 v = ld_f4_hint(a + (long long)r * n, last_use);
					acc[0] += (double)(v.x * w);
					acc[1] += (double)(v.y * w);
					acc[2] += (double)(v.z * w);
					acc[3] += (double)(v.w * w);
				}
			}
			named_sync(2, FUSED_ROLE);
			if (t == 0) {
				__threadfence_block();
				s_done = b + 1;
			}
		}
		// the row groups' sums of each column, in group order
		double *sred = sau;   // Q x S doubles (Q S <= 4 x 256)
		if (act)
#pragma unroll
			for (int e = 0; e < 4; e++) sred[q * S + 4 * j + e] = acc[e];
		named_sync(2, FUSED_ROLE);
		float *gv = vselw(I, gs);
		for (int col = t; col < c1 - c0; col += FUSED_ROLE) {
			double tot = 0.0;
			for (int qq = 0; qq < Q; qq++) tot += sred[qq * S + col];
			gv[c0 + col] = (float)tot;
		}
	}
}

// ---------------------------------------------------------------------------
// dense normal product for rows that fit in shared memory (n <= ROWS_COLS):
// CTA c takes the rows c, c + G, c + 2 G, ... whole.  A row is bulk-copied into
// a ring of shared-memory stages; the CTA forms its dot product with u (each
// thread its products eight at a time in FP32, those sums in FP64), which is
// all that A^T needs of it: the row, still in shared memory, times that value
// is added to the threads' FP64 column sums in registers.  No CTA waits for
// another's rows; the CTAs' column sums are added over clusters of four
// through distributed shared memory (their partials then fit the adjoint's
// buffer), the clusters' by k_dense_rows_red, all in a fixed order.  One barrier
// for R rows: their stages are refilled once the next barrier shows that every
// thread has finished with them.
// Bound: HBM (A once), the conversions of A's elements to double close behind;
// for short rows the chain of shuffles, barrier and launches.  The form above,
// whose reducers wait for bands of rows of all CTAs and read them again from
// L2, took 119 us on 4915 x 16384 (this: 72), 57 on 2765 x 9216 (35), 18.6 on
// 1229 x 4096 (14.7) and 20 on 307 x 1024 (7.5); its error against FP64 was
// 9.0e-8 (this: 5.9e-8).  It stays for wider rows.
// Rows of up to 4096 columns are converted to double once for both uses, so
// their dot products too are in FP64 and the second read of shared memory goes
// (307 x 1024: 10.1 -> 7.5 us); wider rows have no registers for that.
// ---------------------------------------------------------------------------
constexpr int ROWS_THREADS = 512;
constexpr int ROWS_COLS = 8 * 4 * ROWS_THREADS;          // 16384: 32 columns per thread
constexpr int ROWS_SMEM = 212 * 1024;                    // of the stages
constexpr int ROWS_STAGES = 8;                           // at most
constexpr int ROWS_CLUSTER = 4;                          // CTAs whose column sums are added on chip

__device__ __forceinline__ void cluster_sync() {
	asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 bytes of the shared memory of the cluster's CTA `rank`, at the address
// `addr` of this CTA's
__device__ __forceinline__ double2 ld_cluster_d2(unsigned addr, int rank) {
	double2 v;
	asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %2, %3;\n\tld.shared::cluster.v2.f64 {%0, %1}, [a];\n\t}"
	             : "=d"(v.x), "=d"(v.y)
	             : "r"(addr), "r"(rank)
	             : "memory");
	return v;
}
inline int rows_stages(long long n) { return (int)std::min<long long>(ROWS_STAGES, ROWS_SMEM / (4 * n)); }

// NV float4 columns per thread; R rows between barriers (several for short
// rows, whose time is the chain of shuffles and the barrier, not the bytes)
template <int NV, int R>
__global__ void __launch_bounds__(ROWS_THREADS, 1) k_dense_rows(const Inst *tab, int inst, int pred, VecSel us,
                                                                VecSel aus, int stages, int early, double *gpart,
                                                                int *err, unsigned long long *launches) {
	pdl_launch_next();
	if (launches && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(launches, 1ull);
	const Inst &I = tab[inst];
	extern __shared__ __align__(128) unsigned char dsm[];
	__shared__ unsigned long long full[ROWS_STAGES];
	__shared__ double spart[2][R][ROWS_THREADS / 32];
	// a wait gave up: one flag for each parity of the loop, so that a warp which
	// is on to the next rows raises another flag than a slow one still reads
	__shared__ int s_abort[2];
	const OpDev &op = I.op;
	const int m = (int)op.m, n = (int)op.n, n4 = n >> 2;
	const int G = gridDim.x, c = blockIdx.x, rows = c < m ? (m - c + G - 1) / G : 0;
	const float *A = op.A;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const unsigned bar0 = smem_u32(full);
	auto issue = [&](int i) {   // thread 0: this CTA's row i into its stage
		const int st = i % stages;
		mbar_expect_tx(bar0 + 8u * st, 4u * n);
		bulk_g2s(smem_u32(dsm + (size_t)st * n * 4), A + (long long)(c + (long long)i * G) * n, 4u * n, bar0 + 8u * st);
	};
	if (threadIdx.x == 0) {
		s_abort[0] = s_abort[1] = 0;
		for (int st = 0; st < stages; st++) mbar_init(bar0 + 8u * st, 1);
		fence_mbar_init();
		if (early)   // A is written by no kernel of the chain: the first rows before the wait
			for (int i = 0; i < min(stages, rows); i++) issue(i);
	}
	__syncthreads();
	pdl_wait_prev();
	const float4 *u4 = reinterpret_cast<const float4 *>(vsel(I, us));
	constexpr bool EXACT = NV <= 2;   // the row as doubles in registers, dot products in FP64
	float4 uv[NV];
#pragma unroll
	for (int k = 0; k < NV; k++) {
		const int j = threadIdx.x + k * ROWS_THREADS;
		uv[k] = j < n4 ? u4[j] : make_float4(0.f, 0.f, 0.f, 0.f);
	}
	double ud[EXACT ? 4 * NV : 1];
	if (EXACT)
#pragma unroll
		for (int k = 0; k < NV; k++) {
			ud[4 * k] = uv[k].x; ud[4 * k + 1] = uv[k].y;
			ud[4 * k + 2] = uv[k].z; ud[4 * k + 3] = uv[k].w;
		}
	if (!pred_ok(*I.ctrl, pred)) {   // the same in every CTA; copies under way land before the CTA exits
		if (early && warp == 0)
			for (int i = 0; i < min(stages, rows); i++) mbar_wait_warp(bar0 + 8u * i, 0u, err);
		return;
	}
	if (!early && threadIdx.x == 0)
		for (int i = 0; i < min(stages, rows); i++) issue(i);
	float *au = vselw(I, aus);
	double acc[4 * NV];
#pragma unroll
	for (int k = 0; k < 4 * NV; k++) acc[k] = 0.0;
	int i = 0;
	for (int par = 0; i < rows; i += R, par ^= 1) {
		const float4 *row[R];
		double w[R], ad[R][EXACT ? 4 * NV : 1];
#pragma unroll
		for (int r = 0; r < R; r++) {
			const int st = (i + r) % stages;
			row[r] = reinterpret_cast<const float4 *>(dsm + (size_t)st * n * 4);
			w[r] = 0.0;
			if (i + r >= rows) continue;
			const bool ok = mbar_wait_warp(bar0 + 8u * st, (unsigned)((i + r) / stages) & 1u, err);
			if (!ok && lane == 0) s_abort[par] = 1;
			if (!ok) continue;
			if (EXACT) {   // short rows: converted once, products and sums in FP64
#pragma unroll
				for (int k = 0; k < NV; k++) {
					const int j = threadIdx.x + k * ROWS_THREADS;
					const float4 a = j < n4 ? row[r][j] : make_float4(0.f, 0.f, 0.f, 0.f);
					ad[r][4 * k] = a.x; ad[r][4 * k + 1] = a.y;
					ad[r][4 * k + 2] = a.z; ad[r][4 * k + 3] = a.w;
#pragma unroll
					for (int q = 4 * k; q < 4 * k + 4; q++) w[r] = fma(ad[r][q], ud[q], w[r]);
				}
				continue;
			}
			// two float4 (eight products) summed in FP32, those sums in FP64
#pragma unroll
			for (int k = 0; k < NV; k += 2) {
				float p = 0.f;
#pragma unroll
				for (int h = k; h < k + 2 && h < NV; h++) {
					const int j = threadIdx.x + h * ROWS_THREADS;
					if (j < n4) {
						const float4 a = row[r][j];
						p = fmaf(a.x, uv[h].x, p);
						p = fmaf(a.y, uv[h].y, p);
						p = fmaf(a.z, uv[h].z, p);
						p = fmaf(a.w, uv[h].w, p);
					}
				}
				w[r] += (double)p;
			}
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1)
#pragma unroll
			for (int r = 0; r < R; r++) w[r] += __shfl_xor_sync(0xffffffffu, w[r], o);
#pragma unroll
		for (int r = 0; r < R; r++)
			if (lane == r) spart[par][r][warp] = w[r];
		__syncthreads();
		if (s_abort[par]) break;
		if (threadIdx.x == 0 && i > 0) {   // every thread has finished with the rows before: their stages may be refilled
			fence_proxy_async_smem();
			for (int r = i - R + stages; r < min(i + stages, rows); r++) issue(r);
		}
#pragma unroll
		for (int r = 0; r < R; r++) {
			if (i + r >= rows) break;
			double t = 0.0;
#pragma unroll
			for (int q = 0; q < ROWS_THREADS / 32; q++) t += spart[par][r][q];
			const float tf = (float)t;
			if (threadIdx.x == 0) au[c + (long long)(i + r) * G] = tf;
			const double td = (double)tf;
			if (EXACT) {
#pragma unroll
				for (int q = 0; q < 4 * NV; q++) acc[q] = fma(ad[r][q], td, acc[q]);
				continue;
			}
#pragma unroll
			for (int k = 0; k < NV; k++) {
				const int j = threadIdx.x + k * ROWS_THREADS;
				if (j < n4) {
					const float4 a = row[r][j];
					acc[4 * k] = fma((double)a.x, td, acc[4 * k]);
					acc[4 * k + 1] = fma((double)a.y, td, acc[4 * k + 1]);
					acc[4 * k + 2] = fma((double)a.z, td, acc[4 * k + 2]);
					acc[4 * k + 3] = fma((double)a.w, td, acc[4 * k + 3]);
				}
			}
		}
	}
	if (i < rows && warp == 0) {   // a wait gave up: let the copies in flight land (bounded) before the CTA exits
		for (int r = i; r < min(rows, max(i - R, 0) + stages); r++)
			mbar_wait_warp(bar0 + 8u * (r % stages), (unsigned)(r / stages) & 1u, err);
	}
	// the cluster's column sums: each CTA's to its own shared memory (the
	// stages, at least two, hold 8 n bytes), a quarter of the columns added per
	// CTA in rank order
	__syncthreads();
	double2 *own = reinterpret_cast<double2 *>(dsm);
#pragma unroll
	for (int k = 0; k < NV; k++) {
		const int j = threadIdx.x + k * ROWS_THREADS;
		if (j < n4) {
			own[2 * j] = make_double2(acc[4 * k], acc[4 * k + 1]);
			own[2 * j + 1] = make_double2(acc[4 * k + 2], acc[4 * k + 3]);
		}
	}
	cluster_sync();
	double2 *gp = reinterpret_cast<double2 *>(gpart + (long long)(c / ROWS_CLUSTER) * n);
	const int n2 = n >> 1, quarter = (n2 + ROWS_CLUSTER - 1) / ROWS_CLUSTER, q0 = (c % ROWS_CLUSTER) * quarter;
	for (int j = q0 + threadIdx.x; j < min(n2, q0 + quarter); j += ROWS_THREADS) {
		double2 v[ROWS_CLUSTER];
#pragma unroll
		for (int k = 0; k < ROWS_CLUSTER; k++) v[k] = ld_cluster_d2(smem_u32(own + j), k);
#pragma unroll
		for (int k = 1; k < ROWS_CLUSTER; k++) {
			v[0].x += v[k].x;
			v[0].y += v[k].y;
		}
		gp[j] = v[0];
	}
	cluster_sync();   // no CTA leaves while another reads its shared memory
}

// g = the clusters' column sums, 32 columns per block: warp w adds the clusters
// w, w + 8, ... of its lane's column (all of a B200's loaded at once), then warp
// 0 the warps' sums in order
constexpr int ROWS_RED_WARPS = 8;
__global__ void __launch_bounds__(32 * ROWS_RED_WARPS) k_dense_rows_red(const Inst *tab, int inst, int pred, VecSel gs, int G,
                                                        const double *gpart, unsigned long long *launches) {
	pdl_launch_next();
	if (launches && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(launches, 1ull);
	const Inst &I = tab[inst];
	__shared__ double ws[ROWS_RED_WARPS][32];
	const int n = (int)I.op.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col = blockIdx.x * 32 + lane;
	pdl_wait_prev();
	if (!pred_ok(*I.ctrl, pred)) return;
	double s = 0.0;
	if (col < n) {
		constexpr int U = 5, W = ROWS_RED_WARPS;
		for (int k = warp; k < G; k += W * U) {
			double v[U];
#pragma unroll
			for (int q = 0; q < U; q++) v[q] = k + W * q < G ? __ldcg(gpart + (long long)(k + W * q) * n + col) : 0.0;
#pragma unroll
			for (int q = 0; q < U; q++) s += v[q];
		}
	}
	ws[warp][lane] = s;
	__syncthreads();
	if (warp == 0 && col < n) {
		double t = ws[0][lane];
		for (int w = 1; w < ROWS_RED_WARPS; w++) t += ws[w][lane];
		vselw(I, gs)[col] = (float)t;
	}
}

// f(kernel) for the form that rows of n elements take
template <class F>
static void rows_kernel(long long n, F f) {
	const int nv = (int)((n + 4 * ROWS_THREADS - 1) / (4 * ROWS_THREADS));
	if (nv <= 1) f(k_dense_rows<1, 2>);
	else if (nv <= 2) f(k_dense_rows<2, 2>);
	else if (nv <= 4) f(k_dense_rows<4, 1>);
	else if (nv <= 6) f(k_dense_rows<6, 1>);
	else f(k_dense_rows<8, 1>);
}
template <class K>
static cudaLaunchConfig_t rows_config(K kern, long long n, int grid, cudaStream_t s, cudaLaunchAttribute (&at)[2]) {
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)grid);
	cfg.blockDim = dim3(ROWS_THREADS);
	cfg.dynamicSmemBytes = (size_t)rows_stages(n) * n * 4;
	cfg.stream = s;
	at[0].id = cudaLaunchAttributeClusterDimension;
	at[0].val.clusterDim.x = ROWS_CLUSTER;
	at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
	at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[1].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = at;
	cfg.numAttrs = 2;
	TG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM));
	return cfg;
}
int fused_rows_grid(long long n) {
	int clusters = 0;
	rows_kernel(n, [&](auto kern) {
		cudaLaunchAttribute at[2];
		cudaLaunchConfig_t cfg = rows_config(kern, n, ROWS_CLUSTER, nullptr, at);
		cfg.numAttrs = 1;
		TG_CUDA(cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg));
	});
	return std::max(1, clusters) * ROWS_CLUSTER;
}
static void launch_rows(const LaunchCtx &L, const OpBatch &B, const OpBatch::Fused &f, int pred, VecSel x, VecSel y,
                        VecSel z, bool early) {
	auto *ctr = (unsigned long long *)L.launches;
	double *part = reinterpret_cast<double *>(B.dense_part);
	rows_kernel(f.n, [&](auto kern) {
		cudaLaunchAttribute at[2];
		cudaLaunchConfig_t cfg = rows_config(kern, f.n, f.grid, L.stream, at);
		TG_CUDA(cudaLaunchKernelEx(&cfg, kern, L.inst, f.inst, pred, x, y, rows_stages(f.n), early ? 1 : 0, part, B.err, ctr));
	});
	launch_pdl(k_dense_rows_red, (unsigned)((f.n + 31) / 32), 32 * ROWS_RED_WARPS, 0, L.stream, L.inst, f.inst, pred, z,
	           f.grid / ROWS_CLUSTER, (const double *)part, ctr);
}

bool fused_by_rows(long long m, long long n, const float *A) {
	// rows are copied by 16-byte bulk copies: n % 4 == 0 and A 16-byte aligned
	return m >= 1 && n >= 4 && m < (1LL << 31) && n <= ROWS_COLS && n % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
}

int fused_grid() {
	int dev = 0, sms = 0;
	TG_CUDA(cudaGetDevice(&dev));
	TG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
	TG_CUDA(cudaFuncSetAttribute(k_dense_normal, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_DYN_BYTES));
	return std::max(1, std::min(sms, FUSED_GRID_MAX));
}

int fused_rows_per_cta(long long m, long long n, int grid, const float *A, int *slab) {
	// rows are streamed by 16-byte bulk copies: n % 4 == 0 and A 16-byte aligned
	if (m < 1 || n < 1 || m >= (1LL << 31) || n % 4 != 0 || (reinterpret_cast<uintptr_t>(A) & 15) != 0) return 0;
	long long S = (n + grid - 1) / grid;   // slab width, a multiple of 4
	S = (S + 3) / 4 * 4;
	const long long SV = S / 4;
	if (SV > FUSED_ROLE) return 0;        // one float4 per reducer thread and slab row
	const long long Q = FUSED_ROLE / SV;  // row groups
	if (Q * S > (long long)FUSED_GRID_MAX * FUSED_RPC_MAX) return 0;   // their sums reuse the band buffer
	const long long row = 4 * n;
	long long rpc = FUSED_BAND_BYTES / (grid * row);
	rpc = std::max(1LL, std::min<long long>(rpc, FUSED_RPC_MAX));
	if (2 * grid * rpc * row > FUSED_L2_BYTES) return 0;
	*slab = (int)S;
	return (int)rpc;
}

#else   // FP64 build: no one-pass normal product (dense normal products take the gemv kernels)
int fused_grid() { return 1; }
int fused_rows_per_cta(long long, long long, int, const real *, int *) { return 0; }
bool fused_by_rows(long long, long long, const real *) { return false; }
int fused_rows_grid(long long) { return 1; }
#endif
// Kernels that read the instance and its index, which no kernel of a chain
// writes, before they wait for the previous kernel (the caller's own arrays only
// after it: the previous kernel may be the caller's)
#define RAY_PROLOGUE()                                                                \
	pdl_launch_next();                                                                \
	if (launches && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(launches, 1ull);   \
	const int2 tl_ = map.tiles[blockIdx.x];                                           \
	const Inst &I = tab[tl_.x];                                                       \
	const OpDev &op = I.op;
#define RAY_WAIT()                                                                    \
	pdl_wait_prev();                                                                  \
	if (!pred_ok(*I.ctrl, pred)) return;

// ---------------------------------------------------------------------------
// compressed gather: y[line] = w * sum_k val[k] * x[ind[k]] over a line's range
//   kind 0: CSR rows (forward), kind 1: CSC columns (adjoint of CSR),
//   kind 2: ray adjoint (implicit weight = scale, ind = measurement index)
// Small operators are bound by the chain of loads from the instance to the first
// entry, so what no kernel writes of it is read before the wait (us a product,
// before: sparse 97x97 adjoint 6.8 -> 5.5, forward 6.1 -> 5.4, 40x40 4.5 -> 3.5, 160x160
// 13.6 -> 12.5); large ones by the L2's sectors (hemisphere of 32^3 voxels and
// 1.6M rays 80 -> 77.4).
// ---------------------------------------------------------------------------
template <int W>
__global__ void __launch_bounds__(256) k_gather(const Inst *tab, TileMap map, int pred, int kind, VecSel xs,
                                                VecSel ys, unsigned long long *launches) {
	RAY_PROLOGUE();
	const int *ptr, *ind;
	const real *val;
	long long lines, xlen, ylen;
	if (kind == 0) { ptr = op.rptr; ind = op.rind; val = op.rval; lines = op.m; xlen = op.n; ylen = op.m; }
	else if (kind == 1) { ptr = op.cptr; ind = op.cind; val = op.cval; lines = op.n; xlen = op.m; ylen = op.n; }
	else { ptr = op.cptr; ind = op.cind; val = nullptr; lines = I.n; xlen = 0; ylen = 0; }
	constexpr int LPB = 256 / W;   // lines per block
	const unsigned local = (unsigned)tl_.y, lt = (unsigned)((lines + LPB - 1) / LPB), layer = local / lt;
	const long long line = (long long)(local - layer * lt) * LPB + threadIdx.x / W;
	const int gl = threadIdx.x % W;
	// the line's range before the wait, unless the CSR may be the caller's
	int k0 = 0, k1 = 0;
	auto range = [&]() {
		if (line < lines) {
			k0 = ptr[line];
			k1 = ptr[line + 1];
		}
	};
	if (kind) range();
	RAY_WAIT();
	if (!kind) range();
	const real *x = vsel(I, xs) + layer * xlen;
	double acc = 0.0;   // FP64 accumulation of FP32 products
	if (line < lines) {
		// four of the lane's entries per step: their indices, then the four
		// gathers, in flight together; summed in the lane's entry order
		int k = k0 + gl;
		if (val) {
			for (; k + 3 * W < k1; k += 4 * W) {
				int ii[4];
				real vv[4], xx[4];
#pragma unroll
				for (int u = 0; u < 4; u++) {
					ii[u] = __ldg(ind + k + u * W);
					vv[u] = __ldg(val + k + u * W);
				}
#pragma unroll
				for (int u = 0; u < 4; u++) xx[u] = ld_vec(x + ii[u]);
#pragma unroll
				for (int u = 0; u < 4; u++) acc = fma((double)vv[u], (double)xx[u], acc);
			}
			for (; k < k1; k += W) acc = fma((double)__ldg(val + k), (double)ld_vec(x + __ldg(ind + k)), acc);
		} else {
			for (; k + 3 * W < k1; k += 4 * W) {
				int ii[4];
				real xx[4];
#pragma unroll
				for (int u = 0; u < 4; u++) ii[u] = __ldg(ind + k + u * W);
#pragma unroll
				for (int u = 0; u < 4; u++) xx[u] = ld_vec(x + ii[u]);
#pragma unroll
				for (int u = 0; u < 4; u++) acc += xx[u];
			}
			for (; k < k1; k += W) acc += ld_vec(x + __ldg(ind + k));
		}
	}
#pragma unroll
	for (int o = W / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
	if (gl == 0 && line < lines) vselw(I, ys)[layer * ylen + line] = (real)(val ? acc : acc * op.scale);
}

// ---------------------------------------------------------------------------
// rays
// ---------------------------------------------------------------------------
struct RayWalk {
	int x0, y0, z0, sx, sy, sz, out;
	int drive;        // 0 x, 1 y, 2 z
	int M;            // driving length; the ray has M + 1 hits
	int a1, a2;       // |delta| of the two minor axes (in axis order, skipping drive)
	__device__ RayWalk(int4 pk) {
		int dx, dy, dz;
		unpack_ray(pk, x0, y0, z0, dx, dy, dz, out);
		sx = dx < 0 ? -1 : 1; sy = dy < 0 ? -1 : 1; sz = dz < 0 ? -1 : 1;
		int mx = abs(dx), my = abs(dy), mz = abs(dz);
		// 3d/mat_mult.h:241,280 (2D: mz = 0 gives 2d/mat_mult.h:160's le >= m)
		if (mx >= my && mx >= mz) { drive = 0; M = mx; a1 = my; a2 = mz; }
		else if (my >= mx && my >= mz) { drive = 1; M = my; a1 = mx; a2 = mz; }
		else { drive = 2; M = mz; a1 = mx; a2 = my; }
	}
	// linear index of step j given the minor offsets k1, k2
	__device__ __forceinline__ long long index(int j, int k1, int k2, int rvx, long long rvxy) const {
		int x, y, z;
		if (drive == 0) { x = x0 + sx * j; y = y0 + sy * k1; z = z0 + sz * k2; }
		else if (drive == 1) { x = x0 + sx * k1; y = y0 + sy * j; z = z0 + sz * k2; }
		else { x = x0 + sx * k1; y = y0 + sy * k2; z = z0 + sz * j; }
		return (long long)x + (long long)y * rvx + (long long)z * rvxy;
	}
};

// minor-axis offset after j driving steps: floor((2 j a + M - 1) / (2 M)),
// advanced by `stride` steps at a time with exact integer carries
struct MinorStep {
	int q, r, qa, ra, twoM;
	__device__ MinorStep(int j, int a, int M, int stride) {
		if (M == 0) { q = r = qa = ra = 0; twoM = 1; return; }
		twoM = 2 * M;
		int num = 2 * j * a + M - 1;
		q = num / twoM; r = num - q * twoM;
		int inc = 2 * stride * a;
		qa = inc / twoM; ra = inc - qa * twoM;
	}
	__device__ __forceinline__ void advance() {
		q += qa; r += ra;
		if (r >= twoM) { r -= twoM; q++; }
	}
};

// Forward projection, SUBW lanes per ray.  Lane l takes the hits j = l,
// l + SUBW, ...; the linear index advances by SUBW driving steps plus, per
// minor axis, the exact quotient / remainder increments of the closed form
// floor((2 j a + M - 1) / (2 M)) - one add and one compare-carry per axis.
// All index arithmetic is 32-bit (images and volumes are below 2^31 voxels,
// extents below 2^15).
template <int SUBW, bool D3>
__global__ void __launch_bounds__(256) k_ray_fwd(const Inst *tab, TileMap map, int pred, VecSel xs, VecSel ys,
                                                 unsigned long long *launches) {
	RAY_PROLOGUE();
	constexpr int RPB = 256 / SUBW;   // rays per block
	const int gl = threadIdx.x % SUBW;
	const long long ray = (long long)tl_.y * RPB + threadIdx.x / SUBW;
	const real *x = nullptr;   // the image's transpose, else the image (known after the wait)
	double acc = 0.0;   // FP64 accumulation along the ray (of FP32 sums of four hits)
	const bool live = ray < op.nrays;
	int out, x0, y0, z0, dx, dy, dz;
	unpack_ray(op.rays[live ? ray : op.nrays - 1], x0, y0, z0, dx, dy, dz, out);
	const int mx = abs(dx), my = abs(dy), mz = D3 ? abs(dz) : 0;
	const int sx = dx < 0 ? -1 : 1, sy = (dy < 0 ? -1 : 1) * op.rvx;
	const int sz = (dz < 0 ? -1 : 1) * op.rvx * op.rvy;
	// driving axis (3d/mat_mult.h:241,280; 2D: 2d/mat_mult.h:160)
	int M, a1, a2, sd, s1, s2;
	int idx = x0 + y0 * op.rvx + z0 * op.rvx * op.rvy;
	if (mx >= my && mx >= mz) { M = mx; sd = sx; a1 = my; s1 = sy; a2 = mz; s2 = sz; }
	else if (my >= mx && my >= mz) {
		M = my; sd = sy; a1 = mx; s1 = sx; a2 = mz; s2 = sz;
		if (!D3 && op.xT) {   // transposed image: y steps are contiguous
			x = op.xT;
			idx = y0 + x0 * op.tH;
			sd = dy < 0 ? -1 : 1;
			s1 = (dx < 0 ? -1 : 1) * op.tH;
		}
	} else { M = mz; sd = sz; a1 = mx; s1 = sx; a2 = my; s2 = sy; }
	idx += gl * sd;
	const int twoM = 2 * M > 0 ? 2 * M : 1;
	int q1 = 0, r1 = 0, qa1 = 0, ra1 = 0, q2 = 0, r2 = 0, qa2 = 0, ra2 = 0;
	if (M > 0) {
		int num = 2 * gl * a1 + M - 1;
		q1 = num / twoM; r1 = num - q1 * twoM;
		qa1 = (2 * SUBW * a1) / twoM; ra1 = 2 * SUBW * a1 - qa1 * twoM;
		idx += q1 * s1;
		if (D3) {
			num = 2 * gl * a2 + M - 1;
			q2 = num / twoM; r2 = num - q2 * twoM;
			qa2 = (2 * SUBW * a2) / twoM; ra2 = 2 * SUBW * a2 - qa2 * twoM;
			idx += q2 * s2;
		}
	}
	const int dstep = SUBW * sd + qa1 * s1 + (D3 ? qa2 * s2 : 0);
	auto step = [&]() {
		idx += dstep;
		r1 += ra1;
		if (r1 >= twoM) { r1 -= twoM; idx += s1; }
		if (D3) {
			r2 += ra2;
			if (r2 >= twoM) { r2 -= twoM; idx += s2; }
		}
	};
	RAY_WAIT();
	if (!x) x = vsel(I, xs);
	if (live) {
		// four of the lane's hits summed in FP32, those sums in FP64 (one
		// conversion per four hits)
		int j = gl;
		for (; j + 3 * SUBW <= M; j += 4 * SUBW) {
			real v[4];
#pragma unroll
			for (int u = 0; u < 4; u++) {
				v[u] = ld_vec(x + idx);
				step();
			}
			acc += (double)((v[0] + v[1]) + (v[2] + v[3]));
		}
		real rest = 0.f;
		for (; j <= M; j += SUBW) {
			rest += ld_vec(x + idx);
			step();
		}
		acc += (double)rest;
	}
#pragma unroll
	for (int o = SUBW / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
	if (gl == 0 && live) vselw(I, ys)[out] = (real)(acc * op.scale);
}

// Forward projection, one thread per ray (the built-in form where the minor
// axis can be read contiguously).  Neighbouring rays run side by side, so at
// step j a warp's 32 rays sit on one line across the driving axis: with that
// line contiguous in memory (y-driven rays read the image, x-driven ones its
// transpose xT; in 3D x-driven rays read the y-major copy xT, the others the
// volume) a load touches a few cache lines where lanes along the ray touched
// one per minor step.  The Bresenham position is a 32.32 fixed-point number:
// each step adds drive stride << 32 +- inc, inc = a 2^32 / M rounded up (at
// most one unit too large), and the carry out of the fraction is the minor
// step - one 64-bit add, no comparison.  Exact while 2 M (M + 2) < 2^32
// (M <= 46339; extents are below 2^15): floor((2 j a + M - 1) / (2 M)) lies at
// least 1 / (2 M) below the next integer, the accumulated rounding below that.
// The sums are k_ray_fwd<8>'s, in its order: class l of eight holds the hits
// j = l (mod 8), four of them summed in FP32 (missing ones as zeros), those
// sums in FP64 per class, the classes in the shuffle tree's order.
// Bound: 2D by issue (7 warp instructions per hit and lane, 18 before) at 28
// resident warps per SM - 256^2 ring, 2.72e7 hits, with the transpose: 26.0 ->
// 15.8 us; 3D by L1's rate of lines and the latency of its L2 hits (a warp's hits
// spread over about 12 sectors, read once; L1 77 % busy, L2 71, issue 45) -
// 128^3 hemisphere, 1.29e8 hits, with the transpose: 295 -> 147 us.
template <bool D3>
__global__ void __launch_bounds__(RAY1_BLOCK) k_ray_fwd_thread(const Inst *tab, TileMap map, int pred, VecSel xs,
                                                               VecSel ys, unsigned long long *launches) {
	RAY_PROLOGUE();
	const long long ray = (long long)tl_.y * RAY1_BLOCK + threadIdx.x;
	const bool live = ray < op.nrays;
	int x0, y0, z0, dx, dy, dz, out;
	unpack_ray(op.rays_fwd[live ? ray : op.nrays - 1], x0, y0, z0, dx, dy, dz, out);
	const int mx = abs(dx), my = abs(dy), mz = D3 ? abs(dz) : 0;
	const int nx = op.rvx, ny = D3 ? op.rvy : op.tH;
	const real *x = nullptr;   // the transpose, else the image itself (known after the wait)
	// driving axis (3d/mat_mult.h:241,280; 2D: 2d/mat_mult.h:160); a1: the
	// contiguous minor axis, a2: the other one, of stride S2
	int M, a1, a2 = 0, sd, base, S2 = 0;
	bool n1, n2 = false;
	if (mx >= my && mx >= mz) {
		M = mx; a1 = my; n1 = dy < 0; sd = dx < 0 ? -ny : ny;
		base = y0 + x0 * ny;
		if (D3) { a2 = mz; n2 = dz < 0; S2 = nx * ny; base += z0 * S2; }
		x = op.xT;
	} else if (my >= mx && my >= mz) {
		M = my; a1 = mx; n1 = dx < 0; sd = dy < 0 ? -nx : nx;
		base = x0 + y0 * nx;
		if (D3) { a2 = mz; n2 = dz < 0; S2 = nx * ny; base += z0 * S2; }
	} else {
		M = mz; a1 = mx; n1 = dx < 0; sd = (dz < 0 ? -nx : nx) * ny;
		base = x0 + z0 * nx * ny;
		a2 = my; n2 = dy < 0; S2 = nx; base += y0 * S2;
	}
	long long P1 = (long long)base << 32, P2 = 0, d1 = (long long)sd << 32, d2 = 0;
	if (M > 0) {
		// 2^32 / M to 2^-46 relative: a float reciprocal and one Newton step
		const double r0 = (double)__frcp_rn((float)M), r = 4294967296.0 * (r0 * fma(-(double)M, r0, 2.0));
		const long long f0 = (long long)((M - 1) * r * 0.5) + 1;
		const long long inc1 = (long long)(a1 * r) + 1, inc2 = D3 ? (long long)(a2 * r) + 1 : 0;
		P1 += n1 ? 0xffffffffLL - f0 : f0;
		d1 += n1 ? -inc1 : inc1;
		if (D3) {
			P2 = n2 ? 0xffffffffLL - f0 : f0;
			d2 = n2 ? -inc2 : inc2;
		}
	}
	unsigned f1 = (unsigned)P1, f2 = (unsigned)P2;   // fractions, indices, and their steps
	int i1 = (int)(P1 >> 32), i2 = (int)(P2 >> 32);
	const unsigned df1 = (unsigned)d1, df2 = (unsigned)d2;
	const int di1 = (int)(d1 >> 32), di2 = (int)(d2 >> 32);
	auto next = [&]() -> real {
		const real *p = x + (i1 + (D3 ? i2 * S2 : 0));
		asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;" : "+r"(f1), "+r"(i1) : "r"(df1), "r"(di1));
		if (D3) asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;" : "+r"(f2), "+r"(i2) : "r"(df2), "r"(di2));
		return ld_vec(p);
	};
	RAY_WAIT();
	if (!x) x = vsel(I, xs);
	double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
	int left = M + 1;
	// 32 hits a round: rounds that every lane fills, then, warp by warp, the
	// rest with each lane's missing hits as zeros, eight hits at a time (a
	// warp's rays differ in length: taken lane by lane, full and partial
	// rounds would run one after the other)
	while (__all_sync(0xffffffffu, left >= 32)) {
		real s[8], u[8], v[8];
#pragma unroll
		for (int l = 0; l < 8; l++) u[l] = next();
#pragma unroll
		for (int l = 0; l < 8; l++) v[l] = next();
#pragma unroll
		for (int l = 0; l < 8; l++) s[l] = u[l] + v[l];
#pragma unroll
		for (int l = 0; l < 8; l++) u[l] = next();
#pragma unroll
		for (int l = 0; l < 8; l++) v[l] = next();
#pragma unroll
		for (int l = 0; l < 8; l++) acc[l] += (double)(s[l] + (u[l] + v[l]));
		left -= 32;
	}
	while (__any_sync(0xffffffffu, left > 0)) {
		real s[8], u[8], v[8];
#pragma unroll
		for (int l = 0; l < 8; l++) {
			s[l] = l < left ? next() : (real)0;
			u[l] = v[l] = (real)0;
		}
		if (__any_sync(0xffffffffu, left > 8)) {
#pragma unroll
			for (int l = 0; l < 8; l++) s[l] += 8 + l < left ? next() : (real)0;
			if (__any_sync(0xffffffffu, left > 16)) {
#pragma unroll
				for (int l = 0; l < 8; l++) u[l] = 16 + l < left ? next() : (real)0;
				if (__any_sync(0xffffffffu, left > 24))
#pragma unroll
					for (int l = 0; l < 8; l++) v[l] = 24 + l < left ? next() : (real)0;
			}
		}
#pragma unroll
		for (int l = 0; l < 8; l++) acc[l] += (double)(s[l] + (u[l] + v[l]));
		left -= 32;
	}
	if (!live) return;
	const double t = ((acc[0] + acc[4]) + (acc[2] + acc[6])) + ((acc[1] + acc[5]) + (acc[3] + acc[7]));
	vselw(I, ys)[out] = (real)(t * op.scale);
}

// The adjoint by on-the-fly tracing (TVAL3G_RAY_ADJ_ATOMICS): lanes and
// steps as in k_ray_fwd (always the image's own layout), each hit adding
// scale * y[ray] to its pixel with an atomic add into the zeroed output.
// The order of the adds varies from run to run, so the sums are not
// bit-reproducible; the gather adjoints are.
__global__ void __launch_bounds__(256) k_ray_atomic_zero(const Inst *tab, TileMap map, int pred, VecSel ys,
                                                         unsigned long long *launches) {
	OPROLOGUE();
	real *out = vselw(I, ys);
	const long long i0 = local * ATOMIC_ZERO_TILE;
	for (long long i = i0 + threadIdx.x; i < min(I.n, i0 + ATOMIC_ZERO_TILE); i += blockDim.x) out[i] = 0.f;
}

template <bool D3>
__global__ void __launch_bounds__(256) k_ray_adj_atomic(const Inst *tab, TileMap map, int pred, VecSel xs,
                                                        VecSel ys, unsigned long long *launches) {
	OPROLOGUE();
	const OpDev &op = I.op;
	constexpr int SUBW = RAY_SUBW, RPB = 256 / SUBW;
	const int gl = threadIdx.x % SUBW;
	const long long ray = local * RPB + threadIdx.x / SUBW;
	if (ray >= op.nrays) return;
	real *g = vselw(I, ys);
	int x0, y0, z0, dx, dy, dz, out;
	unpack_ray(op.rays[ray], x0, y0, z0, dx, dy, dz, out);
	const real w = vsel(I, xs)[out] * op.scale;
	const int mx = abs(dx), my = abs(dy), mz = D3 ? abs(dz) : 0;
	const int sx = dx < 0 ? -1 : 1, sy = (dy < 0 ? -1 : 1) * op.rvx;
	const int sz = (dz < 0 ? -1 : 1) * op.rvx * op.rvy;
	int M, a1, a2, sd, s1, s2;
	int idx = x0 + y0 * op.rvx + z0 * op.rvx * op.rvy;
	if (mx >= my && mx >= mz) { M = mx; sd = sx; a1 = my; s1 = sy; a2 = mz; s2 = sz; }
	else if (my >= mx && my >= mz) { M = my; sd = sy; a1 = mx; s1 = sx; a2 = mz; s2 = sz; }
	else { M = mz; sd = sz; a1 = mx; s1 = sx; a2 = my; s2 = sy; }
	idx += gl * sd;
	const int twoM = 2 * M > 0 ? 2 * M : 1;
	int r1 = 0, qa1 = 0, ra1 = 0, r2 = 0, qa2 = 0, ra2 = 0;
	if (M > 0) {
		int num = 2 * gl * a1 + M - 1;
		int q = num / twoM;
		r1 = num - q * twoM;
		qa1 = (2 * SUBW * a1) / twoM; ra1 = 2 * SUBW * a1 - qa1 * twoM;
		idx += q * s1;
		if (D3) {
			num = 2 * gl * a2 + M - 1;
			q = num / twoM;
			r2 = num - q * twoM;
			qa2 = (2 * SUBW * a2) / twoM; ra2 = 2 * SUBW * a2 - qa2 * twoM;
			idx += q * s2;
		}
	}
	const int dstep = SUBW * sd + qa1 * s1 + (D3 ? qa2 * s2 : 0);
	for (int j = gl; j <= M; j += SUBW) {
		atomicAdd(g + idx, w);
		idx += dstep;
		r1 += ra1;
		if (r1 >= twoM) { r1 -= twoM; idx += s1; }
		if (D3) {
			r2 += ra2;
			if (r2 >= twoM) { r2 -= twoM; idx += s2; }
		}
	}
}

// xT[y + x*tH] = x[x + y*ld] for the ray forwards, in 3D slice by slice (32x32
// tiles through shared memory; local tile = (z * ceil(tH/32) + ty) * ceil(ld/32) + tx)
__global__ void __launch_bounds__(256) k_transpose2d(const Inst *tab, TileMap map, int pred, VecSel xs,
                                                     unsigned long long *launches) {
	OPROLOGUE();
	__shared__ real tile[32][33];
	const OpDev &op = I.op;
	const int ld = op.rvx, H = op.tH;
	const int ntx = (ld + 31) / 32, nty = (H + 31) / 32;
	const int bx = (int)local % ntx, row = (int)local / ntx, z = row / nty, by = row - z * nty;
	const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
	const real *X = vsel(I, xs) + (long long)z * ld * H;
	real *XT = op.xT + (long long)z * ld * H;
#pragma unroll
	for (int j = 0; j < 32; j += 8) {
		const int x = bx * 32 + tx, y = by * 32 + ty + j;
		if (x < ld && y < H) tile[ty + j][tx] = X[x + y * ld];
	}
	__syncthreads();
#pragma unroll
	for (int j = 0; j < 32; j += 8) {
		const int y = by * 32 + tx, x = bx * 32 + ty + j;
		if (x < ld && y < H) XT[y + x * H] = tile[tx][ty + j];
	}
}

#ifndef TVAL3G_FP64   // tiled ray adjoints: FP32 data only
// ---------------------------------------------------------------------------
// tiled 2D ray adjoint
// ---------------------------------------------------------------------------
__global__ void k_to_int(const long long *in, int *out, long long n);

constexpr int RAYT_THREADS = RAYT * RAYT;   // one thread per pixel of a tile
constexpr int RAYT_WARPS = RAYT_THREADS / 32;

// Twice as many warps as pixel-warps (groups of 32 pixels).  A tile's words
// are one sequence - pixel-warp after pixel-warp, each as long as its longest
// list - cut into one equal run per warp, so that no warp waits at the end for
// the pixel-warp with the longest lists.  A warp leaves its sum of every
// pixel-warp that its run meets; run w and pixel-warp p meet at most once, and
// along the sequence w + p only grows: the slot of their sum.
constexpr int RAYT_ADJ_THREADS = 2 * RAYT_THREADS;
constexpr int RAYT_ADJ_WARPS = RAYT_ADJ_THREADS / 32;
constexpr int RAYT_AHEAD = 4;                            // words a thread loads ahead of use
constexpr int RAYT_BAR_BYTES = 64;                       // the list's barrier, the pixel-warps' word offsets
constexpr int RAYT_SLOTS = RAYT_ADJ_WARPS + RAYT_WARPS - 1;
constexpr int RAYT_SACC_BYTES = RAYT_SLOTS * 32 * 8;     // the runs' sums
static_assert(8 + 4 * (RAYT_WARPS + 1) <= RAYT_BAR_BYTES, "barrier and offsets");
constexpr int RAYT_LIST_CHUNK = 8192;                    // list entries per bulk copy
// rays of a tile's list per part (2D), for images of at most TILE_CUT tiles:
// with fewer tiles than SMs the longest list is the launch's length.  Adjoint
// of rings of (side, transducers) (33, 256), (64, 512), (128, 512), (192, 384),
// back to back, us: whole tiles 20.7 18.6 27.1 19.8; parts of 12288 rays 15.7
// 18.1 25.7 19.8; 8192: 13.5 15.1 19.7 16.8; 6144: 11.3 14.1 17.5 15.9; 4096:
// 10.6 17.1 18.8 16.4.  Of (256, 512), 256 tiles: whole 26.0, 8192 rays 25.6
// with the index in L2 but 5 % slower with it from HBM.
// (The image's tiles count, not the launch's: parts add in another order, and an
// instance gives the same bits alone and in a batch.)
constexpr int TILE_PART = 6144, TILE_CUT = 148;
static_assert(TILE_CUT < 1 << 24, "tile numbers beside part numbers (OpDev::vtile)");
constexpr int TILE_PARTS = 16;                           // parts per tile at most
constexpr int RAYT_ZERO_TILES = 16;                      // tiles without rays zeroed per block

// the list's barrier and the pixel-warps' word offsets, the runs' sums, then the
// list's measurements: slot 0 (the zero that pad entries read) sits 12 bytes past
// a 16-byte boundary so that slots 1.. are aligned for the bulk copy of the list
int tiled_smem_bytes(int tmax) {
	return RAYT_BAR_BYTES + RAYT_SACC_BYTES + 12 + (int)sizeof(float) * (tmax + 1);
}

// a 16-byte index word: read once per product, so it takes no room in L1
__device__ __forceinline__ uint4 ld_word(const uint4 *p) {
	uint4 v;
	asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
	             : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
	             : "l"(p));
	return v;
}

// the eight entries of a 16-byte index word, summed in a fixed tree
__device__ __forceinline__ float word_sum(const float *yt, uint4 q) {
	return ((yt[q.x & 0xffff] + yt[q.x >> 16]) + (yt[q.y & 0xffff] + yt[q.y >> 16])) +
	       ((yt[q.z & 0xffff] + yt[q.z >> 16]) + (yt[q.w & 0xffff] + yt[q.w >> 16]));
}

// g at pixel px (0 .. RAYT^2 - 1, row-major in the tile) of tile (brick) t
__device__ __forceinline__ void tiled_store(const Inst &I, const OpDev &op, VecSel ys, int t, int px, float v) {
	if (op.tile3) {   // brick of BRICK_X x BRICK_Y x BRICK_Z voxels
		const int bxy = op.ntx * op.nty;
		const int x = (t % op.ntx) * BRICK_X + px % BRICK_X;
		const int y = ((t % bxy) / op.ntx) * BRICK_Y + (px / BRICK_X) % BRICK_Y;
		const int z = (t / bxy) * BRICK_Z + px / (BRICK_X * BRICK_Y);
		// (the last layer of bricks may reach beyond the image's end, where the volume is smaller than the image)
		const long long p = x + (long long)y * op.rvx + (long long)z * op.rvx * op.rvy;
		if (x < op.rvx && y < op.rvy && p < I.n) vselw(I, ys)[p] = v;
		return;
	}
	const int x = (t % op.ntx) * RAYT + (px % RAYT), row = (t / op.ntx) * RAYT + (px / RAYT);
	if (x < op.rvx && row < op.tH) vselw(I, ys)[x + row * op.rvx] = v;
}

// g[p] = scale * sum over the rays through p of y[ray] (the transposed
// projection of 2d/mat_mult.h:145-181).  Block per RAYT x RAYT tile (3D: per
// brick): the measurements of the rays crossing the tile are gathered into
// shared memory (slot 0 holds the zero that pad entries read), then the warps
// sum the pixels' entries in ray order - eight per 16-byte word in FP32, the
// words in FP64.  The words come straight from global memory, RAYT_AHEAD ahead
// of use, the first before the gather.  Pixels are taken in order of
// decreasing hit count (OpDev::tperm), so a warp's pixels have lists of nearly
// one length and its words carry little padding.  A 2D tile of an image with
// few tiles is cut into parts (TILE_PART), a block each, whose FP64 sums the
// last of them adds in order.  Deterministic, no atomics on values.
// Bound: the L1 and shared-memory pipes - a gather of 32 scattered
// measurements is 32 tags, a word's eight reads 3.3 wavefronts each - at the
// blocks that the longest list's shared memory lets an SM hold.  Measured
// (back to back): 128^3 hemisphere, 1.29e8 hits, 350 us with the words going
// through per-warp rings in shared memory (one block per SM) and each warp
// owning half of one pixel-warp's words; 231 us without the rings (two blocks),
// 219 with 16 instead of 64 empty tiles per block, 188 with the words cut into
// equal runs.  256^2 ring: 32.4 -> 25.8 us (225 blocks on 148 SMs).
// Lists in the forward's sorted ray order (y permuted first) took 174 us there
// but 16.0 against 13.0 us at 64^3 and 44.5 against 42.3 at 100^3: not kept.
__global__ void __launch_bounds__(RAYT_ADJ_THREADS, 2) k_ray_adj_tiled(const Inst *tab, TileMap map, int pred,
                                                                       VecSel xs, VecSel ys, int *err,
                                                                       unsigned long long *launches) {
	RAY_PROLOGUE();
	const int local = tl_.y;
	extern __shared__ __align__(128) unsigned char smem[];
	if (local >= op.tfull) {
		RAY_WAIT();
		// tiles that no ray crosses (the launch order ends with them): zeros,
		// RAYT_ZERO_TILES tiles per block, none of the list machinery
		// (32-bit indices: tile counts stay below 2^31, and 64-bit ones here
		// cost the whole kernel eight registers)
		const int e0 = op.tfull + (local - op.tfull) * RAYT_ZERO_TILES;
		const int e1 = min(e0 + RAYT_ZERO_TILES, op.tcount);
		const float zero = (float)(0.0 * op.scale);   // the bits a block of this tile would write
		constexpr int HALVES = RAYT_ADJ_THREADS / RAYT_THREADS, EACH = RAYT_ZERO_TILES / HALVES;
		int tz[EACH];   // this half block's tiles, loaded together
#pragma unroll
		for (int k = 0; k < EACH; k++) {
			const int e = e0 + k * HALVES + (int)threadIdx.x / RAYT_THREADS;
			tz[k] = e < e1 ? __ldg(op.tempty + (e - op.tfull)) : -1;
		}
#pragma unroll
		for (int k = 0; k < EACH; k++)
			if (tz[k] >= 0) tiled_store(I, op, ys, tz[k], threadIdx.x % RAYT_THREADS, zero);
		return;
	}
	const int4 vt = __ldg(op.vtile + local);
	const bool cut = op.tpart != nullptr;   // else vt.x is the tile whole: volumes have up to 2^25 bricks
	const int t = cut ? vt.x & 0xffffff : vt.x, parts = cut ? (vt.x >> 24 & 15) + 1 : 1, part = cut ? (int)((unsigned)vt.x >> 28) : 0;
	const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const unsigned bar_list = smem_u32(smem);
	int *sb = reinterpret_cast<int *>(smem + 8);   // the pixel-warps' first words
	double *sacc = reinterpret_cast<double *>(smem + RAYT_BAR_BYTES);
	float *yt = reinterpret_cast<float *>(smem + RAYT_BAR_BYTES + RAYT_SACC_BYTES + 12);
	// the tile's list (a multiple of 4 entries from a 16-byte boundary) is
	// bulk-copied into the measurement slots 1..len, then each slot's
	// measurement index is replaced by its value.  The index depends on no
	// earlier kernel: the copy and the first words are under way before the wait
	const int k0 = vt.y, len = vt.z;
	if (threadIdx.x == 0) {
		mbar_init(bar_list, 1);
		fence_mbar_init();
		mbar_expect_tx(bar_list, (unsigned)len * 4u);
		for (int c0 = 0; c0 < len; c0 += RAYT_LIST_CHUNK)
			bulk_g2s(smem_u32(yt + 1 + c0), op.tmeas + k0 + c0, (unsigned)min(RAYT_LIST_CHUNK, len - c0) * 4u, bar_list);
		yt[0] = 0.f;
	}
	const int *wo = op.woff + vt.w * RAYT_WARPS;
	const int w0 = __ldg(wo), nwords = (__ldg(wo + RAYT_WARPS) - w0) >> 5;   // words per lane
	if (threadIdx.x <= RAYT_WARPS) sb[threadIdx.x] = (__ldg(wo + threadIdx.x) - w0) >> 5;
	auto run = [&](int w) { return (int)((long long)w * nwords / RAYT_ADJ_WARPS); };   // first word of warp w's run
	const int v0 = run(wid), nv = run(wid + 1) - v0;
	const uint4 *src = op.sidx + w0 + 32LL * v0 + lane;
	uint4 q[RAYT_AHEAD];
#pragma unroll
	for (int j = 0; j < RAYT_AHEAD; j++)
		if (j < nv) q[j] = ld_word(src + 32 * j);
	__syncthreads();   // barrier initialisation seen by every thread
	pdl_wait_prev();
	bool ok = mbar_wait_warp(bar_list, 0u, err, op.first_wait_polls ? op.first_wait_polls - 1u : ASYNC_WAIT_LIMIT);
	if (!ok) mbar_wait_warp(bar_list, 0u, err);   // gave up: let the copy land (bounded) before the block exits
	if (!pred_ok(*I.ctrl, pred)) return;
	const float *y = vsel(I, xs);
	if (ok) {   // eight independent gathers in flight per thread
		constexpr int U8 = 8;
		int k = threadIdx.x;
		for (; k + (U8 - 1) * RAYT_ADJ_THREADS < len; k += U8 * RAYT_ADJ_THREADS) {
			float yv[U8];
#pragma unroll
			for (int u = 0; u < U8; u++) yv[u] = y[__float_as_int(yt[1 + k + u * RAYT_ADJ_THREADS])];
#pragma unroll
			for (int u = 0; u < U8; u++) yt[1 + k + u * RAYT_ADJ_THREADS] = yv[u];
		}
		for (; k < len; k += RAYT_ADJ_THREADS) yt[1 + k] = y[__float_as_int(yt[1 + k])];
	}
	__syncthreads();
	if (ok && nv > 0) {
		double acc = 0.0;
		int pw = 0;
		while (sb[pw + 1] <= v0) pw++;   // the pixel-warp of the run's first word
		int end = sb[pw + 1] - v0;
		auto add = [&](int k, uint4 word) {   // word k of the run
			if (k == end) {
				sacc[(wid + pw) * 32 + lane] = acc;
				acc = 0.0;
				do pw++;
				while (sb[pw + 1] - v0 <= k);
				end = sb[pw + 1] - v0;
			}
			acc += (double)word_sum(yt, word);
		};
		int k = 0;
		for (; k + 2 * RAYT_AHEAD <= nv; k += RAYT_AHEAD) {
			uint4 c[RAYT_AHEAD];
#pragma unroll
			for (int j = 0; j < RAYT_AHEAD; j++) {
				c[j] = q[j];
				q[j] = ld_word(src + 32 * (k + RAYT_AHEAD + j));
			}
#pragma unroll
			for (int j = 0; j < RAYT_AHEAD; j++) add(k + j, c[j]);
		}
		// the words loaded, then the last ones
#pragma unroll
		for (int j = 0; j < RAYT_AHEAD; j++)
			if (k + j < nv) {
				add(k + j, q[j]);
				if (k + RAYT_AHEAD + j < nv) q[j] = ld_word(src + 32 * (k + RAYT_AHEAD + j));
			}
		k += RAYT_AHEAD;
#pragma unroll
		for (int j = 0; j < RAYT_AHEAD; j++)
			if (k + j < nv) add(k + j, q[j]);
		sacc[(wid + pw) * 32 + lane] = acc;
	}
	__syncthreads();
	// this thread's pixel: its pixel-warp's sums, run by run
	double acc = 0.0;
	const int b0 = wid < RAYT_WARPS ? sb[wid] : 0, b1 = wid < RAYT_WARPS ? sb[wid + 1] : 0;
	if (b1 > b0) {
		const int wlo = (int)(((long long)RAYT_ADJ_WARPS * b0 + RAYT_ADJ_WARPS - 1) / nwords);
		const int whi = (int)(((long long)RAYT_ADJ_WARPS * (b1 - 1) + RAYT_ADJ_WARPS - 1) / nwords);
		for (int w = wlo; w <= whi; w++)
			if (run(w) < run(w + 1)) acc += sacc[(w + wid) * 32 + lane];   // (fewer words than warps: some runs are empty)
	}
	if (parts > 1) {
		// a part of a tile: the block that finishes last adds the parts' sums in
		// their order (a block whose wait gave up takes its turn all the same: the
		// ticket must come round to zero)
		__shared__ int last;
		double *slot = op.tpart + (long long)__ldg(op.tpoff + local) * RAYT_THREADS + threadIdx.x;
		if (threadIdx.x < RAYT_THREADS) slot[(long long)part * RAYT_THREADS] = acc;
		__threadfence();
		__syncthreads();
		if (threadIdx.x == 0) {
			// (atomicInc wraps to 0 at parts - 1: also when two products overlapped
			// against the rule, the count is back at 0 after both)
			last = atomicInc(op.tticket + t, (unsigned)parts - 1u) == (unsigned)parts - 1u;
		}
		__syncthreads();
		if (!last || threadIdx.x >= RAYT_THREADS) return;
		__threadfence();
		acc = 0.0;
		for (int k = 0; k < parts; k++) acc += __ldcg(slot + (long long)k * RAYT_THREADS);
	}
	if (threadIdx.x >= RAYT_THREADS || !ok) return;
	const int px = __ldg(op.tperm + (long long)t * RAYT_THREADS + threadIdx.x);   // this thread's pixel of the tile
	tiled_store(I, op, ys, t, px, (float)(acc * op.scale));
}

// --- index builder (once per operator) ---------------------------------------
// The rays crossing tile t, as a bitmap over traced-ray ids in shared memory,
// from the pixel-major lists of traced-ray ids (cptr, cind).
// image index of pixel px (0 .. RAYT^2 - 1, row-major) of tile t, or -1 outside the image
__device__ __forceinline__ int tile_pixel(int t, int px, int ntx, int ld, int H) {
	const int x = (t % ntx) * RAYT + px % RAYT, y = (t / ntx) * RAYT + px / RAYT;
	return (x < ld && y < H) ? x + y * ld : -1;
}

__device__ void tile_bitmap(unsigned *bm, int nwords, int p, const int *cptr, const int *cind) {
	for (int w = threadIdx.x; w < nwords; w += blockDim.x) bm[w] = 0u;
	__syncthreads();
	if (p >= 0) {
		const int k1 = cptr[p + 1];
		for (int k = cptr[p]; k < k1; k += 8) {   // eight loads in flight, then their updates
			int r[8];
#pragma unroll
			for (int j = 0; j < 8; j++) r[j] = k + j < k1 ? cind[k + j] : -1;
#pragma unroll
			for (int j = 0; j < 8; j++)
				if (r[j] >= 0) atomicOr(&bm[r[j] >> 5], 1u << (r[j] & 31));
		}
	}
	__syncthreads();
}

// exclusive prefix of the bitmap words' popcounts (pre), by a block of
// RAYT_THREADS: thread i scans the words [w0, w1).  Returns the tile's rays.
__device__ int tile_prefix(const unsigned *bm, int *pre, int nwords, int &w0, int &w1) {
	__shared__ int ws[RAYT_WARPS];
	const int per = (nwords + RAYT_THREADS - 1) / RAYT_THREADS;
	w0 = min(nwords, (int)threadIdx.x * per);
	w1 = min(nwords, w0 + per);
	int c = 0;
	for (int w = w0; w < w1; w++) c += __popc(bm[w]);
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	int inc = c;
	for (int o = 1; o < 32; o <<= 1) {
		const int u = __shfl_up_sync(0xffffffffu, inc, o);
		if (lane >= o) inc += u;
	}
	if (lane == 31) ws[wid] = inc;
	__syncthreads();
	int run = inc - c, total = 0;
	for (int i = 0; i < RAYT_WARPS; i++) {
		if (i < wid) run += ws[i];
		total += ws[i];
	}
	for (int w = w0; w < w1; w++) {
		pre[w] = run;
		run += __popc(bm[w]);
	}
	__syncthreads();
	return total;
}
// position of ray r in the tile's list
__device__ __forceinline__ int tile_pos(const unsigned *bm, const int *pre, int r) {
	return pre[r >> 5] + __popc(bm[r >> 5] & ((1u << (r & 31)) - 1u));
}
// words [v0, v1) of a pixel-warp's nv that part p of `parts` takes
__device__ __forceinline__ void part_words(int nv, int p, int parts, int &v0, int &v1) {
	v0 = nv * p / parts;
	v1 = nv * (p + 1) / parts;
}

// rays per tile (rounded up to a multiple of 4: the pad entries stay 0, a
// valid measurement index that no position refers to); the tile's pixels in
// order of decreasing list length, ties by position (perm[rank] = pixel); the
// parts a tile is cut into (one per `part` rays of its list, at most
// TILE_PARTS), the stretch of the list that the words of each refer to (a
// pixel's positions ascend, so its first and last words' ends bound it; begun
// on a 16-byte boundary) and, per part and warp of ranks, its word count (32 x
// its share of the longest of the warp's lists, in 16-byte words).
// parts[t stride + p] = (list offset in the tile, length, words, parts); stride:
// TILE_PARTS, or 1 where no tile is cut
__global__ void __launch_bounds__(RAYT_THREADS) k_tile_count(int ld, int H, int ntx, int nrays, int part, int stride,
                                                             const int *cptr, const int *cind, long long *tlen, long long *wlen,
                                                             int4 *parts, unsigned char *perm, unsigned *gbm) {
	extern __shared__ unsigned bm[];   // nwords bits, then nwords exclusive prefix counts
	__shared__ int cnt[RAYT_THREADS];
	__shared__ int byrank[RAYT_THREADS], pixel[RAYT_THREADS];
	__shared__ int lo[TILE_PARTS], hi[TILE_PARTS], wsum[TILE_PARTS];
	const int t = blockIdx.x, nwords = (nrays + 31) >> 5;
	int *pre = reinterpret_cast<int *>(bm + nwords);
	int p = tile_pixel(t, threadIdx.x, ntx, ld, H);
	tile_bitmap(bm, nwords, p, cptr, cind);
	if (gbm)
		for (int w = threadIdx.x; w < nwords; w += blockDim.x)
			gbm[(long long)t * nwords + w] = bm[w];   // kept for k_tile_fill
	const int mine = p >= 0 ? cptr[p + 1] - cptr[p] : 0;
	cnt[threadIdx.x] = mine;
	if (threadIdx.x < TILE_PARTS) {
		lo[threadIdx.x] = INT_MAX;
		hi[threadIdx.x] = -1;
		wsum[threadIdx.x] = 0;
	}
	int w0, w1;
	const int total = tile_prefix(bm, pre, nwords, w0, w1);
	int rank = 0;
	for (int q = 0; q < RAYT_THREADS; q++) {
		const int o = cnt[q];
		rank += (o > mine || (o == mine && q < (int)threadIdx.x)) ? 1 : 0;
	}
	perm[(long long)t * RAYT_THREADS + rank] = (unsigned char)threadIdx.x;
	byrank[rank] = mine;
	pixel[rank] = p;
	__syncthreads();
	const int nv = __reduce_max_sync(0xffffffffu, (byrank[threadIdx.x] + 7) >> 3);
	const int np = max(1, min(min(stride, (int)(((long long)total + part - 1) / part)), (byrank[0] + 7) >> 3));
	p = pixel[threadIdx.x];
	const int k0 = p >= 0 ? cptr[p] : 0, k1 = k0 + byrank[threadIdx.x];
	for (int i = 0; i < stride; i++) {
		int v0 = 0, v1 = 0;
		if (i < np) part_words(nv, i, np, v0, v1);
		const int ka = k0 + 8 * v0, kb = min(k1, k0 + 8 * v1);
		if (ka < kb) {
			atomicMin(&lo[i], tile_pos(bm, pre, cind[ka]));
			atomicMax(&hi[i], tile_pos(bm, pre, cind[kb - 1]));
		}
		if ((threadIdx.x & 31) == 0) {
			wlen[((long long)t * stride + i) * RAYT_WARPS + (threadIdx.x >> 5)] = 32LL * (v1 - v0);
			atomicAdd(&wsum[i], v1 - v0);
		}
	}
	__syncthreads();
	if (threadIdx.x < stride) {
		const int i = threadIdx.x, a = hi[i] < 0 ? 0 : lo[i] & ~3;
		parts[(long long)t * stride + i] = make_int4(a, hi[i] < 0 ? 0 : (hi[i] - a + 4) & ~3, wsum[i], np);
	}
	if (threadIdx.x == 0) tlen[t] = (total + 3) / 4 * 4;   // lists start on 16-byte boundaries (bulk copies)
}

// the tile's list (measurement indices in traced order) and its pixels'
// 1-based positions in their part's stretch of it, padded with 0 to the warp's
// word count
__global__ void __launch_bounds__(RAYT_THREADS) k_tile_fill(int ld, int H, int ntx, int nrays, int stride,
                                                            const int *__restrict__ cptr,
                                                            const int *__restrict__ cind,
                                                            const int *__restrict__ live_out,
                                                            const long long *__restrict__ tptr,
                                                            const long long *__restrict__ woff,
                                                            const int4 *__restrict__ parts,
                                                            const unsigned char *__restrict__ perm,
                                                            int *__restrict__ tmeas, uint4 *__restrict__ sidx,
                                                            const unsigned *__restrict__ gbm) {
	extern __shared__ unsigned bm[];   // nwords bits, then nwords exclusive prefix counts
	const int t = blockIdx.x, nwords = (nrays + 31) >> 5;
	int *pre = reinterpret_cast<int *>(bm + nwords);
	// thread = rank: its pixel in the order of decreasing list length
	const int p = tile_pixel(t, perm[(long long)t * RAYT_THREADS + threadIdx.x], ntx, ld, H);
	if (gbm) {   // the bitmap k_tile_count built
		for (int w = threadIdx.x; w < nwords; w += blockDim.x) bm[w] = gbm[(long long)t * nwords + w];
		__syncthreads();
	} else {
		tile_bitmap(bm, nwords, p, cptr, cind);
	}
	int w0, w1;
	tile_prefix(bm, pre, nwords, w0, w1);
	const long long base = tptr[t];
	for (int w = w0; w < w1; w++) {
		unsigned b = bm[w];
		int r = pre[w];
		while (b) {
			const int bit = __ffs(b) - 1;
			b &= b - 1;
			tmeas[base + r++] = live_out[w * 32 + bit];
		}
	}
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	int k = p >= 0 ? cptr[p] : 0;
	const int k1 = p >= 0 ? cptr[p + 1] : 0;
	parts += (long long)t * stride;
	const int np = parts[0].w;
	for (int i = 0; i < np; i++) {
		const long long wl = ((long long)t * stride + i) * RAYT_WARPS + wid;
		const long long v0 = woff[wl];
		const int nv = (int)((woff[wl + 1] - v0) >> 5), first = 1 - parts[i].x;
		for (int v = 0; v < nv; v++, k += 8) {
			int r[8];   // the word's eight loads first, then their positions
#pragma unroll
			for (int j = 0; j < 8; j++) r[j] = k + j < k1 ? cind[k + j] : -1;
			unsigned e[8];
#pragma unroll
			for (int j = 0; j < 8; j++) e[j] = r[j] < 0 ? 0u : (unsigned)(first + tile_pos(bm, pre, r[j]));
			sidx[v0 + 32LL * v + lane] = make_uint4(e[0] | (e[1] << 16), e[2] | (e[3] << 16), e[4] | (e[5] << 16),
			                                        e[6] | (e[7] << 16));
		}
	}
}

// the launch list of a tiled adjoint: the parts of the tiles that rays cross
// (longest work first), then the tiles that none crosses; the slots of the
// tiles that have several parts
struct VTile {
	int tile, part, parts, list, len, words;
	long long id;   // of its word offsets
	double cost() const { return 0.2 * len + 26.0 * words; }   // shared-memory wavefronts: gather, sums
};
static void upload_tiles(cudaStream_t s, std::vector<VTile> &vt, const std::vector<int> &empty, int nt, OpDev &d,
                         std::vector<void *> &owned, long long *bytes) {
	std::stable_sort(vt.begin(), vt.end(), [](const VTile &a, const VTile &b) { return a.cost() > b.cost(); });
	std::vector<int> first((size_t)nt, -1), poff(vt.size() + 1, 0);
	std::vector<int4> h(vt.size() + 1);
	int slots = 0, tmax = 0;
	bool cut = false;
	for (const VTile &v : vt) cut |= v.parts > 1;
	for (size_t i = 0; i < vt.size(); i++) {
		const VTile &v = vt[i];
		h[i] = make_int4(cut ? (int)((unsigned)v.tile | (unsigned)(v.parts - 1) << 24 | (unsigned)v.part << 28) : v.tile, v.list,
		                 v.len, (int)v.id);
		if (v.parts > 1 && first[v.tile] < 0) {
			first[v.tile] = slots;
			slots += v.parts;
		}
		poff[i] = std::max(first[v.tile], 0);
		tmax = std::max(tmax, v.len);
	}
	auto up = [&](const void *src, size_t n, size_t alloc) {
		void *q = dev_alloc(std::max(alloc, (size_t)16), s);
		owned.push_back(q);
		if (n) TG_CUDA(cudaMemcpyAsync(q, src, n, cudaMemcpyHostToDevice, s));
		*bytes += (long long)alloc;
		return q;
	};
	d.vtile = (const int4 *)up(h.data(), sizeof(int4) * vt.size(), sizeof(int4) * vt.size());
	d.tempty = (const int *)up(empty.data(), sizeof(int) * empty.size(), sizeof(int) * empty.size());
	d.tpoff = (const int *)up(poff.data(), sizeof(int) * vt.size(), sizeof(int) * vt.size());
	d.tticket = nullptr;
	d.tpart = nullptr;
	if (slots) {
		d.tticket = (unsigned *)up(nullptr, 0, sizeof(unsigned) * (size_t)nt);
		TG_CUDA(cudaMemsetAsync(d.tticket, 0, sizeof(unsigned) * (size_t)nt, s));
		d.tpart = (double *)up(nullptr, 0, sizeof(double) * (size_t)slots * RAYT_THREADS);
	}
	d.tiled = 1;
	d.tfull = (int)vt.size();
	d.tcount = d.tfull + (int)empty.size();
	d.ntiles = d.tfull + ((int)empty.size() + RAYT_ZERO_TILES - 1) / RAYT_ZERO_TILES;
	d.tmax = tmax;
	TG_CUDA(cudaFuncSetAttribute(k_ray_adj_tiled, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                             tiled_smem_bytes(RAYT_MAX_LIST)));
}

bool build_tiled_index(cudaStream_t s, int ld, int H, int nrays, const int *cptr, const int *cind,
                       const int *live_out, OpDev &d, long long *bytes, long long *kept, std::vector<void *> &owned) {
	if (nrays <= 0 || nrays > RAYT_MAX_RAYS) return false;
	const int ntx = (ld + RAYT - 1) / RAYT, nty = (H + RAYT - 1) / RAYT, nt = ntx * nty;
	const bool cut = nt <= TILE_CUT;
	const int stride = cut ? TILE_PARTS : 1;   // parts of a tile at most
	const long long nw = (long long)nt * stride * RAYT_WARPS;
	const int nwords = (nrays + 31) / 32;
	const int smem = 2 * (int)sizeof(unsigned) * nwords;
	// Each thread walks its own pixel's list of ray ids, so a warp touches 32
	// cache lines per load and reuses each over the next 31 loads: the lines
	// must stay in L1.  With no preference the driver would size shared memory
	// for the most blocks that fit (7 of 32 KB), leaving L1 little room, while
	// there are only nt blocks (256 for a 256x256 image): ask for shared memory
	// for two blocks per SM and leave the rest to L1.
	const int pct = (int)std::min<long long>(100, (2LL * (smem + 4096) * 100 + 232447) / 232448);
	for (const void *f : {(const void *)k_tile_count, (const void *)k_tile_fill}) {
		TG_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
		TG_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, pct));
	}
	long long *tlen = (long long *)dev_alloc(sizeof(long long) * (nt + 1), s);
	long long *tptr = (long long *)dev_alloc(sizeof(long long) * (nt + 1), s);
	long long *wlen = (long long *)dev_alloc(sizeof(long long) * (nw + 1), s);
	long long *woff = (long long *)dev_alloc(sizeof(long long) * (nw + 1), s);
	int4 *parts = (int4 *)dev_alloc(sizeof(int4) * (size_t)nt * stride, s);
	unsigned char *perm = (unsigned char *)dev_alloc((size_t)nt * RAYT_THREADS, s);
	// the tiles' ray bitmaps, kept from the count for the fill when they take
	// at most 512 MB (else the fill builds them again)
	const long long gbm_bytes = (long long)nt * nwords * (long long)sizeof(unsigned);
	unsigned *gbm = gbm_bytes <= (512LL << 20) ? (unsigned *)dev_alloc((size_t)gbm_bytes, s) : nullptr;
	k_tile_count<<<nt, RAYT_THREADS, smem, s>>>(ld, H, ntx, nrays, cut ? TILE_PART : INT_MAX, stride, cptr, cind, tlen, wlen,
	                                            parts, perm, gbm);
	TG_CUDA(cudaGetLastError());
	scan_counts(s, tlen, tptr, nt);
	scan_counts(s, wlen, woff, nw);
	std::vector<long long> h_tptr(nt + 1);
	std::vector<int4> h_parts((size_t)nt * stride);
	long long words = 0;
	TG_CUDA(cudaMemcpyAsync(h_tptr.data(), tptr, sizeof(long long) * (nt + 1), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaMemcpyAsync(h_parts.data(), parts, sizeof(int4) * h_parts.size(), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaMemcpyAsync(&words, woff + nw, sizeof(long long), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaStreamSynchronize(s));
	std::vector<VTile> vt;
	std::vector<int> empty;
	int longest = 0;
	for (int t = 0; t < nt; t++) {
		if (h_tptr[t + 1] == h_tptr[t]) {
			empty.push_back(t);
			continue;
		}
		const int4 *q = &h_parts[(size_t)t * stride];
		int live = 0, at = 0;
		for (int i = 0; i < q[0].w; i++) live += q[i].y > 0;
		for (int i = 0; i < q[0].w; i++)
			if (q[i].y > 0) {
				vt.push_back({t, at++, live, (int)(h_tptr[t] + q[i].x), q[i].y, q[i].z, (long long)t * stride + i});
				longest = std::max(longest, q[i].y);
			}
	}
	const bool ok = longest <= RAYT_MAX_LIST && words < (1LL << 31) && h_tptr[nt] < (1LL << 31);
	if (ok) {
		int *tmeas = (int *)dev_alloc(sizeof(int) * (size_t)std::max(h_tptr[nt], 4LL), s);
		TG_CUDA(cudaMemsetAsync(tmeas, 0, sizeof(int) * (size_t)std::max(h_tptr[nt], 4LL), s));
		uint4 *sidx = (uint4 *)dev_alloc(sizeof(uint4) * (size_t)std::max(words, 1LL), s);
		int *woff32 = (int *)dev_alloc(sizeof(int) * (nw + 1), s);
		owned.push_back(tmeas); owned.push_back(sidx); owned.push_back(woff32); owned.push_back(perm);
		k_tile_fill<<<nt, RAYT_THREADS, smem, s>>>(ld, H, ntx, nrays, stride, cptr, cind, live_out, tptr, woff, parts, perm, tmeas,
		                                           sidx, gbm);
		TG_CUDA(cudaGetLastError());
		k_to_int<<<(unsigned)((nw + 1 + 255) / 256), 256, 0, s>>>(woff, woff32, nw + 1);
		TG_CUDA(cudaGetLastError());
		*bytes = (long long)sizeof(uint4) * words + (long long)sizeof(int) * (h_tptr[nt] + (long long)vt.size() * RAYT_WARPS) +
		         (long long)nt * RAYT_THREADS;
		upload_tiles(s, vt, empty, nt, d, owned, bytes);
		*kept = *bytes + (long long)sizeof(int) * (nw + 1 - (long long)vt.size() * RAYT_WARPS);   // offsets of parts that are not there
		d.ntx = ntx;
		d.nty = nty;
		d.tmeas = tmeas; d.woff = woff32; d.sidx = sidx; d.tperm = perm;
	} else {
		dev_free(perm, s);
	}
	dev_free(gbm, s);
	dev_free(parts, s);
	dev_free(tlen, s);
	dev_free(tptr, s);
	dev_free(wlen, s);
	dev_free(woff, s);
	return ok;
}

// --- 3D brick index (once per operator) --------------------------------------
__global__ void k_entry_rows(long long rows, const int *rptr, int *row_of);
static_assert(BRICK_X * BRICK_Y * BRICK_Z == RAYT_THREADS, "a brick has as many voxels as a 2D tile has pixels");

__device__ __forceinline__ int brick_of(int v, int rvx, int rvy, int nbx, int nby) {
	const int x = v % rvx, y = (v / rvx) % rvy, z = v / (rvx * rvy);
	return x / BRICK_X + (y / BRICK_Y) * nbx + (z / BRICK_Z) * nbx * nby;
}

// run starts: hit k starts a run if it is its ray's first hit or lies in
// another brick than the hit before it (row_of: the ray of every hit)
__global__ void k_run_flags(long long total, const int *rptr, const int *row_of, const int *rind, int rvx, int rvy,
                            int nbx, int nby, long long *flag) {
	for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
	     k += (long long)gridDim.x * blockDim.x) {
		const int r = row_of[k];
		const int b = brick_of(rind[k], rvx, rvy, nbx, nby);
		flag[k] = (k == rptr[r] || b != brick_of(rind[k - 1], rvx, rvy, nbx, nby)) ? 1 : 0;
	}
}

// per run (rs: exclusive scan of the flags): its brick and its ray; the
// identity row pointers of the run -> brick matrix
__global__ void k_run_info(long long total, const long long *flag, const long long *rs, const int *row_of,
                           const int *rind, int rvx, int rvy, int nbx, int nby, int *run_brick, int *run_ray,
                           int *ident, long long runs) {
	for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
	     k += (long long)gridDim.x * blockDim.x)
		if (flag[k]) {
			const long long j = rs[k];
			run_brick[j] = brick_of(rind[k], rvx, rvy, nbx, nby);
			run_ray[j] = row_of[k];
		}
	for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j <= runs; j += (long long)gridDim.x * blockDim.x)
		ident[j] = (int)j;
}

// runs in brick order (bruns, brick offsets bptr): position of each run in
// its brick's list, and the list of measurement indices (padded offsets tptr)
__global__ void k_run_pos(long long runs, const int *bruns, const int *bptr, const int *run_brick, const int *run_ray,
                          const int *live_out, const int *tptr, int *pos_of_run, int *tmeas) {
	for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < runs;
	     j += (long long)gridDim.x * blockDim.x) {
		const int r = bruns[j], b = run_brick[r];
		const int pos = (int)(j - bptr[b]);
		pos_of_run[r] = pos;
		tmeas[tptr[b] + pos] = live_out[run_ray[r]];
	}
}

// per hit in traced order: its 1-based position in its brick's list
__global__ void k_hit_pos(long long total, const long long *rs, const int *pos_of_run, float *posf) {
	for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
	     k += (long long)gridDim.x * blockDim.x)
		posf[k] = (float)(pos_of_run[rs[k + 1] - 1] + 1);
}

__device__ __forceinline__ int brick_voxel(int t, int px, int rvx, int rvy, int rvz, int nbx, int nby) {
	const int bxy = nbx * nby;
	const int x = (t % nbx) * BRICK_X + px % BRICK_X;
	const int y = ((t % bxy) / nbx) * BRICK_Y + (px / BRICK_X) % BRICK_Y;
	const int z = (t / bxy) * BRICK_Z + px / (BRICK_X * BRICK_Y);
	return (x < rvx && y < rvy && z < rvz) ? x + y * rvx + z * rvx * rvy : -1;
}

// per brick: its voxels by decreasing list length (perm[rank] = voxel of the
// brick), the word count of every warp of ranks (32 x its longest list in
// 16-byte words of eight positions)
__global__ void __launch_bounds__(RAYT_THREADS) k_brick_count(int rvx, int rvy, int rvz, int nbx, int nby,
                                                              const int *cptr, long long *wlen, unsigned char *perm) {
	__shared__ int cnt[RAYT_THREADS];
	__shared__ int byrank[RAYT_THREADS];
	const int t = blockIdx.x;
	const int p = brick_voxel(t, threadIdx.x, rvx, rvy, rvz, nbx, nby);
	const int mine = p >= 0 ? cptr[p + 1] - cptr[p] : 0;
	cnt[threadIdx.x] = mine;
	__syncthreads();
	int rank = 0;
	for (int q = 0; q < RAYT_THREADS; q++) {
		const int o = cnt[q];
		rank += (o > mine || (o == mine && q < (int)threadIdx.x)) ? 1 : 0;
	}
	perm[(long long)t * RAYT_THREADS + rank] = (unsigned char)threadIdx.x;
	byrank[rank] = mine;
	__syncthreads();
	const int nv = __reduce_max_sync(0xffffffffu, (byrank[threadIdx.x] + 7) >> 3);
	if ((threadIdx.x & 31) == 0) wlen[(long long)t * RAYT_WARPS + (threadIdx.x >> 5)] = 32LL * nv;
}

// per brick, thread = rank: its voxel's positions packed eight to a 16-byte
// word, the words of a warp's 32 voxels interleaved, padded with 0
__global__ void __launch_bounds__(RAYT_THREADS) k_brick_fill(int rvx, int rvy, int rvz, int nbx, int nby,
                                                             const int *__restrict__ cptr,
                                                             const float *__restrict__ cval,
                                                             const long long *__restrict__ woff,
                                                             const unsigned char *__restrict__ perm,
                                                             uint4 *__restrict__ sidx) {
	const int t = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const int p = brick_voxel(t, perm[(long long)t * RAYT_THREADS + threadIdx.x], rvx, rvy, rvz, nbx, nby);
	const long long wl = (long long)t * RAYT_WARPS + wid;
	const long long v0 = woff[wl];
	const int nv = (int)((woff[wl + 1] - v0) >> 5);
	int k = p >= 0 ? cptr[p] : 0;
	const int k1 = p >= 0 ? cptr[p + 1] : 0;
	for (int v = 0; v < nv; v++, k += 8) {
		unsigned e[8];
#pragma unroll
		for (int j = 0; j < 8; j++) e[j] = k + j < k1 ? (unsigned)cval[k + j] : 0u;
		sidx[v0 + 32LL * v + lane] = make_uint4(e[0] | (e[1] << 16), e[2] | (e[3] << 16), e[4] | (e[5] << 16),
		                                        e[6] | (e[7] << 16));
	}
}

float *brick_positions(cudaStream_t s, int rvx, int rvy, int rvz, int nrays, long long total, const int *rptr,
                       const int *rind, const int *live_out, BrickLists &bl, std::vector<void *> &owned) {
	if (nrays <= 0 || total <= 0) return nullptr;
	bl.nbx = (rvx + BRICK_X - 1) / BRICK_X;
	bl.nby = (rvy + BRICK_Y - 1) / BRICK_Y;
	bl.nbz = (rvz + BRICK_Z - 1) / BRICK_Z;
	const long long nb = (long long)bl.nbx * bl.nby * bl.nbz;
	if (nb >= (1LL << 31)) return nullptr;
	bl.nb = (int)nb;
	const unsigned grid = (unsigned)std::min(8192LL, (total + 255) / 256);
	int *row_of = (int *)dev_alloc(sizeof(int) * (size_t)total, s);
	long long *flag = (long long *)dev_alloc(sizeof(long long) * (size_t)(total + 1), s);
	long long *rs = (long long *)dev_alloc(sizeof(long long) * (size_t)(total + 1), s);
	k_entry_rows<<<(unsigned)(((long long)nrays * 32 + 255) / 256), 256, 0, s>>>(nrays, rptr, row_of);
	k_run_flags<<<grid, 256, 0, s>>>(total, rptr, row_of, rind, rvx, rvy, bl.nbx, bl.nby, flag);
	TG_CUDA(cudaGetLastError());
	scan_counts(s, flag, rs, total);
	long long runs = 0;
	TG_CUDA(cudaMemcpyAsync(&runs, rs + total, sizeof(long long), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaStreamSynchronize(s));
	float *posf = nullptr;
	int *run_brick = (int *)dev_alloc(sizeof(int) * (size_t)runs, s);
	int *run_ray = (int *)dev_alloc(sizeof(int) * (size_t)runs, s);
	int *ident = (int *)dev_alloc(sizeof(int) * (size_t)(runs + 1), s);
	int *bptr = (int *)dev_alloc(sizeof(int) * (size_t)(nb + 1), s);
	int *bruns = (int *)dev_alloc(sizeof(int) * (size_t)runs, s);
	k_run_info<<<grid, 256, 0, s>>>(total, flag, rs, row_of, rind, rvx, rvy, bl.nbx, bl.nby, run_brick, run_ray, ident,
	                                runs);
	TG_CUDA(cudaGetLastError());
	// the runs of every brick in traced (ray) order: the transpose of the
	// run -> brick matrix
	build_transpose(s, runs, nb, runs, ident, run_brick, nullptr, bptr, bruns, nullptr);
	std::vector<int> h_bptr((size_t)nb + 1);
	TG_CUDA(cudaMemcpyAsync(h_bptr.data(), bptr, sizeof(int) * (size_t)(nb + 1), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaStreamSynchronize(s));
	bl.h_tptr.assign((size_t)nb + 1, 0);
	bl.tmax = 0;
	for (long long b = 0; b < nb; b++) {
		const long long len = h_bptr[b + 1] - h_bptr[b];
		bl.tmax = std::max(bl.tmax, len);
		bl.h_tptr[b + 1] = bl.h_tptr[b] + (len + 3) / 4 * 4;
	}
	if (bl.tmax <= RAYT_MAX_LIST && bl.h_tptr[nb] < (1LL << 31)) {
		std::vector<int> t32((size_t)nb + 1);
		for (long long b = 0; b <= nb; b++) t32[b] = (int)bl.h_tptr[b];
		bl.tptr = (int *)dev_alloc(sizeof(int) * (size_t)(nb + 1), s);
		owned.push_back(bl.tptr);
		TG_CUDA(cudaMemcpyAsync(bl.tptr, t32.data(), sizeof(int) * (size_t)(nb + 1), cudaMemcpyHostToDevice, s));
		const long long tl = std::max(bl.h_tptr[nb], 4LL);
		bl.tmeas = (int *)dev_alloc(sizeof(int) * (size_t)tl, s);
		owned.push_back(bl.tmeas);
		TG_CUDA(cudaMemsetAsync(bl.tmeas, 0, sizeof(int) * (size_t)tl, s));
		int *pos_of_run = (int *)dev_alloc(sizeof(int) * (size_t)runs, s);
		k_run_pos<<<(unsigned)std::min(8192LL, (runs + 255) / 256), 256, 0, s>>>(runs, bruns, bptr, run_brick, run_ray,
		                                                                          live_out, bl.tptr, pos_of_run, bl.tmeas);
		posf = (float *)dev_alloc(sizeof(float) * (size_t)total, s);
		k_hit_pos<<<grid, 256, 0, s>>>(total, rs, pos_of_run, posf);
		TG_CUDA(cudaGetLastError());
		dev_free(pos_of_run, s);
	}
	dev_free(row_of, s);
	dev_free(flag, s);
	dev_free(rs, s);
	dev_free(run_brick, s);
	dev_free(run_ray, s);
	dev_free(ident, s);
	dev_free(bptr, s);
	dev_free(bruns, s);
	return posf;
}

bool build_brick_words(cudaStream_t s, int rvx, int rvy, int rvz, const int *cptr, const float *cval,
                       BrickLists &bl, OpDev &d, long long *bytes, std::vector<void *> &owned) {
	const int nb = bl.nb;
	const long long nw = (long long)nb * RAYT_WARPS;
	long long *wlen = (long long *)dev_alloc(sizeof(long long) * (size_t)(nw + 1), s);
	long long *woff = (long long *)dev_alloc(sizeof(long long) * (size_t)(nw + 1), s);
	unsigned char *perm = (unsigned char *)dev_alloc((size_t)nb * RAYT_THREADS, s);
	k_brick_count<<<nb, RAYT_THREADS, 0, s>>>(rvx, rvy, rvz, bl.nbx, bl.nby, cptr, wlen, perm);
	TG_CUDA(cudaGetLastError());
	scan_counts(s, wlen, woff, nw);
	long long words = 0;
	TG_CUDA(cudaMemcpyAsync(&words, woff + nw, sizeof(long long), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaStreamSynchronize(s));
	const bool ok = words < (1LL << 31);
	if (ok) {
		uint4 *sidx = (uint4 *)dev_alloc(sizeof(uint4) * (size_t)std::max(words, 1LL), s);
		int *woff32 = (int *)dev_alloc(sizeof(int) * (size_t)(nw + 1), s);
		owned.push_back(sidx); owned.push_back(woff32); owned.push_back(perm);
		k_brick_fill<<<nb, RAYT_THREADS, 0, s>>>(rvx, rvy, rvz, bl.nbx, bl.nby, cptr, cval, woff, perm, sidx);
		k_to_int<<<(unsigned)((nw + 1 + 255) / 256), 256, 0, s>>>(woff, woff32, nw + 1);
		TG_CUDA(cudaGetLastError());
		*bytes = (long long)sizeof(uint4) * words + (long long)sizeof(int) * (bl.h_tptr[nb] + nw + 1) +
		         (long long)nb * RAYT_THREADS;
		std::vector<VTile> vt;
		std::vector<int> empty;
		for (int t = 0; t < nb; t++) {
			const int len = (int)(bl.h_tptr[t + 1] - bl.h_tptr[t]);
			if (len) vt.push_back({t, 0, 1, (int)bl.h_tptr[t], len, 0, t});
			else empty.push_back(t);
		}
		upload_tiles(s, vt, empty, nb, d, owned, bytes);
		d.tile3 = 1;
		d.ntx = bl.nbx;
		d.nty = bl.nby;
		d.tmeas = bl.tmeas; d.woff = woff32; d.sidx = sidx; d.tperm = perm;
	} else {
		dev_free(perm, s);
	}
	dev_free(wlen, s);
	dev_free(woff, s);
	return ok;
}

#else   // FP64 build: the ray adjoints are the pixel-major gathers
bool build_tiled_index(cudaStream_t, int, int, int, const int *, const int *, const int *, OpDev &, long long *,
                       long long *, std::vector<void *> &) {
	return false;
}
int tiled_smem_bytes(int) { return 0; }
real *brick_positions(cudaStream_t, int, int, int, int, long long, const int *, const int *, const int *, BrickLists &,
                      std::vector<void *> &) {
	return nullptr;
}
bool build_brick_words(cudaStream_t, int, int, int, const int *, const real *, BrickLists &, OpDev &, long long *,
                       std::vector<void *> &) {
	return false;
}
#endif
// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
template <int W>
static void gather_w(cudaStream_t s, const LaunchCtx &L, const TileMap &map, int pred, int kind, VecSel x,
                     VecSel y) {
	launch_pdl(k_gather<W>, map.count, 256, 0, s, L.inst, map, pred, kind, x, y, (unsigned long long *)L.launches);
}
static void gather(const LaunchCtx &L, const TileMap (&maps)[4], int pred, int kind, VecSel x, VecSel y) {
	if (maps[0].count > 0) gather_w<4>(L.stream, L, maps[0], pred, kind, x, y);
	if (maps[1].count > 0) gather_w<8>(L.stream, L, maps[1], pred, kind, x, y);
	if (maps[2].count > 0) gather_w<16>(L.stream, L, maps[2], pred, kind, x, y);
	if (maps[3].count > 0) gather_w<32>(L.stream, L, maps[3], pred, kind, x, y);
	TG_CUDA(cudaGetLastError());
}

void op_forward(const LaunchCtx &L, const OpBatch &B, int pred, VecSel x, VecSel y, bool unfused, bool xT_ready) {
	auto *ctr = (unsigned long long *)L.launches;
#ifndef TVAL3G_FP64
	for (const auto &e : B.mrhs) mrhs_apply(L.stream, L.inst, e.first, pred, *e.second, false, x, y, ctr);
#endif
	const TileMap(&df)[DENSE_FORMS] = unfused ? B.dense_fwd_nf : B.dense_fwd;
	auto dense = [&](auto kern, const TileMap &t) {
		if (t.count > 0) launch_pdl(kern, t.count, 256, 0, L.stream, L.inst, t, pred, x, y, ctr);
	};
	dense(k_dense_fwd<1, 4>, df[DENSE_ONE]);
	dense(k_dense_fwd<4, 4>, df[DENSE_FOUR]);
#ifndef TVAL3G_FP64
	dense(k_dense_fwd_smem<1, 4>, df[DENSE_SHORT]);
	dense(k_dense_fwd_smem<1, 2>, df[DENSE_LONG_ONE]);
	dense(k_dense_fwd_smem<2, 2>, df[DENSE_LONG_TWO]);
#else
	dense(k_dense_fwd<1, 1>, df[DENSE_LONG_ONE]);
#endif
	gather(L, B.csr_fwd, pred, 0, x, y);
	if (B.ray2_transpose.count > 0 && !xT_ready) {
		launch_pdl(k_transpose2d, B.ray2_transpose.count, 256, 0, L.stream, L.inst, B.ray2_transpose, pred, x, ctr);
	}
	if (B.ray3_transpose.count > 0)
		launch_pdl(k_transpose2d, B.ray3_transpose.count, 256, 0, L.stream, L.inst, B.ray3_transpose, pred, x, ctr);
	if (B.ray2_fwd[0].count > 0)
		launch_pdl(k_ray_fwd<4, false>, B.ray2_fwd[0].count, 256, 0, L.stream, L.inst, B.ray2_fwd[0], pred, x, y, ctr);
	if (B.ray2_fwd[1].count > 0)
		launch_pdl(k_ray_fwd<8, false>, B.ray2_fwd[1].count, 256, 0, L.stream, L.inst, B.ray2_fwd[1], pred, x, y, ctr);
	if (B.ray2_fwd[2].count > 0)
		launch_pdl(k_ray_fwd<16, false>, B.ray2_fwd[2].count, 256, 0, L.stream, L.inst, B.ray2_fwd[2], pred, x, y, ctr);
	if (B.ray2_fwd[3].count > 0)
		launch_pdl(k_ray_fwd_thread<false>, B.ray2_fwd[3].count, RAY1_BLOCK, 0, L.stream, L.inst, B.ray2_fwd[3], pred, x, y,
		           ctr);
	if (B.ray3_fwd[3].count > 0)
		launch_pdl(k_ray_fwd_thread<true>, B.ray3_fwd[3].count, RAY1_BLOCK, 0, L.stream, L.inst, B.ray3_fwd[3], pred, x, y,
		           ctr);
	if (B.ray3_fwd[0].count > 0)
		launch_pdl(k_ray_fwd<4, true>, B.ray3_fwd[0].count, 256, 0, L.stream, L.inst, B.ray3_fwd[0], pred, x, y, ctr);
	if (B.ray3_fwd[1].count > 0)
		launch_pdl(k_ray_fwd<8, true>, B.ray3_fwd[1].count, 256, 0, L.stream, L.inst, B.ray3_fwd[1], pred, x, y, ctr);
	if (B.ray3_fwd[2].count > 0)
		launch_pdl(k_ray_fwd<16, true>, B.ray3_fwd[2].count, 256, 0, L.stream, L.inst, B.ray3_fwd[2], pred, x, y, ctr);
}

void op_adjoint(const LaunchCtx &L, const OpBatch &B, int pred, VecSel x, VecSel y, bool unfused) {
	auto *ctr = (unsigned long long *)L.launches;
#ifndef TVAL3G_FP64
	for (const auto &e : B.mrhs) mrhs_apply(L.stream, L.inst, e.first, pred, *e.second, true, x, y, ctr);
#endif
	const TileMap &da = unfused ? B.dense_adj_nf : B.dense_adj, &dr = unfused ? B.dense_red_nf : B.dense_red;
	if (da.count > 0) {
		launch_pdl(k_dense_adj, da.count, 256, 0, L.stream, L.inst, da, pred, x, y, B.dense_part, ctr);
		launch_pdl(k_dense_red, dr.count, 256, 0, L.stream, L.inst, dr, pred, x, y, (const real *)B.dense_part, ctr);
	}
	gather(L, B.csc_adj, pred, 1, x, y);
	gather(L, B.ray_adj, pred, 2, x, y);
	if (B.ray_atomic_zero.count > 0)
		launch_pdl(k_ray_atomic_zero, B.ray_atomic_zero.count, 256, 0, L.stream, L.inst, B.ray_atomic_zero, pred, y, ctr);
	if (B.ray2_adj_atomic.count > 0)
		launch_pdl(k_ray_adj_atomic<false>, B.ray2_adj_atomic.count, 256, 0, L.stream, L.inst, B.ray2_adj_atomic, pred,
		           x, y, ctr);
	if (B.ray3_adj_atomic.count > 0)
		launch_pdl(k_ray_adj_atomic<true>, B.ray3_adj_atomic.count, 256, 0, L.stream, L.inst, B.ray3_adj_atomic, pred,
		           x, y, ctr);
#ifndef TVAL3G_FP64
	if (B.ray_adj_tiled.count > 0) {
		launch_pdl(k_ray_adj_tiled, B.ray_adj_tiled.count, RAYT_ADJ_THREADS, tiled_smem_bytes(B.tiled_tmax), L.stream,
		           L.inst, B.ray_adj_tiled, pred, x, y, B.err, ctr);
	}
#endif
}

void op_fused_normal(const LaunchCtx &L, const OpBatch &B, int pred, VecSel x, VecSel y, VecSel z, bool early) {
#ifndef TVAL3G_FP64
	auto *ctr = (unsigned long long *)L.launches;
	for (const auto &f : B.fused) {
		if (f.bands == 0) {   // whole rows in shared memory
			launch_rows(L, B, f, pred, x, y, z, early);
			continue;
		}
		int *flags = B.fused_flags + f.off, *err = B.err;
		TG_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * f.bands, L.stream));
		int inst = f.inst;
		const Inst *tab = L.inst;
		void *args[] = {(void *)&tab, (void *)&inst, (void *)&pred, (void *)&x, (void *)&y, (void *)&z,
		                (void *)&flags, (void *)&err, (void *)&ctr};
		TG_CUDA(cudaLaunchCooperativeKernel((const void *)k_dense_normal, dim3(B.fused_grid), dim3(FUSED_THREADS),
		                                    args, FUSED_DYN_BYTES, L.stream));
	}
#else
	(void)L; (void)B; (void)pred; (void)x; (void)y; (void)z; (void)early;
#endif
}

void op_normal(const LaunchCtx &L, const OpBatch &B, int pred, VecSel x, VecSel y, VecSel z) {
	op_fused_normal(L, B, pred, x, y, z, false);
	op_forward(L, B, pred, x, y, true, false);
	op_adjoint(L, B, pred, y, z, true);
}

// ---------------------------------------------------------------------------
// one-time builders
// ---------------------------------------------------------------------------
constexpr int SCAN_ITEMS = 4, SCAN_T = 256, SCAN_TILE = SCAN_ITEMS * SCAN_T;

__global__ void k_scan_tiles(const long long *in, long long *out, long long n, long long *tot) {
	__shared__ long long sh[32];
	long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
	long long v[SCAN_ITEMS], s = 0;
	for (int k = 0; k < SCAN_ITEMS; k++) {
		v[k] = (base + k < n) ? in[base + k] : 0;
		s += v[k];
	}
	// exclusive scan of the thread sums
	int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	long long incl = s;
	for (int o = 1; o < 32; o <<= 1) {
		long long t = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o) incl += t;
	}
	if (lane == 31) sh[wid] = incl;
	__syncthreads();
	if (wid == 0) {
		long long t = lane < SCAN_T / 32 ? sh[lane] : 0, ti = t;
		for (int o = 1; o < 32; o <<= 1) {
			long long u = __shfl_up_sync(0xffffffffu, ti, o);
			if (lane >= o) ti += u;
		}
		if (lane < SCAN_T / 32) sh[lane] = ti - t;
	}
	__syncthreads();
	long long run = sh[wid] + incl - s;
	for (int k = 0; k < SCAN_ITEMS; k++) {
		if (base + k < n) out[base + k] = run;
		run += v[k];
	}
	if (threadIdx.x == SCAN_T - 1) tot[blockIdx.x] = sh[wid] + incl;
}

// exclusive scan of the nb tile totals in place, by one block of 1024
// threads (each a contiguous run of totals); out[n] = the grand total
__global__ void __launch_bounds__(1024) k_scan_totals(long long *tot, int nb, long long *out, long long n) {
	__shared__ long long sh[32];
	const int t = threadIdx.x, per = (nb + 1023) / 1024;
	const int b0 = min(nb, t * per), b1 = min(nb, b0 + per);
	long long s = 0;
#pragma unroll 8
	for (int b = b0; b < b1; b++) s += tot[b];
	const int lane = t & 31, wid = t >> 5;
	long long incl = s;
	for (int o = 1; o < 32; o <<= 1) {
		const long long u = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o) incl += u;
	}
	if (lane == 31) sh[wid] = incl;
	__syncthreads();
	if (wid == 0) {
		const long long v = sh[lane];
		long long vi = v;
		for (int o = 1; o < 32; o <<= 1) {
			const long long u = __shfl_up_sync(0xffffffffu, vi, o);
			if (lane >= o) vi += u;
		}
		sh[lane] = vi - v;
	}
	__syncthreads();
	long long run = sh[wid] + incl - s;
	// eight loads before their stores: a load after a store to the same array
	// would wait for the store's data
	for (int b = b0; b < b1; b += 8) {
		long long v[8];
#pragma unroll
		for (int j = 0; j < 8; j++) v[j] = b + j < b1 ? tot[b + j] : 0;
#pragma unroll
		for (int j = 0; j < 8; j++)
			if (b + j < b1) {
				tot[b + j] = run;
				run += v[j];
			}
	}
	if (t == 1023) out[n] = sh[wid] + incl;
}

__global__ void k_scan_add(long long *out, long long n, const long long *tot) {
	long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) out[i] += tot[i / SCAN_TILE];
}

void scan_counts(cudaStream_t s, const long long *cnt, long long *out, long long n) {
	long long nb = (n + SCAN_TILE - 1) / SCAN_TILE;
	if (nb < 1) nb = 1;
	long long *tot = nullptr;
	tot = (decltype(tot))dev_alloc(sizeof(long long) * nb, s);
	k_scan_tiles<<<(unsigned)nb, SCAN_T, 0, s>>>(cnt, out, n, tot);
	k_scan_totals<<<1, 1024, 0, s>>>(tot, (int)nb, out, n);
	if (n > 0) k_scan_add<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(out, n, tot);
	TG_CUDA(cudaGetLastError());
	dev_free(tot, s);
}

__global__ void k_to_int(const long long *in, int *out, long long n) {
	long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) out[i] = (int)in[i];
}

// The transpose is a stable least-significant-digit radix sort of the CSR
// entries by column, 8 bits per pass: the entries arrive in row order, so
// each column's rows come out ascending, with no per-column sort and no
// atomics that would make the order depend on timing.
constexpr int RADIX_T = 256, RADIX_ITEMS = 16, RADIX_TILE = RADIX_T * RADIX_ITEMS;
constexpr int RADIX_WARPS = RADIX_T / 32;

// the row of every entry (warp per row)
__global__ void k_entry_rows(long long rows, const int *rptr, int *row_of) {
	long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	int lane = threadIdx.x & 31;
	if (row >= rows) return;
	for (int k = rptr[row] + lane; k < rptr[row + 1]; k += 32) row_of[k] = (int)row;
}

// digit counts of one tile of entries, hist[digit * tiles + tile]: one add for a
// warp whose entries share their digit (as those of a ray along y, low digit, or
// x, high digit, do), else one each;
// 27M entries of the 256^2 ring's 130816 rays: 57 -> 36 us.  (The warp's groups
// of equal digits by eight ballots: 106; by match.any: 145.)
__global__ void __launch_bounds__(RADIX_T) k_radix_hist(const int *__restrict__ key, long long nnz, int shift,
                                                        long long *__restrict__ hist) {
	__shared__ int cnt[256];
	cnt[threadIdx.x] = 0;
	__syncthreads();
	const long long base = (long long)blockIdx.x * RADIX_TILE + threadIdx.x;
	const int lane = threadIdx.x & 31;
	int kv[RADIX_ITEMS];
#pragma unroll
	for (int j = 0; j < RADIX_ITEMS; j++) kv[j] = base + j * RADIX_T < nnz ? key[base + j * RADIX_T] : 0;
#pragma unroll
	for (int j = 0; j < RADIX_ITEMS; j++) {
		const bool ok = base + j * RADIX_T < nnz;
		const int d = (kv[j] >> shift) & 255;
		const int d0 = __shfl_sync(0xffffffffu, d, 0);
		if (__all_sync(0xffffffffu, ok && d == d0)) {
			if (lane == 0) atomicAdd(&cnt[d0], 32);
		} else if (ok) {
			atomicAdd(&cnt[d], 1);
		}
	}
	__syncthreads();
	hist[(long long)threadIdx.x * gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// Stable scatter of one tile by its digit.  Warp w takes the tile's entries
// w * 32 RADIX_ITEMS .. in order, 32 a round, and ranks them against its own
// counts per digit - the round's lanes of a digit are the bits or-ed into the
// digit's mask - with no barrier until the warps' counts are added up.  The
// entries are placed in shared memory in digit order, then written out in slot
// order: consecutive threads write the consecutive entries of one digit to
// consecutive addresses.
// Bound: latency, so the registers that decide the resident blocks: without
// entry values (three blocks per SM) 276 -> 154 us on the 27M entries above,
// where two blocks took 328 and three barriers a round and match.any 276; HBM
// would take 66.
constexpr int RADIX_DYN_BYTES = RADIX_TILE * (8 + (int)sizeof(real));   // keys, values, entry values
template <bool VAL>   // entry values travel too
__global__ void __launch_bounds__(RADIX_T, VAL ? 2 : 3) k_radix_scatter(const int *__restrict__ key, const int *__restrict__ val,
                                                           const real *__restrict__ fval, long long nnz, int shift,
                                                           const long long *__restrict__ off,
                                                           int *__restrict__ key_out, int *__restrict__ val_out,
                                                           real *__restrict__ fval_out) {
	extern __shared__ int stage[];   // RADIX_TILE keys, then row values, then entry values (fval only)
	int *sk = stage, *sv = stage + RADIX_TILE;
	real *sf = reinterpret_cast<real *>(stage + 2 * RADIX_TILE);
	__shared__ int wcnt[RADIX_WARPS][256];   // counts, then the warps' first slots
	__shared__ unsigned wmask[RADIX_WARPS][256];   // the round's lanes of each digit
	__shared__ long long tile_off[256];      // of the digit's slot 0, were it the tile's first
	__shared__ int wsum[RADIX_WARPS];
	const int t = threadIdx.x, lane = t & 31, w = t >> 5;
	const long long first = off[(long long)t * gridDim.x + blockIdx.x];
#pragma unroll
	for (int q = 0; q < RADIX_WARPS; q++) wcnt[q][t] = wmask[q][t] = 0;
	const long long base = (long long)blockIdx.x * RADIX_TILE;
	const int cnt = (int)min((long long)RADIX_TILE, nnz - base), mine = w * 32 * RADIX_ITEMS + lane;
	key += base;
	val += base;
	int kv[RADIX_ITEMS], vv[RADIX_ITEMS], rk[RADIX_ITEMS];
	real fv[VAL ? RADIX_ITEMS : 1];
#pragma unroll
	for (int j = 0; j < RADIX_ITEMS; j++) {   // every load up front
		const int k = mine + 32 * j;
		const bool ok = k < cnt;
		kv[j] = ok ? key[k] : 0;
		vv[j] = ok ? val[k] : 0;
		if (VAL) fv[j] = ok ? fval[base + k] : 0.f;
	}
	__syncthreads();
#pragma unroll
	for (int j = 0; j < RADIX_ITEMS; j++) {
		const bool ok = mine + 32 * j < cnt;
		const int d = (kv[j] >> shift) & 255;
		if (ok) atomicOr(&wmask[w][d], 1u << lane);
		__syncwarp();
		const unsigned peers = wmask[w][d];
		const int before = wcnt[w][d];
		rk[j] = before + __popc(peers & ((1u << lane) - 1u));
		__syncwarp();
		if (ok && lane == __ffs(peers) - 1) {
			wcnt[w][d] = before + __popc(peers);
			wmask[w][d] = 0u;
		}
		__syncwarp();
	}
	__syncthreads();
	{   // digit t: its warps' first slots, after the tile's entries of smaller digits
		int run = 0;
#pragma unroll
		for (int q = 0; q < RADIX_WARPS; q++) {
			const int c = wcnt[q][t];
			wcnt[q][t] = run;
			run += c;
		}
		int inc = run;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int u = __shfl_up_sync(0xffffffffu, inc, o);
			if (lane >= o) inc += u;
		}
		if (lane == 31) wsum[w] = inc;
		__syncthreads();
		int start = inc - run;
		for (int q = 0; q < w; q++) start += wsum[q];
#pragma unroll
		for (int q = 0; q < RADIX_WARPS; q++) wcnt[q][t] += start;
		tile_off[t] = first - start;
	}
	__syncthreads();
#pragma unroll
	for (int j = 0; j < RADIX_ITEMS; j++)
		if (mine + 32 * j < cnt) {
			const int slot = wcnt[w][(kv[j] >> shift) & 255] + rk[j];
			sk[slot] = kv[j];
			sv[slot] = vv[j];
			if (VAL) sf[slot] = fv[j];
		}
	__syncthreads();
#pragma unroll 4
	for (int i = t; i < cnt; i += RADIX_T) {
		const int kk = sk[i];
		const long long pos = tile_off[(kk >> shift) & 255] + i;
		if (key_out) key_out[pos] = kk;
		val_out[pos] = sv[i];
		if (VAL) fval_out[pos] = sf[i];
	}
}

// the first entry of every column in the sorted keys, a binary search each: 16 us
// on 27M entries and 65536 columns, where finding the changes between
// neighbours, adding up counts and their scan took 86
__global__ void k_col_starts(const int *__restrict__ skey, long long nnz, long long cols, int *__restrict__ cptr) {
	const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (c > cols) return;
	long long lo = 0, hi = nnz;
	while (lo < hi) {
		const long long mid = (lo + hi) >> 1;
		if (skey[mid] < c) lo = mid + 1;
		else hi = mid;
	}
	cptr[c] = (int)lo;
}

void build_transpose(cudaStream_t s, long long rows, long long cols, long long nnz, const int *rptr,
                     const int *rind, const real *rval, int *cptr, int *cind, real *cval) {
	if (nnz <= 0 || rows <= 0) {
		TG_CUDA(cudaMemsetAsync(cptr, 0, sizeof(int) * (cols + 1), s));
		return;
	}
	int bits = 1;
	while (bits < 31 && (1LL << bits) < cols) bits++;
	const int passes = (bits + 7) / 8;
	const long long tiles = (nnz + RADIX_TILE - 1) / RADIX_TILE;
	int *k0 = nullptr, *k1 = nullptr, *v0 = nullptr, *v1 = nullptr;
	real *f0 = nullptr, *f1 = nullptr;
	long long *hist = nullptr, *hoff = nullptr;
	hist = (decltype(hist))dev_alloc(sizeof(long long) * (256 * tiles + 1), s);
	hoff = (decltype(hoff))dev_alloc(sizeof(long long) * (256 * tiles + 1), s);
	v0 = (decltype(v0))dev_alloc(sizeof(int) * nnz, s);
	k0 = (decltype(k0))dev_alloc(sizeof(int) * nnz, s);
	if (passes > 1) {
		k1 = (decltype(k1))dev_alloc(sizeof(int) * nnz, s);
		v1 = (decltype(v1))dev_alloc(sizeof(int) * nnz, s);
		if (rval) {
			f0 = (decltype(f0))dev_alloc(sizeof(real) * nnz, s);
			f1 = (decltype(f1))dev_alloc(sizeof(real) * nnz, s);
		}
	}
	k_entry_rows<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, s>>>(rows, rptr, v0);
	// pass p reads (key, row, value) from the previous pass (the CSR itself
	// first) and writes the next triple of buffers; the last pass writes
	// cind and cval, and its keys for the column offsets
	const int *kin = rind, *vin = v0;
	const real *fin = rval;
	for (int p = 0; p < passes; p++) {
		const bool last = p == passes - 1;
		int *kout = p % 2 == 0 ? k0 : k1;
		int *vout = last ? cind : (p % 2 == 0 ? v1 : v0);
		real *fout = !rval ? nullptr : last ? cval : (p % 2 == 0 ? f0 : f1);
		k_radix_hist<<<(unsigned)tiles, RADIX_T, 0, s>>>(kin, nnz, 8 * p, hist);
		scan_counts(s, hist, hoff, 256 * tiles);
		auto scatter = [&](auto kern, int dyn) {
			TG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn));
			kern<<<(unsigned)tiles, RADIX_T, dyn, s>>>(kin, vin, fin, nnz, 8 * p, hoff, kout, vout, fout);
		};
		if (rval) scatter(k_radix_scatter<true>, RADIX_DYN_BYTES);
		else scatter(k_radix_scatter<false>, RADIX_TILE * 8);
		kin = kout;
		vin = vout;
		fin = fout;
	}
	k_col_starts<<<(unsigned)((cols + 1 + 255) / 256), 256, 0, s>>>(kin, nnz, cols, cptr);
	TG_CUDA(cudaGetLastError());
	for (void *ptr : {(void *)hist, (void *)hoff, (void *)v0, (void *)v1, (void *)k0, (void *)k1, (void *)f0,
	                  (void *)f1})
		if (ptr) dev_free(ptr, s);
}

// The direction key of a ray among those of its start point: driving axis and
// its sign, then the slope along the non-contiguous minor axis in FAN_STRIPS
// strips, then the slope along the contiguous one.  Rays of one strip read few
// lines of the volume at each step: the 128^3 hemisphere's forward took 223 us
// in the geometry's own order (receivers scattered over the sphere) and, with
// 4 / 8 / 16 / 32 / 64 / 128 / 256 strips, 219 / 188 / 166 / 156 / 150 / 147 / 146.
// first: the ray starts a new start point's rays.
constexpr int FAN_STRIPS = 128, FAN_POS = 64;   // with 6 axis-and-sign classes: 16 bits, two radix passes
__global__ void k_ray_fan_key(int nrays, const int4 *rays, int *key, int *id, long long *first) {
	const int r = blockIdx.x * blockDim.x + threadIdx.x;
	if (r >= nrays) return;
	int x0, y0, z0, dx, dy, dz, out;
	const int4 pk = rays[r];
	unpack_ray(pk, x0, y0, z0, dx, dy, dz, out);
	const int mx = abs(dx), my = abs(dy), mz = abs(dz);
	int drive, M, c, o;   // driving length, contiguous and other minor displacement
	bool neg;
	if (mx >= my && mx >= mz) { drive = 0; M = mx; neg = dx < 0; c = dy; o = dz; }
	else if (my >= mx && my >= mz) { drive = 1; M = my; neg = dy < 0; c = dx; o = dz; }
	else { drive = 2; M = mz; neg = dz < 0; c = dx; o = dy; }
	const int m2 = 2 * max(M, 1);
	const int strip = min(FAN_STRIPS - 1, (o + M) * FAN_STRIPS / m2), pos = min(FAN_POS - 1, (c + M) * FAN_POS / m2);
	key[r] = ((drive * 2 + neg) * FAN_STRIPS + strip) * FAN_POS + pos;
	id[r] = r;
	bool start = r == 0;
	if (r > 0) {
		const int4 q = rays[r - 1];
		start = q.x != pk.x || ((q.y ^ pk.y) & 0xffff) != 0;
	}
	first[r] = start ? 1 : 0;
}

// the running count of start points, by original ray, at the sorted rays
__global__ void k_ray_group(int nrays, const int *id, const long long *first, const long long *before, int *key) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < nrays) key[i] = (int)(before[id[i]] + first[id[i]]);
}

__global__ void k_ray_permute(int nrays, const int *id, const int4 *rays, int4 *sorted) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < nrays) sorted[i] = rays[id[i]];
}

// Stable sort of (key, value) pairs by the key's low `bits` bits; the sorted
// values go to vout (the arrays k and v are used up).
static void radix_pairs(cudaStream_t s, int *k, int *v, long long n, int bits, int *kout, int *vout) {
	const long long tiles = (n + RADIX_TILE - 1) / RADIX_TILE;
	long long *hist = (long long *)dev_alloc(sizeof(long long) * (256 * tiles + 1), s);
	long long *hoff = (long long *)dev_alloc(sizeof(long long) * (256 * tiles + 1), s);
	TG_CUDA(cudaFuncSetAttribute(k_radix_scatter<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, RADIX_TILE * 8));
	for (int p = 0; p < (bits + 7) / 8; p++) {
		k_radix_hist<<<(unsigned)tiles, RADIX_T, 0, s>>>(k, n, 8 * p, hist);
		scan_counts(s, hist, hoff, 256 * tiles);
		k_radix_scatter<false><<<(unsigned)tiles, RADIX_T, RADIX_TILE * 8, s>>>(k, v, nullptr, n, 8 * p, hoff, kout, vout, nullptr);
		std::swap(k, kout);
		std::swap(v, vout);
	}
	if (((bits + 7) / 8) % 2 == 0) TG_CUDA(cudaMemcpyAsync(vout, v, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
	TG_CUDA(cudaGetLastError());
	dev_free(hist, s);
	dev_free(hoff, s);
}

int4 *sort_rays_3d(cudaStream_t s, int nrays, const int4 *rays, long long starts) {
	const unsigned grid = (unsigned)((nrays + 255) / 256);
	int *buf = (int *)dev_alloc(sizeof(int) * 4 * (size_t)nrays, s);
	int *k0 = buf, *k1 = buf + nrays, *v0 = k1 + nrays, *v1 = v0 + nrays;
	long long *first = (long long *)dev_alloc(sizeof(long long) * 2 * (size_t)(nrays + 1), s);
	long long *before = first + nrays + 1;
	int4 *sorted = (int4 *)dev_alloc(sizeof(int4) * (size_t)nrays, s);
	k_ray_fan_key<<<grid, 256, 0, s>>>(nrays, rays, k0, v0, first);
	scan_counts(s, first, before, nrays);
	int bits = 1;
	while ((1 << bits) < 6 * FAN_STRIPS * FAN_POS) bits++;
	radix_pairs(s, k0, v0, nrays, bits, k1, v1);   // v1: by direction
	k_ray_group<<<grid, 256, 0, s>>>(nrays, v1, first, before, k0);
	bits = 1;
	while ((1LL << bits) <= std::min<long long>(starts, nrays)) bits++;   // groups count from 1
	radix_pairs(s, k0, v1, nrays, bits, k1, v0);   // v0: by start point, then direction
	k_ray_permute<<<grid, 256, 0, s>>>(nrays, v0, rays, sorted);
	TG_CUDA(cudaGetLastError());
	dev_free(buf, s);
	dev_free(first, s);
	return sorted;
}

__global__ void k_ray_flags(long long cand, const int *up, long long ER, long long *flag) {
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < cand;
	     i += (long long)gridDim.x * blockDim.x)
		flag[i] = up[i % ER] != 0 ? 1 : 0;
}

// err[0] / err[1]: the first candidate (loop order) with an endpoint outside
// the image / a use_path index beyond numPaths
__global__ void k_ray_pack(RayGeo g, long long cand, const long long *flag, const long long *slot, int4 *rays,
                           int *out, unsigned long long *err) {
	const long long ER = (long long)g.E * g.R;
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < cand;
	     i += (long long)gridDim.x * blockDim.x) {
		if (!flag[i]) continue;
		const long long mp = i / ER, er = i - mp * ER;
		const int e = (int)(er / g.R), r = (int)(er - (long long)e * g.R);
		const int u = g.up[er];
		const long long ie = mp * g.E + e, ir = mp * g.R + r;
		const int x0 = g.xe[ie], y0 = g.ye[ie], x1 = g.xr[ir], y1 = g.yr[ir];
		const int z0 = g.is3 ? g.ze[ie] : 0, z1 = g.is3 ? g.zr[ir] : 0;
		const bool inside = x0 >= 0 && x0 < g.nx && x1 >= 0 && x1 < g.nx && y0 >= 0 && y0 < g.ny && y1 >= 0 &&
		                    y1 < g.ny && z0 >= 0 && z0 < g.nz && z1 >= 0 && z1 < g.nz;
		const long long o = g.is3 ? mp * g.numPaths + u - 1 : er;
		const bool path_ok = !g.is3 || (u >= 1 && o < g.mtot);
		if (!inside) atomicMin(err, (unsigned long long)i);
		else if (!path_ok) atomicMin(err + 1, (unsigned long long)i);
		else {
			rays[slot[i]] = pack_ray(x0, y0, z0, x1 - x0, y1 - y0, z1 - z0, (int)o);
			out[slot[i]] = (int)o;
		}
	}
}

void pack_rays(cudaStream_t s, const RayGeo &g, long long cand, long long *nrays, int4 **rays, int **out) {
	long long *flag = (long long *)dev_alloc(sizeof(long long) * (size_t)(cand + 1), s);
	long long *slot = (long long *)dev_alloc(sizeof(long long) * (size_t)(cand + 1), s);
	unsigned long long *err = (unsigned long long *)dev_alloc(2 * sizeof(unsigned long long), s);
	const unsigned grid = (unsigned)std::max(1LL, std::min(8192LL, (cand + 255) / 256));
	if (cand > 0) k_ray_flags<<<grid, 256, 0, s>>>(cand, g.up, (long long)g.E * g.R, flag);
	scan_counts(s, flag, slot, cand);
	TG_CUDA(cudaMemsetAsync(err, 0xff, 2 * sizeof(unsigned long long), s));
	long long nr = 0;
	TG_CUDA(cudaMemcpyAsync(&nr, slot + cand, sizeof(long long), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaStreamSynchronize(s));
	int4 *r = (int4 *)dev_alloc(sizeof(int4) * (size_t)std::max(nr, 1LL), s);
	int *o = (int *)dev_alloc(sizeof(int) * (size_t)std::max(nr, 1LL), s);
	if (cand > 0) k_ray_pack<<<grid, 256, 0, s>>>(g, cand, flag, slot, r, o, err);
	TG_CUDA(cudaGetLastError());
	unsigned long long h_err[2];
	TG_CUDA(cudaMemcpyAsync(h_err, err, sizeof(h_err), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaStreamSynchronize(s));
	dev_free(flag, s);
	dev_free(slot, s);
	dev_free(err, s);
	if (h_err[0] != ~0ull || h_err[1] != ~0ull) {
		dev_free(r, s);
		dev_free(o, s);
		if (h_err[0] <= h_err[1])
			throw Error{TVAL3G_ERR_ARGUMENT, g.is3 ? "Argument error: a ray endpoint lies outside the volume"
			                                       : "Argument error: a ray endpoint lies outside the image"};
		throw Error{TVAL3G_ERR_ARGUMENT, "Argument error: use_path index exceeds numPaths"};
	}
	*nrays = nr;
	*rays = r;
	*out = o;
}

__global__ void k_ray_len(int nrays, const int4 *rays, long long *len) {
	int r = blockIdx.x * blockDim.x + threadIdx.x;
	if (r >= nrays) return;
	RayWalk w(rays[r]);
	len[r] = (long long)w.M + 1;
}

__global__ void k_ray_trace(int nrays, const int4 *rays, int rvx, int rvy, const int *rptr, int *rind) {
	long long ray = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	int lane = threadIdx.x & 31;
	if (ray >= nrays) return;
	RayWalk w(rays[ray]);
	const long long rvxy = (long long)rvx * rvy;
	MinorStep s1(lane, w.a1, w.M, 32), s2(lane, w.a2, w.M, 32);
	const int base = rptr[ray];
	for (int j = lane; j <= w.M; j += 32) {
		rind[base + j] = (int)w.index(j, s1.q, s2.q, rvx, rvxy);
		s1.advance();
		s2.advance();
	}
}

int *trace_rays(cudaStream_t s, int nrays, const int4 *rays, int rvx, int rvy, int *rptr, long long *total_out) {
	long long *len = nullptr, *off = nullptr;
	len = (decltype(len))dev_alloc(sizeof(long long) * (nrays + 1), s);
	off = (decltype(off))dev_alloc(sizeof(long long) * (nrays + 1), s);
	if (nrays > 0) k_ray_len<<<(nrays + 255) / 256, 256, 0, s>>>(nrays, rays, len);
	scan_counts(s, len, off, nrays);
	long long total = 0;
	TG_CUDA(cudaMemcpyAsync(&total, off + nrays, sizeof(long long), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaStreamSynchronize(s));
	*total_out = total;
	if (total >= (1LL << 31) - 1) {
		dev_free(len, s);
		dev_free(off, s);
		throw Error{TVAL3G_ERR_ARGUMENT, "Argument error: the ray operator has more than 2^31-1 hits"};
	}
	k_to_int<<<(unsigned)((nrays + 1 + 255) / 256), 256, 0, s>>>(off, rptr, nrays + 1);
	int *rind = (int *)dev_alloc(sizeof(int) * (size_t)std::max(total, 1LL), s);
	if (nrays > 0) k_ray_trace<<<(unsigned)(((long long)nrays * 32 + 255) / 256), 256, 0, s>>>(nrays, rays, rvx, rvy, rptr, rind);
	TG_CUDA(cudaGetLastError());
	dev_free(len, s);
	dev_free(off, s);
	return rind;
}

TG_END
