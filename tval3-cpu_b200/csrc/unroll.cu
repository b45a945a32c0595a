// Differentiable unrolled TVAL3 (2D): K inner iterations of the solve with
// per-iteration (mu_k, beta_k), gradients of <gU, U_K / scl> with respect to
// b, mu_k and beta_k by a hand-written adjoint.
//
// Forward.  A plan in schedule mode runs the real FP32 solve for exactly K
// inner iterations (tol = 0, no A^T skipping) and records, per instance and
// iteration, the step actually taken (tau times the Armijo backtracking
// factor, or the restart's tau; 2d/tval3_cpu_2d.cpp:425-453,526-576) and
// whether the multipliers were updated after it (2d:673-694,820-842).  These
// decisions are then held fixed: the differentiated function F is the
// iteration map with them as constants (with bs = scl b; iteration 0 uses
// (mu_1, beta_1)):
//
//   U_0 = A^T bs;  sigma_0 = 0;  delta_0 = 0
//   iteration k >= 1:  U_k = U_{k-1} - step_k d_{k-1}
//   state(k): V = D U_k, Z = V - sigma_{k-1} / beta_k, W = S(Z, 1/beta_k),
//             E = V - W, r = A U_k - bs,
//             if outer_k: sigma_k = sigma_{k-1} - beta_k E, delta_k = delta_{k-1} - mu_k r
//             d_k = D^T (E - sigma_k / beta_k) + A^T ((mu_k r - delta_k) / beta_k)
//
// F is replayed on the device in FP64, with a checkpoint of (U, sigma,
// delta, d) every `ckpt` iterations; its U_K / scl is the forward output.
// FP64, because F is only piecewise smooth (the shrinkage switches pixels on
// and off at |Z| = 1/beta): rounding the trajectory's states to FP32 moves
// the exact gradient by up to 8e-4 relative at 128x128 with K = 50 (measured
// on the FP64 restatement), far above the FP32 forward's 2e-6.
//
// Backward.  Segment by segment from the last, the states of the segment are
// recomputed from its checkpoint and the adjoint runs back through them:
// per iteration one forward and one adjoint projector application (FP64
// gathers over the operator's CSR and its device-built CSC; for ray
// operators the traced Bresenham lists), D and D^T, the shrinkage's
// Jacobian-transpose, and FP64 inner products (block partials summed in a
// fixed order) for the mu_k and beta_k gradients.
//
// Layout.  The instances share the operator and the schedule, so up to eight
// of them run side by side: a chunk of W = 1, 2, 4 or 8 instances keeps every
// vector interleaved, element i of instance c at i W + c.  An entry of the
// operator is then read once for the chunk and its gather is one W-double
// segment instead of W scattered sectors, and an iteration is three launches:
// the image stencils (the descent step, D, the shrinkage, D^T with its
// neighbours' shrinkage recomputed), A with the measurement update as its row
// epilogue, A^T with the sum into d (or into the cotangent of U and dd).
// Measured, forward and backward of 8 instances of 128x128 (32768 rays, K =
// 10), the FP32 solve included: 23.1 ms one instance after another with one
// launch per elementary operation (nearly all of it launch latency), 4.6 ms so,
// 3.6 ms with the rows without entries left out, programmatic dependent
// launches and the last segment's states kept from the forward.  What bounds it
// now: the gathers (27 us per product of 3.4e6 entries and 8 instances, 8 TB/s
// of L2 and L1) and the FP32 solve.
#include <algorithm>
#include <cstring>
#include <vector>

#include "plan.cuh"

TG_BEGIN
namespace {

constexpr int EW_BLOCKS = 148 * 8;   // grid-stride kernels: at most one wave of 8 blocks per SM
constexpr int EW_THREADS = 256;
constexpr int NPIX = 4, NMEAS = 3;   // inner products per reverse step
constexpr int MAXW = 8;              // instances side by side
constexpr size_t ARENA_WIDE = (size_t)16 << 30;   // bytes beyond which the chunks get narrower

__device__ __forceinline__ void shrink2(double zx, double zy, double t, bool iso, double &wx, double &wy) {
	if (iso) {
		const double nrm = sqrt(zx * zx + zy * zy);
		const double s = nrm > t ? (nrm - t) / nrm : 0.0;
		wx = s * zx;
		wy = s * zy;
	} else {
		const double ax = fabs(zx) - t, ay = fabs(zy) - t;
		wx = ax > 0.0 ? (zx >= 0.0 ? ax : -ax) : 0.0;
		wy = ay > 0.0 ? (zy >= 0.0 ? ay : -ay) : 0.0;
	}
}

// Z-cotangent and the t-derivative term of W = S(Z, t) for the W-cotangent (wbx, wby)
__device__ __forceinline__ void shrink2_vjp(double zx, double zy, double t, bool iso, double wbx, double wby,
                                            double &zbx, double &zby, double &tbar) {
	if (iso) {
		const double nrm = sqrt(zx * zx + zy * zy);
		if (nrm > t) {
			const double zw = (zx * wbx + zy * wby) / nrm;
			const double a = 1.0 - t / nrm, c = t / (nrm * nrm);
			zbx = a * wbx + c * zx * zw;
			zby = a * wby + c * zy * zw;
			tbar += -zw;
		} else {
			zbx = zby = 0.0;
		}
	} else {
		const bool onx = fabs(zx) > t, ony = fabs(zy) > t;
		zbx = onx ? wbx : 0.0;
		zby = ony ? wby : 0.0;
		if (onx) tbar += (zx >= 0.0 ? -1.0 : 1.0) * wbx;
		if (ony) tbar += (zy >= 0.0 ? -1.0 : 1.0) * wby;
	}
}

template <int NS>
__device__ __forceinline__ void block_partials(double (&v)[NS], double *part) {
	__shared__ double sh[NS][EW_THREADS / 32];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
	for (int s = 0; s < NS; s++) {
		double t = warp_sum(v[s]);
		if (lane == 0) sh[s][w] = t;
	}
	__syncthreads();
	if (threadIdx.x < NS) {
		double t = 0;
		for (int k = 0; k < EW_THREADS / 32; k++) t += sh[threadIdx.x][k];
		part[blockIdx.x * NS + threadIdx.x] = t;
	}
}

// every kernel is launched with programmatic dependent launch (launch_pdl)
#define UNR_PDL()      \
	pdl_launch_next(); \
	pdl_wait_prev();

// a chunk's per-instance pointers and factors (NULL: a pad instance)
struct Lanes {
	const float *in[MAXW] = {};
	float *out[MAXW] = {};
	double a[MAXW] = {};
};

// x[i W + c] = a_c in_c[map[i]] (map NULL: i) / out_c[i] = a_c x[i W + c]
template <int W>
__global__ void k_lanes_in(long long n, const int *map, Lanes L, double *x) {
	UNR_PDL();
	for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n * W; e += (long long)gridDim.x * blockDim.x) {
		const int c = (int)(e & (W - 1));
		x[e] = L.in[c] ? L.a[c] * (double)L.in[c][map ? map[e / W] : e / W] : 0.0;
	}
}
template <int W>
__global__ void k_lanes_out(long long n, Lanes L, const double *x) {
	UNR_PDL();
	for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n * W; e += (long long)gridDim.x * blockDim.x) {
		const int c = (int)(e & (W - 1));
		if (L.out[c]) L.out[c][e / W] = (float)(L.a[c] * x[e]);
	}
}

// One launch's operator rows: y = sum of the row's entries times x, a warp per
// row, lanes (entry, instance); val NULL = every weight w (ray operators: the
// scale factor).  x NULL: the sums are 0.
struct Rows {
	long long rows;
	const int *ptr, *ind;
	const float *val;
	double w;
	const double *x;
};

// the sum of row `row`, instance lane % W, in every lane of the warp
template <int W>
__device__ __forceinline__ double row_sum(const Rows &R, long long row) {
	constexpr int G = 32 / W;   // entries per step
	const int lane = threadIdx.x & 31, c = lane % W;
	double acc = 0.0;
	if (R.x) {
		const int k1 = R.ptr[row + 1];
		int k = R.ptr[row] + lane / W;
		// four entries per lane in flight: their indices, then the gathers
		for (; k + 3 * G < k1; k += 4 * G) {
			int ii[4];
			double vv[4], xx[4];
#pragma unroll
			for (int u = 0; u < 4; u++) {
				ii[u] = __ldg(R.ind + k + u * G);
				vv[u] = R.val ? (double)__ldg(R.val + k + u * G) : R.w;
			}
#pragma unroll
			for (int u = 0; u < 4; u++) xx[u] = ld_vec(R.x + (long long)ii[u] * W + c);
#pragma unroll
			for (int u = 0; u < 4; u++) acc += vv[u] * xx[u];
		}
		for (; k < k1; k += G) acc += (R.val ? (double)__ldg(R.val + k) : R.w) * ld_vec(R.x + (long long)__ldg(R.ind + k) * W + c);
	}
#pragma unroll
	for (int o = 16; o >= W; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
	return acc;
}

// f(row, instance, element, sum) at every row and instance
template <int W, class F>
__device__ __forceinline__ void for_rows(const Rows &R, F f) {
	const int lane = threadIdx.x & 31;
	for (long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < R.rows;
	     row += ((long long)gridDim.x * blockDim.x) >> 5) {
		const double s = row_sum<W>(R, row);
		if (lane < W) f(row, lane, row * W + lane, s);
	}
}

// y = sums [+ add]
template <int W>
__global__ void __launch_bounds__(EW_THREADS) k_rows(Rows R, const double *add, double *y) {
	UNR_PDL();
	for_rows<W>(R, [&](long long, int, long long e, double s) { y[e] = add ? s + add[e] : s; });
}

// forward state, measurements: r = A U - bs, multiplier update of delta,
// q = (mu r - delta) / beta
template <int W>
__global__ void __launch_bounds__(EW_THREADS) k_state_meas(Rows R, const double *bs, const double *dl, double *dlo,
                                                           double *r, double *q, double mu, double beta,
                                                           const int *outer) {
	UNR_PDL();
	for_rows<W>(R, [&](long long, int c, long long e, double s) {
		const double rr = s - bs[e];
		double d = dl ? dl[e] : 0.0;
		if (outer && outer[c]) d -= mu * rr;
		dlo[e] = d;
		r[e] = rr;
		q[e] = (mu * rr - d) / beta;
	});
}

// reverse step, measurements (the sums: A dd); partials: <Ad, r>,
// <Ad, delta - mu r>, <delta_k-bar, r>
template <int W>
__global__ void __launch_bounds__(EW_THREADS) k_rev_meas(Rows R, const double *r, const double *dl, double *dlb,
                                                         double *bsb, double mu, double beta, const int *outer,
                                                         double *rb, double *part) {
	UNR_PDL();
	double acc[NMEAS] = {0, 0, 0};
	for_rows<W>(R, [&](long long, int c, long long e, double a) {
		const double rr = r[e];
		const double db = dlb[e] - a / beta;   // cotangent of delta_k
		double rbv = (mu / beta) * a;
		acc[0] += a * rr;
		acc[1] += a * (dl[e] - mu * rr);
		if (outer && outer[c]) {
			rbv -= mu * db;
			acc[2] += db * rr;
		}
		dlb[e] = db;
		rb[e] = rbv;
		bsb[e] -= rbv;
	});
	block_partials<NMEAS>(acc, part);
}

// U_0 = A^T bs: gb = scl (bsbar + A Ubar), at the rows' measurements
template <int W>
__global__ void __launch_bounds__(EW_THREADS) k_grad_b(Rows R, const int *map, const double *bsb, Lanes L) {
	UNR_PDL();
	for_rows<W>(R, [&](long long row, int c, long long e, double s) {
		if (L.out[c]) L.out[c][map ? map[row] : row] = (float)(L.a[c] * (bsb[e] + s));
	});
}

// a pixel of a p x q image with its periodic neighbours, as element offsets of
// instance c in the interleaved layout
template <int W>
struct Pix {
	long long e, xm, xp, ym, yp;   // itself; x - 1, x + 1, y - 1, y + 1
	int x, y;
	__device__ Pix(int p, int q, unsigned i, int c) {
		y = (int)(i / (unsigned)q);
		x = (int)(i - (unsigned)y * q);
		e = (long long)i * W + c;
		xm = e + (x > 0 ? -1 : q - 1) * W;
		xp = e + (x < q - 1 ? 1 : -(q - 1)) * W;
		ym = e + (long long)(y > 0 ? -q : (p - 1) * q) * W;
		yp = e + (long long)(y < p - 1 ? q : -(p - 1) * q) * W;
	}
};

// D^T at a pixel of (gx, gy): 2d:280-293
template <int W>
__device__ __forceinline__ double dt_pix(const Pix<W> &P, const double *gx, const double *gy) {
	return (gx[P.xm] - gx[P.e]) + (gy[P.ym] - gy[P.e]);
}

// forward state, pixels: the descent step U = U - step d (d NULL: none), V =
// D U (2d:268-293), shrinkage, multiplier update of sigma, G = E - sigma_k /
// beta and t = D^T G, with G at the two neighbours that D^T reads recomputed
// from their own U, d and sigma (a second launch would cost more than that)
template <int W>
__global__ void __launch_bounds__(EW_THREADS) k_state_pix(int p, int q, const double *U, const double *d,
                                                          const double *step, const double *sx, const double *sy,
                                                          double beta, const int *outer, int iso, double *Uo,
                                                          double *sxo, double *syo, double *t) {
	UNR_PDL();
	const double thr = 1.0 / beta;
	const long long n = (long long)p * q;
	for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < n * W; g += (long long)gridDim.x * blockDim.x) {
		const int c = (int)(g & (W - 1));
		const Pix<W> P(p, q, (unsigned)(g / W), c);
		const double a = d ? -step[c] : 0.0;
		const bool o = outer && outer[c];
		auto u = [&](long long e) { return d ? fma(a, d[e], U[e]) : U[e]; };
		auto G = [&](double u0, double ux, double uy, long long e, double &gx, double &gy, double &s_x, double &s_y) {
			const double Vx = ux - u0, Vy = uy - u0;
			double wx, wy;
			s_x = sx ? sx[e] : 0.0;
			s_y = sy ? sy[e] : 0.0;
			shrink2(Vx - s_x / beta, Vy - s_y / beta, thr, iso, wx, wy);
			const double ex = Vx - wx, ey = Vy - wy;
			if (o) {
				s_x -= beta * ex;
				s_y -= beta * ey;
			}
			gx = ex - s_x / beta;
			gy = ey - s_y / beta;
		};
		const double u0 = u(P.e), um = u(P.xm), un = u(P.ym);
		double gx, gy, gxm, gym, s_x, s_y, s1, s2, dummy;
		G(u0, u(P.xp), u(P.yp), P.e, gx, gy, s_x, s_y);
		G(um, u0, u(P.xm + (P.yp - P.e)), P.xm, gxm, dummy, s1, s2);
		G(un, u(P.ym + (P.xp - P.e)), u0, P.ym, dummy, gym, s1, s2);
		Uo[P.e] = u0;
		sxo[P.e] = s_x;
		syo[P.e] = s_y;
		t[P.e] = (gxm - gx) + (gym - gy);
	}
}

// reverse step, pixels (dd NULL: no cotangent of d yet); partials:
// <Dd, sigma_k>, <sigma_k-bar, E>, the shrinkage's t-derivative term,
// <Zbar, sigma_{k-1}>
template <int W>
__global__ void __launch_bounds__(EW_THREADS) k_rev_pix(int p, int q, const double *dd, const double *U,
                                                        const double *s0x, const double *s0y, const double *s1x,
                                                        const double *s1y, double *sbx, double *sby, double beta,
                                                        const int *outer, int iso, double *vbx, double *vby,
                                                        double *part) {
	UNR_PDL();
	const double t = 1.0 / beta;
	const long long n = (long long)p * q;
	double acc[NPIX] = {0, 0, 0, 0};
	for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < n * W; g += (long long)gridDim.x * blockDim.x) {
		const int c = (int)(g & (W - 1));
		const Pix<W> P(p, q, (unsigned)(g / W), c);
		const long long i = P.e;
		const double vx = U[P.xp] - U[i], vy = U[P.yp] - U[i];
		const double z0x = s0x ? s0x[i] : 0.0, z0y = s0y ? s0y[i] : 0.0;
		const double zx = vx - z0x / beta, zy = vy - z0y / beta;
		double wx, wy;
		shrink2(zx, zy, t, iso, wx, wy);
		const double ex = vx - wx, ey = vy - wy;
		const double dx = dd ? dd[P.xp] - dd[i] : 0.0, dy = dd ? dd[P.yp] - dd[i] : 0.0;
		const double sx = sbx[i] - dx / beta, sy = sby[i] - dy / beta;   // cotangent of sigma_k
		double ebx = dx, eby = dy;
		acc[0] += dx * s1x[i] + dy * s1y[i];
		if (outer && outer[c]) {
			ebx -= beta * sx;
			eby -= beta * sy;
			acc[1] += sx * ex + sy * ey;
		}
		double zbx, zby;
		shrink2_vjp(zx, zy, t, iso, -ebx, -eby, zbx, zby, acc[2]);
		acc[3] += zbx * z0x + zby * z0y;
		vbx[i] = ebx + zbx;
		vby[i] = eby + zby;
		sbx[i] = sx - zbx / beta;   // cotangent of sigma_{k-1}
		sby[i] = sy - zby / beta;
	}
	block_partials<NPIX>(acc, part);
}

// Ubar += A^T rb + D^T vb; dd = -step Ubar (step NULL: not needed)
template <int W>
__global__ void __launch_bounds__(EW_THREADS) k_rev_u(Rows R, int p, int q, const double *vbx, const double *vby,
                                                      double *ub, const double *step, double *dd) {
	UNR_PDL();
	for_rows<W>(R, [&](long long row, int c, long long e, double s) {
		const Pix<W> P(p, q, (unsigned)row, c);
		const double u = ub[e] + s + dt_pix(P, vbx, vby);
		ub[e] = u;
		if (step) dd[e] = -step[c] * u;
	});
}

// block k adds the block partials of reverse step k (NPIX + NMEAS sums) to
// sums[k], in a fixed order
__global__ void __launch_bounds__(EW_THREADS) k_rev_sums(const double *pp, const double *pm, int nbp, int nbm,
                                                         double *sums) {
	UNR_PDL();
	const int k = blockIdx.x;
	double v[NPIX + NMEAS] = {};
	for (int b = threadIdx.x; b < nbp; b += EW_THREADS)
#pragma unroll
		for (int s = 0; s < NPIX; s++) v[s] += pp[((long long)k * nbp + b) * NPIX + s];
	for (int b = threadIdx.x; b < nbm; b += EW_THREADS)
#pragma unroll
		for (int s = 0; s < NMEAS; s++) v[NPIX + s] += pm[((long long)k * nbm + b) * NMEAS + s];
	__shared__ double sh[(NPIX + NMEAS) * 32];
	const double t = block_sum_each<NPIX + NMEAS>(v, sh);
	if (threadIdx.x < NPIX + NMEAS) sums[k * (NPIX + NMEAS) + threadIdx.x] += t;
}

}  // namespace

struct UnrolledInst {
	std::vector<double> steps;
	std::vector<int> outer;
	double scl = 1;
};

// one state of a chunk: U, sigma, delta, the residual r = A U - bs (each
// W-interleaved)
struct ChunkState {
	double *U = nullptr, *sx = nullptr, *sy = nullptr, *dl = nullptr, *r = nullptr;
};
// up to MAXW instances side by side
struct Chunk {
	int first = 0, count = 0;            // its instances
	double *bs = nullptr;                // scl b
	double *steps = nullptr;             // K x W
	int *outer = nullptr;                // K x W
	std::vector<ChunkState> ck;          // every C iterations
	std::vector<double *> ckd;           // and their d
};

class Unrolled {
public:
	Unrolled(const tval3g_problem &p, int count, const tval3g_options &o, int K, int ckpt);
	~Unrolled();
	void forward(const float *const *d_b, const double *mu, const double *beta, float *const *d_U, cudaStream_t s);
	void backward(const float *const *d_gU, float *const *d_gb, double *g_mu, double *g_beta, cudaStream_t s);
	const UnrolledInst &inst(int i) const { return in_[i]; }
	int count() const { return count_; }
	int K() const { return K_; }

private:
	int count_, K_, C_, p_, q_, iso_;
	int W_ = 1;               // instances side by side (1, 2, 4 or 8)
	long long n_, m_, nnz_ = 0;
	Plan *plan_ = nullptr;
	// used when the caller passes the legacy default stream: blocking, so it
	// is ordered with that stream's work on both sides
	cudaStream_t own_ = nullptr;
	// the operator as a CSR over measurements and its CSC over pixels.  Rows
	// without entries (a ring's untraced rays, half of them) are left out: their
	// A U is 0, no column reads their q, and their part of every gradient is 0.
	// map_: the measurement of each row kept (NULL: all are kept); m_all_: all
	long long m_all_ = 0;
	int *map_ = nullptr;
	int *rptr_ = nullptr, *rind_ = nullptr, *cptr_ = nullptr, *cind_ = nullptr;
	float *rval_ = nullptr, *cval_ = nullptr;
	double w_ = 1.0;
	std::vector<UnrolledInst> in_;
	std::vector<Chunk> ch_;
	std::vector<double> mu_, beta_;
	std::vector<double> h_steps_;      // uploaded per chunk
	std::vector<int> h_outer_;
	std::vector<float *> eng_u_;       // the FP32 solve's U (decisions only)
	std::vector<void *> allocs_;
	// the states of a segment after its checkpoint, j = 1..C (the forward
	// writes its last segment's here, where the backward begins); d of the
	// last two iterations; seg_chunk_: the chunk whose last segment seg_ holds
	std::vector<ChunkState> seg_;
	const Chunk *seg_chunk_ = nullptr;
	double *dbuf_[2], *t_, *q_meas_;
	double *ub_, *sbx_, *sby_, *dlb_, *bsb_, *dd_, *rb_, *vbx_, *vby_;
	double *pp_, *pm_, *sums_;   // reverse steps' block partials, their sums (K + 1 steps)
	int nbp_ = 0, nbm_ = 0;      // blocks of the pixel and row kernels
	void *dmalloc(size_t bytes);
	// the FP64 buffers, one arena (256-byte aligned pieces)
	char *arena_ = nullptr;
	size_t arena_off_ = 0;
	void layout();
	double *da(long long count);
	ChunkState state_alloc(bool own_r = true);   // false: r goes to rb_, which a forward does not use
	void release();
	Rows rows(bool trans, const double *x) const;
	int row_blocks(bool trans) const;
	template <int W>
	void state(const Chunk &c, int k, const ChunkState &from, const double *d, const ChunkState &to, double *dout,
	           cudaStream_t s);
	template <int W>
	void forward_chunk(Chunk &c, const float *const *d_b, float *const *d_U, cudaStream_t s);
	template <int W>
	void backward_chunk(Chunk &c, const float *const *d_gU, float *const *d_gb, cudaStream_t s);
};

void Unrolled::layout() {
	arena_off_ = 0;
	nbp_ = (int)std::min<long long>(EW_BLOCKS, (n_ * W_ + EW_THREADS - 1) / EW_THREADS);
	ch_.clear();
	seg_.clear();
	rb_ = da(m_ * W_);
	const int nck = (K_ - 1) / C_ + 1;   // segments: states 0, C, 2 C, ... below K start one
	for (int f = 0; f < count_; f += W_) {
		Chunk c;
		c.first = f;
		c.count = std::min(W_, count_ - f);
		c.bs = da(m_ * W_);
		c.steps = da((long long)K_ * W_);
		c.outer = reinterpret_cast<int *>(da((long long)K_ * W_));
		for (int k = 0; k < nck; k++) {
			// r is read of iteration 0's state alone: the later ones, which end a
			// segment too, are recomputed as its last state
			c.ck.push_back(state_alloc(k == 0));
			c.ckd.push_back(da(n_ * W_));
		}
		ch_.push_back(c);
	}
	for (int j = 0; j < std::max(2, std::min(C_, K_)); j++) seg_.push_back(state_alloc());
	for (double **v : {&dbuf_[0], &dbuf_[1], &t_, &ub_, &sbx_, &sby_, &dd_, &vbx_, &vby_}) *v = da(n_ * W_);
	for (double **v : {&q_meas_, &dlb_, &bsb_}) *v = da(m_ * W_);
	pp_ = da((long long)(K_ + 1) * nbp_ * NPIX);
	pm_ = da((long long)(K_ + 1) * nbm_ * NMEAS);
	sums_ = da((long long)(K_ + 1) * (NPIX + NMEAS));
}

double *Unrolled::da(long long count) {
	double *p = arena_ ? reinterpret_cast<double *>(arena_ + arena_off_) : nullptr;
	arena_off_ += (sizeof(double) * (size_t)std::max(count, 1LL) + 255) / 256 * 256;
	return p;
}

void *Unrolled::dmalloc(size_t bytes) {
	void *p = nullptr;
	TG_CUDA(cudaMalloc(&p, std::max(bytes, (size_t)8)));
	allocs_.push_back(p);
	return p;
}

Unrolled::Unrolled(const tval3g_problem &p, int count, const tval3g_options &o, int K, int ckpt)
	: count_(count), K_(K), C_(ckpt) {
	TG_ARG(count >= 1 && K >= 1 && ckpt >= 1, "Argument error: count, K and the checkpoint interval must be >= 1");
	TG_ARG(p.dims == 2 && (p.op_kind == TVAL3G_OP_RAY2D || p.op_kind == TVAL3G_OP_CSR ||
	                       (p.op_kind == TVAL3G_OP_DENSE && p.layers <= 1)) && p.layers <= 1,
	       "Argument error: the unrolled solve is 2D with one layer");
	TG_ARG(!o.nonneg, "Argument error: the unrolled solve has no nonnegativity projection");
	p_ = p.dim_y;
	q_ = p.dim_x;
	iso_ = o.tv_norm != 0;
	tval3g_options oo = o;
	oo.maxit = K;
	oo.tol = 0;                 // exactly K inner iterations
	oo.maxcnt = 1 << 30;
	oo.skipMulRatio = 0;        // g = A^T (A U - b) every iteration
	std::vector<tval3g_problem> probs(count, p);
	std::vector<tval3g_options> opts(count, oo);
	tval3g_operator *op = nullptr;
	try {
		TG_CUDA(cudaStreamCreate(&own_));
		plan_ = new Plan(count, probs.data(), opts.data(), TVAL3G_GRAPH | TVAL3G_TRACE | PLAN_SCHEDULE);
		// the operator's CSR on the host: the traced rays, the caller's CSR, or the dense rows
		std::vector<long long> hp;
		std::vector<int> hi;
		std::vector<float> hv;
		if (p.op_kind == TVAL3G_OP_RAY2D) {
			int rc = tval3g_op_create(&op, &p, 0);
			if (rc != TVAL3G_OK) throw Error{rc, tval3g_last_error()};
			long long rows = 0, cols = 0, nnz = 0;
			tval3g_op_shape(op, &rows, &cols, &nnz);
			m_ = rows;
			n_ = cols;
			hp.resize(m_ + 1);
			hi.resize(std::max(nnz, 1LL));
			rc = tval3g_op_ray_csr(op, hp.data(), hi.data());
			if (rc != TVAL3G_OK) throw Error{rc, tval3g_last_error()};
			tval3g_op_destroy(op);
			op = nullptr;
			w_ = p.scale_factor;
		} else if (p.op_kind == TVAL3G_OP_CSR) {
			m_ = p.m;
			n_ = p.n_cols;
			hp.assign(p.csr_ptr, p.csr_ptr + m_ + 1);
			hi.assign(p.csr_ind, p.csr_ind + p.nnz);
			hv.assign(p.csr_val, p.csr_val + p.nnz);
		} else {
			m_ = p.m;
			n_ = p.n_cols;
			hp.resize(m_ + 1);
			for (long long r = 0; r <= m_; r++) hp[r] = r * n_;
			hi.resize(m_ * n_);
			for (long long k = 0; k < m_ * n_; k++) hi[k] = (int)(k % n_);
			hv.assign(p.A, p.A + m_ * n_);
		}
		TG_ARG(n_ == (long long)p_ * q_, "Argument error: the operator does not match the image");
		nnz_ = hp[m_];
		TG_ARG(nnz_ < (1LL << 31), "Argument error: too many operator entries");
		m_all_ = m_;
		std::vector<int> hp32(1, 0), live;
		for (long long r = 0; r < m_all_; r++)
			if (hp[r + 1] > hp[r]) {
				hp32.push_back((int)hp[r + 1]);
				live.push_back((int)r);
			}
		m_ = (long long)live.size();
		if (m_ < m_all_) {
			map_ = static_cast<int *>(dmalloc(sizeof(int) * (size_t)std::max(m_, 1LL)));
			TG_CUDA(cudaMemcpy(map_, live.data(), sizeof(int) * (size_t)m_, cudaMemcpyHostToDevice));
		}
		rptr_ = static_cast<int *>(dmalloc(sizeof(int) * (m_ + 1)));
		rind_ = static_cast<int *>(dmalloc(sizeof(int) * (size_t)nnz_));
		cptr_ = static_cast<int *>(dmalloc(sizeof(int) * (n_ + 1)));
		cind_ = static_cast<int *>(dmalloc(sizeof(int) * (size_t)nnz_));
		TG_CUDA(cudaMemcpy(rptr_, hp32.data(), sizeof(int) * (m_ + 1), cudaMemcpyHostToDevice));
		TG_CUDA(cudaMemcpy(rind_, hi.data(), sizeof(int) * (size_t)nnz_, cudaMemcpyHostToDevice));
		if (!hv.empty()) {
			rval_ = static_cast<float *>(dmalloc(sizeof(float) * (size_t)nnz_));
			cval_ = static_cast<float *>(dmalloc(sizeof(float) * (size_t)nnz_));
			TG_CUDA(cudaMemcpy(rval_, hv.data(), sizeof(float) * (size_t)nnz_, cudaMemcpyHostToDevice));
		}
		build_transpose(own_, m_, n_, nnz_, rptr_, rind_, rval_, cptr_, cind_, cval_);
		TG_CUDA(cudaStreamSynchronize(own_));
		in_.resize(count);
		for (int i = 0; i < count; i++)
			eng_u_.push_back(static_cast<float *>(dmalloc(sizeof(float) * (size_t)n_)));
		while (W_ < MAXW && W_ < count) W_ *= 2;
		nbm_ = row_blocks(false);
		// one allocation for every buffer: laid out once to size it, then at its
		// address.  A segment's states are kept for the whole chunk: long segments
		// of large images take narrower chunks (down to one instance at a time)
		for (layout(); W_ > 1 && arena_off_ > ARENA_WIDE; layout()) W_ /= 2;
		arena_ = static_cast<char *>(dmalloc(arena_off_));
		layout();
	} catch (...) {
		if (op) tval3g_op_destroy(op);
		release();
		throw;
	}
}

Unrolled::~Unrolled() { release(); }

void Unrolled::release() {
	cudaDeviceSynchronize();
	for (void *p : allocs_) cudaFree(p);
	allocs_.clear();
	delete plan_;
	plan_ = nullptr;
	if (own_) cudaStreamDestroy(own_);
	own_ = nullptr;
}

#define EW(kern, grid, ...) launch_pdl(kern, dim3(grid), dim3(EW_THREADS), 0, s, __VA_ARGS__)

ChunkState Unrolled::state_alloc(bool own_r) {
	ChunkState t;
	t.U = da(n_ * W_);
	t.sx = da(n_ * W_);
	t.sy = da(n_ * W_);
	t.dl = da(m_ * W_);
	t.r = own_r ? da(m_ * W_) : rb_;
	return t;
}

// the rows of A (trans: of A^T) applied to x
Rows Unrolled::rows(bool trans, const double *x) const {
	return Rows{trans ? n_ : m_, trans ? cptr_ : rptr_, trans ? cind_ : rind_, trans ? cval_ : rval_, w_, x};
}
int Unrolled::row_blocks(bool trans) const {
	return (int)std::max(1LL, std::min<long long>(EW_BLOCKS, ((trans ? n_ : m_) * 32 + EW_THREADS - 1) / EW_THREADS));
}

// iteration k (0: the initial state, U given): from the state `from` and its
// d to the state `to` and its d
template <int W>
void Unrolled::state(const Chunk &c, int k, const ChunkState &from, const double *d, const ChunkState &to, double *dout,
                     cudaStream_t s) {
	const int j = std::max(k, 1) - 1;
	const double mu = mu_[j], beta = beta_[j];
	const double *step = k ? c.steps + (long long)j * W : nullptr;
	const int *outer = k ? c.outer + (long long)j * W : nullptr;
	EW(k_state_pix<W>, nbp_, p_, q_, from.U, d, step, from.sx, from.sy, beta, outer, iso_, to.U, to.sx, to.sy, t_);
	EW(k_state_meas<W>, row_blocks(false), rows(false, to.U), c.bs, from.dl, to.dl, to.r, q_meas_, mu, beta, outer);
	EW(k_rows<W>, row_blocks(true), rows(true, q_meas_), t_, dout);
}

template <int W>
void Unrolled::forward_chunk(Chunk &c, const float *const *d_b, float *const *d_U, cudaStream_t s) {
	Lanes L;
	for (int i = 0; i < c.count; i++) {
		const UnrolledInst &I = in_[c.first + i];
		L.in[i] = d_b[c.first + i];
		L.a[i] = I.scl;
	}
	EW(k_lanes_in<W>, nbp_, m_, map_, L, c.bs);
	// U_0 = A^T bs, sigma and delta 0 (NULL); its state is checkpoint 0
	EW(k_rows<W>, row_blocks(true), rows(true, c.bs), nullptr, ub_);
	ChunkState init;
	init.U = ub_;
	ChunkState at = c.ck[0];
	const double *d = c.ckd[0];
	const int last = ((int)c.ck.size() - 1) * C_;   // where the last segment starts
	seg_chunk_ = &c;
	state<W>(c, 0, init, nullptr, at, c.ckd[0], s);
	for (int k = 1; k <= K_; k++) {
		const bool ck = k % C_ == 0 && k < K_;
		const ChunkState to = ck ? c.ck[k / C_] : seg_[k > last ? k - last - 1 : k & 1];
		double *dout = ck ? c.ckd[k / C_] : dbuf_[k & 1];
		state<W>(c, k, at, d, to, dout, s);
		at = to;
		d = dout;
	}
	for (int i = 0; i < c.count; i++) {
		L.out[i] = d_U[c.first + i];
		L.a[i] = 1.0 / in_[c.first + i].scl;
	}
	EW(k_lanes_out<W>, nbp_, n_, L, at.U);
}

template <int W>
void Unrolled::backward_chunk(Chunk &c, const float *const *d_gU, float *const *d_gb, cudaStream_t s) {
	const size_t nb = sizeof(double) * (size_t)(n_ * W), mb = sizeof(double) * (size_t)(m_ * W);
	Lanes L;
	for (int i = 0; i < c.count; i++) {
		L.in[i] = d_gU[c.first + i];
		L.a[i] = 1.0 / in_[c.first + i].scl;
	}
	EW(k_lanes_in<W>, nbp_, n_, nullptr, L, ub_);
	for (double *v : {sbx_, sby_}) TG_CUDA(cudaMemsetAsync(v, 0, nb, s));
	for (double *v : {dlb_, bsb_}) TG_CUDA(cudaMemsetAsync(v, 0, mb, s));
	const double *dd = nullptr;   // the cotangent of d, once there is one
	for (int g = (int)c.ck.size() - 1; g >= 0; g--) {
		const int k0 = g * C_, k1 = std::min(k0 + C_, K_);
		auto st = [&](int k) -> const ChunkState & { return k == k0 ? c.ck[g] : seg_[k - k0 - 1]; };
		if (seg_chunk_ != &c || g + 1 < (int)c.ck.size()) {
			const double *d = c.ckd[g];
			for (int k = k0 + 1; k <= k1; k++) {
				state<W>(c, k, st(k - 1), d, st(k), dbuf_[k & 1], s);
				d = dbuf_[k & 1];
			}
			seg_chunk_ = g + 1 == (int)c.ck.size() ? &c : nullptr;
		}
		for (int k = k1; k >= (g == 0 ? 0 : k0 + 1); k--) {
			const int j = std::max(k, 1) - 1;
			const double mu = mu_[j], beta = beta_[j];
			const double *step = k ? c.steps + (long long)j * W : nullptr;
			const int *outer = k ? c.outer + (long long)j * W : nullptr;
			const ChunkState &S = st(k);
			EW(k_rev_pix<W>, nbp_, p_, q_, dd, S.U, k ? st(k - 1).sx : nullptr, k ? st(k - 1).sy : nullptr, S.sx, S.sy, sbx_,
			   sby_, beta, outer, iso_, vbx_, vby_, pp_ + (long long)k * nbp_ * NPIX);
			EW(k_rev_meas<W>, nbm_, rows(false, dd), S.r, S.dl, dlb_, bsb_, mu, beta, outer, rb_,
			   pm_ + (long long)k * nbm_ * NMEAS);
			EW(k_rev_u<W>, row_blocks(true), rows(true, rb_), p_, q_, vbx_, vby_, ub_, step, dd_);
			dd = dd_;
		}
	}
	for (int i = 0; i < c.count; i++) {
		L.out[i] = d_gb[c.first + i];
		L.a[i] = in_[c.first + i].scl;
		if (map_) TG_CUDA(cudaMemsetAsync(L.out[i], 0, sizeof(float) * (size_t)m_all_, s));
	}
	EW(k_grad_b<W>, row_blocks(false), rows(false, ub_), map_, bsb_, L);
	EW(k_rev_sums, K_ + 1, pp_, pm_, nbp_, nbm_, sums_);
}

// f<W>(...) for the plan's W
#define BY_W(call)                   \
	switch (W_) {                    \
	case 1: call(1); break;          \
	case 2: call(2); break;          \
	case 4: call(4); break;          \
	default: call(8); break;         \
	}

void Unrolled::forward(const float *const *d_b, const double *mu, const double *beta, float *const *d_U,
                       cudaStream_t s) {
	if (!s) s = own_;
	seg_chunk_ = nullptr;
	mu_.assign(mu, mu + K_);
	beta_.assign(beta, beta + K_);
	// the FP32 solve that records the decisions
	plan_->set_schedule(mu, beta);
	std::vector<tval3g_info> info(count_);
	plan_->solve(d_b, nullptr, eng_u_.data(), info.data(), s);
	const std::vector<Ctrl> c = plan_->ctrl();
	std::vector<tval3g_trace_record> tr(K_);
	for (int i = 0; i < count_; i++) {
		TG_ARG(info[i].status == TVAL3G_OK, "Argument error: the forward solve stopped on a non-finite value");
		const int got = plan_->trace(i, tr.data(), K_);
		TG_ARG(got == K_, "Internal error: the forward solve did not run K iterations");
		UnrolledInst &I = in_[i];
		I.steps.resize(K_);
		I.outer.resize(K_);
		for (int k = 0; k < K_; k++) {
			I.steps[k] = tr[k].step;
			I.outer[k] = tr[k].outer != 0;
		}
		I.scl = c[i].scl;
	}
	// replay F in FP64 with checkpoints, chunk by chunk
	for (Chunk &c : ch_) {
		h_steps_.assign((size_t)K_ * W_, 0.0);
		h_outer_.assign((size_t)K_ * W_, 0);
		for (int i = 0; i < c.count; i++)
			for (int k = 0; k < K_; k++) {
				h_steps_[(size_t)k * W_ + i] = in_[c.first + i].steps[k];
				h_outer_[(size_t)k * W_ + i] = in_[c.first + i].outer[k];
			}
		TG_CUDA(cudaMemcpyAsync(c.steps, h_steps_.data(), sizeof(double) * h_steps_.size(), cudaMemcpyHostToDevice, s));
		TG_CUDA(cudaMemcpyAsync(c.outer, h_outer_.data(), sizeof(int) * h_outer_.size(), cudaMemcpyHostToDevice, s));
#define FWD(w) forward_chunk<w>(c, d_b, d_U, s)
		BY_W(FWD)
#undef FWD
	}
	TG_CUDA(cudaStreamSynchronize(s));
}

void Unrolled::backward(const float *const *d_gU, float *const *d_gb, double *g_mu, double *g_beta, cudaStream_t s) {
	TG_ARG(!mu_.empty(), "Argument error: backward before forward");
	if (!s) s = own_;
	constexpr int NS = NPIX + NMEAS;
	std::vector<double> h((size_t)(K_ + 1) * NS);
	TG_CUDA(cudaMemsetAsync(sums_, 0, sizeof(double) * h.size(), s));
	for (size_t i = ch_.size(); i-- > 0;) {   // the last chunk's last segment is still there
		Chunk &c = ch_[i];
#define BWD(w) backward_chunk<w>(c, d_gU, d_gb, s)
		BY_W(BWD)
#undef BWD
	}
	TG_CUDA(cudaMemcpyAsync(h.data(), sums_, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s));
	TG_CUDA(cudaStreamSynchronize(s));
	std::fill(g_mu, g_mu + K_, 0.0);
	std::fill(g_beta, g_beta + K_, 0.0);
	for (int k = K_; k >= 0; k--) {   // iteration 0 uses (mu_1, beta_1)
		const int j = std::max(k, 1) - 1;
		const double *P = &h[(size_t)k * NS], *M = P + NPIX;
		const double beta = beta_[j], b2 = beta * beta;
		g_mu[j] += M[0] / beta - M[2];
		g_beta[j] += P[0] / b2 + M[1] / b2 - P[1] - P[2] / b2 + P[3] / b2;
	}
}

TG_END

using namespace tval3g;

struct tval3g_unrolled {
	Unrolled *u;
};

#define UNR_BEGIN try {
#define UNR_END                                                      \
	}                                                                \
	catch (const Error &e) {                                         \
		set_error(e.msg);                                            \
		return e.code;                                               \
	}                                                                \
	catch (const std::exception &e) {                                \
		set_error(std::string("Internal error: ") + e.what());       \
		return TVAL3G_ERR_INTERNAL;                                  \
	}                                                                \
	return TVAL3G_OK;

extern "C" int tval3g_unrolled_create(tval3g_unrolled **h, const tval3g_problem *prob, int count,
                                      const tval3g_options *opts, int K, int ckpt) {
	UNR_BEGIN
	TG_ARG(h && prob && opts, "Argument error: NULL argument");
	TG_ARG(!prob->complex_data, "Argument error: the unrolled solve takes real data");
	*h = nullptr;
	auto *u = new tval3g_unrolled{nullptr};
	try {
		u->u = new Unrolled(*prob, count, *opts, K, ckpt);
	} catch (...) {
		delete u;
		throw;
	}
	*h = u;
	UNR_END
}

extern "C" int tval3g_unrolled_forward(tval3g_unrolled *h, const float *const *d_b, const double *mu,
                                       const double *beta, float *const *d_U, void *stream) {
	UNR_BEGIN
	TG_ARG(h && h->u && d_b && mu && beta && d_U, "Argument error: NULL argument");
	h->u->forward(d_b, mu, beta, d_U, (cudaStream_t)stream);
	UNR_END
}

extern "C" int tval3g_unrolled_backward(tval3g_unrolled *h, const float *const *d_gU, float *const *d_gb,
                                        double *g_mu, double *g_beta, void *stream) {
	UNR_BEGIN
	TG_ARG(h && h->u && d_gU && d_gb && g_mu && g_beta, "Argument error: NULL argument");
	h->u->backward(d_gU, d_gb, g_mu, g_beta, (cudaStream_t)stream);
	UNR_END
}

extern "C" int tval3g_unrolled_decisions(const tval3g_unrolled *h, int index, double *steps, int *outer,
                                         double *scl) {
	UNR_BEGIN
	TG_ARG(h && h->u && steps && outer && scl, "Argument error: NULL argument");
	TG_ARG(index >= 0 && index < h->u->count(), "Argument error: index out of range");
	const UnrolledInst &I = h->u->inst(index);
	TG_ARG(!I.steps.empty(), "Argument error: decisions before forward");
	for (int k = 0; k < h->u->K(); k++) {
		steps[k] = I.steps[k];
		outer[k] = I.outer[k];
	}
	*scl = I.scl;
	UNR_END
}

extern "C" int tval3g_unrolled_destroy(tval3g_unrolled *h) {
	UNR_BEGIN
	if (h) {
		delete h->u;
		delete h;
	}
	UNR_END
}
