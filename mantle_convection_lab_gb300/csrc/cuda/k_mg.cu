// Converged Stokes solve for uniform meshes: FP64 iterative refinement around
// the reference's Uzawa iteration, whose inner velocity solves run as
// multigrid-preconditioned CG in TI (float for the mixed-precision solver,
// double for the plain FP64 one), or preconditioned MINRES.  One persistent
// kernel per time step (a cooperative grid or one cluster); every loop has a cap.
//
//   refinement (FP64):  R = [F - K d - G p ; G^T d],  stop when |R|/|F| < rtol
//   correction:        the Uzawa loop of citcom_solver (Solver.c:14-249) on
//                      [K G; G^T 0][dd; dp] = [R_m; -R_c], preconditioned by
//                      dividing by BAB (the reference multiplies by BAB,
//                      Solver.c:133-134, which squares the viscosity contrast
//                      instead of cancelling it), run to outer_rtol
//   inner K^-1:         CG preconditioned by one V(nu,nu) cycle: damped Jacobi
//                      smoothing, full-weighting restriction R = P^T, bilinear
//                      prolongation P (coincident / edge / centre weights 1,
//                      1/2, 1/4 as in interp_error, Solver.c:1009-1143),
//                      re-discretised coarse operators with injected
//                      viscosity, dense inverse on the coarsest grid.
//
// The operator is matrix-free (k_march.cuh).
#include <math.h>
#include "k_mg.cuh"
#include "fp64_util.cuh"

namespace mclg {

MCLG_SHAPE_UPLOAD(upload_shape_tables_mg)


template <class T>
struct OpTab {
	T N[4][4], Dx[4][4], Dz[4][4];
	// the two magnitudes of Dx and Dz over the Gauss points, and of the linear
	// interpolation along an edge to a Gauss point (k_march.cuh)
	T axp, axm, azp, azm, p, q;
};
__constant__ OpTab<float> cTf;
__constant__ OpTab<double> cTd;
template <class T> __device__ __forceinline__ const OpTab<T> &tab();
template <> __device__ __forceinline__ const OpTab<float> &tab<float>() { return cTf; }
template <> __device__ __forceinline__ const OpTab<double> &tab<double>() { return cTd; }

// Fill the unit-Jacobian tables: r = dz/dx of the (square-per-level) elements.
void upload_op_tables(const ShapeTables &S, double r, cudaStream_t st)
{
	OpTab<double> d;
	OpTab<float> f;
	const double sr = sqrt(r);
	for (int a = 0; a < 4; a++)
		for (int g = 0; g < 4; g++) {
			d.N[a][g] = S.N[a][g];
			d.Dx[a][g] = S.dNdxi[a][g] * sr;
			d.Dz[a][g] = S.dNdeta[a][g] / sr;
			f.N[a][g] = (float)d.N[a][g];
			f.Dx[a][g] = (float)d.Dx[a][g];
			f.Dz[a][g] = (float)d.Dz[a][g];
		}
	// corner 2 (xi = eta = 1): dN/dxi = (1 + eta_g)/4
	double ap = S.dNdxi[2][0], am = S.dNdxi[2][0];
	for (int g = 1; g < 4; g++) {
		ap = fmax(ap, S.dNdxi[2][g]);
		am = fmin(am, S.dNdxi[2][g]);
	}
	d.axp = ap * sr;
	d.axm = am * sr;
	d.azp = ap / sr;
	d.azm = am / sr;
	d.p = 2.0 * ap;
	d.q = 2.0 * am;
	f.axp = (float)d.axp;
	f.axm = (float)d.axm;
	f.azp = (float)d.azp;
	f.azm = (float)d.azm;
	f.p = (float)d.p;
	f.q = (float)d.q;
	cudaMemcpyToSymbolAsync(cTd, &d, sizeof d, 0, cudaMemcpyHostToDevice, st);
	cudaMemcpyToSymbolAsync(cTf, &f, sizeof f, 0, cudaMemcpyHostToDevice, st);
}

// ---- small helpers ----------------------------------------------------------
__device__ __forceinline__ void span(Part pt, int &start, int &stride)
{
	start = pt.thread();
	stride = pt.size * blockDim.x;
}

__device__ __forceinline__ unsigned spread_bits(unsigned v)
{
	v &= 0xffffu;
	v = (v | (v << 8)) & 0x00ff00ffu;
	v = (v | (v << 4)) & 0x0f0f0f0fu;
	v = (v | (v << 2)) & 0x33333333u;
	v = (v | (v << 1)) & 0x55555555u;
	return v;
}

// Morton index of element (ex, ez) on a uniform mesh: x in the odd bits
// (morton, Tree.c:447-456).
__device__ __forceinline__ int morton(int ex, int ez)
{
	return (int)((spread_bits((unsigned)ex) << 1) | spread_bits((unsigned)ez));
}

// ---- the matrix-free operator -----------------------------------------------
#include "k_march.cuh"

// Inverse diagonal of the level operator (the element diagonals summed).
template <class T, class V>
__device__ void level_invdiag(Part pt, int N, const unsigned char *mask, const T *eta, V *invD, double2 *kdiag64)
{
	const OpTab<T> &O = tab<T>();
	const int n = N + 1;
	int i0, st;
	span(pt, i0, st);
	for (int A = i0; A < n * n; A += st) {
		const int ix = A / n, iz = A - ix * n;
		T du = 0, dw = 0;
		const int eox[4] = {ix - 1, ix - 1, ix, ix}, eoz[4] = {iz - 1, iz, iz, iz - 1}, ea[4] = {2, 3, 0, 1};
#pragma unroll
		for (int q = 0; q < 4; q++) {
			const int ex = eox[q], ez = eoz[q];
			if (ex < 0 || ex >= N || ez < 0 || ez >= N)
				continue;
			const T e[4] = {eta[ez + ex * n], eta[ez + 1 + ex * n], eta[ez + 1 + (ex + 1) * n], eta[ez + (ex + 1) * n]};
			const int a = ea[q];
#pragma unroll
			for (int g = 0; g < 4; g++) {
				T eg = 0;
#pragma unroll
				for (int c = 0; c < 4; c++)
					eg += O.N[c][g] * e[c];
				du += 2 * eg * O.Dx[a][g] * O.Dx[a][g] + eg * O.Dz[a][g] * O.Dz[a][g];
				dw += 2 * eg * O.Dz[a][g] * O.Dz[a][g] + eg * O.Dx[a][g] * O.Dx[a][g];
			}
		}
		const unsigned m = mask[A];
		V v;
		v.x = (m & 1u) ? T(0) : T(1) / du;
		v.y = (m & 2u) ? T(0) : T(1) / dw;
		invD[A] = v;
		if (kdiag64)
			kdiag64[A] = make_double2((m & 1u) ? 1.0 : (double)du, (m & 2u) ? 1.0 : (double)dw);
	}
}

// b_c = P^T r_f over the coarse nodes (full weighting 1, 1/2, 1/4).
template <class T, class V>
__device__ void restrict_res(Part pt, const MGLevel<T> &F, const MGLevel<T> &C)
{
	int i0, st;
	span(pt, i0, st);
	for (int A = i0; A < C.n * C.n; A += st) {
		const int cx = A / C.n, cz = A - cx * C.n;
		T su = 0, sw = 0;
#pragma unroll
		for (int dx = -1; dx <= 1; dx++)
#pragma unroll
			for (int dz = -1; dz <= 1; dz++) {
				const int fx = 2 * cx + dx, fz = 2 * cz + dz;
				if (fx < 0 || fx >= F.n || fz < 0 || fz >= F.n)
					continue;
				const T wgt = (dx == 0 ? T(1) : T(0.5)) * (dz == 0 ? T(1) : T(0.5));
				const V r = F.r[fz + fx * F.n];
				su += wgt * r.x;
				sw += wgt * r.y;
			}
		const unsigned m = C.mask[A];
		V o;
		o.x = (m & 1u) ? T(0) : su;
		o.y = (m & 2u) ? T(0) : sw;
		C.b[A] = o;
	}
}

// ---- coarsest grid: dense inverse -------------------------------------------
// The operator's inverse on the coarsest grid lives in the leading block's
// shared memory for the whole solve where it fits (a 4 x 4 grid has 50 dofs),
// in global memory otherwise (8 x 8: 162 dofs).  Inverting in place in shared
// memory takes 50 ranks of 2500 FP64 multiply-adds; as an augmented elimination
// in global memory the set-up of a solve took 0.57 ms.

// Tasks of each level's passes, on one block (0) and on the whole team (1).
struct Splits {
	Split lev[2][kMaxLev];
};

template <class T>
struct SolveShared {
	Splits sp;
	double m[kCoarseShared * kCoarseShared];   // the matrix, then its inverse in T in the same place
	T b[kCoarseShared];
	__device__ T *inv() { return reinterpret_cast<T *>(m); }
};

// Assemble the coarsest operator densely (FP64) into M (rows of nd), identity
// rows and columns on the Dirichlet dofs, and invert it in place by
// Gauss-Jordan (SPD: no pivoting); one block.
template <class T>
__device__ __noinline__ void coarse_invert(const MGHier<T> &H, double *M)
{
	const MGLevel<T> &L = H.lv[H.nlev - 1];
	const OpTab<double> &O = tab<double>();
	const int nd = H.cnd, n = L.n, N = L.N;
	for (int k = threadIdx.x; k < nd * nd; k += blockDim.x)
		M[k] = 0.0;
	__syncthreads();
	// elements of one colour (parities of ex, ez) share no node
	for (int col = 0; col < 4; col++) {
		const int w = (N - (col >> 1) + 1) / 2, h = (N - (col & 1) + 1) / 2;
		for (int k = threadIdx.x; k < w * h * 64; k += blockDim.x) {
			const int e = k >> 6, p = (k >> 3) & 7, q = k & 7;
			const int ex = 2 * (e / h) + (col >> 1), ez = 2 * (e % h) + (col & 1);
			const int cn[4] = {ez + ex * n, ez + 1 + ex * n, ez + 1 + (ex + 1) * n, ez + (ex + 1) * n};
			const int a = p >> 1, i = p & 1, b = q >> 1, j = q & 1;
			double kv = 0.0;
			for (int g = 0; g < 4; g++) {
				double eg = 0.0;
				for (int c = 0; c < 4; c++)
					eg += O.N[c][g] * (double)L.eta[cn[c]];
				double t;
				if (i == 0 && j == 0)
					t = 2 * O.Dx[a][g] * O.Dx[b][g] + O.Dz[a][g] * O.Dz[b][g];
				else if (i == 1 && j == 1)
					t = 2 * O.Dz[a][g] * O.Dz[b][g] + O.Dx[a][g] * O.Dx[b][g];
				else if (i == 0)
					t = O.Dz[a][g] * O.Dx[b][g];
				else
					t = O.Dx[a][g] * O.Dz[b][g];
				kv += eg * t;
			}
			const int r = 2 * cn[a] + i, c = 2 * cn[b] + j;
			const bool dr = (L.mask[cn[a]] >> i) & 1u, dc = (L.mask[cn[b]] >> j) & 1u;
			if (!dr && !dc)
				M[r * nd + c] += kv;
		}
		__syncthreads();
	}
	for (int r = threadIdx.x; r < nd; r += blockDim.x)
		if ((L.mask[r >> 1] >> (r & 1)) & 1u)
			M[r * nd + r] = 1.0;
	__syncthreads();
	__shared__ double ipiv;
	for (int k = 0; k < nd; k++) {
		if (threadIdx.x == 0) {
			ipiv = 1.0 / M[k * nd + k];
			M[k * nd + k] = 1.0;
		}
		__syncthreads();
		const double s = ipiv;
		for (int c = threadIdx.x; c < nd; c += blockDim.x)
			M[k * nd + c] *= s;
		__syncthreads();
		// a row per warp: its factor is read before any lane clears it
		const int lane = threadIdx.x & 31;
		for (int r = threadIdx.x >> 5; r < nd; r += blockDim.x >> 5) {
			if (r == k)
				continue;
			const double f = M[r * nd + k];
			__syncwarp();
			for (int c = lane; c < nd; c += 32)
				M[r * nd + c] = (c == k ? 0.0 : M[r * nd + c]) - f * M[k * nd + c];
			__syncwarp();
		}
		__syncthreads();
	}
}

template <class T>
__device__ void coarse_build(const MGHier<T> &H, SolveShared<T> &cs)
{
	const bool sh = H.cnd <= kCoarseShared;
	double *M = sh ? cs.m : H.cwork;
	const int n2 = H.cnd * H.cnd;
	coarse_invert<T>(H, M);
	if (!sh) {
		for (int k = threadIdx.x; k < n2; k += blockDim.x)
			H.cinv[k] = (T)M[k];
		__syncthreads();
		return;
	}
	constexpr int kPer = (kCoarseShared * kCoarseShared + kBlock - 1) / kBlock;
	const int nt = blockDim.x;
	T v[kPer];
#pragma unroll
	for (int u = 0; u < kPer; u++)
		v[u] = (int)threadIdx.x + u * nt < n2 ? (T)M[threadIdx.x + u * nt] : T(0);
	__syncthreads();
#pragma unroll
	for (int u = 0; u < kPer; u++)
		if ((int)threadIdx.x + u * nt < n2)
			cs.inv()[threadIdx.x + u * nt] = v[u];
	__syncthreads();
}

// x = inverse * b, four lanes per row (interleaved columns); one block.
template <class T, class V>
__device__ void coarse_solve(const MGHier<T> &H, SolveShared<T> &cs, V *x)
{
	const MGLevel<T> &L = H.lv[H.nlev - 1];
	const int nd = H.cnd;
	const bool sh = nd <= kCoarseShared;
	const T *b = reinterpret_cast<const T *>(L.b), *inv = sh ? cs.inv() : H.cinv;
	T *xo = reinterpret_cast<T *>(x);
	if (sh) {
		for (int i = threadIdx.x; i < nd; i += blockDim.x)
			cs.b[i] = b[i];
		__syncthreads();
		b = cs.b;
	}
	const int part = threadIdx.x & 3;
	for (int i0 = 0; i0 < nd; i0 += blockDim.x / 4) {
		const int i = i0 + (threadIdx.x >> 2);
		T s = 0;
		if (i < nd)
			for (int j = part; j < nd; j += 4)
				s += inv[i * nd + j] * b[j];
		s += __shfl_xor_sync(0xffffffffu, s, 1);
		s += __shfl_xor_sync(0xffffffffu, s, 2);
		if (i < nd && part == 0)
			xo[i] = s;
	}
	__syncthreads();
}

// ---- one V(nu,nu) cycle: out0 = B rhs0 -----------------------------------------
// Levels below nblk run on the whole team (team barriers); the small levels
// from nblk down run inside block 0 alone (block barriers).  Every block walks
// the same buffer bookkeeping so that all of them know where each level's
// result lies; only the active blocks do the work.
template <class T>
__device__ __forceinline__ Pass<T> level_pass(const MGLevel<T> &L, const typename V2T<T>::t *b)
{
	Pass<T> P;
	P.N = L.N;
	P.mask = L.mask;
	P.eta = L.eta;
	P.invD = L.invD;
	P.b = b;
	P.x = P.xc = P.x0 = nullptr;
	P.out = P.xout = P.bout = nullptr;
	P.nc = 0;
	P.omega = P.wload = P.c0 = T(0);
	P.cx = T(1);
	P.dotv = nullptr;
	P.dotb = false;
	return P;
}

template <class T>
__device__ __forceinline__ int sweeps(const MGHier<T> &H, int l)
{
	return l < H.lfine ? H.nu : H.nu_c;
}

// The buffer that holds level l's iterate after its passes on the way down
// (sweeps from the second on alternate), and its result on the way up.  Formed
// from the level's sweep count where it is needed: a table of them would lie
// on the stack, which misses L1 after every team barrier.
template <class T>
__device__ __forceinline__ typename V2T<T>::t *x_down(const MGHier<T> &H, int l)
{
	const int nu = sweeps(H, l);
	return nu > 2 && (nu & 1) ? H.lv[l].xb : H.lv[l].xa;
}
template <class T>
__device__ __forceinline__ typename V2T<T>::t *x_up(const MGHier<T> &H, int l)
{
	if (l == H.nlev - 1)
		return H.lv[l].xa;
	const bool b = (x_down(H, l) == H.lv[l].xb) != (sweeps(H, l) & 1);
	return b ? H.lv[l].xb : H.lv[l].xa;
}

template <class T>
__device__ __forceinline__ void level_down(Sync &sy, const Splits &sp, const MGHier<T> &H, int l,
                                           const typename V2T<T>::t *rhs0, bool wide)
{
	typedef typename V2T<T>::t V;
	const MGLevel<T> &L = H.lv[l];
	const int nu = sweeps(H, l);
	V *x = L.xa, *xt = L.xb;
	// below the finest level the right-hand side P^T r of the finer level is
	// formed in this level's first pass (and stored for its later passes)
	Pass<T> P = level_pass<T>(L, l == 0 ? rhs0 : L.b);
	if (l >= 1) {
		P.xc = H.lv[l - 1].r;
		P.nc = H.lv[l - 1].n;
		P.bout = L.b;
	}
	const Part pt = sy.part(wide);
	const Split &split = sp.lev[wide][l];
	if (nu == 1) {
		// one sweep from zero, x = omega D^-1 b, formed inside the residual pass
		P.wload = H.omega;
		P.out = L.r;
		P.xout = x;
		if (l >= 1)
			march<T, PASS_RESID, XS_ZERO_R, false>(P, pt, split, nullptr);
		else
			march<T, PASS_RESID, XS_ZERO, false>(P, pt, split, nullptr);
		sy.sync(wide);
	} else {
		// sweep 1 (from zero) fused into sweep 2; the Chebyshev pair from zero is
		// x1 = w1 D^-1 b, x2 = c1 x1 + w2 D^-1 (b - A x1)
		const bool ch = H.cheb && nu == 2;
		P.wload = ch ? H.w1 : H.omega;
		P.omega = ch ? H.w2 : H.omega;
		P.cx = ch ? H.c1 : T(1);
		P.out = x;
		if (l >= 1)
			march<T, PASS_SMOOTH, XS_ZERO_R, false>(P, pt, split, nullptr);
		else
			march<T, PASS_SMOOTH, XS_ZERO, false>(P, pt, split, nullptr);
		sy.sync(wide);
		P.cx = T(1);
		P.omega = H.omega;
		for (int s = 2; s < nu; s++) {
			P.x = x;
			P.out = xt;
			march<T, PASS_SMOOTH, XS_PLAIN, false>(P, pt, split, nullptr);
			sy.sync(wide);
			V *tmp = x;
			x = xt;
			xt = tmp;
		}
		P.x = x;
		P.out = L.r;
		march<T, PASS_RESID, XS_PLAIN, false>(P, pt, split, nullptr);
		sy.sync(wide);
	}
	// the next level forms its right-hand side from L.r in its first pass,
	// except the coarsest (a dense solve)
	if (l + 1 == H.nlev - 1) {
		restrict_res<T, V>(pt, L, H.lv[l + 1]);
		sy.sync(wide);
	}
}

// With dot (level 0 only), the last sweep also accumulates this thread's
// share of out0.dotv (out0.rhs0 without dotv) into *dot and is not followed by
// a barrier: the caller's reduction provides it.
template <class T>
__device__ __forceinline__ void level_up(Sync &sy, const Splits &sp, const MGHier<T> &H, int l,
                                         const typename V2T<T>::t *rhs0, typename V2T<T>::t *out0, bool wide,
                                         const double2 *dotv, double *dot)
{
	typedef typename V2T<T>::t V;
	const MGLevel<T> &L = H.lv[l];
	V *x = x_down(H, l);
	V *xt = (x == L.xa) ? L.xb : L.xa;
	const int nu = sweeps(H, l);
	const Part pt = sy.part(wide);
	const Split &split = sp.lev[wide][l];
	Pass<T> P = level_pass<T>(L, l == 0 ? rhs0 : L.b);
	P.xc = x_up(H, l + 1);
	P.nc = H.lv[l + 1].n;
	// the coarse-grid correction x + P xc is formed inside the first post-smoothing
	// sweep; the Chebyshev pair keeps that iterate (x0) in L.r, free on the way up,
	// for x2 = c1 x1 - c0 x0 + w2 D^-1 (b - A x1)
	const bool ch = H.cheb && nu == 2;
	for (int s = 0; s < nu; s++) {
		const bool last = l == 0 && s == nu - 1;
		V *dst = last ? out0 : xt;
		double *dp = last ? dot : nullptr;
		P.x = x;
		P.out = dst;
		P.dotv = dp ? dotv : nullptr;
		P.dotb = dp && !dotv;
		if (s == 0) {
			P.omega = ch ? H.w1 : H.omega;
			P.xout = ch ? L.r : nullptr;
			march<T, PASS_SMOOTH, XS_PROLONG, false>(P, pt, split, dp);
		} else if (ch) {
			P.omega = H.w2;
			P.cx = H.c1;
			P.c0 = H.c0;
			P.x0 = L.r;
			P.xout = nullptr;
			march<T, PASS_SMOOTH, XS_PLAIN, true>(P, pt, split, dp);
		} else {
			P.omega = H.omega;
			march<T, PASS_SMOOTH, XS_PLAIN, false>(P, pt, split, dp);
		}
		if (!dp)
			sy.sync(wide);
		xt = x;
		x = dst;
	}
}

// Everything below is inlined, once for each correction solve: the passes use
// most of a thread's registers, and as calls they saved and restored them on
// the stack on every level (25 of 98 us per MINRES iteration at 64^2).
//
// out0 = B rhs0.  *dot receives this thread's share of out0.dotv (of out0.rhs0
// without dotv) and the cycle ends without a barrier: the caller reduces *dot,
// which synchronises the team.  While the leading block works on the smallest
// levels, the others run aside().
template <class T, class Aside>
__device__ __forceinline__ void vcycle(Sync &sy, SolveShared<T> &cs, const MGHier<T> &H,
                                       const typename V2T<T>::t *rhs0, typename V2T<T>::t *out0, const double2 *dotv,
                                       double *dot, Aside aside)
{
	typedef typename V2T<T>::t V;
	const int lc = H.nlev - 1;
	// first block-local level (the coarsest always is; in one block all are)
	const int nb = sy.size > 1 ? (H.nblk < lc ? H.nblk : lc) : 0;
	const bool b0 = sy.leader();
	*dot = 0.0;
#pragma unroll 1
	for (int l = 0; l < lc; l++)
		if (l < nb || b0)
			level_down<T>(sy, cs.sp, H, l, rhs0, l < nb);
	if (b0)
		coarse_solve<T, V>(H, cs, H.lv[lc].xa);
	else
		aside();
#pragma unroll 1
	for (int l = lc - 1; l >= 0; l--) {
		if (l == nb - 1)
			sy.sync();   // block 0's coarse-level results become visible to every block
		if (l < nb || b0)
			level_up<T>(sy, cs.sp, H, l, rhs0, out0, l < nb, dotv, dot);
	}
}

// ---- inner solve: CG preconditioned by one V-cycle, all in T -----------------
// x = K^-1 b to rtol; b is overwritten.  The recurrences' scalars are formed by
// one thread of each block while the others wait for its broadcast: a division
// or a square root on every thread costs the FP64 pipe (2 lanes per clock and
// SM) about a microsecond each.  The V-cycle's last sweep forms <z, r>, and the
// operator pass the new direction p = z + beta p (into the other of two buffers:
// its neighbours still read the old one).
template <class T>
__device__ __noinline__ int pcg_inner(Sync &team, SolveShared<T> &cs, const MGHier<T> &H, typename V2T<T>::t *b,
                                      typename V2T<T>::t *x, double rtol, int maxit)
{
	typedef typename V2T<T>::t V;
	Sync sy = team;
	__shared__ double rho, bb0, co;
	const MGLevel<T> &L = H.lv[0];
	auto nodes = [&] { return H.lv[0].n * H.lv[0].n; };
	{
		const int tid = sy.tid(), nth = sy.nth(), nn = nodes();
		double bb[1] = {0.0};
		for (int A = tid; A < nn; A += nth) {
			const V bv = b[A];
			H.pr[A] = bv;
			V zero;
			zero.x = T(0);
			zero.y = T(0);
			x[A] = zero;
			const double b0 = widen(bv.x), b1 = widen(bv.y);
			bb[0] += b0 * b0 + b1 * b1;
		}
		sy.reduce_then<1>(bb, [&](const double (&v)[1]) { bb0 = v[0]; });
	}
	if (!(bb0 > 0.0)) {
		team = sy;
		return 0;
	}
	V *p = H.pp, *po = b;
	int it = 0;
	while (it < maxit) {
		double rz[1], pq[1];
		vcycle<T>(sy, cs, H, H.pr, H.pz, nullptr, rz, [] {});
		sy.reduce_then<1>(rz, [&](const double (&v)[1]) {
			co = it > 0 ? v[0] / rho : 0.0;
			rho = v[0];
		});
		Pass<T> P = level_pass<T>(L, nullptr);
		P.x = H.pz;
		P.xc = po;
		P.wload = (T)co;
		P.xout = p;
		P.out = H.pq;
		march<T, PASS_MATVEC, XS_AXPY, false>(P, sy.part(true), cs.sp.lev[1][0], pq);
		sy.reduce_then<1>(pq, [&](const double (&v)[1]) { co = rho / v[0]; });
		const double alpha = co;
		const T al = (T)alpha;
		double rr[1] = {0.0};
		const int tid = sy.tid(), nth = sy.nth(), nn = nodes();
		V *r = H.pr;
		const V *q = H.pq;
		for (int A = tid; A < nn; A += nth) {
			V xv = x[A], rv = r[A];
			const V pv = p[A], qv = q[A];
			xv.x += al * pv.x;
			xv.y += al * pv.y;
			rv.x -= al * qv.x;
			rv.y -= al * qv.y;
			x[A] = xv;
			r[A] = rv;
			const double r0 = widen(rv.x), r1 = widen(rv.y);
			rr[0] += r0 * r0 + r1 * r1;
		}
		sy.reduce<1>(rr);
		it++;
		V *t = p;
		p = po;
		po = t;
		if (!(rr[0] > rtol * rtol * bb0) || !isfinite(alpha))
			break;
	}
	sy.sync();
	team = sy;
	return it;
}

// ---- FP64 operators on the fine uniform mesh -----------------------------------
__device__ __forceinline__ void g_entries(double hx, double hz, int a, double &g0, double &g1)
{
	element_g(cS, hz, hx, a, g0, g1);
}

// Element vectors of the solve (residual, Lanczos, preconditioner, direction)
// are x-major, e = ez + ex*N0, so that a warp's elements along z are adjacent;
// only the pressure itself (a.p and its candidates and history) is in the
// mesh's Morton order.

// y = G s at every node (masked); s x-major, free dofs only.
__device__ void gmul64(int N0, const unsigned char *mask, const GTab &gt, const double *s, double2 *y, int tid,
                       int nth)
{
	const int n = N0 + 1;
	for (int A = tid; A < n * n; A += nth) {
		const int ix = A / n, iz = A - ix * n;
		double s0 = 0.0, s1 = 0.0;
		const int eox[4] = {ix - 1, ix - 1, ix, ix}, eoz[4] = {iz - 1, iz, iz, iz - 1}, ea[4] = {2, 3, 0, 1};
#pragma unroll
		for (int q = 0; q < 4; q++) {
			const int ex = eox[q], ez = eoz[q];
			if (ex < 0 || ex >= N0 || ez < 0 || ez >= N0)
				continue;
			const double se = s[ez + ex * N0];
			s0 += gt.g0[ea[q]] * se;
			s1 += gt.g1[ea[q]] * se;
		}
		const unsigned m = mask[A];
		y[A] = make_double2((m & 1u) ? 0.0 : s0, (m & 2u) ? 0.0 : s1);
	}
}

// (G^T u)_e at element (ex, ez), free dofs in ascending equation order.
__device__ __forceinline__ double gtmul64_elem(int N0, const unsigned char *mask, const GTab &gt,
                                               const double2 *u, int ex, int ez)
{
	const int n = N0 + 1;
	const int cn[4] = {ez + ex * n, ez + 1 + ex * n, ez + 1 + (ex + 1) * n, ez + (ex + 1) * n};
	double s = 0.0;
#pragma unroll
	for (int c = 0; c < 4; c++) {
		const int a = kSortedCorner[c];
		const double g0 = gt.g0[a], g1 = gt.g1[a];
		const double2 ua = u[cn[a]];
		const unsigned m = mask[cn[a]];
		if (!(m & 1u))
			s += g0 * ua.x;
		if (!(m & 2u))
			s += g1 * ua.y;
	}
	return s;
}

template <class TI>
__device__ __forceinline__ Pass<double> fine_pass64(const MGArgs<TI> &a, const double2 *d, const double *p)
{
	Pass<double> P;
	P.N = a.N0;
	P.mask = a.mask0;
	P.eta = a.vis;
	P.x = d;
	P.b = P.invD = P.xc = P.x0 = nullptr;
	P.out = P.xout = P.bout = nullptr;
	P.nc = 0;
	P.omega = P.wload = P.c0 = 0.0;
	P.cx = 1.0;
	P.dotv = nullptr;
	P.dotb = false;
	P.gp = p;
	P.gp_morton = 1;
	P.g0 = a.gt.g0[0];
	P.g1 = a.gt.g1[0];
	return P;
}

// FP64 residual R = [F - K d - G p ; G^T d] into a.R, a.Rc; rs = {|R_m|^2, |R_c|^2, |F|^2}
// summed over the team (every block holds the same values on return).  One
// pass: as three loops with two team barriers between them it took 0.61 ms at
// 1024^2.
template <class TI>
__device__ void stokes_residual(const MGArgs<TI> &a, Sync &sy, const Split &split0, const double2 *d, const double *p, double (&rs)[3])
{
	Pass<double> P = fine_pass64(a, d, p);
	P.F = a.F;
	P.out64 = a.R;
	P.gt_out = a.Rc;
	march<double, PASS_RES64, XS_PLAIN, false>(P, sy.part(true), split0, rs);
	sy.reduce<3>(rs);
}

// ---- MINRES vector kernels (FP64) ---------
// Separate functions so that their registers do not compete with the solver's
// state.  Bound by the FP64 pipe and HBM together at 1024^2 (the velocity and
// direction updates: 11 and 12 FP64 operations, 120 and 112 B per node and
// element), so each trip's loads are issued before the previous trip's
// arithmetic; conversions to and from TI go through widen / narrow.

// v_old <- az ig - dg v - gg v_old (velocity, with its TI copy into bI) and the
// same for the pressure part with Ahp, whose preconditioned vector z_p = v_p / BAB
// is formed with it; returns this thread's share of z_p.v_p.
template <class VI>
__device__ __noinline__ void minres_v_nodes(int nn, int tid, int nth, const double2 *__restrict__ az_,
                                            const double2 *__restrict__ v_, double2 *__restrict__ vo_,
                                            VI *__restrict__ bI, double ig, double dg, double gg)
{
	typedef decltype(VI().x) TI;
	double2 az, v, vo;
	auto load = [&](int A) {
		if (A < nn) {
			az = az_[A];
			v = v_[A];
			vo = vo_[A];
		}
	};
	load(tid);
	for (int A = tid; A < nn; A += nth) {
		const double2 caz = az, cv = v, cvo = vo;
		load(A + nth);
		const double2 vn = make_double2(caz.x * ig - dg * cv.x - gg * cvo.x, caz.y * ig - dg * cv.y - gg * cvo.y);
		vo_[A] = vn;
		VI w;
		w.x = narrow_to<TI>(vn.x);
		w.y = narrow_to<TI>(vn.y);
		bI[A] = w;
	}
}

__device__ __noinline__ double minres_v_elems(int ne, int tid, int nth, const double *__restrict__ ah_,
                                              const double *__restrict__ p0_, double *__restrict__ p1_,
                                              const double *__restrict__ ibab, double *__restrict__ zp1_, double ig,
                                              double dg, double gg)
{
	double ah, p0, p1, ib, acc = 0.0;
	auto load = [&](int e) {
		if (e < ne) {
			ah = ah_[e];
			p0 = p0_[e];
			p1 = p1_[e];
			ib = ibab[e];
		}
	};
	load(tid);
	for (int e = tid; e < ne; e += nth) {
		const double cah = ah, c0 = p0, c1 = p1, cib = ib;
		load(e + nth);
		const double vn = cah * ig - dg * c0 - gg * c1, z = vn * cib;
		p1_[e] = vn;
		zp1_[e] = z;
		acc += z * vn;
	}
	return acc;
}

// w_old <- z - k3 w_old - k2 w for the velocity (z in TI) and the pressure
// parts, and the solution's update: steps 0 none, 1 x += s0 w_new, 2
// x += s1 w + s0 w_new.
template <class VI>
__device__ __noinline__ void minres_w_nodes(int steps, int nn, int tid, int nth, const VI *__restrict__ z_,
                                            double2 *__restrict__ wo_, const double2 *__restrict__ w_,
                                            double2 *__restrict__ x_, double k3, double k2, double s0,
                                            double s1)
{
	VI z;
	double2 wo, w, x = make_double2(0.0, 0.0);
	auto load = [&](int A) {
		if (A < nn) {
			z = z_[A];
			wo = wo_[A];
			w = w_[A];
			if (steps > 0)
				x = x_[A];
		}
	};
	load(tid);
	for (int A = tid; A < nn; A += nth) {
		const VI cz = z;
		const double2 co = wo, cw = w;
		double2 cx = x;
		load(A + nth);
		const double2 wn = make_double2(widen(cz.x) - k3 * co.x - k2 * cw.x, widen(cz.y) - k3 * co.y - k2 * cw.y);
		wo_[A] = wn;
		if (steps > 0) {
			if (steps > 1) {
				cx.x += s1 * cw.x;
				cx.y += s1 * cw.y;
			}
			x_[A] = make_double2(cx.x + s0 * wn.x, cx.y + s0 * wn.y);
		}
	}
}

__device__ __noinline__ void minres_w_elems(int steps, int ne, int tid, int nth, const double *__restrict__ z_,
                                            double *__restrict__ wo_, const double *__restrict__ w_,
                                            double *__restrict__ x_, double k3, double k2, double s0,
                                            double s1)
{
	double z, wo, w, x = 0.0;
	auto load = [&](int e) {
		if (e < ne) {
			z = z_[e];
			wo = wo_[e];
			w = w_[e];
			if (steps > 0)
				x = x_[e];
		}
	};
	load(tid);
	for (int e = tid; e < ne; e += nth) {
		const double cz = z, co = wo, cw = w;
		double cx = x;
		load(e + nth);
		const double wn = cz - k3 * co - k2 * cw;
		wo_[e] = wn;
		if (steps > 0) {
			if (steps > 1)
				cx += s1 * cw;
			x_[e] = cx + s0 * wn;
		}
	}
}

// x += s w, the last pending step of a solve that ends before its next update
__device__ __noinline__ void minres_x_update(int nn, int ne, int tid, int nth, const double2 *__restrict__ w_,
                                             double2 *__restrict__ x_, const double *__restrict__ wp_,
                                             double *__restrict__ xp_, double s)
{
	for (int A = tid; A < nn; A += nth) {
		const double2 w = w_[A], x = x_[A];
		x_[A] = make_double2(x.x + s * w.x, x.y + s * w.y);
	}
	for (int e = tid; e < ne; e += nth)
		xp_[e] += s * wp_[e];
}

// z = M^-1 v for M = diag(one V-cycle of K, BAB): the velocity part goes
// through the TI hierarchy (z_u stays in TI), the pressure part is multiplied
// by 1/BAB (a.bab holds the reciprocal).  Returns <z, v> over the team.
template <class TI>
__device__ double block_precond(const MGArgs<TI> &a, Sync &sy, SolveShared<TI> &cs, const double2 *vu, const double *vp,
                                typename V2T<TI>::t *zu, double *zp)
{
	typedef typename V2T<TI>::t VI;
	const MGHier<TI> &H = a.H;
	const int tid = sy.tid(), nth = sy.nth();
	const int N0 = a.N0, n0 = N0 + 1, nn = n0 * n0, ne = N0 * N0;
	VI *bI = H.lv[0].b;
	for (int A = tid; A < nn; A += nth) {
		const double2 v = vu[A];
		VI w;
		w.x = narrow_to<TI>(v.x);
		w.y = narrow_to<TI>(v.y);
		bI[A] = w;
	}
	sy.sync();
	double dot[1] = {0.0};
	vcycle<TI>(sy, cs, H, bI, zu, vu, &dot[0], [] {});   // the last sweep forms <z_u, v_u>
	for (int e = tid; e < ne; e += nth) {
		const double z = vp[e] * a.bab[e];
		zp[e] = z;
		dot[0] += z * vp[e];
	}
	sy.reduce<1>(dot);
	return dot[0];
}

// Y = K u + G p and Yc = G^T u in FP64 (the Stokes operator applied to (u, p);
// p in Morton order).  Ends with a team barrier.
template <class TI>
__device__ void stokes_apply(const MGArgs<TI> &a, Sync &sy, const Split &split0, const double2 *u, const double *p, double2 *Y, double *Yc)
{
	Pass<double> P = fine_pass64(a, u, p);
	P.out64 = Y;
	P.gt_out = Yc;
	march<double, PASS_STOKES, XS_PLAIN, false>(P, sy.part(true), split0, nullptr);
	sy.sync();
}

// warm_start=4: the start of the solve is the member of
//     x(alpha, beta) = h1 + alpha (h1 - h2) + beta (h1 - 2 h2 + h3)
// (h1, h2, h3 the last three solutions) whose residual under this step's
// operator is smallest in the norm the MINRES correction works in,
// |r|_M^2 = <r, M^-1 r> with M = diag(V-cycle, BAB): a least-squares problem in
// (alpha, beta) from the residual r0 at h1 and the operator applied to the two
// differences, a_k = A D_k; with M symmetric only M^-1 a_1 and M^-1 a_2 are
// needed.  The family holds the previous solution (0, 0), the linear (1, 0)
// and the quadratic (1, 1) extrapolation in time.  (In the plain L2 norm the
// minimiser chose coefficients of 10^5 along the second difference, whose
// operator image is tiny, and the solves diverged.)  ndir = 1 uses h1, h2 only
// (beta = 0).  Coefficients outside [-4, 8] fall back to the linear
// extrapolation.  Scratch: the MINRES and inner-CG vectors, free until the
// correction solve starts.
// Measured on the 1024^2 viscosity-contrast workload: the minimiser picks the
// quadratic member, MINRES needs about half the iterations of the linear start
// for some ten steps, then more and more (the error the solves leave behind is
// carried on and amplified from step to step), 111 against 100 per step over
// 30 steps; warm_start=3 stays the default there.
template <class TI>
__device__ __noinline__ void warm_guess(const MGArgs<TI> &a, Sync &sy, SolveShared<TI> &cs, int ndir)
{
	typedef typename V2T<TI>::t VI;
	const int tid = sy.tid(), nth = sy.nth();
	const int N0 = a.N0, n0 = N0 + 1, nn = n0 * n0, ne = N0 * N0;
	double2 *U1 = a.mw[0], *U2 = a.mw[1], *Y1 = a.mv[0], *Y2 = a.mv[1];
	double *P1 = a.mwp[0], *P2 = a.mwp[1], *Yc1 = a.mvp[0], *Yc2 = a.mvp[1];
	VI *Z1 = a.H.px, *Z2 = a.H.pr;
	double *Zp1 = a.mzp[0], *Zp2 = a.mzp[1];
	double rs[3];
	stokes_residual(a, sy, cs.sp.lev[1][0], a.h1d, a.h1p, rs);   // a.R = F - K h1 - G p1, a.Rc = G^T h1
	for (int A = tid; A < nn; A += nth) {
		const double2 x1 = a.h1d[A], x2 = a.h2d[A];
		U1[A] = make_double2(x1.x - x2.x, x1.y - x2.y);
		if (ndir == 2) {
			const double2 x3 = a.h3d[A];
			U2[A] = make_double2(x1.x - 2.0 * x2.x + x3.x, x1.y - 2.0 * x2.y + x3.y);
		}
	}
	for (int e = tid; e < ne; e += nth) {
		P1[e] = a.h1p[e] - a.h2p[e];
		if (ndir == 2)
			P2[e] = a.h1p[e] - 2.0 * a.h2p[e] + a.h3p[e];
	}
	sy.sync();
	stokes_apply(a, sy, cs.sp.lev[1][0], U1, P1, Y1, Yc1);
	if (ndir == 2)
		stokes_apply(a, sy, cs.sp.lev[1][0], U2, P2, Y2, Yc2);
	// M^-1 a_k (the preconditioner's pressure part divides by BAB); the signs of
	// the continuity parts follow r = [F - K d - G p ; -G^T d]
	double q[5];   // <a1, M^-1 a1>, <a2, M^-1 a1>, <a2, M^-1 a2>, <r0, M^-1 a1>, <r0, M^-1 a2>
	q[0] = block_precond(a, sy, cs, Y1, Yc1, Z1, Zp1);
	q[2] = ndir == 2 ? block_precond(a, sy, cs, Y2, Yc2, Z2, Zp2) : 0.0;
	double c[3] = {0.0, 0.0, 0.0};
	for (int A = tid; A < nn; A += nth) {
		const double2 r = a.R[A];
		const VI z1 = Z1[A];
		c[1] += (double)z1.x * r.x + (double)z1.y * r.y;
		if (ndir == 2) {
			const double2 y2 = Y2[A];
			const VI z2 = Z2[A];
			c[0] += (double)z1.x * y2.x + (double)z1.y * y2.y;
			c[2] += (double)z2.x * r.x + (double)z2.y * r.y;
		}
	}
	for (int e = tid; e < ne; e += nth) {
		const double rc = -a.Rc[e];
		c[1] += Zp1[e] * rc;
		if (ndir == 2) {
			c[0] += Zp1[e] * Yc2[e];
			c[2] += Zp2[e] * rc;
		}
	}
	sy.reduce<3>(c);
	q[1] = c[0];
	q[3] = c[1];
	q[4] = c[2];
	// every thread holds the same q: the same coefficients and branches
	double al = q[0] > 0.0 ? q[3] / q[0] : 1.0, be = 0.0;
	if (ndir == 2) {
		const double det = q[0] * q[2] - q[1] * q[1];
		if (det > 1e-12 * q[0] * q[2]) {
			al = (q[3] * q[2] - q[4] * q[1]) / det;
			be = (q[4] * q[0] - q[3] * q[1]) / det;
		}
	}
	if (!isfinite(al) || !isfinite(be) || al < -4.0 || al > 8.0 || be < -4.0 || be > 8.0) {
		al = 1.0;
		be = 0.0;
	}
	for (int A = tid; A < nn; A += nth) {
		const double2 x1 = a.h1d[A], u1 = U1[A];
		double2 d = make_double2(x1.x + al * u1.x, x1.y + al * u1.y);
		if (ndir == 2) {
			const double2 u2 = U2[A];
			d.x += be * u2.x;
			d.y += be * u2.y;
		}
		a.d[A] = d;
	}
	for (int e = tid; e < ne; e += nth)
		a.p[e] = a.h1p[e] + al * P1[e] + (ndir == 2 ? be * P2[e] : 0.0);
	if (tid == 0) {
		a.sc->warm_a = al;
		a.sc->warm_b = be;
	}
	sy.sync();
}

// The scalars of the MINRES recurrences, formed by one thread of each block
// (all blocks hold the same sums, so all form the same values).
struct MinresScal {
	double gam, gam_prev, eta, eta0, delta, c_prev, c_cur, s_prev, s_cur;
	double ig, dg, gg, k2, k3, step, step1;   // step1: the step of the iteration before
	double k1, k1p;   // factors of the directions w(j) = k1 y(j) and w(j-1) = k1p y(j-1)
	int stop;   // 1: last iteration; 2: breakdown before the update; 4: a non-finite value
};

// Correction solve by preconditioned MINRES (the Lanczos-based algorithm of
// Elman, Silvester and Wathen, "Finite Elements and Fast Iterative Solvers",
// Alg. 4.1) on [K G; G^T 0][x_u; x_p] = [R_m; -R_c] from a zero start, with
// the block-diagonal SPD preconditioner diag(V-cycle, BAB).  K is applied in
// TI, G in FP64 and G^T in float pairs (gt_elem), in one pass over the mesh; Lanczos and
// direction vectors are FP64 and x_u, x_p accumulate in a.dd, a.dpv.  The FP64
// refinement around this solve restores full accuracy.  Stops when the
// M^-1-norm of the residual has dropped by rtol.  Returns the iterations.
template <class TI>
__device__ __noinline__ int minres_correction(const MGArgs<TI> &a, Sync &team, SolveShared<TI> &cs, double rtol,
                                              int maxit)
{
	typedef typename V2T<TI>::t VI;
	__shared__ MinresScal ms;
	// Nothing that lives through a barrier is held in a local array, and sizes and
	// pointers are read from the arguments in shared memory where they are used:
	// what does not fit the registers goes to the stack, which misses L1 after every
	// team barrier.
	Sync sy = team;
	const MGHier<TI> &H = a.H;
	auto nodes = [&] { return (a.N0 + 1) * (a.N0 + 1); };
	auto elems = [&] { return a.N0 * a.N0; };
	double pdot = 0.0;
	{
		const double2 zero2 = make_double2(0.0, 0.0);
		const int tid = sy.tid(), nth = sy.nth(), nn = nodes(), ne = elems();
		for (int A = tid; A < nn; A += nth) {
			const double2 r = a.R[A];
			a.mv[0][A] = r;
			VI w;
			w.x = narrow_to<TI>(r.x);
			w.y = narrow_to<TI>(r.y);
			H.lv[0].b[A] = w;
			a.mv[1][A] = zero2;
			a.mw[0][A] = zero2;
			a.mw[1][A] = zero2;
			a.dd[A] = zero2;
		}
		for (int e = tid; e < ne; e += nth) {
			const double v = -a.Rc[e], z = v * a.bab[e];
			a.mvp[0][e] = v;
			a.mzp[0][e] = z;
			pdot += z * v;
			a.mvp[1][e] = 0.0;
			a.mwp[0][e] = 0.0;
			a.mwp[1][e] = 0.0;
			a.dpv[e] = 0.0;
		}
	}
	sy.sync();
	// index cv: z(j), v(j); 1-cv: v(j-1).  cw: w(j); 1-cw: w(j-1).  it = -1: z(0) = M^-1 v(0)
	int cv = 1, cw = 0, it = -1;
	// The direction update is needed only by the next one, and the pressure part of
	// the Lanczos update by the reduction after the V-cycle: on a team they run in
	// the V-cycle, on the blocks that would wait for the leading block's small
	// levels (8 us of an iteration at 64^2, 17 at 1024^2).  Not where that block runs
	// the whole cycle: its last sweep would overwrite the z that is still read.
	// steps: the pending direction update's (-1: none).
	const bool defer = sy.size >= 4 && H.nblk > 0;
	int steps = -1;
#pragma unroll 1
	while (it < maxit) {
		if (it >= 0) {
			// A z(j), unscaled (z~ = z / gam): K z_u + G z_p into a.Kd, G^T z_u into
			// a.Ahp, and their product with (z_u, z_p)
			double dl[1];
			Pass<TI> P = level_pass<TI>(H.lv[0], nullptr);
			P.out64 = a.Kd;
			P.gt_out = a.Ahp;
			P.g0 = a.gt.g0[0];
			P.g1 = a.gt.g1[0];
			P.gp_morton = 0;
			P.x = a.mzu[cv];
			P.gp = a.mzp[cv];
			march<TI, PASS_STOKES, XS_PLAIN, false>(P, sy.part(true), cs.sp.lev[1][0], dl);
			sy.reduce_then<1>(dl, [&](const double (&v)[1]) {
				ms.delta = v[0] * ms.ig * ms.ig;
				ms.dg = ms.delta * ms.ig;
			});
			// v(j+1) = A z~ - (delta/gam) v(j) - (gam/gam_prev) v(j-1), into v(j-1)'s
			// buffer, its TI copy as the V-cycle's right-hand side, and z_p(j+1)
			minres_v_nodes<VI>(nodes(), sy.tid(), sy.nth(), a.Kd, a.mv[cv], a.mv[1 - cv], H.lv[0].b, ms.ig, ms.dg, ms.gg);
			if (!defer)
				pdot = minres_v_elems(elems(), sy.tid(), sy.nth(), a.Ahp, a.mvp[cv], a.mvp[1 - cv], a.bab, a.mzp[1 - cv],
				                      ms.ig, ms.dg, ms.gg);
			sy.sync();
		}
		double dot[1];
		vcycle<TI>(sy, cs, H, H.lv[0].b, a.mzu[1 - cv], a.mv[1 - cv], &dot[0], [&] {
			if (!defer || it < 0)
				return;
			// the previous iteration's direction update (its z(j-1) and z_p(j-1) lie in
			// the buffers that this iteration's z(j+1) overwrites: z_u after this point,
			// z_p below by the same thread), and the pressure part of the Lanczos update
			const Part pt{sy.rank - 1, sy.size - 1};
			const int tid = pt.thread(), nth = pt.size * (int)blockDim.x;
			if (steps >= 0) {
				minres_w_nodes<VI>(steps, nodes(), tid, nth, a.mzu[1 - cv], a.mw[cw], a.mw[1 - cw], a.dd, ms.k3,
				                   ms.k2, ms.step, ms.step1);
				minres_w_elems(steps, elems(), tid, nth, a.mzp[1 - cv], a.mwp[cw], a.mwp[1 - cw], a.dpv, ms.k3,
				               ms.k2, ms.step, ms.step1);
			}
			pdot = minres_v_elems(elems(), tid, nth, a.Ahp, a.mvp[cv], a.mvp[1 - cv], a.bab, a.mzp[1 - cv], ms.ig, ms.dg,
			                      ms.gg);
		});
		dot[0] += pdot;
		pdot = 0.0;
		sy.reduce_then<1>(dot, [&](const double (&v)[1]) {
			const double gn2 = fmax(v[0], 0.0);
			const double gam_next = sqrt(gn2);
			if (it < 0) {
				ms.gam = gam_next;
				ms.gam_prev = 1.0;
				ms.eta = ms.eta0 = gam_next;
				ms.c_prev = ms.c_cur = 1.0;
				ms.s_prev = ms.s_cur = 0.0;
				ms.ig = 1.0 / gam_next;
				ms.gg = gam_next;
				ms.k1 = ms.k1p = 0.0;
				ms.stop = v[0] > 0.0 ? 0 : 3;
				return;
			}
			// Givens rotations
			const double a0 = ms.c_cur * ms.delta - ms.c_prev * ms.s_cur * ms.gam;
			const double a1s = a0 * a0 + gn2;
			const double a2 = ms.s_cur * ms.delta + ms.c_prev * ms.c_cur * ms.gam;
			const double a3 = ms.s_prev * ms.gam;
			const double ia1 = rsqrt(a1s);
			ms.stop = 0;
			if (!(a1s > 0.0) || !isfinite(a1s)) {
				ms.stop = isfinite(a1s) ? 2 : 6;
				return;
			}
			const double c_next = a0 * ia1, s_next = gam_next * ia1;
			// w(j+1) = (z(j)/gam - a3 w(j-1) - a2 w(j)) / a1; x += c_next eta w(j+1).  Kept
			// are the directions y without the factor k1 = 1/(gam a1), which goes into the
			// steps: y(j+1) = z(j) - k3 y(j-1) - k2 y(j), an FP64 operation less for every
			// value (244 against 248 us per iteration at 1024^2)
			const double k1 = ms.ig * ia1;
			ms.k3 = a3 * ms.gam * ms.k1p;
			ms.k2 = a2 * ms.gam * ms.k1;
			ms.k1p = ms.k1;
			ms.k1 = k1;
			ms.step1 = ms.step;
			ms.step = c_next * ms.eta * k1;
			ms.eta = -s_next * ms.eta;
			ms.gam_prev = ms.gam;
			ms.gam = gam_next;
			ms.c_prev = ms.c_cur;
			ms.c_cur = c_next;
			ms.s_prev = ms.s_cur;
			ms.s_cur = s_next;
			if (!isfinite(ms.eta))
				ms.stop = 5;
			else if (!(fabs(ms.eta) > rtol * ms.eta0) || !(gam_next > 0.0))
				ms.stop = 1;
		});
		if (it < 0) {
			it = 0;
			if (ms.stop)
				break;
			cv = 0;
			continue;
		}
		const int stop = ms.stop;
		if ((stop & 4) && sy.tid() == 0)
			atomicOr(&a.sc->status, 2);
		if (stop & 2) {
			if (it & 1)   // the pending step along w(j)
				minres_x_update(nodes(), elems(), sy.tid(), sy.nth(), a.mw[cw], a.dd, a.mwp[cw], a.dpv, ms.step);
			break;
		}
		// into w(j-1)'s buffer; the solution takes the steps of two iterations at a time
		// (x += step w(j) + step' w(j+1), the same additions in the same order), or what
		// is pending when the loop ends
		const bool last = stop || it + 1 >= maxit;
		steps = (it & 1) ? 2 : last ? 1 : 0;
		if (!defer || last) {
			minres_w_nodes<VI>(steps, nodes(), sy.tid(), sy.nth(), a.mzu[cv], a.mw[1 - cw], a.mw[cw], a.dd, ms.k3,
			                   ms.k2, ms.step, ms.step1);
			minres_w_elems(steps, elems(), sy.tid(), sy.nth(), a.mzp[cv], a.mwp[1 - cw], a.mwp[cw], a.dpv, ms.k3,
			               ms.k2, ms.step, ms.step1);
		}
		it++;
		cv = 1 - cv;
		cw = 1 - cw;
		if (stop)
			break;
		// the next step's 1/gam and gam/gam_prev, off the other threads' path; they are
		// read after the next reduction's broadcast
		if (threadIdx.x == 0) {
			ms.ig = 1.0 / ms.gam;
			ms.gg = ms.gam / ms.gam_prev;
		}
		// no barrier here: the next operator pass reads z(j+1) and z_p(j+1),
		// complete since the reduction, and touches none of the vectors that the
		// updates write
	}
	sy.sync();
	team = sy;
	return it;
}

// p += dp, dp x-major and p in the mesh's Morton order
__device__ void add_pressure(int N0, const double *dp, double *p, int tid, int nth)
{
	for (int e = tid; e < N0 * N0; e += nth) {
		const int ex = e / N0, ez = e - ex * N0;
		p[morton(ex, ez)] += dp[e];
	}
}

// ---- one converged Stokes solve ----------------------------------------------------
// The whole solve of one time step: per-step setup of the hierarchy, FP64
// refinement, correction solves.  Runs on the cooperative grid (one model) or
// inside one block (one model of a batch), as `sy` says.
template <class TI>
__device__ void stokes_solve(const MGArgs<TI> &a, Sync &sy)
{
	typedef typename V2T<TI>::t VI;
	__shared__ SolveShared<TI> cs;   // this block's working data of the solve
	const MGHier<TI> &H = a.H;
	const int tid = sy.tid(), nth = sy.nth();
	const int N0 = a.N0, n0 = N0 + 1, nn = n0 * n0, ne = N0 * N0;
	int *status = &a.sc->status;
	const GTab &gt = a.gt;

	for (int l = threadIdx.x; l < a.H.nlev; l += blockDim.x) {
		cs.sp.lev[0][l].set(a.H.lv[l].n, blockDim.x / 32);
		cs.sp.lev[1][l].set(a.H.lv[l].n, sy.size * (blockDim.x / 32));
	}
	// -- per-step setup: viscosity on every level, inverse diagonals, BAB, coarse inverse
	for (int A = tid; A < nn; A += nth)
		H.lv[0].eta[A] = (TI)a.vis[A];
	sy.sync();
	for (int l = 1; l < H.nlev; l++) {
		const MGLevel<TI> &C = H.lv[l], &F = H.lv[l - 1];
		for (int A = tid; A < C.n * C.n; A += nth) {
			const int cx = A / C.n, cz = A - cx * C.n;
			if (H.eta_avg == 0) {
				C.eta[A] = F.eta[2 * cz + 2 * cx * F.n];
			} else {
				double s = 0.0, wsum = 0.0;
				for (int dx = -1; dx <= 1; dx++)
					for (int dz = -1; dz <= 1; dz++) {
						const int fx = 2 * cx + dx, fz = 2 * cz + dz;
						if (fx < 0 || fx >= F.n || fz < 0 || fz >= F.n)
							continue;
						const double w = (dx == 0 ? 1.0 : 0.5) * (dz == 0 ? 1.0 : 0.5);
						const double ev = (double)F.eta[fz + fx * F.n];
						s += w * (H.eta_avg == 2 ? log(ev) : ev);
						wsum += w;
					}
				s /= wsum;
				C.eta[A] = (TI)(H.eta_avg == 2 ? exp(s) : s);
			}
		}
		sy.sync();
	}
	for (int l = 0; l < H.nlev; l++)
		level_invdiag<TI, VI>(sy.part(true), H.lv[l].N, H.lv[l].mask, H.lv[l].eta, H.lv[l].invD, nullptr);
	level_invdiag<double, double2>(sy.part(true), N0, a.mask0, a.vis, a.invD64, a.kdiag64);
	sy.sync();
	for (int e = tid; e < ne; e += nth) {
		const int ex = e / N0, ez = e - ex * N0;
		const int cn[4] = {ez + ex * n0, ez + 1 + ex * n0, ez + 1 + (ex + 1) * n0, ez + (ex + 1) * n0};
		double s = 0.0;
#pragma unroll
		for (int c = 0; c < 4; c++) {
			const int ac = kSortedCorner[c];
			double g0, g1;
			g_entries(a.hx, a.hz, ac, g0, g1);
			const double2 kd = a.kdiag64[cn[ac]];
			const unsigned m = a.mask0[cn[ac]];
			if (!(m & 1u))
				s += g0 * g0 / kd.x;
			if (!(m & 2u))
				s += g1 * g1 / kd.y;
		}
		a.bab[e] = 1.0 / s;   // the solvers multiply by 1/BAB
	}
	if (sy.leader())
		coarse_build<TI>(H, cs);
	sy.sync();

	int refine = 0, outer_total = 0, inner_total = 0, capped = 0;
	double res_m = 0.0, res_c = 0.0, fnorm = 1.0;
	if (a.method == 1 && a.h1d != nullptr) {
		const int nh = a.sc->nsolved < 3 ? a.sc->nsolved : 3;   // solutions in the history
		if (nh >= 2)
			warm_guess<TI>(a, sy, cs, nh - 1);
	}
	if (a.d_alt != nullptr) {
		// Two candidate guesses: (d, p) from the network and (d_alt, p_alt),
		// the previous step's solution.  Keep the one with the smaller FP64
		// residual; a non-finite network guess always loses.
		double rl[3], rp[3];
		stokes_residual(a, sy, cs.sp.lev[1][0], a.d, a.p, rl);
		stokes_residual(a, sy, cs.sp.lev[1][0], a.d_alt, a.p_alt, rp);
		const double el = rl[0] + rl[1], ep = rp[0] + rp[1];
		const bool learned = isfinite(el) && (a.guess_force || el < ep);
		if (!learned) {
			for (int A = tid; A < nn; A += nth)
				a.d[A] = a.d_alt[A];
			for (int e = tid; e < ne; e += nth)
				a.p[e] = a.p_alt[e];
		}
		if (tid == 0) {
			a.sc->guess_used = learned ? 1 : 0;
			a.sc->res_learned = sqrt(el / rl[2]);
			a.sc->res_prev = sqrt(ep / rp[2]);
		}
		sy.sync();
	}
	while (true) {
		// -- FP64 residual R = [F - K d - G p ; G^T d]
		double rs[3];
		stokes_residual(a, sy, cs.sp.lev[1][0], a.d, a.p, rs);
		// a zero load (|F| = 0): the residual is measured absolutely
		fnorm = rs[2] > 0.0 ? sqrt(rs[2]) : 1.0;
		res_m = sqrt(rs[0]) / fnorm;
		res_c = sqrt(rs[1]) / fnorm;
		const double res = sqrt(rs[0] + rs[1]) / fnorm;
		if (!isfinite(res)) {
			if (tid == 0)
				atomicOr(status, 2);
			break;
		}
		if (!(res >= a.rtol))
			break;
		if (refine >= a.max_refine) {
			capped = 1;
			break;
		}
		refine++;

		if (a.method == 1) {
			// -- correction solve: MINRES on [K G; G^T 0][dd; dp] = [R_m; -R_c].
			// Far from the target (res > 1e4 rtol) a pass reduces by 1e-2,
			// where MINRES converges fastest; close to it, by what is left to
			// reach rtol (with a factor 2 margin), but not below outer_rtol.
			const double prt = res > 1e4 * a.rtol ? 1e-2 : fmax(a.outer_rtol, 0.5 * a.rtol / res);
			const int it = minres_correction<TI>(a, sy, cs, prt, a.max_outer);
			outer_total += it;
			inner_total += it + 1;
			for (int A = tid; A < nn; A += nth) {
				const double2 c = a.dd[A];
				double2 v = a.d[A];
				v.x += c.x;
				v.y += c.y;
				a.d[A] = v;
			}
			add_pressure(N0, a.dpv, a.p, tid, nth);
			sy.sync();
			continue;
		}

		// -- correction solve: Uzawa on [K G; G^T 0][dd; dp] = [R_m; -R_c]
		VI *bI = H.lv[0].b, *xI = H.px;   // level-0 buffers double as CG input/output here
		for (int A = tid; A < nn; A += nth) {
			const double2 r = a.R[A];
			VI v;
			v.x = narrow_to<TI>(r.x);
			v.y = narrow_to<TI>(r.y);
			bI[A] = v;
		}
		sy.sync();
		inner_total += pcg_inner<TI>(sy, cs, H, bI, xI, a.inner_rtol, a.max_inner);
		for (int A = tid; A < nn; A += nth) {
			const VI v = xI[A];
			a.dd[A] = make_double2(widen(v.x), widen(v.y));
		}
		sy.sync();
		double *r0 = a.r0, *r1 = a.r1, *r2 = a.r2, *z0 = a.z0, *z1 = a.z1, *s1 = a.s1, *s2 = a.s2;
		double c0[1] = {0.0};
		for (int e = tid; e < ne; e += nth) {
			const int ex = e / N0, ez = e - ex * N0;
			const double v = a.Rc[e] + gtmul64_elem(N0, a.mask0, gt, a.dd, ex, ez);
			r1[e] = v;
			a.dpv[e] = 0.0;
			c0[0] += v * v;
		}
		sy.reduce<1>(c0);
		const double rnorm0 = sqrt(c0[0]);
		double rnorm = rnorm0;
		int cycle = 0;
		while (cycle < a.max_outer && rnorm > a.outer_rtol * rnorm0 && rnorm > 0.0) {
			double rz[2] = {0.0, 0.0};
			for (int e = tid; e < ne; e += nth) {
				const double z = r1[e] * a.bab[e];
				z1[e] = z;
				rz[0] += r1[e] * z;
				if (cycle > 0)
					rz[1] += r0[e] * z0[e];
			}
			sy.reduce<2>(rz);
			const double delta = cycle == 0 ? 0.0 : rz[0] / rz[1];
			for (int e = tid; e < ne; e += nth)
				s2[e] = cycle == 0 ? z1[e] : z1[e] + delta * s1[e];
			sy.sync();
			gmul64(N0, a.mask0, gt, s2, a.u1, tid, nth);
			for (int A = tid; A < nn; A += nth) {
				const double2 v = a.u1[A];
				VI w;
				w.x = narrow_to<TI>(v.x);
				w.y = narrow_to<TI>(v.y);
				bI[A] = w;
			}
			sy.sync();
			inner_total += pcg_inner<TI>(sy, cs, H, bI, xI, a.inner_rtol, a.max_inner);
			for (int A = tid; A < nn; A += nth) {
				const VI v = xI[A];
				a.u1[A] = make_double2(widen(v.x), widen(v.y));
			}
			sy.sync();
			double sa[1] = {0.0};
			for (int e = tid; e < ne; e += nth) {
				const int ex = e / N0, ez = e - ex * N0;
				const double t = gtmul64_elem(N0, a.mask0, gt, a.u1, ex, ez);
				a.Ahp[e] = t;
				sa[0] += s2[e] * t;
			}
			sy.reduce<1>(sa);
			const double alpha = rz[0] / sa[0];
			double rr[1] = {0.0};
			for (int e = tid; e < ne; e += nth) {
				const double v = r1[e] - alpha * a.Ahp[e];
				r2[e] = v;
				a.dpv[e] += alpha * s2[e];
				rr[0] += v * v;
			}
			for (int A = tid; A < nn; A += nth) {
				const double2 u = a.u1[A];
				double2 v = a.dd[A];
				v.x -= alpha * u.x;
				v.y -= alpha * u.y;
				a.dd[A] = v;
			}
			sy.reduce<1>(rr);
			rnorm = sqrt(rr[0]);
			cycle++;
			double *sh = s1; s1 = s2; s2 = sh;
			sh = r0; r0 = r1; r1 = r2; r2 = sh;
			sh = z0; z0 = z1; z1 = sh;
			if (!isfinite(alpha) || !isfinite(rnorm)) {
				if (tid == 0)
					atomicOr(status, 2);
				break;
			}
		}
		outer_total += cycle;
		// apply the correction in FP64
		for (int A = tid; A < nn; A += nth) {
			const double2 c = a.dd[A];
			double2 v = a.d[A];
			v.x += c.x;
			v.y += c.y;
			a.d[A] = v;
		}
		add_pressure(N0, a.dpv, a.p, tid, nth);
		sy.sync();
	}
	if (capped && tid == 0)
		atomicOr(status, 1);
	// nodal velocity (v_to_nodes, Solver.c:1319-1343)
	for (int A = tid; A < nn; A += nth) {
		const double2 dv = a.d[A];
		const unsigned m = a.mask0[A];
		a.V[A] = make_double2((m & 1u) ? a.vbcval[A] : dv.x, (m & 2u) ? a.vbcval[nn + A] : dv.y);
	}
	if (tid == 0) {
		a.sc->uzawa_cycles = outer_total;
		a.sc->cg_cycles = inner_total;
		a.sc->refine_passes = refine;
		if (a.sc->nsolved < 1000000)
			a.sc->nsolved++;
		a.sc->res_m = res_m;
		a.sc->res_c = res_c;
		a.sc->dv = 0.0;
		a.sc->dp = 0.0;
	}
}

// Most threads per block: 512 in FP32 (two blocks of 256 per SM on a grid, one of
// 512 in a single model's cluster); the FP64 passes hold twice the registers and
// are bound by the FP64 pipe, which 256 threads keep busy.
template <class TI> constexpr int kSolveThreads = sizeof(TI) == 4 ? 512 : 256;

// One model on the whole cooperative grid, or on one cluster (a.cluster).
template <class TI>
__global__ void __launch_bounds__(kSolveThreads<TI>, 1) k_stokes_mg(const __grid_constant__ MGArgs<TI> a)
{
	__shared__ MGArgs<TI> sa;
	__shared__ double cpart[2 * kRedWidth];
	load_args(sa, a);
	cg::cluster_group cl = cg::this_cluster();
	Sync sy = sa.cluster ? Sync::of(SYNC_CLUSTER, cpart, blockIdx.x, gridDim.x)
	                     : Sync::of(SYNC_GRID, sa.red.part, blockIdx.x, gridDim.x);
	stokes_solve<TI>(sa, sy);
	if (sa.cluster)
		cl.sync();   // no block leaves while another reads its partials
}

// A batch of independent models.  Launched with clusters of `cs` blocks
// (cs = 1: plain blocks); each cluster takes the next model from the queue
// (ordered largest first by the host) and solves it alone with cluster
// barriers, so the launch is an ordinary one and clusters never wait on each
// other.  The cluster's rank-0 block draws from the queue and every block
// reads the draw from its shared memory; all blocks of a cluster leave the
// loop on the same draw.
template <class TI>
__global__ void __launch_bounds__(kSolveThreads<TI>, 1) k_stokes_mg_batch(const MGArgs<TI> *models, int nmodels,
                                                                              int *queue)
{
	__shared__ MGArgs<TI> sa;
	__shared__ int next;
	__shared__ double cpart[2 * kRedWidth];
	cg::cluster_group cl = cg::this_cluster();
	const int cs = (int)cl.num_blocks(), rank = (int)cl.block_rank();
	for (;;) {
		if (rank == 0 && threadIdx.x == 0)
			next = atomicAdd(queue, 1);
		if (cs > 1) {
			cl.sync();
			const int m = *cl.map_shared_rank(&next, 0);
			cl.sync();   // every block has read the draw before the next one
			if (m >= nmodels)
				break;
			load_args(sa, models[m]);
			Sync sy = Sync::of(SYNC_CLUSTER, cpart, rank, cs);
			stokes_solve<TI>(sa, sy);
			cl.sync();   // no block starts the next model (or leaves) while another reads its partials
		} else {
			__syncthreads();
			const int m = next;
			__syncthreads();
			if (m >= nmodels)
				break;
			load_args(sa, models[m]);
			Sync sy = Sync::of(SYNC_BLOCK, nullptr, 0, 1);
			stokes_solve<TI>(sa, sy);
			__syncthreads();
		}
	}
}

void *stokes_mg_kernel(int fp64) { return fp64 ? (void *)k_stokes_mg<double> : (void *)k_stokes_mg<float>; }
void *stokes_mg_batch_kernel(int fp64)
{
	return fp64 ? (void *)k_stokes_mg_batch<double> : (void *)k_stokes_mg_batch<float>;
}

}  // namespace mclg
