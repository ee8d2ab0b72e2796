// Converged Stokes solve on quadtree meshes with hanging nodes; see k_qt.cuh.
// One persistent kernel per time step.  Vectors are node layout
// (both components of a node together); a primal vector stores its reduced
// dofs and is read through the constraints (qt_val), a dual vector (operator
// output, residual) is zero outside the reduced dofs.
#include <math.h>
#include "k_qt.cuh"
#include "fp64_util.cuh"

namespace mclg {

MCLG_SHAPE_UPLOAD(upload_shape_tables_qt)

// ---- values through the constraints ----------------------------------------------
// dof (2*node + component) of a primal vector: stored if reduced, the weighted
// sum of its reduced dofs if constrained, 0 if fixed.
template <class T, class X>
__device__ __forceinline__ X qt_val(const QtLevel<T> &L, const X *__restrict__ xf, int dof)
{
	const unsigned char k = L.kind[dof];
	if (k == 1)
		return xf[dof];
	X s = X(0);
	if (k == 2)
		for (int i = L.ex_off[dof]; i < L.ex_off[dof + 1]; i++)
			s += (X)L.ex_w[i] * xf[L.ex_src[i]];
	return s;
}

// Both components of node B of a primal vector through the constraints (the
// rare path of a row: a column with a constrained component).
template <class T, class X>
__device__ __noinline__ typename Q2T<X>::t qt_val2(const QtLevel<T> &L, const X *__restrict__ xf, int B)
{
	typename Q2T<X>::t v;
	v.x = qt_val(L, xf, 2 * B);
	v.y = qt_val(L, xf, 2 * B + 1);
	return v;
}

// Both rows of node j of K x~ (x~ the expanded x), with K in the level's TI
// blocks or its FP64 blocks.  Columns go in chunks of four: the chunk's index
// and block loads, then its gathers, are issued before any is used (a short
// chunk is padded with the node itself and a zero block).
template <class T, class K4, class X>
__device__ __forceinline__ void qt_rows(const QtLevel<T> &L, const K4 *__restrict__ K, const X *__restrict__ xf, int j,
                                        X &y0, X &y1)
{
	typedef typename Q2T<X>::t X2;
	const X2 *x2 = reinterpret_cast<const X2 *>(xf);
	X s0 = X(0), s1 = X(0);
	const int n = L.cnt[j];
	for (int k0 = 0; k0 < n; k0 += 4) {
		int Bf[4];
		K4 kb[4];
		X2 xv[4];
#pragma unroll
		for (int u = 0; u < 4; u++) {
			const bool in = k0 + u < n;
			Bf[u] = in ? L.nb[(size_t)(k0 + u) * L.nno + j] : j;
			kb[u] = in ? K[(size_t)(k0 + u) * L.nno + j] : K4{};
		}
#pragma unroll
		for (int u = 0; u < 4; u++)
			xv[u] = x2[Bf[u] & ~kQtCon];
#pragma unroll
		for (int u = 0; u < 4; u++) {
			if (Bf[u] & kQtCon)
				xv[u] = qt_val2(L, xf, Bf[u] & ~kQtCon);
			s0 += (X)kb[u].x * xv[u].x + (X)kb[u].y * xv[u].y;
			s1 += (X)kb[u].z * xv[u].x + (X)kb[u].w * xv[u].y;
		}
	}
	y0 = s0;
	y1 = s1;
}

// (C^T K C x) at both dofs of node A: the node's own rows plus the rows of
// the constrained dofs whose expansion holds them; 0 outside reduced dofs.
template <class T, class K4, class X>
__device__ __forceinline__ void qt_op_node(const QtLevel<T> &L, const K4 *__restrict__ K, const X *__restrict__ xf,
                                           int A, X &y0, X &y1)
{
	X y[2];
	qt_rows(L, K, xf, A, y[0], y[1]);
#pragma unroll
	for (int c = 0; c < 2; c++) {
		const int dof = 2 * A + c;
		if (L.kind[dof] != 1) {
			y[c] = X(0);
			continue;
		}
		for (int i = L.fo_off[dof]; i < L.fo_off[dof + 1]; i++) {
			const int h = L.fo_dof[i];
			X h0, h1;
			qt_rows(L, K, xf, h >> 1, h0, h1);
			y[c] += (X)L.fo_w[i] * ((h & 1) ? h1 : h0);
		}
	}
	y0 = y[0];
	y1 = y[1];
}

// Sources of the x a V-cycle pass reads at a node: the stored vector, or the
// first Jacobi sweep from zero, omega D^-1 b, formed where it is read (so the
// pass after it needs no barrier for it) with the operations, in the order, of
// the pass it replaces.  (Forming the prolongation x + P xc the same way inside
// the first sweep up was measured 2x slower on configuration 2: every
// neighbour's prolongation is recomputed through a deeper chain of gathers.)
template <class TI>
struct QtXStored {
	typedef typename Q2T<TI>::t X2;
	const X2 *x;
	__device__ __forceinline__ X2 operator()(int B) const { return x[B]; }
};

template <class TI>
struct QtXFirst {
	typedef typename Q2T<TI>::t X2;
	const X2 *b;
	const TI *invD;
	TI omega;
	__device__ __forceinline__ X2 operator()(int B) const
	{
		const X2 bv = b[B], dv = reinterpret_cast<const X2 *>(invD)[B];
		X2 o;
		o.x = omega * dv.x * bv.x;
		o.y = omega * dv.y * bv.y;
		return o;
	}
};

// (C^T K C x) at both dofs of node A from the assembled reduced operator: a
// plain node-block ELL row (x's constrained and fixed entries are stored as 0
// and the reduced columns hold every coupling); x read through src.  A row's
// first kChunk columns (all of an interior row between equal elements) are in
// flight together: after a team barrier every load is an L2 access.
template <class TI, class XS>
__device__ __forceinline__ void qt_kr_node_src(const QtLevel<TI> &L, const XS &src, int A, TI &y0, TI &y1)
{
	typedef typename Q2T<TI>::t X2;
	typedef typename V4T<TI>::t K4;
	constexpr int kChunk = sizeof(TI) == 4 ? 9 : 4;
	TI s0 = TI(0), s1 = TI(0);
	const int n = L.rcnt[A];
	for (int k0 = 0; k0 == 0 || k0 < n; k0 += kChunk) {   // (the first chunk does not wait for n)
		int B[kChunk];
		K4 kb[kChunk];
#pragma unroll
		for (int u = 0; u < kChunk; u++) {
			const bool in = k0 + u < L.rnbw;   // (columns past the row's end are the row node with a zero block)
			B[u] = in ? L.rnb[(size_t)(k0 + u) * L.nno + A] : A;
			kb[u] = in ? L.Kr[(size_t)(k0 + u) * L.nno + A] : K4{};
		}
		X2 xv[kChunk];
#pragma unroll
		for (int u = 0; u < kChunk; u++)
			xv[u] = src(B[u]);
#pragma unroll
		for (int u = 0; u < kChunk; u++) {
			s0 += kb[u].x * xv[u].x + kb[u].y * xv[u].y;
			s1 += kb[u].z * xv[u].x + kb[u].w * xv[u].y;
		}
	}
	y0 = s0;
	y1 = s1;
}

template <class TI>
__device__ __forceinline__ void qt_kr_node(const QtLevel<TI> &L, const TI *__restrict__ xf, int A, TI &y0, TI &y1)
{
	const QtXStored<TI> src{reinterpret_cast<const typename Q2T<TI>::t *>(xf)};
	qt_kr_node_src(L, src, A, y0, y1);
}

// s = sum of w[i] x[src[i]] over [i0, i1), C entries at a time: their indices,
// then their gathers in flight together (a list's loop waits for both in turn).
template <int C, class T>
__device__ __forceinline__ T qt_gather(const int *__restrict__ src, const T *__restrict__ w, const T *__restrict__ x,
                                       int i0, int i1)
{
	T s = T(0);
	for (int i = i0; i < i1; i += C) {
		int j[C];
		T ww[C], xv[C];
#pragma unroll
		for (int u = 0; u < C; u++) {
			const bool in = i + u < i1;
			j[u] = src[in ? i + u : i0];
			ww[u] = in ? w[i + u] : T(0);
		}
#pragma unroll
		for (int u = 0; u < C; u++)
			xv[u] = x[j[u]];
#pragma unroll
		for (int u = 0; u < C; u++)
			s += i + u < i1 ? ww[u] * xv[u] : T(0);
	}
	return s;
}

// G p at node A on the finest level: an element's entries are +-dz_deta and
// +-dx_dxi by corner (the sums over the Gauss points that element_g forms, 8
// FP64 operations a corner, come to one of the two half-widths).
__device__ __forceinline__ void qt_gmul(const DevLevel &L, const double *__restrict__ p, int A, double &y0, double &y1)
{
	double s0 = 0.0, s1 = 0.0;
	const int n = L.p2n_cnt[A];
	int e[4], a[4];
#pragma unroll
	for (int k = 0; k < 4; k++) {
		e[k] = L.p2n_el[k * L.nno + A];
		a[k] = L.p2n_a[k * L.nno + A];
	}
	double pe[4], hz[4], hx[4];
#pragma unroll
	for (int k = 0; k < 4; k++) {
		const int ek = k < n ? e[k] : e[0];
		pe[k] = p[ek];
		hz[k] = L.dzh[ek];
		hx[k] = L.dxh[ek];
	}
#pragma unroll
	for (int k = 0; k < 4; k++)
		if (k < n) {
			s0 += (a[k] < 2 ? hz[k] : -hz[k]) * pe[k];
			s1 += (a[k] == 0 || a[k] == 3 ? hx[k] : -hx[k]) * pe[k];
		}
	y0 = s0;
	y1 = s1;
}

// (C^T G p) at both dofs of node A (FP64, the finest level)
template <class T>
__device__ __forceinline__ void qt_g_node(const QtLevel<T> &Q, const DevLevel &L, const double *__restrict__ p, int A,
                                          double &y0, double &y1)
{
	const uchar2 k = reinterpret_cast<const uchar2 *>(Q.kind)[A];
	const int f0 = Q.fo_off[2 * A], f1 = Q.fo_off[2 * A + 1], f2 = Q.fo_off[2 * A + 2];
	qt_gmul(L, p, A, y0, y1);
	y0 = k.x == 1 ? y0 : 0.0;
	y1 = k.y == 1 ? y1 : 0.0;
	// the rows of the constrained dofs that hold this node, both components' lists
	// in one, two entries at a time with their loads in flight together
	const int ie = k.y == 1 ? f2 : f1;
	for (int i = k.x == 1 ? f0 : f1; i < ie; i += 2) {
		int h[2], e[2][4], a[2][4], n[2];
		double w[2], pe[2][4], g[2][4];
#pragma unroll
		for (int u = 0; u < 2; u++) {
			const bool in = i + u < ie;
			h[u] = Q.fo_dof[in ? i + u : i];
			w[u] = in ? (double)Q.fo_w[i + u] : 0.0;
		}
#pragma unroll
		for (int u = 0; u < 2; u++) {
			const int B = h[u] >> 1;
			n[u] = vfree(L, B, h[u] & 1) ? L.p2n_cnt[B] : 0;
#pragma unroll
			for (int q = 0; q < 4; q++) {
				e[u][q] = L.p2n_el[q * L.nno + B];
				a[u][q] = L.p2n_a[q * L.nno + B];
			}
		}
#pragma unroll
		for (int u = 0; u < 2; u++) {
			const double *hh = (h[u] & 1) ? L.dxh : L.dzh;
#pragma unroll
			for (int q = 0; q < 4; q++) {
				const int eq = q < n[u] ? e[u][q] : e[u][0];
				pe[u][q] = p[eq];
				g[u][q] = hh[eq];
			}
		}
#pragma unroll
		for (int u = 0; u < 2; u++) {
			double s = 0.0;
#pragma unroll
			for (int q = 0; q < 4; q++)
				if (q < n[u]) {
					const bool pos = (h[u] & 1) ? (a[u][q] == 0 || a[u][q] == 3) : a[u][q] < 2;
					s += (pos ? g[u][q] : -g[u][q]) * pe[u][q];
				}
			if (i + u < ie)
				(i + u < f1 ? y0 : y1) += w[u] * s;
		}
	}
}

// Component c of an element's four corners through the constraints, x as stored
// on entry (k: the corners' kinds).  A few elements along the edges of refinement
// have constrained corners and would hold up the whole pass: the corners' lists go
// two entries at a time with every corner's loads in flight together, instead of a
// chain of three accesses for each corner and component in turn.
template <int c, class T, class X>
__device__ __forceinline__ void qt_constrained(const QtLevel<T> &Q, const X *__restrict__ xf, const int (&n)[4],
                                               const uchar2 (&k)[4], X (&x)[4])
{
	int i0[4], i1[4];
	bool any = false;
#pragma unroll
	for (int a = 0; a < 4; a++) {
		const unsigned char ka = c ? k[a].y : k[a].x;
		x[a] = ka == 1 ? x[a] : X(0);
		i0[a] = i1[a] = 0;
		if (ka == 2) {
			i0[a] = Q.ex_off[2 * n[a] + c];
			i1[a] = Q.ex_off[2 * n[a] + c + 1];
			any = true;
		}
	}
	while (any) {
		int s[8];
		X w[8], v[8];
#pragma unroll
		for (int q = 0; q < 8; q++) {
			const int i = i0[q >> 1] + (q & 1);
			const bool in = i < i1[q >> 1];
			s[q] = in ? Q.ex_src[i] : -1;
			w[q] = in ? (X)Q.ex_w[i] : X(0);
		}
#pragma unroll
		for (int q = 0; q < 8; q++)
			v[q] = s[q] >= 0 ? xf[s[q]] : X(0);
		any = false;
#pragma unroll
		for (int a = 0; a < 4; a++) {
			if (s[2 * a] >= 0)
				x[a] += w[2 * a] * v[2 * a];
			if (s[2 * a + 1] >= 0)
				x[a] += w[2 * a + 1] * v[2 * a + 1];
			i0[a] += 2;
			any |= i0[a] < i1[a];
		}
	}
}

// (G^T C u)_e of a primal vector u (flat, X) on the finest level
template <class T, class X>
__device__ __forceinline__ double qt_gt_elem(const QtLevel<T> &Q, const DevLevel &L, const X *__restrict__ uf, int e)
{
	int n[4];
	X u[4], w[4];
	uchar2 k[4];
#pragma unroll
	for (int a = 0; a < 4; a++)
		n[a] = L.ienl[a * L.nel + e];
#pragma unroll
	for (int a = 0; a < 4; a++) {
		const typename Q2T<X>::t v = reinterpret_cast<const typename Q2T<X>::t *>(uf)[n[a]];
		k[a] = reinterpret_cast<const uchar2 *>(Q.kind)[n[a]];
		u[a] = v.x;
		w[a] = v.y;
	}
	qt_constrained<0>(Q, uf, n, k, u);
	qt_constrained<1>(Q, uf, n, k, w);
	return gt_elem(u[0], u[1], u[2], u[3], w[0], w[1], w[2], w[3], L.dzh[e], L.dxh[e]);
}

// ---- the V-cycle (TI) -------------------------------------------------------------
// One damped Jacobi sweep on the constrained operator: xo = xi + w D^-1 (b - A xi),
// xi read through src.
template <class TI, class XS>
__device__ __forceinline__ typename Q2T<TI>::t qt_sweep_node(const QtLevel<TI> &L, TI omega, const XS &src, int A)
{
	typedef typename Q2T<TI>::t V;
	TI y0, y1;
	const V x = src(A), b = L.b[A], dg = reinterpret_cast<const V *>(L.invD)[A];   // invD is 0 off the reduced dofs
	const uchar2 k = reinterpret_cast<const uchar2 *>(L.kind)[A];
	qt_kr_node_src(L, src, A, y0, y1);
	V o;
	o.x = k.x == 1 ? x.x + omega * dg.x * (b.x - y0) : TI(0);
	o.y = k.y == 1 ? x.y + omega * dg.y * (b.y - y1) : TI(0);
	return o;
}

template <class TI, class XS>
__device__ __forceinline__ void qt_sweep_src(const QtLevel<TI> &L, TI omega, const XS &src,
                                             typename Q2T<TI>::t *xo, int tid, int nth)
{
	for (int A = tid; A < L.nno; A += nth)
		xo[A] = qt_sweep_node(L, omega, src, A);
}

template <class TI>
__device__ __forceinline__ void qt_sweep(const QtLevel<TI> &L, TI omega, const typename Q2T<TI>::t *xi,
                                         typename Q2T<TI>::t *xo, int tid, int nth)
{
	const QtXStored<TI> src{xi};
	qt_sweep_src(L, omega, src, xo, tid, nth);
}

// The part of the solve's team running a part of the V-cycle: the whole team,
// or its leading block alone for the smallest levels (block barriers instead
// of team barriers).
struct QtTeam {
	Sync *sy;
	bool wide;
	int tid, nth;
	__device__ void sync()
	{
		if (wide)
			sy->sync();
		else
			__syncthreads();
	}
};

// Buffer index holding a level's result: the coarsest solve writes x[0]; a
// finer level runs smooth-1 sweeps from the first one, then smooth after the
// correction, so it ends in x[(2 smooth - 1) & 1].
template <class TI>
__device__ __forceinline__ int qt_final(const QtHier<TI> &H, int l)
{
	return l == 0 ? 0 : (2 * H.smooth - 1) & 1;
}

// Level l on the way down: smoothing from zero, residual, restriction into l-1.
// The first sweep from zero, x0 = w D^-1 b, is formed where the next pass reads
// it (the residual, or the second sweep), so it costs no barrier of its own.
template <class TI>
__device__ __forceinline__ void qt_down(const QtHier<TI> &H, int l, QtTeam &t)
{
	typedef typename Q2T<TI>::t V;
	const QtLevel<TI> &L = H.lv[l];
	const QtXFirst<TI> first{L.b, L.invD, H.omega};
	int cur;
	if (H.smooth == 1) {
		// x0 stored for the way up, and the residual b - A x0 in the same pass
		V *x0 = L.x[0];
		for (int A = t.tid; A < L.nno; A += t.nth) {
			TI y0, y1;
			qt_kr_node_src(L, first, A, y0, y1);
			x0[A] = first(A);
			const V b = L.b[A];
			const uchar2 k = reinterpret_cast<const uchar2 *>(L.kind)[A];
			V r;
			r.x = k.x == 1 ? b.x - y0 : TI(0);
			r.y = k.y == 1 ? b.y - y1 : TI(0);
			L.r[A] = r;
		}
		cur = 0;
		t.sync();
	} else {
		qt_sweep_src(L, H.omega, first, L.x[1], t.tid, t.nth);   // sweeps 1 and 2
		cur = 1;
		t.sync();
		for (int s = 2; s < H.smooth; s++) {
			qt_sweep(L, H.omega, L.x[cur], L.x[1 - cur], t.tid, t.nth);
			cur = 1 - cur;
			t.sync();
		}
		const TI *xf = reinterpret_cast<const TI *>(L.x[cur]);
		for (int A = t.tid; A < L.nno; A += t.nth) {
			TI y0, y1;
			qt_kr_node(L, xf, A, y0, y1);
			const V b = L.b[A];
			const uchar2 k = reinterpret_cast<const uchar2 *>(L.kind)[A];
			V r;
			r.x = k.x == 1 ? b.x - y0 : TI(0);
			r.y = k.y == 1 ? b.y - y1 : TI(0);
			L.r[A] = r;
		}
		t.sync();
	}
	const QtLevel<TI> &C = H.lv[l - 1];
	const TI *rf = reinterpret_cast<const TI *>(L.r);
	TI *cb = reinterpret_cast<TI *>(C.b);
	for (int d = t.tid; d < 2 * C.nno; d += t.nth) {   // restriction: P^T by rows
		cb[d] = qt_gather<9, TI>(C.r_src, C.r_w, rf, C.r_off[d], C.r_off[d + 1]);
	}
	t.sync();
}

// Level l on the way up: prolongation of level l-1's result added, smoothing.
// With zout (the finest level) the last sweep writes there, adds this thread's
// share of zout.v to *dot and is not followed by a barrier: the caller's
// reduction provides it.
template <class TI>
__device__ __forceinline__ void qt_up(const QtHier<TI> &H, int l, QtTeam &t, typename Q2T<TI>::t *zout = nullptr,
                                      const double2 *v = nullptr, double *dot = nullptr)
{
	typedef typename Q2T<TI>::t V;
	const QtLevel<TI> &L = H.lv[l];
	int cur = (H.smooth - 1) & 1;
	const TI *xc = reinterpret_cast<const TI *>(H.lv[l - 1].x[qt_final(H, l - 1)]);
	TI *xf = reinterpret_cast<TI *>(L.x[cur]);
	for (int d = t.tid; d < 2 * L.nno; d += t.nth) {
		const int i0 = L.p_off[d], i1 = L.p_off[d + 1];
		const TI x0 = xf[d];
		if (i0 < i1)
			xf[d] = x0 + qt_gather<4, TI>(L.p_src, L.p_w, xc, i0, i1);
	}
	t.sync();
	for (int s = 0; s < H.smooth; s++) {
		if (zout != nullptr && s == H.smooth - 1) {
			const QtXStored<TI> src{L.x[cur]};
			double acc = 0.0;
			for (int A = t.tid; A < L.nno; A += t.nth) {
				const double2 va = v[A];
				const V o = qt_sweep_node(L, H.omega, src, A);
				zout[A] = o;
				acc += widen(o.x) * va.x + widen(o.y) * va.y;
			}
			*dot += acc;
			return;
		}
		qt_sweep(L, H.omega, L.x[cur], L.x[1 - cur], t.tid, t.nth);
		cur = 1 - cur;
		t.sync();
	}
}

// coarsest level: the dense inverse on its reduced dofs, a warp per four rows
// with its lanes along them (a thread per row read the matrix in columns 4*nc
// bytes apart: 8.3 us of a 128 us iteration for 126 unknowns)
template <class TI>
__device__ __forceinline__ void qt_coarse_solve(const QtHier<TI> &H, QtTeam &t)
{
	__shared__ TI sb[kQtMaxCoarse];
	const QtLevel<TI> &C = H.lv[0];
	const TI *bf = reinterpret_cast<const TI *>(C.b);
	TI *xf = reinterpret_cast<TI *>(C.x[0]);
	const int nc = H.nc, lane = threadIdx.x & 31;
	for (int j = threadIdx.x; j < nc; j += blockDim.x)
		sb[j] = bf[H.cdof[j]];
	__syncthreads();
	for (int i0 = 4 * (t.tid >> 5); i0 < nc; i0 += 4 * (t.nth >> 5)) {
		TI s[4] = {TI(0), TI(0), TI(0), TI(0)};
		const TI *row = H.cinv + (size_t)i0 * nc;
#pragma unroll 4
		for (int j = lane; j < nc; j += 32) {
			const TI b = sb[j];
#pragma unroll
			for (int u = 0; u < 4; u++)
				if (i0 + u < nc)
					s[u] += row[(size_t)u * nc + j] * b;
		}
#pragma unroll
		for (int u = 0; u < 4; u++) {
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
				s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
			if (lane == u && i0 + u < nc)
				xf[H.cdof[i0 + u]] = s[u];
		}
	}
	t.sync();
}

// z = V-cycle(b) with b in the finest level's b; *dot receives this thread's
// share of z.v.  Ends without a barrier (the caller's reduction follows).  While
// the leading block works on the smallest levels, the others run aside().
template <class TI, class Aside>
__device__ __forceinline__ void qt_vcycle(Sync &sy, const QtHier<TI> &H, typename Q2T<TI>::t *z, const double2 *v,
                                          double *dot, Aside aside)
{
	typedef typename Q2T<TI>::t V;
	const int top = H.nlev - 1, nb = H.nblk < top ? H.nblk : top;   // the finest level always runs on the team
	QtTeam team{&sy, true, sy.tid(), sy.nth()};
	*dot = 0.0;
#pragma unroll 1
	for (int l = top; l >= (nb > 1 ? nb : 1); l--)
		qt_down(H, l, team);
	if (nb > 0) {
		if (sy.leader()) {
			QtTeam blk{&sy, false, (int)threadIdx.x, (int)blockDim.x};
#pragma unroll 1
			for (int l = nb - 1; l >= 1; l--)
				qt_down(H, l, blk);
			qt_coarse_solve(H, blk);
#pragma unroll 1
			for (int l = 1; l < nb; l++)
				qt_up(H, l, blk);
		} else {
			aside();
		}
		sy.sync();
	} else {
		qt_coarse_solve(H, team);
	}
#pragma unroll 1
	for (int l = nb > 1 ? nb : 1; l <= top; l++)
		qt_up(H, l, team, l == top ? z : nullptr, v, dot);
	if (top == 0) {   // the dense solve is the whole cycle
		const QtLevel<TI> &Q = H.lv[0];
		for (int A = team.tid; A < Q.nno; A += team.nth) {
			const V o = Q.x[0][A];
			const double2 va = v[A];
			z[A] = o;
			*dot += widen(o.x) * va.x + widen(o.y) * va.y;
		}
	}
}

// Dense inverse of the coarsest level's constrained operator on its reduced
// dofs (FP64): the rows of C^T K C from their contribution lists, inverted by
// Gauss-Jordan (SPD: no pivoting) by the whole team, a warp per row.  The matrix
// alternates between two buffers, so that a pivot takes one team barrier.  One
// block alone took 1.1 ms per solve at 126 unknowns: an FP64 inversion of that
// size is 2 million multiply-adds on one SM's two FP64 lanes.
template <class TI>
__device__ __noinline__ void qt_coarse_build(Sync &sy, const QtHier<TI> &H)
{
	const QtLevel<TI> &C = H.lv[0];
	const int nc = H.nc, tid = sy.tid(), nth = sy.nth(), lane = threadIdx.x & 31;
	double *M = H.cwork, *N = H.cwork + (size_t)nc * nc, *at = H.cvec;   // at: a dof's row, -1 off the reduced dofs
	const double *K64f = reinterpret_cast<const double *>(C.K64);
	for (int k = tid; k < nc * nc; k += nth)
		M[k] = 0.0;
	for (int k = tid; k < 2 * C.nno; k += nth)
		at[k] = -1.0;
	sy.sync();
	for (int j = tid; j < nc; j += nth)
		at[H.cdof[j]] = (double)j;
	sy.sync();
	for (int A = tid; A < C.nno; A += nth) {
		const int i1 = C.rc_off[A + 1];
		for (int i = C.rc_off[A]; i < i1;) {
			const int t = C.rc_tgt[i], slot = t >> 2, cc = t & 3;
			double v = 0.0;
			for (; i < i1 && C.rc_tgt[i] == t; i++)
				v += (double)C.rc_w[i] * K64f[C.rc_src[i]];
			const int r = (int)at[2 * A + (cc >> 1)], c = (int)at[2 * C.rnb[(size_t)slot * C.nno + A] + (cc & 1)];
			if (r >= 0 && c >= 0)
				M[(size_t)r * nc + c] = v;
		}
	}
	sy.sync();
	for (int k = 0; k < nc; k++) {
		const double *pk = M + (size_t)k * nc;
		const double ip = (tid >> 5) < nc ? 1.0 / pk[k] : 0.0;   // (warps with rows only: see QtScal)
		for (int r = tid >> 5; r < nc; r += nth >> 5) {
			const double *row = M + (size_t)r * nc;
			double *out = N + (size_t)r * nc;
			const double f = row[k] * ip;
#pragma unroll 4
			for (int c = lane; c < nc; c += 32) {
				const double p = pk[c], m = row[c];
				out[c] = r == k ? (c == k ? ip : p * ip) : (c == k ? -f : m - f * p);
			}
		}
		sy.sync();
		double *t = M;
		M = N;
		N = t;
	}
	for (int k = tid; k < nc * nc; k += nth)
		H.cinv[k] = (TI)M[k];
	sy.sync();
}

// ---- FP64 residual and the preconditioner ------------------------------------------
// R = [C^T (F - K d - G p) ; G^T C d] (FP64); rs = |R_m|^2, |R_c|^2, |C^T F|^2.
template <class TI>
__device__ void qt_residual(Sync &sy, const QtArgs<TI> &a, const double2 *d, const double *p, double (&rs)[3])
{
	const int tid = sy.tid(), nth = sy.nth();
	const DevLevel &L = a.L;
	const QtLevel<TI> &Q = a.H.lv[a.H.nlev - 1];
	const double *df = reinterpret_cast<const double *>(d);
	const double *Ff = reinterpret_cast<const double *>(a.F);
	rs[0] = rs[1] = rs[2] = 0.0;
	for (int A = tid; A < L.nno; A += nth) {
		double k0, k1, g0, g1;
		qt_op_node(Q, Q.K64, df, A, k0, k1);
		qt_g_node(Q, L, p, A, g0, g1);
		double f[2] = {0.0, 0.0};
		for (int c = 0; c < 2; c++) {   // C^T F
			const int dof = 2 * A + c;
			if (Q.kind[dof] != 1)
				continue;
			f[c] = Ff[dof];
			for (int i = Q.fo_off[dof]; i < Q.fo_off[dof + 1]; i++)
				f[c] += (double)Q.fo_w[i] * Ff[Q.fo_dof[i]];
		}
		const double2 r = make_double2(Q.kind[2 * A] == 1 ? f[0] - k0 - g0 : 0.0,
		                               Q.kind[2 * A + 1] == 1 ? f[1] - k1 - g1 : 0.0);
		a.R[A] = r;
		rs[0] += r.x * r.x + r.y * r.y;
		rs[2] += f[0] * f[0] + f[1] * f[1];
	}
	for (int e = tid; e < L.nel; e += nth) {
		const double c = qt_gt_elem(Q, L, df, e);
		a.Rc[e] = c;
		rs[1] += c * c;
	}
	sy.reduce<3>(rs);
}

// The scalars of the MINRES recurrences, formed by one thread of each block: a
// division or a square root on every thread costs the FP64 pipe about a
// microsecond each.
struct QtScal {
	double gam, gam_prev, eta, eta0, delta, c_prev, c_cur, s_prev, s_cur;
	double ig, dg, gg, k1, k2, k3, step, step1;   // step1: the step of the iteration before
	int stop;   // 1: last iteration; 2: breakdown before the update; 4: a non-finite value
};

// The vector updates of the MINRES iteration (inlined: as calls they left no
// registers to the loop's state, whose accesses on the stack miss L1 after every
// team barrier: 157 against 117 us per iteration).

// v_p(j+1) = A z - dg v_p(j) - gg v_p(j-1) into v_p(j-1)'s buffer and z_p = v_p / BAB;
// returns this thread's share of z_p.v_p
__device__ __forceinline__ double qt_v_elems(int ne, int tid, int nth, const double *Ahp, const double *p0, double *p1,
                                             const double *ibab, double *z1, double ig, double dg, double gg)
{
	double acc = 0.0;
	for (int e = tid; e < ne; e += nth) {
		const double vn = Ahp[e] * ig - dg * p0[e] - gg * p1[e], z = vn * ibab[e];
		p1[e] = vn;
		z1[e] = z;
		acc += z * vn;
	}
	return acc;
}

// w(j+1) = (z~(j) - a3 w(j-1) - a2 w(j)) / a1 into w(j-1)'s buffer, and the steps of
// the solution: 0 none, 1 x += step w(j+1), 2 x += step1 w(j) + step w(j+1)
template <class V>
__device__ __forceinline__ void qt_w_update(int steps, int nn, int ne, int tid, int nth, const QtScal &ms, const V *z,
                                            double2 *wo, const double2 *wc, double2 *xu, const double *zp, double *po,
                                            const double *pc, double *xp)
{
	const double k1 = ms.k1, k2 = ms.k2, k3 = ms.k3, s0 = ms.step, s1 = ms.step1;
	for (int A = tid; A < nn; A += nth) {
		const V zz = z[A];
		const double2 o = wo[A], w = wc[A];
		double2 x = make_double2(0.0, 0.0);
		if (steps > 0)
			x = xu[A];
		const double2 wn = make_double2(widen(zz.x) * k1 - k3 * o.x - k2 * w.x, widen(zz.y) * k1 - k3 * o.y - k2 * w.y);
		wo[A] = wn;
		if (steps > 1) {
			x.x += s1 * w.x;
			x.y += s1 * w.y;
		}
		if (steps > 0)
			xu[A] = make_double2(x.x + s0 * wn.x, x.y + s0 * wn.y);
	}
	for (int e = tid; e < ne; e += nth) {
		const double w = pc[e];
		double x = steps > 0 ? xp[e] : 0.0;
		const double wn = zp[e] * k1 - k3 * po[e] - k2 * w;
		po[e] = wn;
		if (steps > 1)
			x += s1 * w;
		if (steps > 0)
			xp[e] = x + s0 * wn;
	}
}

// Correction solve by preconditioned MINRES (Elman, Silvester and Wathen,
// "Finite Elements and Fast Iterative Solvers", Alg. 4.1) on the constrained
// system [C^T K C, C^T G; G^T C, 0][x_u; x_p] = [R_m; -R_c] from zero, with the
// preconditioner diag(V-cycle, BAB); K in TI, G to FP64 accuracy, Lanczos and
// direction vectors FP64; x into a.dd, a.dpv, two iterations' steps at a time.
template <class TI>
__device__ __noinline__ int qt_minres(Sync &team, const QtArgs<TI> &a, double rtol, int maxit)
{
	typedef typename Q2T<TI>::t V;
	__shared__ QtScal ms;
	Sync sy = team;
	const DevLevel &L = a.L;
	const QtLevel<TI> &Q = a.H.lv[a.H.nlev - 1];
	double pdot = 0.0;
	{
		const double2 zero2 = make_double2(0.0, 0.0);
		const int tid = sy.tid(), nth = sy.nth(), nn = L.nno, ne = L.nel;
		for (int A = tid; A < nn; A += nth) {
			const double2 r = a.R[A];
			a.mv[0][A] = r;
			V w;
			w.x = narrow_to<TI>(r.x);
			w.y = narrow_to<TI>(r.y);
			Q.b[A] = w;
			a.mv[1][A] = zero2;
			a.mw[0][A] = zero2;
			a.mw[1][A] = zero2;
			a.dd[A] = zero2;
		}
		for (int e = tid; e < ne; e += nth) {
			const double v = -a.Rc[e], z = v * a.ibab[e];
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
	// levels (111 against 117 us per iteration at 85k nodes, a step of eight
	// ensemble members 27.4 against 28.5 ms).
	// steps: the pending direction update's (-1: none).
	const bool defer = sy.size >= 4 && a.H.nblk > 0 && a.H.nlev > 1;
	int steps = -1;
#pragma unroll 1
	while (it < maxit) {
		if (it >= 0) {
			const int tid = sy.tid(), nth = sy.nth();
			double dl[1] = {0.0};
			{
				const V *z = a.mz[cv];
				const double *zp = a.mzp[cv];
				const TI *zf = reinterpret_cast<const TI *>(z);
				// nodes and elements in one range: with two loops each would end in a
				// trip for the few left over
				const int nn = L.nno, ni = nn + L.nel;
				for (int A = tid; A < ni; A += nth) {
					if (A >= nn) {
						const int e = A - nn;
						const double t = qt_gt_elem(Q, L, zf, e);
						a.Ahp[e] = t;
						dl[0] += t * zp[e];
						continue;
					}
					TI k0, k1;
					double g0, g1;
					const V zz = z[A];
					qt_kr_node(Q, zf, A, k0, k1);
					qt_g_node(Q, L, zp, A, g0, g1);
					const double2 az = make_double2(widen(k0) + g0, widen(k1) + g1);
					a.Kd[A] = az;
					dl[0] += az.x * widen(zz.x) + az.y * widen(zz.y);
				}
			}
			sy.reduce_then<1>(dl, [&](const double (&v)[1]) {
				ms.delta = v[0] * ms.ig * ms.ig;
				ms.dg = ms.delta * ms.ig;
			});
			// v(j+1) into v(j-1)'s buffer, its TI copy as the V-cycle's right-hand side,
			// and z_p(j+1) = v_p(j+1) / BAB
			const double ig = ms.ig, dg = ms.dg, gg = ms.gg;
			{
				const double2 *v = a.mv[cv];
				double2 *vo = a.mv[1 - cv];
				for (int A = tid; A < L.nno; A += nth) {
					const double2 az = a.Kd[A], vc = v[A], vp = vo[A];
					const double2 vn = make_double2(az.x * ig - dg * vc.x - gg * vp.x, az.y * ig - dg * vc.y - gg * vp.y);
					vo[A] = vn;
					V w;
					w.x = narrow_to<TI>(vn.x);
					w.y = narrow_to<TI>(vn.y);
					Q.b[A] = w;
				}
			}
			pdot = 0.0;
			if (!defer)
				pdot = qt_v_elems(L.nel, tid, nth, a.Ahp, a.mvp[cv], a.mvp[1 - cv], a.ibab, a.mzp[1 - cv], ig, dg, gg);
			sy.sync();
		}
		double dot[1];
		qt_vcycle(sy, a.H, a.mz[1 - cv], a.mv[1 - cv], &dot[0], [&] {
			if (!defer || it < 0)
				return;
			// the previous iteration's direction update (its z(j-1) and z_p(j-1) lie in
			// the buffers that this iteration's z(j+1) overwrites: z_u after this point,
			// z_p below by the same thread), and the pressure part of the Lanczos update
			const Part pt{sy.rank - 1, sy.size - 1};
			const int tid = pt.thread(), nth = pt.size * (int)blockDim.x;
			if (steps >= 0)
				qt_w_update(steps, L.nno, L.nel, tid, nth, ms, a.mz[1 - cv], a.mw[cw], a.mw[1 - cw], a.dd, a.mzp[1 - cv],
				            a.mwp[cw], a.mwp[1 - cw], a.dpv);
			pdot = qt_v_elems(L.nel, tid, nth, a.Ahp, a.mvp[cv], a.mvp[1 - cv], a.ibab, a.mzp[1 - cv], ms.ig, ms.dg,
			                  ms.gg);
		});
		dot[0] += pdot;
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
				ms.stop = v[0] > 0.0 ? 0 : 3;
				return;
			}
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
			ms.step1 = ms.step;
			ms.k1 = ms.ig * ia1;
			ms.k2 = a2 * ia1;
			ms.k3 = a3 * ia1;
			ms.step = c_next * ms.eta;
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
		const int tid = sy.tid(), nth = sy.nth();
		const int stop = ms.stop;
		if ((stop & 4) && tid == 0)
			atomicOr(&a.sc->status, kStatNan);
		if (stop & 2) {
			if (it & 1) {   // the pending step along w(j)
				const double s = ms.step;
				for (int A = tid; A < L.nno; A += nth) {
					const double2 w = a.mw[cw][A], x = a.dd[A];
					a.dd[A] = make_double2(x.x + s * w.x, x.y + s * w.y);
				}
				for (int e = tid; e < L.nel; e += nth)
					a.dpv[e] += s * a.mwp[cw][e];
			}
			break;
		}
		const bool last = stop || it + 1 >= maxit;
		steps = (it & 1) ? 2 : last ? 1 : 0;   // the solution takes two iterations' steps at a time
		if (!defer || last)
			qt_w_update(steps, L.nno, L.nel, tid, nth, ms, a.mz[cv], a.mw[1 - cw], a.mw[cw], a.dd, a.mzp[cv],
			            a.mwp[1 - cw], a.mwp[cw], a.dpv);
		it++;
		cv = 1 - cv;
		cw = 1 - cw;
		if (stop)
			break;
		if (threadIdx.x == 0) {   // for the next step; read after the next reduction's broadcast
			ms.ig = 1.0 / ms.gam;
			ms.gg = ms.gam / ms.gam_prev;
		}
		// no barrier here: the next operator pass reads z(j+1) and z_p(j+1), complete
		// since the reduction, and writes none of the vectors the updates above read
	}
	sy.sync();
	team = sy;
	return it;
}

// The whole converged solve of one refined model on the team `sy`.
template <class TI>
__device__ void qt_solve(const QtArgs<TI> &a, Sync &sy)
{
	const int tid = sy.tid(), nth = sy.nth();
	const QtHier<TI> &H = a.H;
	const DevLevel &L = a.L;
	int *status = &a.sc->status;

	for (int e = tid; e < L.nel; e += nth)
		a.ibab[e] = 1.0 / a.bab[e];
	// -- per step: every level's reduced operator C^T K C in TI, and its diagonal
	for (int l = 0; l < H.nlev; l++) {
		const QtLevel<TI> &Q = H.lv[l];
		const double *K64f = reinterpret_cast<const double *>(Q.K64);
		TI *Krf = reinterpret_cast<TI *>(Q.Kr);
		for (int A = tid; A < Q.nno; A += nth) {
			for (int u = 0; u < Q.rnbw; u++) {
				const size_t b = ((size_t)u * Q.nno + A) * 4;
				Krf[b] = Krf[b + 1] = Krf[b + 2] = Krf[b + 3] = TI(0);
			}
			int self = -1;
			for (int u = 0; u < Q.rcnt[A]; u++)
				if (Q.rnb[(size_t)u * Q.nno + A] == A)
					self = u;
			double dgl[2] = {0.0, 0.0};
			const int i1 = Q.rc_off[A + 1];
			for (int i = Q.rc_off[A]; i < i1;) {
				const int t = Q.rc_tgt[i];
				double v = 0.0;
				for (; i < i1 && Q.rc_tgt[i] == t; i++)
					v += (double)Q.rc_w[i] * K64f[Q.rc_src[i]];
				const int slot = t >> 2, cc = t & 3;
				Krf[((size_t)slot * Q.nno + A) * 4 + cc] = (TI)v;
				if (slot == self && (cc == 0 || cc == 3))
					dgl[cc == 3] = v;
			}
			for (int c = 0; c < 2; c++)
				Q.invD[2 * A + c] = Q.kind[2 * A + c] == 1 && dgl[c] > 0.0 ? (TI)(1.0 / dgl[c]) : TI(0);
		}
	}
	sy.sync();
	qt_coarse_build(sy, H);

	int refine = 0, minres_total = 0, vcycles = 0, capped = 0;
	double res_m = 0.0, res_c = 0.0;
	while (true) {
		double rs[3];
		qt_residual(sy, a, a.d, a.p, rs);
		// a zero load (|C^T F| = 0): the residual is measured absolutely
		const double fnorm = rs[2] > 0.0 ? sqrt(rs[2]) : 1.0;
		res_m = sqrt(rs[0]) / fnorm;
		res_c = sqrt(rs[1]) / fnorm;
		const double res = sqrt(rs[0] + rs[1]) / fnorm;
		if (!isfinite(res)) {
			if (tid == 0)
				atomicOr(status, kStatNan);
			break;
		}
		if (!(res >= a.rtol))
			break;
		if (refine >= a.max_refine) {
			capped = 1;
			break;
		}
		refine++;
		// far from the target a pass reduces by 1e-2, close to it by what is
		// left (factor 2 margin), not below outer_rtol
		const double prt = res > 1e4 * a.rtol ? 1e-2 : fmax(a.outer_rtol, 0.5 * a.rtol / res);
		const int it = qt_minres(sy, a, prt, a.max_outer);
		minres_total += it;
		vcycles += it + 1;
		for (int A = tid; A < L.nno; A += nth) {
			const double2 c = a.dd[A];
			double2 v = a.d[A];
			v.x += c.x;
			v.y += c.y;
			a.d[A] = v;
		}
		for (int e = tid; e < L.nel; e += nth)
			a.p[e] += a.dpv[e];
		sy.sync();
	}
	if (capped && tid == 0)
		atomicOr(status, kStatCap);
	// the hanging nodes' values, and the velocity with its boundary values (v_to_nodes)
	const QtLevel<TI> &Q = H.lv[H.nlev - 1];
	double *df = reinterpret_cast<double *>(a.d);
	for (int A = tid; A < L.nno; A += nth) {
		double v[2];
		for (int c = 0; c < 2; c++)
			v[c] = qt_val(Q, (const double *)df, 2 * A + c);
		a.V[A] = make_double2(vfree(L, A, 0) ? v[0] : L.vbcval[A], vfree(L, A, 1) ? v[1] : L.vbcval[L.nno + A]);
	}
	sy.sync();
	for (int A = tid; A < L.nno; A += nth)
		for (int c = 0; c < 2; c++)
			if (Q.kind[2 * A + c] == 2)
				df[2 * A + c] = vfree(L, A, c) ? (c ? a.V[A].y : a.V[A].x) : 0.0;
	if (tid == 0) {
		StepScalars *sc = a.sc;
		sc->uzawa_cycles = minres_total;
		sc->cg_cycles = vcycles;
		sc->refine_passes = refine;
		sc->res_m = res_m;
		sc->res_c = res_c;
		sc->dv = 0.0;
		sc->dp = 0.0;
	}
}

// One refined model on the whole cooperative grid, or on one cluster.
template <class TI>
__global__ void __launch_bounds__(kTeamThreads) k_stokes_qt(const __grid_constant__ QtArgs<TI> a)
{
	__shared__ QtArgs<TI> sa;
	load_args(sa, a);
	__shared__ double cpart[2 * kRedWidth];
	Sync sy = sa.cluster ? Sync::of(SYNC_CLUSTER, cpart, blockIdx.x, gridDim.x)
	                     : Sync::of(SYNC_GRID, sa.red.part, blockIdx.x, gridDim.x);
	qt_solve<TI>(sa, sy);
	if (sa.cluster)
		cg::this_cluster().sync();   // no block leaves while another reads its partials
}

// A batch of independent refined models, launched with clusters of `cs`
// blocks (cs = 1: plain blocks).  Each cluster takes the next model from the
// queue (ordered largest first by the host) and solves it alone with cluster
// barriers, so clusters never wait on one another.  The rank-0 block draws and
// every block reads the draw from its shared memory.
template <class TI>
__global__ void __launch_bounds__(kBlock) k_stokes_qt_batch(const QtArgs<TI> *models, int nmodels, int *queue)
{
	__shared__ QtArgs<TI> sa;
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
			qt_solve<TI>(sa, sy);
			cl.sync();   // no block starts the next model (or leaves) while another reads its partials
		} else {
			__syncthreads();
			const int m = next;
			__syncthreads();
			if (m >= nmodels)
				break;
			load_args(sa, models[m]);
			Sync sy = Sync::of(SYNC_BLOCK, nullptr, 0, 1);
			qt_solve<TI>(sa, sy);
			__syncthreads();
		}
	}
}

// linear extrapolation of the last two solutions: x = 2 x1 - x2
__global__ void __launch_bounds__(kBlock) k_qt_extrapolate(int n2, int ne, const double *d1, const double *d2,
                                                           const double *p1, const double *p2, double *d, double *p)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n2)
		d[i] = 2.0 * d1[i] - d2[i];
	if (i < ne)
		p[i] = 2.0 * p1[i] - p2[i];
}

// d1 <- d - (d1 - d2): the history shift of the second step after a remesh
__global__ void __launch_bounds__(kBlock) k_qt_shift(int n2, int ne, const double *d, const double *p, double *d1,
                                                     double *p1, const double *d2, const double *p2)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n2)
		d1[i] = d[i] - d1[i] + d2[i];
	if (i < ne)
		p1[i] = p[i] - p1[i] + p2[i];
}

// Coarse-level viscosity from the finer level around the same node: the value
// there (avg 0), or the mean (1) or log-mean (2) over the node and its matrix
// neighbours on the finer level, weighted 1 (the node), 1/2 (a neighbour
// along an axis), 1/4 (a diagonal neighbour) -- full weighting where the
// finer level is uniform.
__global__ void __launch_bounds__(kBlock) k_qt_inject(int n, const int *map, const double *src, double *dst, int avg,
                                                      int nno_f, const int *nb_f, const unsigned char *cnt_f,
                                                      const double *X_f)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	const int a = map[i];
	if (avg == 0) {
		dst[i] = src[a];
		return;
	}
	const double xa = X_f[a], za = X_f[nno_f + a];
	double s = 0.0, ws = 0.0;
	for (int k = 0; k < cnt_f[a]; k++) {
		const int B = nb_f[(size_t)k * nno_f + a] & ~kQtCon;
		const bool ax = X_f[B] == xa, az = X_f[nno_f + B] == za;
		const double w = (ax && az) ? 1.0 : (ax || az) ? 0.5 : 0.25;
		s += w * (avg == 2 ? log(src[B]) : src[B]);
		ws += w;
	}
	s /= ws;
	dst[i] = avg == 2 ? exp(s) : s;
}

void *qt_kernel(int fp64) { return fp64 ? (void *)k_stokes_qt<double> : (void *)k_stokes_qt<float>; }
void *qt_batch_kernel(int fp64)
{
	return fp64 ? (void *)k_stokes_qt_batch<double> : (void *)k_stokes_qt_batch<float>;
}

}  // namespace mclg
