// Converged Stokes solve on quadtree meshes with hanging nodes; see k_qt.cuh.
// One persistent kernel per time step.  Vectors are node layout
// (both components of a node together); a primal vector stores its reduced
// dofs and is read through the constraints (qt_val), a dual vector (operator
// output, residual) is zero outside the reduced dofs.
//
// Order of operations.  The pressure's least determined modes on a mesh of many
// refinement levels follow the rounding of the iterates: on a mesh of 85k nodes
// half an ulp on the temperature moves P by 3e-10 .. 1.2e-8, whatever the stop that
// FP64 allows.  So every value that reaches the iterates is formed by one fixed
// sequence of operations, and every sum in one fixed order (QtSync), whichever team
// runs the solve and however a pass cuts its work.  What a pass is free to choose is
// which thread does a node's work, what is in flight together, and when a vector
// update runs.
#include <math.h>
#include "k_qt.cuh"
#include "fp64_util.cuh"

namespace mclg {

MCLG_SHAPE_UPLOAD(upload_shape_tables_qt)

// ---- rounding -----------------------------------------------------------------------
// Where a multiply-add could be formed in more than one way, the way is stated.
__device__ __forceinline__ float madd(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double madd(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }

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
		o.x = mul(mul(omega, dv.x), bv.x);
		o.y = mul(mul(omega, dv.y), bv.y);
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

// a b - c d - e f, as every recurrence of vectors here rounds it
__device__ __forceinline__ double lin3(double a, double b, double c, double d, double e, double f)
{
	return __fma_rn(-e, f, __fma_rn(a, b, -__dmul_rn(c, d)));
}

// acc + (a b + c d), as every sum of products over nodes rounds it
__device__ __forceinline__ double add2(double acc, double a, double b, double c, double d)
{
	return __dadd_rn(acc, __fma_rn(a, b, __dmul_rn(c, d)));
}

// s = sum of w[i] x[src[i]] over [i0, i1) in the list's order, C entries at a time:
// their indices, then their gathers in flight together (a list's loop waits for
// both in turn).
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
			s = i + u < i1 ? madd(ww[u], xv[u], s) : s;
	}
	return s;
}

// G's entries of an element (element_g) by corner: the magnitudes of component 0 are
// those of corners 0 (0 and 3) and 1 (1 and 2), of component 1 those of corners 0
// (0 and 1) and 2 (2 and 3); the sums over the Gauss points that give them run
// through the same products in the same order.  8 FP64 operations a corner, formed
// once per solve (a.ge[4 e ..]) instead of at every corner that an iteration visits.
// They are the half-widths to within their last bit.
__device__ __forceinline__ void qt_g_table(const DevLevel &L, int e, double *ge)
{
	double g0, g1, h0, h1, k0, k1;
	element_g(cS, L.dzh[e], L.dxh[e], 0, g0, g1);
	element_g(cS, L.dzh[e], L.dxh[e], 1, h0, h1);
	element_g(cS, L.dzh[e], L.dxh[e], 2, k0, k1);
	ge[4 * (size_t)e] = g0;
	ge[4 * (size_t)e + 1] = h0;
	ge[4 * (size_t)e + 2] = g1;
	ge[4 * (size_t)e + 3] = -k1;
}
template <int c>
__device__ __forceinline__ int qt_g_slot(int a)
{
	return c ? 2 + (a >> 1) : (a == 1 || a == 2);
}
template <int c>
__device__ __forceinline__ bool qt_g_pos(int a)
{
	return c ? a == 0 || a == 3 : a < 2;
}

// G p at node A on the finest level, its elements in order (gmul_node).
__device__ __forceinline__ void qt_gmul(const DevLevel &L, const double *__restrict__ ge, const double *__restrict__ p,
                                        int A, double &y0, double &y1)
{
	double s0 = 0.0, s1 = 0.0;
	const int n = L.p2n_cnt[A];
	int e[4], a[4];
#pragma unroll
	for (int k = 0; k < 4; k++) {
		e[k] = L.p2n_el[k * L.nno + A];
		a[k] = L.p2n_a[k * L.nno + A];
	}
	double pe[4], h0[4], h1[4];
#pragma unroll
	for (int k = 0; k < 4; k++) {
		const int ek = k < n ? e[k] : e[0], ak = k < n ? a[k] : 0;
		const double *g = ge + 4 * (size_t)ek;
		pe[k] = p[ek];
		h0[k] = g[qt_g_slot<0>(ak)];
		h1[k] = g[qt_g_slot<1>(ak)];
	}
#pragma unroll
	for (int k = 0; k < 4; k++)
		if (k < n) {
			s0 = madd(qt_g_pos<0>(a[k]) ? h0[k] : -h0[k], pe[k], s0);
			s1 = madd(qt_g_pos<1>(a[k]) ? h1[k] : -h1[k], pe[k], s1);
		}
	y0 = s0;
	y1 = s1;
}

// (C^T G p) at both dofs of node A (FP64, the finest level)
template <class T>
__device__ __forceinline__ void qt_g_node(const QtLevel<T> &Q, const DevLevel &L, const double *__restrict__ ge,
                                          const double *__restrict__ p, int A, double &y0, double &y1)
{
	const uchar2 k = reinterpret_cast<const uchar2 *>(Q.kind)[A];
	const int f0 = Q.fo_off[2 * A], f1 = Q.fo_off[2 * A + 1], f2 = Q.fo_off[2 * A + 2];
	qt_gmul(L, ge, p, A, y0, y1);
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
			const int c = h[u] & 1;
#pragma unroll
			for (int q = 0; q < 4; q++) {
				const bool in = q < n[u];
				const int eq = in ? e[u][q] : e[u][0], aq = in ? a[u][q] : 0;
				pe[u][q] = p[eq];
				g[u][q] = ge[4 * (size_t)eq + (c ? qt_g_slot<1>(aq) : qt_g_slot<0>(aq))];
			}
		}
#pragma unroll
		for (int u = 0; u < 2; u++) {
			double s = 0.0;
#pragma unroll
			for (int q = 0; q < 4; q++)
				if (q < n[u]) {
					const bool pos = (h[u] & 1) ? qt_g_pos<1>(a[u][q]) : qt_g_pos<0>(a[u][q]);
					s = madd(pos ? g[u][q] : -g[u][q], pe[u][q], s);
				}
			if (i + u < ie) {
				if (i + u < f1)
					y0 = madd(w[u], s, y0);
				else
					y1 = madd(w[u], s, y1);
			}
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
				x[a] = madd(w[2 * a], v[2 * a], x[a]);
			if (s[2 * a + 1] >= 0)
				x[a] = madd(w[2 * a + 1], v[2 * a + 1], x[a]);
			i0[a] += 2;
			any |= i0[a] < i1[a];
		}
	}
}

// (G^T C u)_e of a primal vector u (flat, X) on the finest level, in FP64: the
// corners in ascending order of their equations.
template <class T, class X>
__device__ __forceinline__ double qt_gt_elem(const QtLevel<T> &Q, const DevLevel &L, const double *__restrict__ ge,
                                             const X *__restrict__ uf, int e)
{
	int n[4];
	X u[4], w[4];
	uchar2 k[4];
	double g[4];
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
	{
		const double2 *g2 = reinterpret_cast<const double2 *>(ge) + 2 * (size_t)e;
		const double2 ga = g2[0], gb = g2[1];
		g[0] = ga.x;
		g[1] = ga.y;
		g[2] = gb.x;
		g[3] = gb.y;
	}
	qt_constrained<0>(Q, uf, n, k, u);
	qt_constrained<1>(Q, uf, n, k, w);
	double s = 0.0;
#pragma unroll
	for (int q = 0; q < 4; q++) {
		const int a = q < 2 ? q : 5 - q;   // kSortedCorner: 0, 1, 3, 2
		const double g0 = g[qt_g_slot<0>(a)], g1 = g[qt_g_slot<1>(a)];
		s = madd(qt_g_pos<0>(a) ? g0 : -g0, widen(u[a]), s);
		s = madd(qt_g_pos<1>(a) ? g1 : -g1, widen(w[a]), s);
	}
	return s;
}

// ---- sums over the team -----------------------------------------------------------
// The order of a single model's sums is that of blocks of 256 threads that take the
// nodes, then the elements, in their own order: butterflies over 32 threads (distances
// 16 .. 1), over a block's eight warps (4, 2, 1), and over the blocks (the same tree
// over blocks 0 .. 255, those from 256 on added to them first).  A grid runs just so:
// id() numbers its threads.  A cluster deals its warps over 16 blocks of 512 threads,
// each node having a thread of its own, and runs its sums through the same tree.
// A batch's teams, whose size is chosen by timing them, sum in the order of their own.
constexpr int kQtPartials = 3 * (kTeamThreads / 32);   // a block's partials of one reduction
struct QtSync : Sync {
	static constexpr int kWarps = kTeamThreads / 32, kPad = 36;   // (stride 36: warps 0 .. 3 in different banks)
	bool single;   // a single model (else a batch)
	__device__ static double *scratch()
	{
		__shared__ double sh[3 * kWarps * kPad];
		return sh;
	}
	__device__ int id() const { return mode == SYNC_GRID ? rank * (int)blockDim.x + (int)threadIdx.x : tid(); }
	// f(sums) on thread 0 of each block; what it writes to shared memory is visible
	// to the block on return.  A warp takes eight warps' values through shared memory,
	// so that the halves that a butterfly would drop cost nothing: 12 FP64 additions
	// of one warp for a block of 256 instead of 40 (the FP64 pipe has two lanes per
	// clock and SM).
	template <int NV, class F>
	__device__ __forceinline__ void reduce_then(const double (&v)[NV], F f)
	{
		static_assert(NV <= 3, "scratch");
		double *sh = scratch();
		const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
		for (int k = 0; k < NV; k++)
			sh[(k * kWarps + w) * kPad + lane] = v[k];
		__syncthreads();
		double t[NV];
#pragma unroll
		for (int k = 0; k < NV; k++)
			t[k] = 0.0;
		if (w < (int)(blockDim.x >> 8)) {   // warp w: the sums of warps 8 w .. 8 w + 7, four lanes each
#pragma unroll
			for (int k = 0; k < NV; k++) {
				const double *s = sh + (k * kWarps + 8 * w + (lane >> 2)) * kPad + (lane & 3);
				t[k] = ((s[0] + s[16]) + (s[8] + s[24])) + ((s[4] + s[20]) + (s[12] + s[28]));
				t[k] += __shfl_xor_sync(0xffffffffu, t[k], 2);
				t[k] += __shfl_xor_sync(0xffffffffu, t[k], 1);
			}
		}
		if (single && mode == SYNC_CLUSTER) {
			// partials[flip][k][warp]; group g of 32 threads is warp g / 16 of block g % 16
			double *mine = partials + flip * kQtPartials;
			if (w < 2 && (lane & 3) == 0)
#pragma unroll
				for (int k = 0; k < NV; k++)
					mine[k * kWarps + 8 * w + (lane >> 2)] = t[k];
			cg::cluster_group cl = cg::this_cluster();
			cl.sync();
			if (w == 0) {   // lane b: groups 8 b .. 8 b + 7
#pragma unroll
				for (int k = 0; k < NV; k++) {
					double x[8];
#pragma unroll
					for (int q = 0; q < 8; q++)
						x[q] = cl.map_shared_rank(mine, (lane & 1) * 8 + q)[k * kWarps + (lane >> 1)];
					t[k] = warp_sum(((x[0] + x[4]) + (x[2] + x[6])) + ((x[1] + x[5]) + (x[3] + x[7])));
				}
			}
			flip ^= 1;
		} else {
			if (w == 0)
#pragma unroll
				for (int k = 0; k < NV; k++)
					t[k] = eight(t[k]);
			if (mode == SYNC_GRID) {
				double *buf = partials + (size_t)flip * kMaxCoopBlocks * kRedWidth;
				if (threadIdx.x == 0)
#pragma unroll
					for (int k = 0; k < NV; k++)
						buf[k * kMaxCoopBlocks + rank] = t[k];
				cg::this_grid().sync();
				if (w == 0) {
#pragma unroll
					for (int k = 0; k < NV; k++) {
						const double *src = buf + k * kMaxCoopBlocks;
						const int b0 = (lane >> 2) * 32 + (lane & 3);
						double x[8];
#pragma unroll
						for (int m = 0; m < 8; m++)
							x[m] = b0 + 4 * m < size ? src[b0 + 4 * m] : 0.0;
						for (int o = 256; o < size; o += 256) {
							double y[8];
#pragma unroll
							for (int m = 0; m < 8; m++)
								y[m] = o + b0 + 4 * m < size ? src[o + b0 + 4 * m] : 0.0;
#pragma unroll
							for (int m = 0; m < 8; m++)
								x[m] += y[m];
						}
						double s = ((x[0] + x[4]) + (x[2] + x[6])) + ((x[1] + x[5]) + (x[3] + x[7]));
						s += __shfl_xor_sync(0xffffffffu, s, 2);
						s += __shfl_xor_sync(0xffffffffu, s, 1);
						t[k] = eight(s);
					}
				}
				flip ^= 1;
			} else if (mode == SYNC_CLUSTER) {
				double *mine = partials + flip * kQtPartials;
				if (threadIdx.x == 0)
#pragma unroll
					for (int k = 0; k < NV; k++)
						mine[k] = t[k];
				cg::cluster_group cl = cg::this_cluster();
				cl.sync();
				if (w == 0) {
					const double *other = cl.map_shared_rank(mine, lane < size ? lane : 0);
#pragma unroll
					for (int k = 0; k < NV; k++) {
						t[k] = warp_sum(lane < size ? other[k] : 0.0);
					}
				}
				flip ^= 1;   // the next reduction writes the other buffer (see GridRed)
			}
		}
		if (threadIdx.x == 0)
			f(t);
		__syncthreads();
	}
	// The sums in every thread.
	template <int NV>
	__device__ __forceinline__ void reduce(double (&v)[NV])
	{
		__shared__ double out[NV];
		reduce_then<NV>(v, [&](const double (&t)[NV]) {
#pragma unroll
			for (int k = 0; k < NV; k++)
				out[k] = t[k];
		});
#pragma unroll
		for (int k = 0; k < NV; k++)
			v[k] = out[k];
	}
	// the sum over eight warps from lanes of four each
	static __device__ double eight(double v)
	{
		v += __shfl_xor_sync(0xffffffffu, v, 16);
		v += __shfl_xor_sync(0xffffffffu, v, 8);
		v += __shfl_xor_sync(0xffffffffu, v, 4);
		return v;
	}
	static __device__ QtSync of(int mode, double *partials, int rank, int size, bool single)
	{
		QtSync s;
		static_cast<Sync &>(s) = Sync::of(mode, partials, rank, size);
		s.single = single;
		return s;
	}
};

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
	o.x = k.x == 1 ? madd(mul(omega, dg.x), b.x - y0, x.x) : TI(0);
	o.y = k.y == 1 ? madd(mul(omega, dg.y), b.y - y1, x.y) : TI(0);
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
	QtSync *sy;
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
// With zout (the finest level) the last sweep writes there and leaves this thread's
// share of zout.v in *dot (nodes by QtSync::id), and is not followed by a barrier:
// the caller's reduction provides it.
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
			for (int A = t.sy->id(); A < L.nno; A += t.nth) {
				const double2 va = v[A];
				const V o = qt_sweep_node(L, H.omega, src, A);
				zout[A] = o;
				acc = add2(acc, widen(o.x), va.x, widen(o.y), va.y);
			}
			*dot = acc;
			return;
		}
		qt_sweep(L, H.omega, L.x[cur], L.x[1 - cur], t.tid, t.nth);
		cur = 1 - cur;
		t.sync();
	}
}

// coarsest level: the dense inverse on its reduced dofs, a thread per row, each row's
// products in order.  The inverse is stored by columns, so that a warp's rows are
// adjacent (by rows, 4*nc bytes apart, it took 8.3 us of a 128 us iteration for 126
// unknowns, now 3 .. 4), and sixteen columns are in flight together; more of them, or
// the next sixteen ahead, cost the solver its registers (133 .. 160 against 124 us).
template <class TI>
__device__ __forceinline__ void qt_coarse_solve(const QtHier<TI> &H, QtTeam &t)
{
	__shared__ TI sb[kQtMaxCoarse];
	const QtLevel<TI> &C = H.lv[0];
	const TI *bf = reinterpret_cast<const TI *>(C.b);
	TI *xf = reinterpret_cast<TI *>(C.x[0]);
	const int nc = H.nc;
	for (int j = threadIdx.x; j < nc; j += blockDim.x)
		sb[j] = bf[H.cdof[j]];
	__syncthreads();
	constexpr int kCols = 16;
	for (int i = t.tid; i < nc; i += t.nth) {
		TI s = TI(0);
		for (int j0 = 0; j0 < nc; j0 += kCols) {
			TI m[kCols];
#pragma unroll
			for (int u = 0; u < kCols; u++)
				m[u] = j0 + u < nc ? H.cinv[(size_t)(j0 + u) * nc + i] : TI(0);
#pragma unroll
			for (int u = 0; u < kCols; u++)
				if (j0 + u < nc)
					s = madd(m[u], sb[j0 + u], s);
		}
		xf[H.cdof[i]] = s;
	}
	t.sync();
}

// z = V-cycle(b) with b in the finest level's b; *dot receives this thread's
// share of z.v (nodes by QtSync::id).  Ends without a barrier (the caller's reduction follows).  While
// the leading block works on the smallest levels, the others run aside().
template <class TI, class Aside>
__device__ __forceinline__ void qt_vcycle(QtSync &sy, const QtHier<TI> &H, typename Q2T<TI>::t *z, const double2 *v,
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
		for (int A = sy.id(); A < Q.nno; A += team.nth) {
			const V o = Q.x[0][A];
			const double2 va = v[A];
			z[A] = o;
			*dot = add2(*dot, widen(o.x), va.x, widen(o.y), va.y);
		}
	}
}

// Entry (row dof d, column dof j) of C^T K C on a level: qt_op_node applied to the
// unit vector of j.
template <class T>
__device__ double qt_unit_val(const QtLevel<T> &L, int dof, int j)
{
	const unsigned char k = L.kind[dof];
	if (k == 1)
		return dof == j ? 1.0 : 0.0;
	double s = 0.0;
	if (k == 2)
		for (int i = L.ex_off[dof]; i < L.ex_off[dof + 1]; i++)
			if (L.ex_src[i] == j)
				s += (double)L.ex_w[i];
	return s;
}
template <class T>
__device__ double qt_unit_row(const QtLevel<T> &L, int d, int j)
{
	const int A = d >> 1, n = L.cnt[A];
	double s = 0.0;
	for (int k = 0; k < n; k++) {
		const int B = L.nb[(size_t)k * L.nno + A] & ~kQtCon;
		const double4 kb = L.K64[(size_t)k * L.nno + A];
		const double x = qt_unit_val(L, 2 * B, j), y = qt_unit_val(L, 2 * B + 1, j);
		s += (d & 1) ? kb.z * x + kb.w * y : kb.x * x + kb.y * y;
	}
	return s;
}
template <class T>
__device__ __noinline__ double qt_unit_entry(const QtLevel<T> &L, int d, int j)
{
	double y = qt_unit_row(L, d, j);
	for (int i = L.fo_off[d]; i < L.fo_off[d + 1]; i++)
		y = madd((double)L.fo_w[i], qt_unit_row(L, L.fo_dof[i], j), y);
	return y;
}

// Dense inverse of the coarsest level's constrained operator on its reduced
// dofs (FP64), by Gauss-Jordan (SPD: no pivoting) by the whole team, a warp per
// row: the pivot's row divided by the pivot, then taken from the others.  The
// matrix alternates between two buffers, so that a pivot takes one team barrier;
// the warp that forms the next pivot's row divides it as well (every warp dividing
// it for itself cost a batch's cluster 6 us of its FP64 pipes a pivot).  One block
// alone took 1.1 ms per solve at 126 unknowns: an FP64 inversion of that size is 2
// million multiply-adds on one SM's two FP64 lanes.
template <class TI>
__device__ __noinline__ void qt_coarse_build(QtSync &sy, const QtHier<TI> &H)
{
	const QtLevel<TI> &C = H.lv[0];
	const int nc = H.nc, tid = sy.tid(), nth = sy.nth(), lane = threadIdx.x & 31;
	const size_t n2 = (size_t)nc * nc;
	double *M = H.cwork, *N = M + n2, *pk = N + n2, *pn = pk + nc;   // pk, pn: this pivot's row divided, the next one's
	for (int k = tid; k < nc * nc; k += nth)
		M[k] = qt_unit_entry(C, H.cdof[k / nc], H.cdof[k % nc]);
	sy.sync();
	if (tid >> 5 == 0)
		for (int c = lane; c < nc; c += 32)
			pk[c] = (c == 0 ? 1.0 : M[c]) / M[0];
	sy.sync();
	for (int k = 0; k < nc; k++) {
		for (int r = tid >> 5; r < nc; r += nth >> 5) {
			const double *row = M + (size_t)r * nc;
			double *out = N + (size_t)r * nc;
			const double f = row[k];
			auto entry = [&](int c) {
				const double p = pk[c], m = c == k ? 0.0 : row[c];
				return r == k ? p : f != 0.0 ? madd(-f, p, m) : m;
			};
			const bool next = r == k + 1;
			const double piv = next ? entry(r) : 1.0;
#pragma unroll 4
			for (int c = lane; c < nc; c += 32) {
				const double v = entry(c);
				out[c] = v;
				if (next)
					pn[c] = (c == r ? 1.0 : v) / piv;
			}
		}
		sy.sync();
		double *t = M;
		M = N;
		N = t;
		t = pk;
		pk = pn;
		pn = t;
	}
	for (int k = tid; k < nc * nc; k += nth)
		H.cinv[(size_t)(k % nc) * nc + k / nc] = (TI)M[k];   // by columns
	sy.sync();
}

// ---- FP64 residual and the preconditioner ------------------------------------------
// R = [C^T (F - K d - G p) ; G^T C d] (FP64); rs = |R_m|^2, |R_c|^2, |C^T F|^2.
template <class TI>
__device__ void qt_residual(QtSync &sy, const QtArgs<TI> &a, const double2 *d, const double *p, double (&rs)[3])
{
	const int tid = sy.id(), nth = sy.nth();
	const DevLevel &L = a.L;
	const QtLevel<TI> &Q = a.H.lv[a.H.nlev - 1];
	const double *df = reinterpret_cast<const double *>(d);
	const double *Ff = reinterpret_cast<const double *>(a.F);
	rs[0] = rs[1] = rs[2] = 0.0;
	for (int A = tid; A < L.nno; A += nth) {
		double k0, k1, g0, g1;
		qt_op_node(Q, Q.K64, df, A, k0, k1);
		qt_g_node(Q, L, a.ge, p, A, g0, g1);
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
		rs[0] = add2(rs[0], r.x, r.x, r.y, r.y);
		rs[2] = add2(rs[2], f[0], f[0], f[1], f[1]);
	}
	for (int e = tid; e < L.nel; e += nth) {
		const double c = qt_gt_elem(Q, L, a.ge, df, e);
		a.Rc[e] = c;
		rs[1] = madd(c, c, rs[1]);
	}
	sy.reduce<3>(rs);
}

// The scalars of the MINRES recurrences, formed by one thread of each block: a
// division or a square root on every thread costs the FP64 pipe about a
// microsecond each.
struct QtScal {
	double gam, gam_prev, eta, eta0, delta, c_prev, c_cur, s_prev, s_cur;
	double ig, dg, gg;               // of the Lanczos step: 1/gam, delta/gam, gam/gam_prev
	double wig, a2, a3, ia1, step;   // of the direction update: 1/gam, the rotations' entries, 1/a1, the solution's step
	double step1;                    // the step of the iteration before
	int stop;   // 1: last iteration; 2: breakdown before the update; 4: a non-finite value
};

// The vector updates of the MINRES iteration (inlined: as calls they left no
// registers to the loop's state, whose accesses on the stack miss L1 after every
// team barrier: 157 against 117 us per iteration).

// v_p(j+1) = A z - dg v_p(j) - gg v_p(j-1) into v_p(j-1)'s buffer and z_p = v_p / BAB
__device__ __forceinline__ void qt_v_elems(int ne, int tid, int nth, const double *Ahp, const double *p0, double *p1,
                                           const double *bab, double *z1, double ig, double dg, double gg)
{
	for (int e = tid; e < ne; e += nth) {
		const double vn = lin3(Ahp[e], ig, dg, p0[e], gg, p1[e]);
		p1[e] = vn;
		z1[e] = vn / bab[e];
	}
}

// w(j+1) = (z~(j) / gam - a3 w(j-1) - a2 w(j)) / a1 into w(j-1)'s buffer, and the steps
// of the solution: 0 none, 1 x += step w(j+1), 2 x += step1 w(j) + step w(j+1)
template <class V>
__device__ __forceinline__ void qt_w_update(int steps, int nn, int ne, int tid, int nth, const QtScal &ms, const V *z,
                                            double2 *wo, const double2 *wc, double2 *xu, const double *zp, double *po,
                                            const double *pc, double *xp)
{
	const double ig = ms.wig, a2 = ms.a2, a3 = ms.a3, ia1 = ms.ia1, s0 = ms.step, s1 = ms.step1;
	for (int A = tid; A < nn; A += nth) {
		const V zz = z[A];
		const double2 o = wo[A], w = wc[A];
		double2 x = make_double2(0.0, 0.0);
		if (steps > 0)
			x = xu[A];
		const double2 wn = make_double2(lin3(widen(zz.x), ig, a3, o.x, a2, w.x) * ia1,
		                                lin3(widen(zz.y), ig, a3, o.y, a2, w.y) * ia1);
		wo[A] = wn;
		if (steps > 1) {
			x.x = madd(s1, w.x, x.x);
			x.y = madd(s1, w.y, x.y);
		}
		if (steps > 0)
			xu[A] = make_double2(madd(s0, wn.x, x.x), madd(s0, wn.y, x.y));
	}
	for (int e = tid; e < ne; e += nth) {
		const double w = pc[e];
		double x = steps > 0 ? xp[e] : 0.0;
		const double wn = lin3(zp[e], ig, a3, po[e], a2, w) * ia1;
		po[e] = wn;
		if (steps > 1)
			x = madd(s1, w, x);
		if (steps > 0)
			xp[e] = madd(s0, wn, x);
	}
}

// Correction solve by preconditioned MINRES (Elman, Silvester and Wathen,
// "Finite Elements and Fast Iterative Solvers", Alg. 4.1) on the constrained
// system [C^T K C, C^T G; G^T C, 0][x_u; x_p] = [R_m; -R_c] from zero, with the
// preconditioner diag(V-cycle, BAB); K in TI, G and G^T in FP64, Lanczos and
// direction vectors FP64; x into a.dd, a.dpv, two iterations' steps at a time.
template <class TI>
__device__ __noinline__ int qt_minres(QtSync &team, const QtArgs<TI> &a, double rtol, int maxit)
{
	typedef typename Q2T<TI>::t V;
	__shared__ QtScal ms;
	QtSync sy = team;
	const DevLevel &L = a.L;
	const QtLevel<TI> &Q = a.H.lv[a.H.nlev - 1];
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
			const double v = -a.Rc[e];
			a.mvp[0][e] = v;
			a.mzp[0][e] = v / a.bab[e];
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
			const int tid = sy.id(), nth = sy.nth();
			double dl[1] = {0.0};
			{
				const V *z = a.mz[cv];
				const double *zp = a.mzp[cv];
				const TI *zf = reinterpret_cast<const TI *>(z);
				for (int A = tid; A < L.nno; A += nth) {
					TI k0, k1;
					double g0, g1;
					const V zz = z[A];
					qt_kr_node(Q, zf, A, k0, k1);
					qt_g_node(Q, L, a.ge, zp, A, g0, g1);
					const double2 az = make_double2(widen(k0) + g0, widen(k1) + g1);
					a.Kd[A] = az;
					dl[0] = add2(dl[0], az.x, widen(zz.x), az.y, widen(zz.y));
				}
				for (int e = tid; e < L.nel; e += nth) {
					const double t = qt_gt_elem(Q, L, a.ge, zf, e);
					a.Ahp[e] = t;
					dl[0] = madd(t, zp[e], dl[0]);
				}
			}
			sy.reduce_then<1>(dl, [&](const double (&v)[1]) {
				ms.delta = v[0] / (ms.gam * ms.gam);
				ms.dg = ms.delta / ms.gam;
			});
			// v(j+1) into v(j-1)'s buffer, its TI copy as the V-cycle's right-hand side,
			// and z_p(j+1) = v_p(j+1) / BAB
			const double ig = ms.ig, dg = ms.dg, gg = ms.gg;
			{
				const double2 *v = a.mv[cv];
				double2 *vo = a.mv[1 - cv];
				for (int A = tid; A < L.nno; A += nth) {
					const double2 az = a.Kd[A], vc = v[A], vp = vo[A];
					const double2 vn = make_double2(lin3(az.x, ig, dg, vc.x, gg, vp.x), lin3(az.y, ig, dg, vc.y, gg, vp.y));
					vo[A] = vn;
					V w;
					w.x = narrow_to<TI>(vn.x);
					w.y = narrow_to<TI>(vn.y);
					Q.b[A] = w;
				}
			}
			if (!defer)
				qt_v_elems(L.nel, tid, nth, a.Ahp, a.mvp[cv], a.mvp[1 - cv], a.bab, a.mzp[1 - cv], ig, dg, gg);
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
			qt_v_elems(L.nel, tid, nth, a.Ahp, a.mvp[cv], a.mvp[1 - cv], a.bab, a.mzp[1 - cv], ms.ig, ms.dg, ms.gg);
		});
		{
			const double *zp = a.mzp[1 - cv], *vp = a.mvp[1 - cv];
			const int nth = sy.nth();
			for (int e = sy.id(); e < L.nel; e += nth)
				dot[0] = madd(zp[e], vp[e], dot[0]);
		}
		sy.reduce_then<1>(dot, [&](const double (&v)[1]) {
			const double gam_next = sqrt(fmax(v[0], 0.0));
			if (it < 0) {
				ms.gam = gam_next;
				ms.gam_prev = 1.0;
				ms.eta = ms.eta0 = gam_next;
				ms.c_prev = ms.c_cur = 1.0;
				ms.s_prev = ms.s_cur = 0.0;
				ms.ig = 1.0 / gam_next;
				ms.gg = gam_next;   // (gam_prev = 1)
				ms.stop = v[0] > 0.0 ? 0 : 3;
				return;
			}
			const double cs = __dmul_rn(ms.c_prev, ms.s_cur), cc = __dmul_rn(ms.c_prev, ms.c_cur);
			const double a0 = __fma_rn(ms.c_cur, ms.delta, -__dmul_rn(cs, ms.gam));
			const double a1 = sqrt(__fma_rn(a0, a0, __dmul_rn(gam_next, gam_next)));
			const double a2 = __fma_rn(cc, ms.gam, __dmul_rn(ms.s_cur, ms.delta));
			const double a3 = ms.s_prev * ms.gam;
			ms.stop = 0;
			if (!(a1 > 0.0) || !isfinite(a1)) {
				ms.stop = isfinite(a1) ? 2 : 6;
				return;
			}
			const double c_next = a0 / a1, s_next = gam_next / a1;
			ms.step1 = ms.step;
			ms.wig = ms.ig;
			ms.a2 = a2;
			ms.a3 = a3;
			ms.ia1 = 1.0 / a1;
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
					a.dd[A] = make_double2(madd(s, w.x, x.x), madd(s, w.y, x.y));
				}
				for (int e = tid; e < L.nel; e += nth)
					a.dpv[e] = madd(s, a.mwp[cw][e], a.dpv[e]);
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
__device__ void qt_solve(const QtArgs<TI> &a, QtSync &sy)
{
	const int tid = sy.tid(), nth = sy.nth();
	const QtHier<TI> &H = a.H;
	const DevLevel &L = a.L;
	int *status = &a.sc->status;

	for (int e = tid; e < L.nel; e += nth)
		qt_g_table(L, e, a.ge);
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
__global__ void __launch_bounds__(kTeamThreads, 1) k_stokes_qt(const __grid_constant__ QtArgs<TI> a)
{
	__shared__ QtArgs<TI> sa;
	load_args(sa, a);
	__shared__ double cpart[2 * kQtPartials];
	QtSync sy = sa.cluster ? QtSync::of(SYNC_CLUSTER, cpart, blockIdx.x, gridDim.x, true)
	                       : QtSync::of(SYNC_GRID, sa.red.part, blockIdx.x, gridDim.x, true);
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
__global__ void __launch_bounds__(kBlock, 2) k_stokes_qt_batch(const QtArgs<TI> *models, int nmodels, int *queue)
{
	__shared__ QtArgs<TI> sa;
	__shared__ int next;
	__shared__ double cpart[2 * kQtPartials];
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
			QtSync sy = QtSync::of(SYNC_CLUSTER, cpart, rank, cs, false);
			qt_solve<TI>(sa, sy);
			cl.sync();   // no block starts the next model (or leaves) while another reads its partials
		} else {
			__syncthreads();
			const int m = next;
			__syncthreads();
			if (m >= nmodels)
				break;
			load_args(sa, models[m]);
			QtSync sy = QtSync::of(SYNC_BLOCK, nullptr, 0, 1, false);
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
