// Matrix-free Q1 viscous operator on a uniform level, one warp per task
// (included by k_mg.cu inside namespace mclg).
//
// A task is a strip of 30 nodes along z (the contiguous direction of the node
// numbering A = iz + ix*n) by a few columns along x.  A warp holds 32 nodes of
// a column, one per lane (the 30 owned ones and one halo node at each end; 16 in
// a paired task, see Split), and walks along x: at each column every lane forms its element's corner
// forces from its own and its upper neighbour's nodal values (shuffles), adds
// them to the two columns' accumulators, and finishes the left column's rows.
// No shared memory, no block barrier, no atomics; every sum has a fixed order.
//
// The element forces use the tensor structure of the 2 x 2 Gauss points: du/dx
// depends only on the point's z index and du/dz only on its x index, so two
// values of each derivative serve the four points, and the stresses are summed
// over one index before the other is applied.  About 85 multiply-adds per
// element and 8 additions per node; with D = diag(2 eta, 2 eta, eta) and
// unit-Jacobian derivatives it is the element matrix of get_element_K
// (Build_matrix.c:192-271).
//
// Bound and choice: a tile of 16 x 32 nodes staged in shared memory, with 12
// stresses per element stored and gathered, took three block barriers and about
// 75 shared-memory accesses and 800 instructions for two nodes; one pass at
// 1024^2 took 47 us and one at 16^2 .. 64^2 6 .. 8 us, of which a grid barrier
// is 1.2.  The column walk issues about 120 instructions per column of 30 nodes.
#pragma once

constexpr int kOwn = 30;       // nodes of a strip that the warp owns (lanes 1..30)
constexpr int kOwnPair = 14;   // ... of a paired task (lanes 17..30)

// How a level's strips and columns are cut into tasks for a number of warps;
// formed once per solve (the divisions took a tenth of a small level's pass).
//
// Where every node column of 14-node strips has a warp of its own, tasks are
// paired: the half-warps form the element columns left and right of one node
// column at the same time and the left one's forces are handed over by shuffles,
// in place of two steps one after the other (the same sums).  Such a level's pass
// is a chain of dependent operations, not throughput: per iteration 129 against
// 169 us at 128^2 in FP64, 34.3 against 37.1 at 64^2, 70.8 against 75.0 at 256^2
// and 248 against 255 at 1024^2 in FP32.  With two paired tasks a warp the work
// counts again (137, 36.7, 70.9 and 247 us), with four it loses everywhere.
struct Split {
	int strips, Lx, ntasks, pair;
	float inv;   // 1/strips: t/strips for t < 2^22 as the truncated product with (t + 1/2)
	__device__ void set(int n, int nwarps)
	{
		strips = (n + kOwnPair - 1) / kOwnPair;
		pair = strips * n <= nwarps;
		if (!pair)
			strips = (n + kOwn - 1) / kOwn;
		int chunks = nwarps / strips;   // the columns are cut into as many chunks as there are warps for them
		chunks = chunks < 1 ? 1 : chunks > n ? n : chunks;   // (n: one column a task, when paired)
		Lx = (n + chunks - 1) / chunks;
		ntasks = strips * ((n + Lx - 1) / Lx);
		inv = 1.0f / (float)strips;
	}
};

enum {
	PASS_MATVEC = 0,   // out = A x; *dot = this thread's share of x.(A x) (with xout, x as formed is
	                   // stored there)
	PASS_RESID = 1,    // out = b - A x (with xout, x as formed is stored there)
	PASS_SMOOTH = 2,   // out = cx x - c0 x0 + omega D^-1 (b - A x) (cx = 1, no x0: damped
	                   // Jacobi; the Chebyshev recurrence otherwise; with xout, x as formed is
	                   // stored there; *dot = this thread's share of out.dotv, or of out.b
	                   // with dotb)
	PASS_STOKES = 3,   // out64 = A x + G gp, gt_out = G^T x per element (x-major);
	                   // *dot = this thread's share of x.out64 + gp.gt_out
	PASS_RES64 = 4     // out64 = F - A x - G gp, gt_out = G^T x; dot[0..2] = this thread's
	                   // shares of |out64|^2, |gt_out|^2, |F|^2
};

// How a pass forms its input x at a node:
//   XS_PLAIN    x
//   XS_ZERO     wload D^-1 b         (the first sweep from a zero guess)
//   XS_PROLONG  x + P xc             (coarse-grid correction, bilinear P)
//   XS_ZERO_R   wload D^-1 b with b = P^T r_f formed from the finer level's
//               residual (xc = r_f, nc = its nodes per side); the pass also
//               writes b for its own nodes (bout), for the level's later passes
//   XS_AXPY     x + wload xc         (CG's direction; xc is not read into it when wload is 0)
// Forming them where the pass reads them saves a barrier and a pass over memory
// on every multigrid level.
enum { XS_PLAIN = 0, XS_ZERO = 1, XS_PROLONG = 2, XS_ZERO_R = 3, XS_AXPY = 4 };

template <class T>
struct Pass {
	typedef typename V2T<T>::t V;
	int N;                       // elements per side
	const unsigned char *mask;
	const T *eta;
	const V *x, *b, *invD, *xc, *x0;
	V *out, *xout, *bout;
	int nc;
	T omega, wload, cx, c0;
	const double2 *dotv;
	bool dotb;
	// PASS_STOKES, PASS_RES64
	const double *gp;
	double2 *out64;
	double *gt_out;
	const double2 *F;
	double g0, g1;               // G of an element's first corner (hz, hx); the others by sign
	int gp_morton;               // gp in Morton order (else x-major, e = ez + ex*N)
};

// What a lane holds of one column: x as the pass forms it (0 at Dirichlet
// dofs), viscosity, mask, the epilogue's operands, and (c) the coarse or fine
// values that x is formed from.
template <class T, class V, int NC>
struct Column {
	V x, b, d, x0, c[NC];
	T e;
	unsigned m;
};

template <class T, int MODE, int XS, bool X0>
__device__ __forceinline__ void march(const Pass<T> &P, Part pt, const Split &sp, double *dot)
{
	typedef typename V2T<T>::t V;
	constexpr int NC = XS == XS_ZERO_R ? 9 : XS == XS_PROLONG ? 4 : 1;
	typedef Column<T, V, NC> Col;
	constexpr unsigned kAll = 0xffffffffu;
	constexpr bool kStokes = MODE == PASS_STOKES || MODE == PASS_RES64;
	constexpr bool kNeedB = MODE == PASS_RESID || MODE == PASS_SMOOTH;
	const OpTab<T> &O = tab<T>();
	const T axp = O.axp, axm = O.axm, azp = O.azp, azm = O.azm, ip = O.p, iq = O.q;
	const int N = P.N, n = N + 1;
	const int lane = threadIdx.x & 31;
	const int nwarps = pt.size * (int)(blockDim.x >> 5);
	const int strips = sp.strips, Lx = sp.Lx, ntasks = sp.ntasks;
	const float inv = sp.inv;
	const bool pair = sp.pair != 0;
	const int zlane = pair ? lane & 15 : lane, zlast = pair ? 15 : 31, half = pair ? lane >> 4 : 0;
	double dacc = 0.0, racc = 0.0, facc = 0.0;

	// consecutive tasks go to different blocks, so that a small level uses many SMs
	for (int t = (threadIdx.x >> 5) * pt.size + pt.rank; t < ntasks; t += nwarps) {
		const int c = (int)(((float)t + 0.5f) * inv), s = t - c * strips;
		const int gz = s * (zlast - 1) - 1 + zlane, xs = c * Lx, xe = pair ? xs + half : min(xs + Lx, n);
		const bool zin = gz >= 0 && gz < n;
		const bool own = zin && zlane >= 1 && zlane < zlast;
		const bool ein = gz >= 0 && gz < N && zlane < zlast;   // this lane's element lies in the box
		const T pl = ein ? ip : T(0), ql = ein ? iq : T(0);
		const int gzc = min(max(gz, 0), n - 1);

		// The loads of column ix, and the operands its rows need later.  No branch:
		// outside the box a lane loads the nearest node and form() takes its value
		// out, so that the loads of several columns are in flight together.
		auto load = [&](int ix, Col &k) {
			const int ixc = min(max(ix, 0), n - 1);
			const int A = gzc + ixc * n;
			k.m = P.mask[A];
			k.e = P.eta[A];
			if (XS == XS_PLAIN || XS == XS_PROLONG || XS == XS_AXPY)
				k.x = P.x[A];
			if (XS == XS_AXPY)
				k.c[0] = P.xc[A];
			if (XS == XS_ZERO || (kNeedB && XS != XS_ZERO_R))
				k.b = P.b[A];
			if (XS == XS_ZERO || XS == XS_ZERO_R || MODE == PASS_SMOOTH)
				k.d = P.invD[A];
			if (X0)
				k.x0 = P.x0[A];
			if (XS == XS_PROLONG) {
				const int a0 = (gzc >> 1) + (ixc >> 1) * P.nc, up = gzc & 1, rt = (ixc & 1) * P.nc;
				k.c[0] = P.xc[a0];
				k.c[1] = P.xc[a0 + up];
				k.c[2] = P.xc[a0 + rt];
				k.c[3] = P.xc[a0 + rt + up];
			}
			if (XS == XS_ZERO_R) {
				// P^T r_f over the 3 x 3 fine nodes around (2 ix, 2 gz); those outside
				// the box are read at the box's edge and weighted 0
				const int nf = P.nc;
#pragma unroll
				for (int q = 0; q < 9; q++) {
					const int fx = min(max(2 * ixc + q / 3 - 1, 0), nf - 1), fz = min(max(2 * gzc + q % 3 - 1, 0), nf - 1);
					k.c[q % NC] = P.xc[fz + fx * nf];
				}
			}
		};
		auto form = [&](int ix, Col &k) {
			const bool in = zin && ix >= 0 && ix < n;
			if (!in) {
				k.m = 3u;
				k.e = T(0);
			}
			if (XS == XS_ZERO_R) {
				const T wl = ix > 0 ? T(0.5) : T(0), wr = ix < n - 1 ? T(0.5) : T(0);
				const T wd = gz > 0 ? T(0.5) : T(0), wu = gz < n - 1 ? T(0.5) : T(0);
				const V *c = k.c;
				k.b.x = (wl * (wd * c[0 % NC].x + c[1 % NC].x + wu * c[2 % NC].x) + (wd * c[3 % NC].x + c[4 % NC].x + wu * c[5 % NC].x)) +
				        wr * (wd * c[6 % NC].x + c[7 % NC].x + wu * c[8 % NC].x);
				k.b.y = (wl * (wd * c[0 % NC].y + c[1 % NC].y + wu * c[2 % NC].y) + (wd * c[3 % NC].y + c[4 % NC].y + wu * c[5 % NC].y)) +
				        wr * (wd * c[6 % NC].y + c[7 % NC].y + wu * c[8 % NC].y);
				k.b.x = (k.m & 1u) ? T(0) : k.b.x;
				k.b.y = (k.m & 2u) ? T(0) : k.b.y;
			}
			if (XS == XS_ZERO || XS == XS_ZERO_R) {
				k.x.x = P.wload * k.d.x * k.b.x;
				k.x.y = P.wload * k.d.y * k.b.y;
			}
			if (XS == XS_AXPY && P.wload != T(0)) {
				k.x.x += P.wload * k.c[0].x;
				k.x.y += P.wload * k.c[0].y;
			}
			if (XS == XS_PROLONG) {
				k.x.x += T(0.25) * ((k.c[0].x + k.c[1 % NC].x) + (k.c[2 % NC].x + k.c[3 % NC].x));
				k.x.y += T(0.25) * ((k.c[0].y + k.c[1 % NC].y) + (k.c[2 % NC].y + k.c[3 % NC].y));
			}
			k.x.x = (k.m & 1u) ? T(0) : k.x.x;
			k.x.y = (k.m & 2u) ? T(0) : k.x.y;
		};

		Col cur, nx, prev;
		load(xs - 1 + half, prev);   // the first columns are in flight together
		load(xs + half, cur);
		load(xs + 1 + half, nx);
		form(xs - 1 + half, prev);
		// left edge of the element column: this lane's and the upper neighbour's
		// values, the viscosity at the edge's two Gauss points
		T u0n = __shfl_down_sync(kAll, prev.x.x, 1), w0n = __shfl_down_sync(kAll, prev.x.y, 1);
		T en = __shfl_down_sync(kAll, prev.e, 1);
		T eL0 = pl * prev.e + ql * en, eL1 = ql * prev.e + pl * en;
		T E0u = u0n - prev.x.x, E0w = w0n - prev.x.y;
		T lou = T(0), low = T(0), upu = T(0), upw = T(0);
		double cL = 0.0, dL = 0.0;

#pragma unroll 1
		for (int ix = xs + half;;) {
			const int ex = ix - 1;
			const bool exin = ex >= 0 && ex < N;
			double pe = 0.0;
			if (kStokes && exin && ein)
				pe = P.gp[P.gp_morton ? morton(ex, gz) : gz + ex * N];
			// operands of the left column's rows that are not needed before
			double2 dv = make_double2(0.0, 0.0);
			const bool row = own && ex >= xs;
			const int A = gz + ex * n;
			if (row && MODE == PASS_SMOOTH && P.dotv)
				dv = P.dotv[A];
			if (row && MODE == PASS_RES64)
				dv = P.F[A];
			form(ix, cur);
			const T u0 = prev.x.x, w0 = prev.x.y, u1 = cur.x.x, w1 = cur.x.y;
			const T u1n = __shfl_down_sync(kAll, u1, 1), w1n = __shfl_down_sync(kAll, w1, 1);
			const T e1n = __shfl_down_sync(kAll, cur.e, 1);
			const T eR0 = pl * cur.e + ql * e1n, eR1 = ql * cur.e + pl * e1n;
			const T E1u = u1n - u1, E1w = w1n - w1;
			T f0u = T(0), f0w = T(0), f1u = T(0), f1w = T(0), f2u = T(0), f2w = T(0), f3u = T(0), f3w = T(0);
			if (exin) {
				// viscosity at the Gauss points (i along x, j along z)
				const T e00 = ip * eL0 + iq * eR0, e10 = iq * eL0 + ip * eR0;
				const T e01 = ip * eL1 + iq * eR1, e11 = iq * eL1 + ip * eR1;
				const T D0u = u1 - u0, D1u = u1n - u0n, D0w = w1 - w0, D1w = w1n - w0n;
				const T ux0 = axp * D0u + axm * D1u, ux1 = axm * D0u + axp * D1u;
				const T wx0 = axp * D0w + axm * D1w, wx1 = axm * D0w + axp * D1w;
				const T uz0 = azp * E0u + azm * E1u, uz1 = azm * E0u + azp * E1u;
				const T wz0 = azp * E0w + azm * E1w, wz1 = azm * E0w + azp * E1w;
				const T X0_ = T(2) * ux0 * (eL0 + eR0), X1_ = T(2) * ux1 * (eL1 + eR1);
				const T Z0_ = T(2) * wz0 * (e00 + e01), Z1_ = T(2) * wz1 * (e10 + e11);
				const T s00 = e00 * (uz0 + wx0), s01 = e01 * (uz0 + wx1);
				const T s10 = e10 * (uz1 + wx0), s11 = e11 * (uz1 + wx1);
				const T S0 = s00 + s01, S1 = s10 + s11, T0 = s00 + s10, T1 = s01 + s11;
				const T Pm = axp * X0_ + axm * X1_, Pp = axm * X0_ + axp * X1_;
				const T Qm = azp * S0 + azm * S1, Qp = azm * S0 + azp * S1;
				const T Rm = azp * Z0_ + azm * Z1_, Rp = azm * Z0_ + azp * Z1_;
				const T Hm = axp * T0 + axm * T1, Hp = axm * T0 + axp * T1;
				f0u = -(Pm + Qm);
				f1u = Qm - Pp;
				f2u = Pp + Qp;
				f3u = Pm - Qp;
				f0w = -(Rm + Hm);
				f1w = Rm - Hp;
				f2w = Rp + Hp;
				f3w = Hm - Rp;
			}
			if (pair) {   // the left element column's forces on the node column, from the other half
				lou = __shfl_xor_sync(kAll, f3u, 16);
				low = __shfl_xor_sync(kAll, f3w, 16);
				upu = __shfl_xor_sync(kAll, f2u, 16);
				upw = __shfl_xor_sync(kAll, f2w, 16);
			}
			// the left column's rows: lower corner of this element, upper corner of the one below
			const T su = upu + f1u, sw = upw + f1w;
			const T fu_ = (lou + f0u) + __shfl_up_sync(kAll, su, 1), fw_ = (low + f0w) + __shfl_up_sync(kAll, sw, 1);
			lou = f3u;
			low = f3w;
			upu = f2u;
			upw = f2w;
			double c1 = 0.0, d1 = 0.0, s0 = 0.0, s1 = 0.0;
			if (kStokes) {
				// G gp: the difference of the right and left element pairs' sums, and of
				// the upper and lower pairs'
				const double pd = __shfl_up_sync(kAll, pe, 1);
				c1 = pe + pd;
				d1 = pe - pd;
				if (pair) {
					cL = __shfl_xor_sync(kAll, c1, 16);
					dL = __shfl_xor_sync(kAll, d1, 16);
				}
				s0 = c1 - cL;
				s1 = d1 + dL;
				cL = c1;
				dL = d1;
				if (row && exin && ein) {
					const double g = gt_elem(u0, u0n, u1n, u1, w0, w0n, w1n, w1, P.g0, P.g1);
					P.gt_out[gz + ex * N] = g;
					if (MODE == PASS_STOKES)
						dacc += g * pe;
					else
						racc += g * g;
				}
			}
			if (row) {
				const unsigned m = prev.m;
				const T fu = (m & 1u) ? T(0) : fu_, fw = (m & 2u) ? T(0) : fw_;
				if (kStokes) {
					double ax = (m & 1u) ? 0.0 : P.g0 * s0 + widen(fu), ay = (m & 2u) ? 0.0 : P.g1 * s1 + widen(fw);
					if (MODE == PASS_STOKES) {
						dacc += ax * widen(u0) + ay * widen(w0);
					} else {
						ax = dv.x - ax;
						ay = dv.y - ay;
						dacc += ax * ax + ay * ay;
						facc += dv.x * dv.x + dv.y * dv.y;
					}
					P.out64[A] = make_double2(ax, ay);
				} else {
					V o;
					if (MODE == PASS_MATVEC) {
						o.x = fu;
						o.y = fw;
						dacc += widen(u0) * widen(fu) + widen(w0) * widen(fw);
					} else if (MODE == PASS_RESID) {
						o.x = (m & 1u) ? T(0) : prev.b.x - fu;
						o.y = (m & 2u) ? T(0) : prev.b.y - fw;
					} else {
						T px = P.cx * u0, py = P.cx * w0;
						if (X0) {
							px -= P.c0 * prev.x0.x;
							py -= P.c0 * prev.x0.y;
						}
						o.x = (m & 1u) ? T(0) : px + P.omega * prev.d.x * (prev.b.x - fu);
						o.y = (m & 2u) ? T(0) : py + P.omega * prev.d.y * (prev.b.y - fw);
						if (P.dotv)
							dacc += widen(o.x) * dv.x + widen(o.y) * dv.y;
						else if (P.dotb)
							dacc += widen(o.x) * widen(prev.b.x) + widen(o.y) * widen(prev.b.y);
					}
					P.out[A] = o;
					if (P.xout)
						P.xout[A] = prev.x;
					if (XS == XS_ZERO_R)
						P.bout[A] = prev.b;
				}
			}
			if (++ix > xe)
				break;
			prev = cur;
			u0n = u1n;
			w0n = w1n;
			E0u = E1u;
			E0w = E1w;
			eL0 = eR0;
			eL1 = eR1;
			cur = nx;
			load(ix + 1, nx);
		}
	}
	if (dot) {
		dot[0] = dacc;
		if (MODE == PASS_RES64) {
			dot[1] = racc;
			dot[2] = facc;
		}
	}
}
