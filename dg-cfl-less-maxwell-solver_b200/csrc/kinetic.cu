// HP-2: the CFL-less kinetic-relaxation step (src/dg/relaxation.c:93-174).
//
// The reference, per step: boundary dofs <- f_eq(w_I(x, t + dt/2));
// for every field iw and velocity iv: sol = M2_iv wn; solve M1_iv sol (KLU);
// swap; relax every dof: f <- omega f_eq(w(f)) + (1 - omega) f.
// With M1 = I + theta dt A and M2 = I - (1 - theta) dt A (relaxation.c:79-83),
// M2 = (1/theta) I - ((1 - theta)/theta) M1, hence
//   M1^-1 M2 f = (1/theta) y - ((1 - theta)/theta) f,   y = M1^-1 f,
// so one block forward substitution per velocity replaces the SpMV + LU
// solve.  M1 is block lower-triangular in a downwind element order (an element
// row couples only to its upwind neighbours, simulation.c:493-604); the host
// builds the level schedule of that order once per velocity and the sweep
// runs level by level, all velocities and all 6 fields of a level in one
// launch.  Per element and velocity the diagonal block is
//   D = I + (theta dt / det) Minv (V + sum_outflow s+ E_f S E_f^T),
//   V_ij = -(v . c_ij), s = v . vn (the L-side scaled normal of each face),
// inverted once at attach in FP64 (G = D^-1); a sweep item computes
//   y_e = G (f_e - (theta dt / det) Minv sum_inflow s- E_f S y_nb|_f).
//
// Sweep order: the state of (element e, velocity v) lives at item index
// k = pos[e * nv + v], its position in the level-sorted item list, so the
// items of one level are contiguous in memory and an item finds everything
// it needs in its records (inflow neighbour items, permutations, v . vn,
// theta dt / det).
//
// Mixed precision (GDN_CUDA_FP32_REFINE): FP64 state, FP32 sweeps, FP64
// residual r = f - b - M1 y computed matrix-free from the FP64 geometry, then
// FP32 correction sweeps M1 d = r with zero boundary data, y += d.
#include <climits>
#include <type_traits>

#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>
#include <cuda_pipeline_primitives.h>

#include "aux.h"
#include "kernels.h"

namespace gdn {

// own-side v.vn of every element face for every velocity, from the L-side
// normal of each face in the reference's operation order (simulation.c:
// 520-540 + kinetic_num_flux_upwind): the R side gets exactly -s.
__global__ void kin_face_s_kernel(const int *__restrict__ face2elem, long long nf, const double *__restrict__ geom,
								  KinModel km, double *__restrict__ sown64)
{
	const long long F = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (F >= nf)
		return;
	const long long eL = face2elem[4 * F], eR = face2elem[4 * F + 2];
	const int fL = face2elem[4 * F + 1], fR = face2elem[4 * F + 3];
	double cod[3][3], vn[3];
	for (int a = 0; a < 3; a++)
		for (int b = 0; b < 3; b++)
			cod[a][b] = geom[eL * 10 + 3 * a + b];
	gdn_face_normal(cod, c_tab_d.ref_normal, fL, vn);
	for (int v = 0; v < km.nv; v++) {
		const double s = gdn_dot_lr(km.vi + 3 * v, vn);
		sown64[(eL * km.nv + v) * 4 + fL] = s;
		if (eR >= 0)
			sown64[(eR * km.nv + v) * 4 + fR] = -s;
	}
}

// inflow mask: bit f set when element e depends on its neighbour across f
__global__ void kin_mask_kernel(const double *__restrict__ sown64, const int *__restrict__ nb, long long ne, int nv,
								unsigned char *__restrict__ mask)
{
	const long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (u >= ne * nv)
		return;
	const long long e = u / nv;
	unsigned char m = 0;
	for (int f = 0; f < 4; f++)
		if (nb[e * 4 + f] >= 0 && sown64[u * 4 + f] < 0.0)
			m |= (unsigned char)(1 << f);
	mask[u] = m;
}

__global__ void kin_iota_kernel(int *a, long long n)
{
	const long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (u < n)
		a[u] = (int)u;
}

// after the sort: pos = inverse of items, level_off[l] = first item of level l
__global__ void kin_schedule_finish_kernel(const int *__restrict__ items, const int *__restrict__ lev_sorted,
										   long long n, int *__restrict__ pos, int *__restrict__ level_off)
{
	const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (k >= n)
		return;
	pos[items[k]] = (int)k;
	const int l = lev_sorted[k];
	if (k == 0 || lev_sorted[k - 1] != l)
		level_off[l] = (int)k;
	if (k == n - 1)
		level_off[l + 1] = (int)n;
}

static int launch_kin_kahn(const unsigned char *mask, const int *nb, const double *sown64, long long ne, int nv,
						   int *indeg, int *level, int *front0, int *front1, unsigned *ctl, long long spin_limit,
						   cudaStream_t s);

int kin_device_schedule(const unsigned char *mask, const int *nb, const double *sown64, long long ne, int nv,
						int *items, int *pos, std::vector<int> &level_off, long long spin_limit, cudaStream_t s)
{
	const long long nu = ne * nv;
	const unsigned g = (unsigned)((nu + 255) / 256);
	int *level = nullptr, *lev_sorted = nullptr, *iota = nullptr, *indeg = nullptr, *loff = nullptr;
	unsigned *ctl = nullptr;
	void *tmp = nullptr;
	size_t tmp_bytes = 0;
	int rc = GDN_CUDA_OK;
	int maxlev = 0;
	auto cleanup = [&]() {
		dev_free(level, s);
		dev_free(lev_sorted, s);
		dev_free(iota, s);
		dev_free(indeg, s);
		dev_free(ctl, s);
		dev_free(loff, s);
		dev_free(tmp, s);
	};
#define GDN_SCHED_TRY(expr)                                                                                           \
	do {                                                                                                           \
		cudaError_t _e = (expr);                                                                                   \
		if (_e != cudaSuccess) {                                                                                   \
			cleanup();                                                                                             \
			return gdn_cuda_fail(_e, #expr, __FILE__, __LINE__);                                                  \
		}                                                                                                          \
	} while (0)
	GDN_SCHED_TRY(dev_alloc(reinterpret_cast<void **>(&level), nu * sizeof(int), s));
	GDN_SCHED_TRY(dev_alloc(reinterpret_cast<void **>(&lev_sorted), nu * sizeof(int), s));
	GDN_SCHED_TRY(dev_alloc(reinterpret_cast<void **>(&iota), nu * sizeof(int), s));
	GDN_SCHED_TRY(dev_alloc(reinterpret_cast<void **>(&indeg), nu * sizeof(int), s));
	GDN_SCHED_TRY(dev_alloc(reinterpret_cast<void **>(&ctl), 8 * sizeof(unsigned), s));
	GDN_SCHED_TRY(cudaMemsetAsync(ctl, 0, 8 * sizeof(unsigned), s));
	// levels: Kahn's algorithm, the two frontiers in the sort buffers
	{
		const int lrc = launch_kin_kahn(mask, nb, sown64, ne, nv, indeg, level, lev_sorted, iota, ctl, spin_limit, s);
		if (lrc != GDN_CUDA_OK) {
			cleanup();
			return lrc;
		}
		unsigned hctl[8];
		GDN_SCHED_TRY(cudaMemcpyAsync(hctl, ctl, sizeof(hctl), cudaMemcpyDeviceToHost, s));
		GDN_SCHED_TRY(cudaStreamSynchronize(s));
		if (hctl[4]) {
			cleanup();
			return gdn_set_error(GDN_CUDA_ERR_TIMEOUT, "attach: the level schedule's grid barrier timed out");
		}
		if ((long long)hctl[6] != nu) {
			cleanup();
			return gdn_set_error(GDN_CUDA_ERR_CYCLE, "attach: the upwind element graph has a cycle");
		}
	}
	kin_iota_kernel<<<g, 256, 0, s>>>(iota, nu);
	GDN_SCHED_TRY(cudaGetLastError());
	// stable sort of the items by level: within a level the item order is
	// ascending e * nv + v, as the host schedule had it
	int bits = 1;
	{
		int *dmax = reinterpret_cast<int *>(ctl + 7);
		GDN_SCHED_TRY(cub::DeviceReduce::Max(nullptr, tmp_bytes, level, dmax, (int)nu, s));
		GDN_SCHED_TRY(dev_alloc(reinterpret_cast<void **>(&tmp), tmp_bytes, s));
		GDN_SCHED_TRY(cub::DeviceReduce::Max(tmp, tmp_bytes, level, dmax, (int)nu, s));
		GDN_SCHED_TRY(cudaMemcpyAsync(&maxlev, dmax, sizeof(int), cudaMemcpyDeviceToHost, s));
		GDN_SCHED_TRY(cudaStreamSynchronize(s));
		dev_free(tmp, s);
		tmp = nullptr;
		while ((1 << bits) <= maxlev)
			bits++;
	}
	GDN_SCHED_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, level, lev_sorted, iota, items, (int)nu, 0,
												  bits, s));
	GDN_SCHED_TRY(dev_alloc(reinterpret_cast<void **>(&tmp), tmp_bytes, s));
	GDN_SCHED_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, level, lev_sorted, iota, items, (int)nu, 0, bits,
												  s));
	GDN_SCHED_TRY(dev_alloc(reinterpret_cast<void **>(&loff), (maxlev + 2) * sizeof(int), s));
	kin_schedule_finish_kernel<<<g, 256, 0, s>>>(items, lev_sorted, nu, pos, loff);
	GDN_SCHED_TRY(cudaGetLastError());
	level_off.assign(maxlev + 2, 0);
	GDN_SCHED_TRY(cudaMemcpyAsync(level_off.data(), loff, (maxlev + 2) * sizeof(int), cudaMemcpyDeviceToHost, s));
	GDN_SCHED_TRY(cudaStreamSynchronize(s));
#undef GDN_SCHED_TRY
	cleanup();
	return rc;
}

// Tables of the block setup, FP64, filled at attach (kin_upload_block_tables):
// MD[d][r][j] = (Minv D_d)[r][j] and MS[f][r][jj] = sum_ii Minv[r][f2n(f, ii)]
// S[ii][jj], so that row r of Minv F is formed from its own row of each.
__constant__ double c_kin_md[3][10][10];
__constant__ double c_kin_ms[4][10][6];

int kin_upload_block_tables(const gdn_cuda_tables *t)
{
	double md[3][10][10], ms[4][10][6];
	for (int d = 0; d < 3; d++)
		for (int r = 0; r < 10; r++)
			for (int j = 0; j < 10; j++) {
				double acc = 0.0;
				for (int k = 0; k < 10; k++)
					acc += t->inv_mass[r][k] * t->internal[k][j][d];
				md[d][r][j] = acc;
			}
	for (int f = 0; f < 4; f++)
		for (int r = 0; r < 10; r++)
			for (int jj = 0; jj < 6; jj++) {
				double acc = 0.0;
				for (int ii = 0; ii < 6; ii++)
					acc += t->inv_mass[r][f2n(f, ii)] * t->face_scal[ii][jj];
				ms[f][r][jj] = acc;
			}
	GDN_CUDA_TRY(cudaMemcpyToSymbol(c_kin_md, md, sizeof(md)));
	GDN_CUDA_TRY(cudaMemcpyToSymbol(c_kin_ms, ms, sizeof(ms)));
	return GDN_CUDA_OK;
}

// G = D^-1 per (element, velocity), FP64 Gauss-Jordan with partial pivoting
// on [D | I], written at the item's sweep position with theta dt / det.
// D = I + c Minv F with F = V + sum_outflow s+ E_f S E_f^T, V_ij = -(v . c_ij),
// row r of Minv F formed directly from the precomputed rows of Minv D_d and
// Minv E_f S.  Ten lanes per item, three items per warp (lanes 30 and 31 idle),
// lane r holding row r of [D | I] in registers (no local memory).
// - Pivot of column k: the largest |a| among the rows not yet used, ties to the
//   smallest position.  A shuffle tree over the item's lanes takes the maximum
//   of |a| as a 64-bit pattern (non-negative doubles order as their bits; +1
//   keeps every candidate above the rows already used); a ballot names the
//   lanes that hold it, and only when two do (anywhere in the warp) a second
//   tree takes the smallest position among them.
// - The normalised pivot row is broadcast through shared memory, and every
//   other row eliminates column k.
// - Rows are not moved: each lane keeps the position its row would have in the
//   row-swapping algorithm, so the pivots are those of the textbook version.
// - Columns left of the pivot are not updated: they no longer feed a pivot or
//   the inverse.
// - The right half is kept in pivot order: slot t holds the column of the row
//   that was the pivot at step t.  Before step k only slots 0..k-1 can differ
//   from the identity (a column of I stays a unit column until its row is a
//   pivot), so step k updates 9 - k left columns and k + 1 slots, and every
//   value equals the one the full [D | I] elimination computes.  The slots go
//   back to their columns when G is written.
constexpr int kBlkThreads = 256;			  // 8 warps, 24 items per CTA
constexpr int kBlkItems = kBlkThreads / 32 * 3;
template <typename GT>
__global__ void __launch_bounds__(kBlkThreads, 4)
	kin_blocks_kernel(const double *__restrict__ geom, const double *__restrict__ sown64,
					  const int *__restrict__ pos, long long ne, KinModel km, double theta,
					  const int *__restrict__ einst, const double *__restrict__ dt_tab, GT *__restrict__ G,
					  GT *__restrict__ rcoef, double4 *__restrict__ ru64, double4 *__restrict__ rs64,
					  int *__restrict__ bad)
{
	__shared__ double sMD[3][10][10], sMS[4][10][6];
	__shared__ __align__(16) double sPiv[kBlkItems][20]; // pivot row of each item
	for (int q = threadIdx.x; q < 300; q += blockDim.x)
		(&sMD[0][0][0])[q] = (&c_kin_md[0][0][0])[q];
	for (int q = threadIdx.x; q < 240; q += blockDim.x)
		(&sMS[0][0][0])[q] = (&c_kin_ms[0][0][0])[q];
	__syncthreads();
	const int lane = threadIdx.x & 31, slot = lane / 10; // slot 3: the two idle lanes
	const bool row = slot < 3;
	const int base = 10 * slot, r = lane - base, seg = row ? 10 : 2;
	const unsigned segmask = row ? 0x3ffu << base : 0xc0000000u;
	const int witem = (threadIdx.x >> 5) * 3 + (row ? slot : 0);
	double *piv = sPiv[witem];
	const long long nu = ne * km.nv;
	const long long u0 = blockIdx.x * (long long)kBlkItems + witem;
	const bool item = row && u0 < nu;
	const long long u = u0 < nu ? u0 : nu - 1; // lanes past the end shadow the last item
	const int rr = row ? r : 0;
	const long long e = u / km.nv;
	const int v = (int)(u % km.nv);
	const double *vv = km.vi + 3 * v;
	double cod[3][3];
#pragma unroll
	for (int a = 0; a < 3; a++)
#pragma unroll
		for (int b = 0; b < 3; b++)
			cod[a][b] = geom[e * 10 + 3 * a + b];
	const double det = geom[e * 10 + 9];
	// u_k = sum_l v_l codtau[l][k]:  v . c_ij = sum_k u_k int d_k phi_i phi_j
	double uk[3];
#pragma unroll
	for (int k = 0; k < 3; k++)
		uk[k] = vv[0] * cod[0][k] + vv[1] * cod[1][k] + vv[2] * cod[2][k];
	double sp[4];
#pragma unroll
	for (int f = 0; f < 4; f++) {
		const double sf = sown64[u * 4 + f];
		sp[f] = sf > 0.0 ? sf : 0.0;
	}
	const double c = theta * dt_tab[einst ? einst[e] : 0] / det;
	const long long kk = pos[u];
	if (item && r == 0) { // the item's records (a singular block fails the attach)
		rcoef[kk] = (GT)c;
		if (ru64) {
			ru64[kk] = make_double4(uk[0], uk[1], uk[2], c);
			rs64[kk] = make_double4(sown64[u * 4], sown64[u * 4 + 1], sown64[u * 4 + 2], sown64[u * 4 + 3]);
		}
	}
	// row rr of [I + c Minv F | I]
	double a[20];
#pragma unroll
	for (int j = 0; j < 10; j++) {
		double acc = -(uk[0] * sMD[0][rr][j] + uk[1] * sMD[1][rr][j] + uk[2] * sMD[2][rr][j]);
#pragma unroll
		for (int f = 0; f < 4; f++)
#pragma unroll
			for (int jj = 0; jj < 6; jj++)
				if (f2n(f, jj) == j)
					acc += sp[f] * sMS[f][rr][jj];
		a[j] = (rr == j ? 1.0 : 0.0) + c * acc;
		a[10 + j] = 0.0; // slot j, filled from step j on
	}
	int posn = rr;	// this row's position in the row-swapping algorithm
	unsigned long long col = 0; // 4 bits per step t: the row (= column of I) that was the pivot
	bool singular = false;
#pragma unroll
	for (int k = 0; k < 10; k++) {
		// pivot: the largest |a[k]| among positions >= k, ties to the smallest position
		const bool cand = row && posn >= k;
		const unsigned long long val = cand ? (unsigned long long)__double_as_longlong(fabs(a[k])) + 1ull : 0ull;
		unsigned long long best = val;
#pragma unroll
		for (int off = 1; off < 16; off <<= 1) {
			const int src = r + off < seg ? lane + off : lane;
			const unsigned long long ob = __shfl_sync(0xffffffffu, best, src);
			best = ob > best ? ob : best;
		}
		best = __shfl_sync(0xffffffffu, best, base);
		const unsigned win = __ballot_sync(0xffffffffu, val == best) & segmask;
		int blane = __ffs(win) - 1;
		if (__any_sync(0xffffffffu, row && (win & (win - 1)) != 0)) { // a tie: the smallest position
			int key = val == best ? posn * 32 + lane : 0x7fffffff;
#pragma unroll
			for (int off = 1; off < 16; off <<= 1) {
				const int src = r + off < seg ? lane + off : lane;
				const int ok = __shfl_sync(0xffffffffu, key, src);
				key = ok < key ? ok : key;
			}
			blane = __shfl_sync(0xffffffffu, key, base) & 31;
		}
		const int bpos = __shfl_sync(0xffffffffu, posn, blane);
		col |= (unsigned long long)(blane - base) << (4 * k);
		// the rows at position k and at the pivot's position trade places
		const bool pivot = row && lane == blane;
		if (row && posn == k)
			posn = bpos;
		else if (pivot)
			posn = k;
		if (pivot) {
			if (a[k] == 0.0) {
				singular = true;
			} else {
				const double inv = 1.0 / a[k];
#pragma unroll
				for (int q = k + 1; q < 10; q++) {
					a[q] *= inv;
					piv[q] = a[q];
				}
#pragma unroll
				for (int t = 0; t < k; t++) {
					a[10 + t] *= inv;
					piv[10 + t] = a[10 + t];
				}
				a[10 + k] = inv; // 1 x inv
				piv[10 + k] = inv;
			}
		}
		singular = __shfl_sync(0xffffffffu, (int)singular, blane) != 0 || singular;
		__syncwarp();
		const double m = a[k];
		if (row && lane != blane && m != 0.0) {
#pragma unroll
			for (int q = k + 1; q < 10; q++)
				a[q] -= m * piv[q];
#pragma unroll
			for (int t = 0; t <= k; t++)
				a[10 + t] -= m * piv[10 + t];
		}
		__syncwarp(); // the pivot row is read before the next step overwrites it
	}
	if (!item)
		return;
	if (singular) {
		atomicMax(bad, 1);
		return;
	}
	// by columns (entry (i, j) at 10 j + i): the sweep takes rows in pairs, and
	// the item's ten lanes write one contiguous column at a time
	GT *Gk = G + kk * 100 + posn;
#pragma unroll
	for (int t = 0; t < 10; t++)
		Gk[((col >> (4 * t)) & 15) * 10] = (GT)a[10 + t];
}

// per-item records of the sweep
template <typename GT>
__global__ void kin_records_kernel(const int *__restrict__ items, const int *__restrict__ pos,
								   const double *__restrict__ sown64, const int *__restrict__ nb,
								   const int *__restrict__ perm, long long nitems, int nv, int4 *__restrict__ rnb,
								   int4 *__restrict__ rpm, GT *__restrict__ rs)
{
	const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (k >= nitems)
		return;
	const long long u = items[k];
	const long long e = u / nv;
	const int v = (int)(u % nv);
	int n[4], pm[4];
	for (int f = 0; f < 4; f++) {
		const double s = sown64[u * 4 + f];
		const int nbv = nb[e * 4 + f];
		pm[f] = perm[e * 4 + f];
		rs[k * 4 + f] = (GT)s;
		if (!(s < 0.0))
			n[f] = INT_MIN; // outflow or tangent: no coupling
		else if (nbv >= 0)
			n[f] = pos[(long long)nbv * nv + v];
		else
			n[f] = nbv; // -(boundary face + 1)
	}
	rnb[k] = make_int4(n[0], n[1], n[2], n[3]);
	rpm[k] = make_int4(pm[0], pm[1], pm[2], pm[3]);
}

template <typename GT>
int launch_kin_setup(const int *face2elem, long long nf, const double *geom, const int *nb, long long ne,
					 const KinModel &km, double *sown64, unsigned char *mask, cudaStream_t s)
{
	kin_face_s_kernel<<<(unsigned)((nf + 255) / 256), 256, 0, s>>>(face2elem, nf, geom, km, sown64);
	GDN_CUDA_TRY(cudaGetLastError());
	const long long nu = ne * km.nv;
	kin_mask_kernel<<<(unsigned)((nu + 255) / 256), 256, 0, s>>>(sown64, nb, ne, km.nv, mask);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

template <typename GT>
int launch_kin_blocks(const double *geom, const double *sown64, const int *items, const int *pos, const int *nb,
					  const int *perm, long long ne, const KinModel &km, double theta, const int *einst,
					  const double *dt_tab, GT *G, GT *rcoef, int4 *rnb, int4 *rpm, GT *rs, double4 *ru64,
					  double4 *rs64, int *bad, cudaStream_t s)
{
	const long long nu = ne * km.nv;
	kin_blocks_kernel<GT><<<(unsigned)((nu + kBlkItems - 1) / kBlkItems), kBlkThreads, 0, s>>>(
		geom, sown64, pos, ne, km, theta, einst, dt_tab, G, rcoef, ru64, rs64, bad);
	GDN_CUDA_TRY(cudaGetLastError());
	kin_records_kernel<GT><<<(unsigned)((nu + 255) / 256), 256, 0, s>>>(items, pos, sown64, nb, perm, nu, km.nv, rnb,
																		rpm, rs);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}
template int launch_kin_setup<double>(const int *, long long, const double *, const int *, long long,
									  const KinModel &, double *, unsigned char *, cudaStream_t);
template int launch_kin_blocks<double>(const double *, const double *, const int *, const int *, const int *,
									   const int *, long long, const KinModel &, double, const int *, const double *,
									   double *, double *, int4 *, int4 *, double *, double4 *, double4 *, int *,
									   cudaStream_t);
template int launch_kin_blocks<float>(const double *, const double *, const int *, const int *, const int *,
									  const int *, long long, const KinModel &, double, const int *, const double *,
									  float *, float *, int4 *, int4 *, float *, double4 *, double4 *, int *,
									  cudaStream_t);

// f_eq of the analytic data at every boundary face node for every velocity,
// at t + dt/2 (relaxation.c:99, dg_update_boundary with use_feq), formed from
// the device time with the host's rounding.  bt[((bf * nv + v) * 6 + c) * 6 + jj].
__global__ void kin_boundary_trace_kernel(const double *__restrict__ bxyz, long long nbf, Batch b, KinModel km,
										  double *__restrict__ bt)
{
	const long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (u >= nbf * 6)
		return;
	const long long bf = u / 6;
	const int jj = (int)(u % 6);
	const int inst = b.bfinst ? b.bfinst[bf] : 0;
	const double t_half = __dadd_rn(b.t[inst], __dmul_rn(0.5, b.dt[inst]));
	double x[3] = {bxyz[3 * u], bxyz[3 * u + 1], bxyz[3 * u + 2]}, we[6], Aw[6];
	exact_w(b.data[inst], x, t_half, we);
	for (int v = 0; v < km.nv; v++) {
		double n[3] = {km.vi[3 * v], km.vi[3 * v + 1], km.vi[3 * v + 2]};
		maxwell_A<double>(n, we, Aw);
		for (int c = 0; c < 6; c++)
			bt[((bf * km.nv + v) * 6 + c) * 6 + jj] = we[c] / km.nv + km.feq_c * Aw[c];
	}
}

int launch_kin_boundary_trace(const double *bxyz, long long nbf, const Batch &b, int nv, const double *vi,
							  double feq_c, double *bt, cudaStream_t s)
{
	if (nbf <= 0)
		return GDN_CUDA_OK;
	KinModel km;
	km.nv = nv;
	for (int i = 0; i < 3 * NV_MAX; i++)
		km.vi[i] = vi[i];
	km.feq_c = feq_c;
	kin_boundary_trace_kernel<<<(unsigned)((nbf * 6 + 255) / 256), 256, 0, s>>>(bxyz, nbf, b, km, bt);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

// 10 consecutive values of one field of one item, converted to T.  The item
// offsets k*60 + c*10 keep float pairs 8-byte, double pairs 16-byte and
// bfloat16 pairs 4-byte aligned.
template <typename S, typename T>
__device__ __forceinline__ void load10(const S *p, T v[10])
{
	if constexpr (std::is_same<S, float>::value) {
		const float2 *q = reinterpret_cast<const float2 *>(p);
#pragma unroll
		for (int i = 0; i < 5; i++) {
			const float2 a = q[i];
			v[2 * i] = (T)a.x;
			v[2 * i + 1] = (T)a.y;
		}
	} else if constexpr (std::is_same<S, double>::value) {
		const double2 *q = reinterpret_cast<const double2 *>(p);
#pragma unroll
		for (int i = 0; i < 5; i++) {
			const double2 a = q[i];
			v[2 * i] = (T)a.x;
			v[2 * i + 1] = (T)a.y;
		}
	} else {
		const __nv_bfloat162 *q = reinterpret_cast<const __nv_bfloat162 *>(p);
#pragma unroll
		for (int i = 0; i < 5; i++) {
			const float2 a = __bfloat1622float2(q[i]);
			v[2 * i] = (T)a.x;
			v[2 * i + 1] = (T)a.y;
		}
	}
}

template <typename S, typename T>
__device__ __forceinline__ void store10(S *p, const T v[10])
{
	if constexpr (std::is_same<S, float>::value) {
		float2 *q = reinterpret_cast<float2 *>(p);
#pragma unroll
		for (int i = 0; i < 5; i++)
			q[i] = make_float2((float)v[2 * i], (float)v[2 * i + 1]);
	} else if constexpr (std::is_same<S, double>::value) {
		double2 *q = reinterpret_cast<double2 *>(p);
#pragma unroll
		for (int i = 0; i < 5; i++)
			q[i] = make_double2((double)v[2 * i], (double)v[2 * i + 1]);
	} else {
		__nv_bfloat162 *q = reinterpret_cast<__nv_bfloat162 *>(p);
#pragma unroll
		for (int i = 0; i < 5; i++)
			q[i] = __floats2bfloat162_rn((float)v[2 * i], (float)v[2 * i + 1]);
	}
}

// Block forward substitution, a warp per five items.  Six lanes serve an item,
// one per field c (lanes 30 and 31 idle):
//   t = sum_inflow s E_f S tr_f,  r = f - coef Minv t,  y = G r.
// The sweep's limit is the memory instructions of an item, not its arithmetic:
// with lane = item every access of a warp touched 32 items 240 bytes apart, 32
// L1 lookups per instruction, and a level of 14 k items took ~7 us on lookups
// alone.  Here every global access moves 16-byte pieces of an item's
// contiguous 240-byte (FP32) rows, six lanes side by side:
//   stage   G and f of the item into shared memory (cp.async), its records
//           into registers (data no sweep step writes);
//   wait    the caller waits for the item's upwind neighbours;
//   solve   the whole row of each inflow neighbour (three at most) into shared
//           memory through L2, one round trip; the face permutation then picks
//           the traces out of the row there; y leaves through shared memory in
//           the same 16-byte pieces.
// An item has at most three inflow faces where the two sides of a face agree (sum
// s = 0).  The attach takes meshes whose sides differ, and there it can have four:
// the traces of face 3 are then read one by one (all_inflow).
// G is read by its six lanes at one address (broadcast), one wavefront per
// 16 bytes; a warp shares nothing with other warps, so there is no CTA barrier.
// ms per step before (lane = item, 32 items per CTA) and after, the fastest
// grouping of each (jittered meshes, d3q4): 17^3 FP64 0.76 / 0.46, 24^3 FP32 with
// one refinement 3.03 / 1.40, 40^3 FP64 2.83 / 1.83, 64^3 FP32 5.83 / 3.71.
constexpr int kSwSlots = 5; // items per warp

// Warps per CTA (static shared memory below 48 KB) and items per CTA.
template <typename T>
struct SweepCfg {
	static constexpr int warps = sizeof(T) == 4 ? 4 : 3;
	static constexpr int threads = 32 * warps;
	static constexpr int items = kSwSlots * warps;
	// G row stride: the five items' 16-byte reads in distinct banks
	static constexpr int gstride = sizeof(T) == 4 ? 100 : 102;
};
int kin_group_items(int fp64)
{
	return fp64 ? SweepCfg<double>::items : SweepCfg<float>::items;
}

template <typename F, typename T>
struct alignas(16) SweepWarp {
	T G[kSwSlots * SweepCfg<T>::gstride];
	T tr[kSwSlots * 180]; // per item: three neighbour rows [6][10]; then its y
	F f[kSwSlots * 60];
};

template <typename T, int ACC>
struct SweepLane {
	long long k;
	int slot, c;
	bool act;
	int nbk[4], pmk[4];
	unsigned inflow; // faces with a trace
	T s[4], coef;
	double2 ya[ACC == 2 ? 5 : 1];
};

// the item has four inflow faces: face 3 has no place among the three rows
template <typename T, int ACC>
__device__ __forceinline__ bool all_inflow(const SweepLane<T, ACC> &in)
{
	return in.inflow == 15u;
}

// nloc (1 to 5) items k0 .. k0 + nloc - 1, or with `list` list[k0 ..].
template <typename F, typename T, int ACC, bool BD>
__device__ __forceinline__ void warp_stage(const KinSweepParams &p, long long k0, int nloc, const int *list,
										   SweepWarp<F, T> &sh, SweepLane<T, ACC> &in)
{
	constexpr int GV = 16 / sizeof(T), GP = 100 / GV;
	constexpr int FB = 60 * sizeof(F) % 16 == 0 ? 16 : 8, FV = FB / sizeof(F), FP = 60 / FV;
	const int lane = threadIdx.x & 31;
	const int slot = lane < 30 ? lane / 6 : kSwSlots - 1, c = lane - 6 * (lane / 6);
	in.slot = slot;
	in.c = c;
	in.act = lane < 30 && slot < nloc;
	const long long kk = k0 + (in.act ? slot : 0);
	const long long k = list ? (long long)list[kk] : kk;
	in.k = k;
	if (in.act) {
		const T *G = reinterpret_cast<const T *>(p.G) + k * 100;
		const F *f = reinterpret_cast<const F *>(p.f) + k * 60;
#pragma unroll
		for (int i = 0; i < (GP + 5) / 6; i++)
			if (c + 6 * i < GP)
				__pipeline_memcpy_async(sh.G + slot * SweepCfg<T>::gstride + (c + 6 * i) * GV, G + (c + 6 * i) * GV, 16);
#pragma unroll
		for (int i = 0; i < (FP + 5) / 6; i++)
			if (c + 6 * i < FP)
				__pipeline_memcpy_async(sh.f + slot * 60 + (c + 6 * i) * FV, f + (c + 6 * i) * FV, FB);
	}
	__pipeline_commit();
	const int4 nb4 = p.rnb[k];
	const int4 pm4 = p.rpm[k];
	in.nbk[0] = nb4.x, in.nbk[1] = nb4.y, in.nbk[2] = nb4.z, in.nbk[3] = nb4.w;
	in.pmk[0] = pm4.x, in.pmk[1] = pm4.y, in.pmk[2] = pm4.z, in.pmk[3] = pm4.w;
	in.coef = reinterpret_cast<const T *>(p.rcoef)[k];
	const T *rs = reinterpret_cast<const T *>(p.rs) + k * 4;
#pragma unroll
	for (int f = 0; f < 4; f++)
		in.s[f] = rs[f];
	if (ACC == 2) {
		const double2 *ya = reinterpret_cast<const double2 *>(p.yacc + k * 60);
#pragma unroll
		for (int i = 0; i < 5; i++)
			in.ya[i] = ya[c + 6 * i];
	}
	in.inflow = 0;
#pragma unroll
	for (int f = 0; f < 4; f++)
		if (in.nbk[f] >= 0 || (BD && in.nbk[f] != INT_MIN))
			in.inflow |= 1u << f;
	if (!in.act)
		in.inflow = 0;
	if (BD) { // boundary inflow faces: f_eq of the data, in face order
#pragma unroll
		for (int f = 0; f < 4; f++)
			if ((in.inflow >> f & 1) && in.nbk[f] < 0 && !(f == 3 && all_inflow(in))) {
				const int r = __popc(in.inflow & ((1u << f) - 1));
				const int v = p.items[k] % p.nv;
				const double *b = p.bt + (((long long)(-in.nbk[f] - 1) * p.nv + v) * 6 + c) * 6;
#pragma unroll
				for (int jj = 0; jj < 6; jj++)
					sh.tr[slot * 180 + r * 60 + c * 10 + jj] = (T)b[jj];
				in.pmk[f] = 0x543210;
			}
	}
}

// y = G r with G by columns; FP32 in packed row pairs
template <typename T>
__device__ __forceinline__ void block_product(const T *G, const T r[10], T y[10])
{
#pragma unroll
	for (int i = 0; i < 10; i++)
		y[i] = T(0);
	const double2 *g = reinterpret_cast<const double2 *>(G);
#pragma unroll
	for (int q = 0; q < 50; q++) {
		const double2 gv = g[q];
		y[2 * q % 10] += gv.x * r[2 * q / 10];
		y[2 * q % 10 + 1] += gv.y * r[2 * q / 10];
	}
}
template <>
__device__ __forceinline__ void block_product<float>(const float *G, const float r[10], float y[10])
{
	float2 acc[5];
#pragma unroll
	for (int i = 0; i < 5; i++)
		acc[i] = make_float2(0.f, 0.f);
	const float4 *g = reinterpret_cast<const float4 *>(G);
#pragma unroll
	for (int q = 0; q < 25; q++) {
		const float4 gv = g[q];
		const int a = 4 * q, b = 4 * q + 2;
		acc[a % 10 / 2] = __ffma2_rn(make_float2(gv.x, gv.y), make_float2(r[a / 10], r[a / 10]), acc[a % 10 / 2]);
		acc[b % 10 / 2] = __ffma2_rn(make_float2(gv.z, gv.w), make_float2(r[b / 10], r[b / 10]), acc[b % 10 / 2]);
	}
#pragma unroll
	for (int i = 0; i < 5; i++) {
		y[2 * i] = acc[i].x;
		y[2 * i + 1] = acc[i].y;
	}
}

// "Not written yet" in the solution array of the row-driven sweeps: all bits of
// a value set, a NaN that no arithmetic returns by itself; written() keeps one
// that was handed in (a payload of the state) out of the array.
__device__ __forceinline__ bool unwritten(float v)
{
	return __float_as_uint(v) == 0xffffffffu;
}
__device__ __forceinline__ bool unwritten(double v)
{
	return __double_as_longlong(v) == -1ll;
}
__device__ __forceinline__ float written(float v)
{
	return unwritten(v) ? __uint_as_float(0x7fffffffu) : v;
}
__device__ __forceinline__ double written(double v)
{
	return unwritten(v) ? __longlong_as_double(0x7fffffffffffffffll) : v;
}

// A lane's pieces of a row [6][10] that another CTA of the same launch writes or
// reads: 16 bytes at 96 i bytes from p (lane c starts at 16 c), moved by relaxed
// accesses of whole values.  A vector access counts as one access per element, so
// the element type is the value's: a double is never seen in halves.
template <typename T>
struct RowPart;
template <>
struct RowPart<double> {
	double2 v[5];
	// on: else v stays as it is
	__device__ __forceinline__ void load_relaxed(const double *p, int, bool on)
	{
		asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %11, 0;\n\t"
					 "@q ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%10];\n\t"
					 "@q ld.relaxed.gpu.global.v2.f64 {%2, %3}, [%10+96];\n\t"
					 "@q ld.relaxed.gpu.global.v2.f64 {%4, %5}, [%10+192];\n\t"
					 "@q ld.relaxed.gpu.global.v2.f64 {%6, %7}, [%10+288];\n\t"
					 "@q ld.relaxed.gpu.global.v2.f64 {%8, %9}, [%10+384];\n\t}"
					 : "+d"(v[0].x), "+d"(v[0].y), "+d"(v[1].x), "+d"(v[1].y), "+d"(v[2].x), "+d"(v[2].y),
					   "+d"(v[3].x), "+d"(v[3].y), "+d"(v[4].x), "+d"(v[4].y)
					 : "l"(p), "r"((int)on));
	}
	__device__ __forceinline__ void store_relaxed(double *p, int) const
	{
#pragma unroll
		for (int i = 0; i < 5; i++)
			asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p + 12 * i), "d"(v[i].x), "d"(v[i].y)
						 : "memory");
	}
	__device__ __forceinline__ void load(const double *p, int)
	{
#pragma unroll
		for (int i = 0; i < 5; i++)
			v[i] = *reinterpret_cast<const double2 *>(p + 12 * i);
	}
	__device__ __forceinline__ void store(double *p, int) const
	{
#pragma unroll
		for (int i = 0; i < 5; i++)
			*reinterpret_cast<double2 *>(p + 12 * i) = v[i];
	}
};
// 15 pieces: the third is that of lanes 0 to 2
template <>
struct RowPart<float> {
	float4 v[3];
	__device__ __forceinline__ void load_relaxed(const float *p, int c, bool on)
	{
		asm volatile("{\n\t.reg .pred q, r;\n\tsetp.ne.s32 q, %13, 0;\n\tsetp.ne.s32 r, %14, 0;\n\t"
					 "@q ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%12];\n\t"
					 "@q ld.relaxed.gpu.global.v4.f32 {%4, %5, %6, %7}, [%12+96];\n\t"
					 "@r ld.relaxed.gpu.global.v4.f32 {%8, %9, %10, %11}, [%12+192];\n\t}"
					 : "+f"(v[0].x), "+f"(v[0].y), "+f"(v[0].z), "+f"(v[0].w), "+f"(v[1].x), "+f"(v[1].y), "+f"(v[1].z),
					   "+f"(v[1].w), "+f"(v[2].x), "+f"(v[2].y), "+f"(v[2].z), "+f"(v[2].w)
					 : "l"(p), "r"((int)on), "r"((int)(on && c < 3)));
	}
	__device__ __forceinline__ void store_relaxed(float *p, int c) const
	{
#pragma unroll
		for (int i = 0; i < 3; i++)
			if (i < 2 || c < 3)
				asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + 24 * i), "f"(v[i].x),
							 "f"(v[i].y), "f"(v[i].z), "f"(v[i].w)
							 : "memory");
	}
	__device__ __forceinline__ void load(const float *p, int c)
	{
#pragma unroll
		for (int i = 0; i < 3; i++)
			if (i < 2 || c < 3)
				v[i] = *reinterpret_cast<const float4 *>(p + 24 * i);
	}
	__device__ __forceinline__ void store(float *p, int c) const
	{
#pragma unroll
		for (int i = 0; i < 3; i++)
			if (i < 2 || c < 3)
				*reinterpret_cast<float4 *>(p + 24 * i) = v[i];
	}
};
__device__ __forceinline__ float load_relaxed(const float *p)
{
	float v;
	asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ double load_relaxed(const double *p)
{
	double v;
	asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
	return v;
}

// the neighbour item of the r-th inflow face (-1: none, or a boundary face)
template <typename T, int ACC>
__device__ __forceinline__ void inflow_rows(const SweepLane<T, ACC> &in, int nr[3])
{
	nr[0] = nr[1] = nr[2] = -1;
	int cnt = 0;
#pragma unroll
	for (int f = 0; f < 4; f++)
		if (in.inflow >> f & 1) {
			const int n = in.nbk[f] >= 0 ? in.nbk[f] : -1;
			nr[0] = cnt == 0 ? n : nr[0];
			nr[1] = cnt == 1 ? n : nr[1];
			nr[2] = cnt == 2 ? n : nr[2];
			cnt++;
		}
}

// trace jj of face 3 of an item with four inflow faces, from where it is
template <typename F, typename T, int ACC, bool BD>
__device__ __forceinline__ T last_trace(const KinSweepParams &p, const SweepLane<T, ACC> &in, int jj)
{
	if (in.nbk[3] >= 0)
		return load_relaxed(reinterpret_cast<const T *>(p.y) + (long long)in.nbk[3] * 60 + in.c * 10 +
							((in.pmk[3] >> (4 * jj)) & 15));
	const int v = p.items[in.k] % p.nv;
	return BD ? (T)p.bt[(((long long)(-in.nbk[3] - 1) * p.nv + v) * 6 + in.c) * 6 + jj] : T(0);
}

// The inflow neighbours' whole rows into shared memory through L2 (L1 is not
// coherent with other SMs' writes made during the launch), then the lane's
// traces x[f] (zero on faces without inflow).  Call after warp_stage.  FLOW:
// the rows may be being written, so they are read by relaxed loads, all of them
// in flight before the first goes to shared memory; else the rows are complete
// and are copied asynchronously.
template <typename F, typename T, int ACC, bool BD, bool FLOW>
__device__ __forceinline__ void warp_gather(const KinSweepParams &p, const SweepLane<T, ACC> &in, const int nr[3],
											SweepWarp<F, T> &sh, T x[4][6])
{
	constexpr int YV = 16 / sizeof(T), YP = 60 / YV;
	T *tr0 = sh.tr + in.slot * 180;
	const T *y = reinterpret_cast<const T *>(p.y);
	if (FLOW) {
		// predicated loads on zeroed registers: branches (FP32 1.28 against 1.25 ms per
		// 40^3 step), and registers that a skipped load leaves undefined stay alive
		// around the loops and spill (1.71)
		RowPart<T> v[3] = {};
#pragma unroll
		for (int r = 0; r < 3; r++)
			v[r].load_relaxed(y + (long long)nr[r] * 60 + in.c * YV, in.c, nr[r] >= 0);
#pragma unroll
		for (int r = 0; r < 3; r++)
			if (nr[r] >= 0)
				v[r].store(tr0 + r * 60 + in.c * YV, in.c);
	} else {
#pragma unroll
		for (int r = 0; r < 3; r++)
			if (nr[r] >= 0) {
				const T *row = y + (long long)nr[r] * 60;
#pragma unroll
				for (int i = 0; i < (YP + 5) / 6; i++)
					if (in.c + 6 * i < YP)
						__pipeline_memcpy_async(tr0 + r * 60 + (in.c + 6 * i) * YV, row + (in.c + 6 * i) * YV, 16);
			}
	}
	__pipeline_commit();
	__pipeline_wait_prior(0);
	__syncwarp();
#pragma unroll
	for (int f = 0; f < 4; f++) {
#pragma unroll
		for (int jj = 0; jj < 6; jj++)
			x[f][jj] = T(0); // not a value of an earlier fetch: x is dead while the rows are waited for
		if (in.inflow >> f & 1) {
			if (f == 3 && all_inflow(in)) {
#pragma unroll 1
				for (int jj = 0; jj < 6; jj++) {
					const T v = last_trace<F, T, ACC, BD>(p, in, jj);
					x[3][0] = jj == 0 ? v : x[3][0];
					x[3][1] = jj == 1 ? v : x[3][1];
					x[3][2] = jj == 2 ? v : x[3][2];
					x[3][3] = jj == 3 ? v : x[3][3];
					x[3][4] = jj == 4 ? v : x[3][4];
					x[3][5] = jj == 5 ? v : x[3][5];
				}
				continue;
			}
			const T *row = tr0 + __popc(in.inflow & ((1u << f) - 1)) * 60 + in.c * 10;
#pragma unroll
			for (int jj = 0; jj < 6; jj++)
				x[f][jj] = row[(in.pmk[f] >> (4 * jj)) & 15];
		}
	}
}

// Row-driven wait and gather: the rows are their own readiness flags.  Every
// value of y is "unwritten" when the solve starts and is written once, whole, by
// a relaxed store of its size; every trace is read by a relaxed load of that size
// and is ready when it is not "unwritten".  Nothing else passes between the CTAs,
// so no flag, fence or ordering between the values of a row is needed.  (Rows copied
// by cp.async are not atomic by the memory model; ms per step with them / as here:
// 17^3 FP64 0.424 / 0.461, 40^3 FP64 1.73 / 1.83, 40^3 FP32 1.23 / 1.28, 64^3 FP32
// 3.62 / 3.71.  FP64 traces straight from L2: 17^3 0.511, 40^3 2.18.  A fence and a flag per warp: 17^3 0.67, 64^3 4.4.)
// One lane per row polls the row's last value until it is written; then the rows
// are fetched, and polled on should a trace still be missing.  Most warps are
// ahead of their inputs, so what waiting costs the others counts: lanes leave the
// poll with their row, and no row is fetched in vain (fetching first and polling
// all rows on: 40^3 FP64 1.83 against 1.73 ms per step, FP32 1.28 against 1.24).
// false when *err is set, or after spin_limit polls (then *err is set here),
// so a lost producer ends the launch instead of hanging it.
template <typename F, typename T, int ACC, bool BD>
__device__ __forceinline__ bool warp_gather_wait(const KinSweepParams &p, const SweepLane<T, ACC> &in, const int nr[3],
												 SweepWarp<F, T> &sh, T x[4][6], int *err, long long spin_limit)
{
	const int mine = in.c == 0 ? nr[0] : (in.c == 1 ? nr[1] : (in.c == 2 ? nr[2] : (in.c == 3 && all_inflow(in) ? in.nbk[3] : -1)));
	const T *last = reinterpret_cast<const T *>(p.y) + (long long)(mine >= 0 ? mine : 0) * 60 + 59;
	bool waiting = mine >= 0;
	for (long long it = 0;; it++) {
		for (;; it++) {
			if (waiting)
				waiting = unwritten(load_relaxed(last));
			if (!__any_sync(0xffffffffu, waiting))
				break;
			if ((it & 63) == 63 && __any_sync(0xffffffffu, *(const volatile int *)err != 0))
				return false;
			if (it >= spin_limit) {
				if ((threadIdx.x & 31) == 0)
					atomicExch(err, 1);
				return false;
			}
		}
		warp_gather<F, T, ACC, BD, true>(p, in, nr, sh, x);
		bool missing = false;
#pragma unroll
		for (int f = 0; f < 4; f++)
			if ((in.inflow >> f & 1) && in.nbk[f] >= 0) { // boundary values carry no mark
#pragma unroll
				for (int jj = 0; jj < 6; jj++)
					missing |= unwritten(x[f][jj]);
			}
		if (!__any_sync(0xffffffffu, missing))
			return true;
		if (it >= spin_limit) {
			if ((threadIdx.x & 31) == 0)
				atomicExch(err, 1);
			return false;
		}
	}
}

// After the gather: solve, y (and the FP64 accumulator) stored.
// SPARSE: the tables have the P2 structural zeros; FLOW: row-driven sweep.  The
// products are the plain sums over the tables: their symmetric forms
// (lift_minv_sym) cancel more, and cost FP32 sweeps a factor two in error.
template <typename F, typename T, int ACC, bool SPARSE, bool FLOW>
__device__ __forceinline__ void warp_solve(const KinSweepParams &p, const SweepLane<T, ACC> &in, const T x[4][6],
										   SweepWarp<F, T> &sh)
{
	constexpr int YV = 16 / sizeof(T);
	const Tables<T> &tb = tab<T>();
	const int slot = in.slot, c = in.c;
	T *tr0 = sh.tr + slot * 180;
	T y[10];
	{
		// t_i = sum over the inflow faces through node i of s_f (S tr_f)_ii
		T t[10];
#pragma unroll
		for (int i = 0; i < 10; i++)
			t[i] = T(0);
#pragma unroll
		for (int f = 0; f < 4; f++)
			if (in.inflow >> f & 1) {
#pragma unroll
				for (int ii = 0; ii < 6; ii++) {
					T acc = T(0);
#pragma unroll
					for (int jj = 0; jj < 6; jj++)
						if (!SPARSE || (smask(ii) >> jj & 1))
							acc += tb.S[ii][jj] * x[f][jj];
					t[f2n(f, ii)] += acc * in.s[f];
				}
			}
		T mt[10], r[10];
		lift_minv<T>(tb, t, mt);
		load10<F, T>(sh.f + slot * 60 + c * 10, r);
#pragma unroll
		for (int i = 0; i < 10; i++)
			r[i] -= in.coef * mt[i];
		block_product<T>(sh.G + slot * SweepCfg<T>::gstride, r, y);
	}
	if (FLOW) {
#pragma unroll
		for (int i = 0; i < 10; i++)
			y[i] = written(y[i]);
	}
	__syncwarp(); // the item's rows are read: its y takes their place
	if (in.act)
		store10<T, T>(tr0 + c * 10, y);
	__syncwarp();
	if (in.act) {
		T *yo = reinterpret_cast<T *>(p.y) + in.k * 60 + c * YV;
		RowPart<T> v;
		v.load(tr0 + c * YV, c);
		if (FLOW)
			v.store_relaxed(yo, c);
		else
			v.store(yo, c);
		if (ACC != 0) {
			double2 *ya = reinterpret_cast<double2 *>(p.yacc + in.k * 60);
#pragma unroll
			for (int i = 0; i < 5; i++) {
				const T *v = tr0 + 2 * (c + 6 * i);
				ya[c + 6 * i] = ACC == 1 ? make_double2((double)v[0], (double)v[1])
										 : make_double2(in.ya[ACC == 2 ? i : 0].x + (double)v[0],
														in.ya[ACC == 2 ? i : 0].y + (double)v[1]);
			}
		}
	}
	__syncwarp(); // the warp's shared memory is free for its next items
}

// the warp's share of the CTA's group [k0, k1): items k .. k + n - 1 (n <= 0: none)
__device__ __forceinline__ int warp_items(long long k0, long long k1, long long &k)
{
	k = k0 + kSwSlots * (threadIdx.x >> 5);
	const long long n = k1 - k;
	return n < kSwSlots ? (int)n : kSwSlots;
}

// One level per launch, with programmatic dependent launch: the next level's
// CTAs stage their items (data no sweep level writes) while this level runs,
// and wait (griddepcontrol.wait) only before they read the upwind rows.  The first
// level is an ordinary launch (launch_kin_sweep).
template <typename F, typename Y, typename T, int ACC, bool BD, bool SPARSE>
__global__ void __launch_bounds__(SweepCfg<T>::threads) kin_sweep_kernel(KinSweepParams p)
{
	__shared__ SweepWarp<F, T> sh[SweepCfg<T>::warps];
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	long long k;
	const int n = warp_items((long long)p.item_begin + (long long)blockIdx.x * SweepCfg<T>::items, p.item_end, k);
	if (n <= 0)
		return;
	SweepLane<T, ACC> in;
	warp_stage<F, T, ACC, BD>(p, k, n, nullptr, sh[threadIdx.x >> 5], in);
	int nr[3];
	T x[4][6];
	inflow_rows(in, nr);
	asm volatile("griddepcontrol.wait;" ::: "memory");
	warp_gather<F, T, ACC, BD, false>(p, in, nr, sh[threadIdx.x >> 5], x);
	warp_solve<F, T, ACC, SPARSE, false>(p, in, x, sh[threadIdx.x >> 5]);
}

// Grid-wide barrier of a cooperative launch (all CTAs co-resident).  *count
// only grows during the launch (it is cleared before the launch): barrier j
// is passed once it reaches (j + 1) x gridDim.x arrivals.  Arrivals are
// release-ordered, polls acquire-ordered.  The wait is bounded: after
// spin_limit polls the CTA sets *err and leaves, and so does every other CTA
// once it sees *err, so a lost CTA ends the launch instead of hanging it.
__device__ __forceinline__ bool grid_barrier(unsigned *count, unsigned target, int *err, long long spin_limit)
{
	__shared__ int s_ok;
	__syncthreads();
	if (threadIdx.x == 0) {
		volatile int *verr = err;
		int ok = 1;
		asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
		long long it = 0;
		for (;;) {
			unsigned v;
			asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
			if (v >= target)
				break;
			if (*verr || ++it > spin_limit) {
				atomicExch(err, 1);
				ok = 0;
				break;
			}
			__nanosleep(16);
		}
		s_ok = ok && !*verr;
	}
	__syncthreads();
	return s_ok != 0;
}

// Level schedule by Kahn's algorithm, one level per grid barrier, in one
// cooperative launch.  indeg[u] = the upwind dependencies of item u not yet
// placed; the items of level l are listed in one frontier, and placing one
// releases its downwind items (across the faces it flows out of: s > 0 there,
// s < 0 on the other side, so each dependency edge is counted once on each
// end).  An item whose last dependency is placed at level l enters level
// l + 1, so level(u) = the longest upwind chain ending at u.  ctl: [0] barrier
// arrivals, [1..3] frontier sizes of levels l mod 3, [4] error, [5] levels,
// [6] items placed (fewer than all: a cycle).
constexpr int kKahnThreads = 512; // one CTA per SM: the barrier's arrivals, not the work, set a level's time
__global__ void __launch_bounds__(kKahnThreads)
	kin_kahn_kernel(const unsigned char *__restrict__ mask, const int *__restrict__ nb,
					const double *__restrict__ sown64, long long ne, int nv, int *__restrict__ indeg,
					int *__restrict__ level, int *front0, int *front1, unsigned *ctl, long long spin_limit)
{
	const long long nu = ne * nv;
	const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	const long long nthreads = (long long)gridDim.x * blockDim.x;
	const int lane = threadIdx.x & 31;
	const unsigned lt = (1u << lane) - 1u;
	unsigned *bar = ctl, *cnt = ctl + 1;
	int *err = reinterpret_cast<int *>(ctl + 4);
	// level 0: the items without upwind dependencies (warp-aggregated appends)
	for (long long b = tid - lane; b < nu; b += nthreads) {
		const long long u = b + lane;
		int d = 0;
		if (u < nu) {
			d = __popc(mask[u]);
			indeg[u] = d;
		}
		const bool push = u < nu && d == 0;
		const unsigned bal = __ballot_sync(0xffffffffu, push);
		unsigned base = 0;
		if (lane == 0 && bal)
			base = atomicAdd(cnt, __popc(bal));
		base = __shfl_sync(0xffffffffu, base, 0);
		if (push) {
			front0[base + __popc(bal & lt)] = (int)u;
			level[u] = 0;
		}
	}
	if (!grid_barrier(bar, gridDim.x, err, spin_limit))
		return;
	int *cur = front0, *nxt = front1;
	long long placed = 0;
	int l = 0;
	for (;; l++) {
		const unsigned n = *(volatile unsigned *)(cnt + l % 3);
		if (n == 0)
			break;
		placed += n;
		if (tid == 0)
			cnt[(l + 2) % 3] = 0; // level l - 1's size: read by every CTA before the last barrier
		for (long long b = tid - lane; b < n; b += nthreads) {
			const long long i = b + lane;
			const long long u = i < n ? cur[i] : 0;
			const long long e = u / nv;
			const int v = (int)(u % nv);
#pragma unroll
			for (int f = 0; f < 4; f++) {
				bool push = false;
				int w = 0;
				if (i < n) {
					const int we = nb[e * 4 + f];
					if (we >= 0 && sown64[u * 4 + f] > 0.0) {
						w = (int)((long long)we * nv + v);
						push = atomicSub(indeg + w, 1) == 1;
					}
				}
				const unsigned bal = __ballot_sync(0xffffffffu, push);
				unsigned base = 0;
				if (lane == 0 && bal)
					base = atomicAdd(cnt + (l + 1) % 3, __popc(bal));
				base = __shfl_sync(0xffffffffu, base, 0);
				if (push) {
					nxt[base + __popc(bal & lt)] = w;
					level[w] = l + 1;
				}
			}
		}
		if (!grid_barrier(bar, (unsigned)(l + 2) * gridDim.x, err, spin_limit))
			return;
		int *t = cur;
		cur = nxt;
		nxt = t;
	}
	if (tid == 0) {
		ctl[5] = (unsigned)l;
		ctl[6] = (unsigned)placed;
	}
}

// cooperative launch of kin_kahn_kernel with every CTA resident
static int launch_kin_kahn(const unsigned char *mask, const int *nb, const double *sown64, long long ne, int nv,
						   int *indeg, int *level, int *front0, int *front1, unsigned *ctl, long long spin_limit,
						   cudaStream_t s)
{
	int dev = 0, nsm = 0, per = 0;
	GDN_CUDA_TRY(cudaGetDevice(&dev));
	GDN_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
	GDN_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kin_kahn_kernel, kKahnThreads, 0));
	if (per < 1)
		return gdn_set_error(GDN_CUDA_ERR_CUDA, "attach: the level schedule kernel cannot be resident");
	const long long nu = ne * nv;
	long long grid = nsm;
	const long long need = (nu + kKahnThreads - 1) / kKahnThreads;
	if (grid > need)
		grid = need;
	if (grid < 1)
		grid = 1;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)grid);
	cfg.blockDim = dim3(kKahnThreads);
	cfg.stream = s;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	GDN_CUDA_TRY(cudaLaunchKernelEx(&cfg, kin_kahn_kernel, mask, nb, sown64, ne, nv, indeg, level, front0, front1,
									ctl, spin_limit));
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

// All levels of one transport solve in one cooperative launch: the CTAs walk
// the levels in order, one group of items at a time, with a grid barrier
// between levels.  A CTA stages its first group of level l before it waits at
// the barrier that ends level l - 1.
template <typename F, typename Y, typename T, int ACC, bool BD, bool SPARSE>
__global__ void __launch_bounds__(SweepCfg<T>::threads)
	kin_levels_kernel(KinSweepParams p, const int *__restrict__ level_off, int nlevels, unsigned *bar, int *err,
					  long long spin_limit)
{
	__shared__ SweepWarp<F, T> sh[SweepCfg<T>::warps];
	for (int l = 0; l < nlevels; l++) {
		const long long b = level_off[l], e = level_off[l + 1];
		const long long ng = (e - b + SweepCfg<T>::items - 1) / SweepCfg<T>::items;
		bool pending = l > 0; // the barrier ending level l - 1 is still to pass
		const unsigned target = (unsigned)l * gridDim.x;
		for (long long g = blockIdx.x; g < ng; g += gridDim.x) {
			long long k;
			const int n = warp_items(b + g * SweepCfg<T>::items, e, k);
			SweepLane<T, ACC> in;
			if (n > 0)
				warp_stage<F, T, ACC, BD>(p, k, n, nullptr, sh[threadIdx.x >> 5], in);
			if (pending && !grid_barrier(bar, target, err, spin_limit))
				return;
			pending = false;
			if (n > 0) {
				int nr[3];
				T x[4][6];
				inflow_rows(in, nr);
				warp_gather<F, T, ACC, BD, false>(p, in, nr, sh[threadIdx.x >> 5], x);
				warp_solve<F, T, ACC, SPARSE, false>(p, in, x, sh[threadIdx.x >> 5]);
			}
		}
		if (pending && !grid_barrier(bar, target, err, spin_limit))
			return;
	}
}

// The whole transport solve in one cooperative launch, driven by the rows
// themselves (warp_gather_wait) instead of a barrier per level.  groups[] lists
// items in sweep order in groups of one CTA's items, never straddling a level.
// Without `group_off`, CTA b takes the groups b, b + gridDim.x, ... of the
// whole sweep; with it, the groups group_off[b] .. group_off[b + 1] - 1 of its
// own spatial part (their items in list[]; parts: equal ranges of elements
// along a Morton curve of their centroids, all velocities of an element in one
// part).  Each warp takes its five items of a group on its own.  All CTAs are
// co-resident and walk their groups in sweep order, so the unfinished item of
// lowest level always has its inputs and a warp at work on it: the solve
// progresses, and its critical path is the longest upwind chain, not the level
// count times a launch.
// Registers: 5 CTAs per SM fit at 96 (FP32) and 128 (FP64), 4 with an accumulator
// (128).  FP64 is launched at 4 (kin_flow_grid); compiled for 4 it has more registers
// and no gain (ms per step 4^3 d3q6 0.0946 / 0.0950, 17^3 0.460 / 0.460, 40^3 1.829 /
// 1.831).
template <typename F, typename Y, typename T, int ACC, bool BD, bool SPARSE>
__global__ void __launch_bounds__(SweepCfg<T>::threads, sizeof(T) == 8 || ACC == 0 ? 5 : 4)
	kin_flow_kernel(KinSweepParams p, const int2 *__restrict__ groups, int ngroups, const int *__restrict__ list,
					const int *__restrict__ group_off, int *err, long long spin_limit)
{
	__shared__ SweepWarp<F, T> sh[SweepCfg<T>::warps];
	const int g0 = group_off ? group_off[blockIdx.x] : blockIdx.x;
	const int g1 = group_off ? group_off[blockIdx.x + 1] : ngroups;
	const int dg = group_off ? 1 : gridDim.x;
	for (int g = g0; g < g1; g += dg) {
		const int2 gr = groups[g];
		long long k;
		const int n = warp_items(gr.x, gr.y, k);
		// the warp's next items into L2: block inverses, right-hand side, records
		// (40^3 FP64 1.89 -> 1.85, 17^3 0.445 -> 0.432 ms per step)
		if (!list && g + dg < g1) {
			const int2 gn = groups[g + dg];
			long long kn;
			const int nn = warp_items(gn.x, gn.y, kn);
			if (nn > 0) {
				const int lane = threadIdx.x & 31;
				if (lane == 0)
					prefetch_l2(reinterpret_cast<const T *>(p.G) + kn * 100, nn * 100 * sizeof(T));
				else if (lane == 1 && 60 * sizeof(F) % 16 == 0)
					prefetch_l2(reinterpret_cast<const F *>(p.f) + kn * 60, nn * 60 * sizeof(F));
				else if (lane == 2)
					prefetch_l2(p.rnb + kn, nn * sizeof(int4));
				else if (lane == 3)
					prefetch_l2(p.rpm + kn, nn * sizeof(int4));
				else if (lane == 4)
					prefetch_l2(reinterpret_cast<const T *>(p.rs) + kn * 4, nn * 4 * sizeof(T));
			}
		}
		if (n <= 0)
			continue;
		SweepLane<T, ACC> in;
		warp_stage<F, T, ACC, BD>(p, k, n, list, sh[threadIdx.x >> 5], in);
		int nr[3];
		T x[4][6];
		inflow_rows(in, nr);
		if (!warp_gather_wait<F, T, ACC, BD>(p, in, nr, sh[threadIdx.x >> 5], x, err, spin_limit))
			return; // *err is set; the state of this solve is invalid
		warp_solve<F, T, ACC, SPARSE, true>(p, in, x, sh[threadIdx.x >> 5]);
	}
}

// Morton code (10 bits per axis) of each element's vertex centroid in the box
// [lo, lo + 1 / inv_ext)
__device__ __forceinline__ unsigned spread10(unsigned x)
{
	x &= 1023u;
	x = (x | (x << 16)) & 0x030000FFu;
	x = (x | (x << 8)) & 0x0300F00Fu;
	x = (x | (x << 4)) & 0x030C30C3u;
	x = (x | (x << 2)) & 0x09249249u;
	return x;
}
__global__ void kin_morton_kernel(const int *__restrict__ e2q, const double *__restrict__ node, long long ne,
								  double3 lo, double3 inv_ext, unsigned *__restrict__ code, int *__restrict__ elem)
{
	const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (e >= ne)
		return;
	double c[3] = {0.0, 0.0, 0.0};
	for (int i = 0; i < 4; i++)
		for (int a = 0; a < 3; a++)
			c[a] += 0.25 * node[3LL * e2q[10 * e + i] + a];
	const double l[3] = {lo.x, lo.y, lo.z}, s[3] = {inv_ext.x, inv_ext.y, inv_ext.z};
	unsigned q[3];
	for (int a = 0; a < 3; a++) {
		const double t = (c[a] - l[a]) * s[a] * 1024.0;
		q[a] = t <= 0.0 ? 0u : (t >= 1023.0 ? 1023u : (unsigned)t);
	}
	code[e] = spread10(q[0]) | (spread10(q[1]) << 1) | (spread10(q[2]) << 2);
	elem[e] = (int)e;
}
// part of each element from its rank along the curve; part of each item
__global__ void kin_part_of_elem_kernel(const int *__restrict__ elem_sorted, long long ne, int nparts,
										int *__restrict__ part_of_elem)
{
	const long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (r < ne)
		part_of_elem[elem_sorted[r]] = (int)(r * nparts / ne);
}
__global__ void kin_part_of_item_kernel(const int *__restrict__ items, const int *__restrict__ part_of_elem,
										long long nitems, int nv, int *__restrict__ part_key, int *__restrict__ iota)
{
	const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (k >= nitems)
		return;
	part_key[k] = part_of_elem[items[k] / nv];
	iota[k] = (int)k;
}
// Spatial parts of the item list (kin_flow_kernel): nparts compact element
// parts; on return plist (device, [nitems]: items of part 0 in sweep order,
// then part 1, ...) and pkey_host (host, [nitems]: the part of plist[i]) are set.
int kin_build_parts(const int *e2q, const double *node, long long ne, const double lo[3], const double hi[3],
					const int *items, long long nitems, int nv, int nparts, int *plist,
					std::vector<int> &plist_host, std::vector<int> &pkey_host, cudaStream_t s)
{
	unsigned *code = nullptr, *code_s = nullptr;
	int *elem = nullptr, *elem_s = nullptr, *pe = nullptr, *pkey = nullptr, *pkey_s = nullptr, *iota = nullptr;
	void *tmp = nullptr;
	size_t tb = 0, tb2 = 0;
	auto cleanup = [&]() {
		dev_free(code, s);
		dev_free(code_s, s);
		dev_free(elem, s);
		dev_free(elem_s, s);
		dev_free(pe, s);
		dev_free(pkey, s);
		dev_free(pkey_s, s);
		dev_free(iota, s);
		dev_free(tmp, s);
	};
#define GDN_PARTS_TRY(expr)                                                                                           \
	do {                                                                                                           \
		cudaError_t _e = (expr);                                                                                   \
		if (_e != cudaSuccess) {                                                                                   \
			cleanup();                                                                                             \
			return gdn_cuda_fail(_e, #expr, __FILE__, __LINE__);                                                  \
		}                                                                                                          \
	} while (0)
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&code), ne * sizeof(unsigned), s));
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&code_s), ne * sizeof(unsigned), s));
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&elem), ne * sizeof(int), s));
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&elem_s), ne * sizeof(int), s));
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&pe), ne * sizeof(int), s));
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&pkey), nitems * sizeof(int), s));
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&pkey_s), nitems * sizeof(int), s));
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&iota), nitems * sizeof(int), s));
	double3 l = make_double3(lo[0], lo[1], lo[2]), ie;
	ie.x = 1.0 / (hi[0] - lo[0] > 0.0 ? hi[0] - lo[0] : 1.0);
	ie.y = 1.0 / (hi[1] - lo[1] > 0.0 ? hi[1] - lo[1] : 1.0);
	ie.z = 1.0 / (hi[2] - lo[2] > 0.0 ? hi[2] - lo[2] : 1.0);
	const unsigned ge = (unsigned)((ne + 255) / 256), gi = (unsigned)((nitems + 255) / 256);
	kin_morton_kernel<<<ge, 256, 0, s>>>(e2q, node, ne, l, ie, code, elem);
	GDN_PARTS_TRY(cudaGetLastError());
	GDN_PARTS_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, code, code_s, elem, elem_s, (int)ne, 0, 30, s));
	GDN_PARTS_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb2, pkey, pkey_s, iota, plist, (int)nitems, 0, 31, s));
	GDN_PARTS_TRY(dev_alloc(reinterpret_cast<void **>(&tmp), tb > tb2 ? tb : tb2, s));
	tb = tb > tb2 ? tb : tb2;
	GDN_PARTS_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, code, code_s, elem, elem_s, (int)ne, 0, 30, s));
	kin_part_of_elem_kernel<<<ge, 256, 0, s>>>(elem_s, ne, nparts, pe);
	GDN_PARTS_TRY(cudaGetLastError());
	kin_part_of_item_kernel<<<gi, 256, 0, s>>>(items, pe, nitems, nv, pkey, iota);
	GDN_PARTS_TRY(cudaGetLastError());
	int bits = 1;
	while ((1 << bits) <= nparts)
		bits++;
	// stable: within a part the items keep their sweep order
	GDN_PARTS_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, pkey, pkey_s, iota, plist, (int)nitems, 0, bits, s));
	plist_host.resize(nitems);
	pkey_host.resize(nitems);
	GDN_PARTS_TRY(cudaMemcpyAsync(plist_host.data(), plist, nitems * sizeof(int), cudaMemcpyDeviceToHost, s));
	GDN_PARTS_TRY(cudaMemcpyAsync(pkey_host.data(), pkey_s, nitems * sizeof(int), cudaMemcpyDeviceToHost, s));
	GDN_PARTS_TRY(cudaStreamSynchronize(s));
#undef GDN_PARTS_TRY
	cleanup();
	return GDN_CUDA_OK;
}

template <typename F, typename Y, typename T>
int launch_kin_sweep(const KinSweepParams &p, int acc, int bdata, int sparse, cudaStream_t s)
{
	const long long n = (long long)p.item_end - p.item_begin;
	if (n <= 0)
		return GDN_CUDA_OK;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)((n + SweepCfg<T>::items - 1) / SweepCfg<T>::items));
	cfg.blockDim = dim3(SweepCfg<T>::threads);
	cfg.dynamicSmemBytes = 0;
	cfg.stream = s;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	// The first level stages what the kernels just before it wrote (boundary data,
	// right-hand side), ahead of griddepcontrol.wait: it is an ordinary launch, which
	// starts after them.  A later level starts after the first has.
	cfg.numAttrs = p.item_begin > 0 ? 1 : 0;
#define GDN_SWEEP(A, B, SP) GDN_CUDA_TRY(cudaLaunchKernelEx(&cfg, kin_sweep_kernel<F, Y, T, A, B, SP>, p))
	if (acc == 0 && bdata) {
		if (sparse)
			GDN_SWEEP(0, true, true);
		else
			GDN_SWEEP(0, true, false);
	} else if (acc == 1 && bdata) {
		if (sparse)
			GDN_SWEEP(1, true, true);
		else
			GDN_SWEEP(1, true, false);
	} else if (acc == 2 && !bdata) {
		if (sparse)
			GDN_SWEEP(2, false, true);
		else
			GDN_SWEEP(2, false, false);
	} else {
		return gdn_set_error(GDN_CUDA_ERR_INVALID, "kinetic sweep: unsupported accumulate / boundary mode");
	}
#undef GDN_SWEEP
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}
template <typename F, typename Y, typename T>
int launch_kin_levels(const KinSweepParams &p, const int *level_off, int nlevels, int grid, unsigned *bar, int *err,
					  long long spin, int acc, int bdata, int sparse, cudaStream_t s)
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)grid);
	cfg.blockDim = dim3(SweepCfg<T>::threads);
	cfg.dynamicSmemBytes = 0;
	cfg.stream = s;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	GDN_CUDA_TRY(cudaMemsetAsync(bar, 0, sizeof(unsigned), s));
#define GDN_LEVELS(A, B, SP)                                                                                          \
	GDN_CUDA_TRY(cudaLaunchKernelEx(&cfg, kin_levels_kernel<F, Y, T, A, B, SP>, p, level_off, nlevels, bar, err, spin))
	if (acc == 0 && bdata) {
		if (sparse)
			GDN_LEVELS(0, true, true);
		else
			GDN_LEVELS(0, true, false);
	} else if (acc == 1 && bdata) {
		if (sparse)
			GDN_LEVELS(1, true, true);
		else
			GDN_LEVELS(1, true, false);
	} else if (acc == 2 && !bdata) {
		if (sparse)
			GDN_LEVELS(2, false, true);
		else
			GDN_LEVELS(2, false, false);
	} else {
		return gdn_set_error(GDN_CUDA_ERR_INVALID, "kinetic sweep: unsupported accumulate / boundary mode");
	}
#undef GDN_LEVELS
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

template <typename F, typename Y, typename T>
int launch_kin_flow(const KinSweepParams &p, const int2 *groups, int ngroups, const int *list, const int *group_off,
					int grid, long long nitems, int *err, long long spin, int acc, int bdata, int sparse,
					cudaStream_t s)
{
	if (ngroups <= 0)
		return GDN_CUDA_OK;
	// every row unwritten (clearing it in the relaxation, which reads y anyway,
	// measured slower: 3.79 against 3.62 ms per 64^3 FP32 step)
	GDN_CUDA_TRY(cudaMemsetAsync(p.y, 0xff, (size_t)nitems * 60 * sizeof(Y), s));
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)grid);
	cfg.blockDim = dim3(SweepCfg<T>::threads);
	cfg.stream = s;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
#define GDN_FLOW(A, B, SP)                                                                                            \
	GDN_CUDA_TRY(cudaLaunchKernelEx(&cfg, kin_flow_kernel<F, Y, T, A, B, SP>, p, groups, ngroups, list, group_off,   \
									err, spin))
	if (acc == 0 && bdata) {
		if (sparse)
			GDN_FLOW(0, true, true);
		else
			GDN_FLOW(0, true, false);
	} else if (acc == 1 && bdata) {
		if (sparse)
			GDN_FLOW(1, true, true);
		else
			GDN_FLOW(1, true, false);
	} else if (acc == 2 && !bdata) {
		if (sparse)
			GDN_FLOW(2, false, true);
		else
			GDN_FLOW(2, false, false);
	} else {
		return gdn_set_error(GDN_CUDA_ERR_INVALID, "kinetic sweep: unsupported accumulate / boundary mode");
	}
#undef GDN_FLOW
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

// CTAs of the row-driven sweep that fit on the device at once
template <typename F, typename Y, typename T>
int kin_flow_grid(int device, int acc, int sparse, int *grid)
{
	int nsm = 0, per = 0;
	GDN_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
	const void *fn;
	if (sparse)
		fn = acc == 0   ? (const void *)kin_flow_kernel<F, Y, T, 0, true, true>
			 : acc == 1 ? (const void *)kin_flow_kernel<F, Y, T, 1, true, true>
						: (const void *)kin_flow_kernel<F, Y, T, 2, false, true>;
	else
		fn = acc == 0   ? (const void *)kin_flow_kernel<F, Y, T, 0, true, false>
			 : acc == 1 ? (const void *)kin_flow_kernel<F, Y, T, 1, true, false>
						: (const void *)kin_flow_kernel<F, Y, T, 2, false, false>;
	GDN_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, SweepCfg<T>::threads, 0));
	// FP32 20 warps per SM, FP64 12 (4 CTAs of 3): with fewer a level is taken in
	// parts, more only poll (ms per step, FP64 4 / 5 CTAs: 17^3 0.460 / 0.466, 32^3
	// 1.164 / 1.177, 40^3 1.829 / 1.825; 64^3 FP32 for 2, 3, 4, 5, before the polls of
	// warp_gather_wait were thinned out: 4.46, 3.93, 3.79, 3.62)
	const int cap = sizeof(T) == 4 ? 5 : 4;
	*grid = nsm * (per > cap ? cap : (per > 0 ? per : 1));
	return GDN_CUDA_OK;
}

// CTAs of the persistent level loop that fit on the device at once
template <typename F, typename Y, typename T>
int kin_levels_grid(int device, int acc, int sparse, int *grid)
{
	int nsm = 0, per = 0;
	GDN_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
	const void *fn;
	if (sparse)
		fn = acc == 0   ? (const void *)kin_levels_kernel<F, Y, T, 0, true, true>
			 : acc == 1 ? (const void *)kin_levels_kernel<F, Y, T, 1, true, true>
						: (const void *)kin_levels_kernel<F, Y, T, 2, false, true>;
	else
		fn = acc == 0   ? (const void *)kin_levels_kernel<F, Y, T, 0, true, false>
			 : acc == 1 ? (const void *)kin_levels_kernel<F, Y, T, 1, true, false>
						: (const void *)kin_levels_kernel<F, Y, T, 2, false, false>;
	GDN_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, SweepCfg<T>::threads, 0));
	// at most 3 CTAs per SM, about one per group of a 64^3 level: fewer arrivals
	// per grid barrier (ms per step for 1, 2, 3, 4 CTAs per SM: 64^3 FP32 8.31,
	// 6.41, 5.98, 5.89; 40^3 FP64 3.69, 3.06, 3.07, 3.10)
	*grid = nsm * (per > 3 ? 3 : per);
	return GDN_CUDA_OK;
}

#define GDN_LEVELS_INST(F, Y, T)                                                                                      \
	template int launch_kin_levels<F, Y, T>(const KinSweepParams &, const int *, int, int, unsigned *, int *,         \
											long long, int, int, int, cudaStream_t);                                     \
	template int kin_levels_grid<F, Y, T>(int, int, int, int *);                                                      \
	template int launch_kin_flow<F, Y, T>(const KinSweepParams &, const int2 *, int, const int *, const int *, int,   \
										  long long, int *, long long, int, int, int, cudaStream_t);                     \
	template int kin_flow_grid<F, Y, T>(int, int, int, int *);
GDN_LEVELS_INST(double, double, double)
GDN_LEVELS_INST(float, float, float)
GDN_LEVELS_INST(__nv_bfloat16, float, float)
GDN_LEVELS_INST(double, float, float)
#undef GDN_LEVELS_INST

template int launch_kin_sweep<double, double, double>(const KinSweepParams &, int, int, int, cudaStream_t);
template int launch_kin_sweep<float, float, float>(const KinSweepParams &, int, int, int, cudaStream_t);
template int launch_kin_sweep<__nv_bfloat16, float, float>(const KinSweepParams &, int, int, int, cudaStream_t);
template int launch_kin_sweep<double, float, float>(const KinSweepParams &, int, int, int, cudaStream_t);

// FP64 residual of the transport system of every item (no level order: it
// only reads y), a lane per item and a warp per field:
//   r = f - y - coef Minv (V y + sum_outflow s E S E^T y + sum_inflow s E S tr)
// with V_ij = -(u . D_ij), u_k = v . codtau[:, k], tr the upwind neighbour's
// y or the boundary f_eq.  This is f - b - M1 y with M1 as the blocks kernel
// builds it, from the FP64 u, theta dt / det and v.vn it records per item.
constexpr int kResThreads = 192;
template <bool SPARSE>
__global__ void __launch_bounds__(kResThreads) kin_residual_kernel(KinResidualParams p)
{
	const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
	const long long k = (long long)blockIdx.x * 32 + lane;
	if (k >= p.nitems)
		return;
	const Tables<double> &tb = c_tab_d;
	const int4 nb4 = p.rnb[k];
	const int4 pm4 = p.rpm[k];
	const int nbk[4] = {nb4.x, nb4.y, nb4.z, nb4.w};
	const int pmk[4] = {pm4.x, pm4.y, pm4.z, pm4.w};
	double tr[4][6];
#pragma unroll
	for (int f = 0; f < 4; f++) {
		const int nbv = nbk[f];
		if (nbv >= 0) {
			const double *yn = p.yacc + (long long)nbv * 60 + c * 10;
#pragma unroll
			for (int jj = 0; jj < 6; jj++)
				tr[f][jj] = yn[(pmk[f] >> (4 * jj)) & 15];
		} else if (nbv != INT_MIN) {
			const int v = p.items[k] % p.nv;
			const double *b = p.bt + (((long long)(-nbv - 1) * p.nv + v) * 6 + c) * 6;
#pragma unroll
			for (int jj = 0; jj < 6; jj++)
				tr[f][jj] = b[jj];
		} else {
#pragma unroll
			for (int jj = 0; jj < 6; jj++)
				tr[f][jj] = 0.0;
		}
	}
	double yk[10], fv[10];
	load10<double, double>(p.yacc + k * 60 + c * 10, yk);
	load10<double, double>(p.f + k * 60 + c * 10, fv);
	const double4 ru = p.ru64[k]; // u_0, u_1, u_2, theta dt / det
	const double4 s4 = p.rs64[k];
	const double s[4] = {s4.x, s4.y, s4.z, s4.w};
	// V y = -(u_0 D_0 y + u_1 D_1 y + u_2 D_2 y)
	double t[10];
#pragma unroll
	for (int i = 0; i < 10; i++) {
		double g[3];
#pragma unroll
		for (int q = 0; q < 3; q++) {
			double acc = 0.0;
#pragma unroll
			for (int j = 0; j < 10; j++)
				if (!SPARSE || (dmask(q, i) >> j & 1))
					acc += tb.D[q][i][j] * yk[j];
			g[q] = acc;
		}
		t[i] = -(ru.x * g[0] + ru.y * g[1] + ru.z * g[2]);
	}
#pragma unroll
	for (int f = 0; f < 4; f++) {
		const bool out = s[f] > 0.0;
#pragma unroll
		for (int ii = 0; ii < 6; ii++) {
			double acc = 0.0;
#pragma unroll
			for (int jj = 0; jj < 6; jj++)
				if (!SPARSE || (smask(ii) >> jj & 1))
					acc += tb.S[ii][jj] * (out ? yk[f2n(f, jj)] : tr[f][jj]);
			t[f2n(f, ii)] += acc * s[f];
		}
	}
	float rr[10];
#pragma unroll
	for (int i = 0; i < 10; i++) {
		double acc = 0.0;
#pragma unroll
		for (int j = 0; j < 10; j++)
			acc += tb.Minv[i][j] * t[j];
		rr[i] = (float)(fv[i] - yk[i] - ru.w * acc);
	}
	store10<float, float>(p.r + k * 60 + c * 10, rr);
}

int launch_kin_residual(const KinResidualParams &p, int sparse, cudaStream_t s)
{
	if (p.nitems <= 0)
		return GDN_CUDA_OK;
	const unsigned grid = (unsigned)((p.nitems + 31) / 32);
	if (sparse)
		kin_residual_kernel<true><<<grid, kResThreads, 0, s>>>(p);
	else
		kin_residual_kernel<false><<<grid, kResThreads, 0, s>>>(p);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

// x = a_y y + a_f f (the Crank-Nicolson transport result), then the
// relaxation of dg_apply_relaxation (dg.c:109-147): w = sum_v x_v,
// f <- omega f_eq(w) + (1 - omega) x.  A thread per (element, node).
template <typename F, typename Y, typename T, int NV>
__global__ void kin_relax_kernel(KinRelaxParams p)
{
	const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (t >= p.ne * 10)
		return;
	const long long e = t / 10;
	const int i = (int)(t % 10);
	F *f = reinterpret_cast<F *>(p.f);
	const Y *yv = reinterpret_cast<const Y *>(p.y);
	T x[NV][6], w[6];
	long long base[NV];
#pragma unroll
	for (int c = 0; c < 6; c++)
		w[c] = T(0);
#pragma unroll
	for (int v = 0; v < NV; v++) {
		base[v] = (long long)p.pos[e * NV + v] * 60 + i;
#pragma unroll
		for (int c = 0; c < 6; c++) {
			const long long o = base[v] + c * 10;
			const T xv = (T)p.a_y * (T)Store<Y>::load(yv + o) + (T)p.a_f * (T)Store<F>::load(f + o);
			x[v][c] = xv;
			w[c] += xv;
		}
	}
	const T om = (T)p.omega, om1 = T(1) - (T)p.omega, fc = (T)p.feq_c, inv_nv = T(1) / T(NV);
#pragma unroll
	for (int v = 0; v < NV; v++) {
		const T n[3] = {(T)p.vi[3 * v], (T)p.vi[3 * v + 1], (T)p.vi[3 * v + 2]};
		T Aw[6];
		maxwell_A<T>(n, w, Aw);
#pragma unroll
		for (int c = 0; c < 6; c++) {
			const T feq = w[c] * inv_nv + fc * Aw[c];
			Store<F>::store(f + base[v] + c * 10, om * feq + om1 * x[v][c]);
		}
	}
}

template <typename F, typename Y, typename T>
int launch_kin_relax(const KinRelaxParams &p, cudaStream_t s)
{
	const unsigned nblk = (unsigned)((p.ne * 10 + 255) / 256);
	if (p.nv == 4)
		kin_relax_kernel<F, Y, T, 4><<<nblk, 256, 0, s>>>(p);
	else
		kin_relax_kernel<F, Y, T, 6><<<nblk, 256, 0, s>>>(p);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}
template int launch_kin_relax<double, double, double>(const KinRelaxParams &, cudaStream_t);
template int launch_kin_relax<float, float, float>(const KinRelaxParams &, cudaStream_t);
template int launch_kin_relax<__nv_bfloat16, float, float>(const KinRelaxParams &, cudaStream_t);

} // namespace gdn
