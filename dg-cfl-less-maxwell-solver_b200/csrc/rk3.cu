// HP-1: one fused kernel per low-storage RK3 stage.
//
// The reference (src/dg/explicit.c:75-96) does, per stage i:
//   dg_update_boundary(t + C_i dt); temp = F w; dw = M^-1 temp;
//   k2 = A_i k2 - dt dw; w += B_i k2
// with F and M^-1 assembled as global CSR matrices (simulation.c:218-491).
// Here the same operator is applied matrix-free, element by element:
//   R = (curl H, -curl E)          volume: -sum_j A(c_ij) w_j with
//                                  c_ij = codtau . int d(phi_i) phi_j
//                                  (simulation.c:263-324), so the physical
//                                  derivative of a field is codtau applied to
//                                  the three reference derivatives D_k w
//     + sum_faces S F_upwind(w_own, w_nb, vn)   (simulation.c:356-491)
//   dw = (1/det) Minv R            (simulation.c:241-243)
// Face fluxes are computed by each element with its own outward normal; the
// upwind flux is antisymmetric under (wL, wR, n) -> (wR, wL, -n), so this is
// the reference's +/- pair up to rounding.  Boundary neighbours read the
// analytic data at the face-node coordinates and the stage time
// (dg_update_boundary, dg.c:76-106), in tables that the step before wrote
// (rk3_trace_block).
//
// Device layout: the state, k2 and the geometry are stored in tiles of 32
// elements, value-major inside a tile (rk3_tix), elements in the order of
// rk3_order_kernel.  Lane = element throughout, so every per-element access of
// a warp is whole rows.  With the P2 tables the derivative tables factor through
// the P1 basis (d(phi_i) is linear) and the products with Q4, S and Minv through
// their symmetry (rk3_tables_factor):
//   FP32  rk3_elem_kernel: a thread per element;
//   FP64  rk3_half_kernel: a thread per element and half (E or H), or where more
//         warps count (rk3_default_variant) rk3_stage_kernel (FACT).
// Other tables run rk3_stage_kernel too, a CTA of 6 warps per tile:
//   0  every thread starts the gathers of its 24 neighbour-trace values
//      (face node jj = warp of the 4 faces), asynchronously into its own flux
//      slots in shared memory (cp.async; FP64 with few CTAs per SM: into
//      registers), so that phase 1 hides their latency;
//   1  warp c (field c): the 10 nodal values of field c in registers (kept
//      for the RK update); without FACT also the two physical derivatives the
//      curl needs, by the table products, to shared memory;
//   2  warp jj: the upwind flux at face node jj of the 4 faces (own traces from
//      the tile) to shared memory;
//   -- the one barrier --
//   3  warp c: R_c = curl part + sum_faces S F_c, lift by Minv, RK update with
//      k2 (loaded before the barrier), coalesced stores.
//
// A step is three launches.  The boundary data of a step's three stages is
// written by extra CTAs of the last stage of the step before (rk3_trace_block;
// by launch_rk3_traces after the state was set), and the stages are programmatic
// dependent launches: a stage's CTAs start while the stage before ends, load
// what no stage writes (connectivity, geometry) and wait before the rest.
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace gdn {

// Structural nonzeros of int d_k(phi_i) phi_j for the P2 basis (bit j of
// row i), and of the P2 triangle mass.  Checked against the tables at attach
// (entries outside the pattern must be below 1e-15 in magnitude).
__host__ __device__ constexpr unsigned dmask(int k, int i)
{
	constexpr unsigned short m[3][10] = {{0x3ff, 0x3ff, 0x000, 0x000, 0x1e3, 0x3fb, 0x3fb, 0x3f7, 0x3f7, 0x000},
										 {0x3ff, 0x000, 0x3ff, 0x000, 0x3fd, 0x3fd, 0x2b5, 0x3f7, 0x000, 0x3f7},
										 {0x3ff, 0x000, 0x000, 0x3ff, 0x3fd, 0x000, 0x3fb, 0x359, 0x3fd, 0x3fb}};
	return m[k][i];
}
__host__ __device__ constexpr unsigned smask(int i)
{
	constexpr unsigned char m[6] = {0x17, 0x27, 0x0f, 0x3c, 0x39, 0x3a};
	return m[i];
}
// the reference's P2 face-node convention (t10.c:37-42)
__host__ __device__ constexpr int f2n(int f, int j)
{
	constexpr int m[4][6] = {{0, 3, 2, 7, 9, 6}, {0, 1, 3, 4, 8, 7}, {0, 2, 1, 6, 5, 4}, {1, 2, 3, 5, 9, 8}};
	return m[f][j];
}

// P2 edge nodes 4..9 and their end vertices (t10.c:37-42 face-node lists)
__host__ __device__ constexpr int edge_end(int e, int side)
{
	constexpr int m[6][2] = {{0, 1}, {1, 2}, {0, 2}, {0, 3}, {1, 3}, {2, 3}};
	return m[e][side];
}

// Physical weak derivative sum_k g_k . D_k w of a P2 field along one
// direction through the P1 basis: d(phi_i) is linear, so
// int d(phi_i) w_h = (vertex i) g_i (4 u_i - s), (edge p-q) 4 (g_p u_q + g_q u_p)
// with u_l = int lambda_l w_h, s = sum_l u_l and g_l the derivative of
// lambda_l along the direction.  v = 4 u; t = v - s (vertex terms).
template <typename T>
__device__ __forceinline__ void p1_weak_derivative(const T cd[3], const T v[4], const T t[4], T out[10])
{
	const T g[4] = {-(cd[0] + cd[1] + cd[2]), cd[0], cd[1], cd[2]};
#pragma unroll
	for (int i = 0; i < 4; i++)
		out[i] = g[i] * t[i];
#pragma unroll
	for (int e = 0; e < 6; e++) {
		const int a = edge_end(e, 0), b = edge_end(e, 1);
		out[4 + e] = g[a] * v[b] + g[b] * v[a];
	}
}

// Vertex sum, edge sum and, per vertex, the sum over its three edges of a P2
// nodal vector.
template <typename T>
__device__ __forceinline__ void p2_sums(const T x[10], T &sv, T &se, T ev[4])
{
	sv = (x[0] + x[1]) + (x[2] + x[3]);
	se = ((x[4] + x[5]) + (x[6] + x[7])) + (x[8] + x[9]);
#pragma unroll
	for (int l = 0; l < 4; l++) {
		T acc = T(0);
		bool first = true;
#pragma unroll
		for (int e = 0; e < 6; e++)
			if (edge_end(e, 0) == l || edge_end(e, 1) == l) {
				acc = first ? x[4 + e] : acc + x[4 + e];
				first = false;
			}
		ev[l] = acc;
	}
}

// v = Q4 w and t = v - sum(v) / 4 through the symmetry of Q4 (q4_sym: qa on
// two vertices, qb on a vertex and an edge through it, qc on a vertex and an
// edge off it): v_l = (qa sv + qc se) - qa w_l + (qb - qc) ev_l.
template <typename T>
__device__ __forceinline__ void q4_apply_sym(const Tables<T> &tb, const T w[10], T v[4], T t[4])
{
	T sv, se, ev[4];
	p2_sums<T>(w, sv, se, ev);
	const T base = tb.q4_sym[0] * sv + tb.q4_sym[1] * se;
	const T s = tb.q4_sym[4] * sv + tb.q4_sym[5] * se; // sum(v) / 4
#pragma unroll
	for (int l = 0; l < 4; l++) {
		v[l] = base + tb.q4_sym[2] * w[l] + tb.q4_sym[3] * ev[l];
		t[l] = v[l] - s;
	}
}

// dw = Minv R through the symmetry of Minv (minv_sym), 58 operations instead
// of 100: vertex i: m0 sv + m1 se + m3 R_i + m4 ev_i; edge p-q: m1 sv + m2 se
// + m4 (R_p + R_q) + m5 R_e + m6 (ev_p + ev_q).
template <typename T>
__device__ __forceinline__ void lift_minv_sym(const Tables<T> &tb, const T R[10], T dw[10])
{
	T sv, se, ev[4];
	p2_sums<T>(R, sv, se, ev);
	const T bv = tb.minv_sym[0] * sv + tb.minv_sym[1] * se;
	const T be = tb.minv_sym[1] * sv + tb.minv_sym[2] * se;
#pragma unroll
	for (int i = 0; i < 4; i++)
		dw[i] = bv + tb.minv_sym[3] * R[i] + tb.minv_sym[4] * ev[i];
#pragma unroll
	for (int e = 0; e < 6; e++) {
		const int a = edge_end(e, 0), b = edge_end(e, 1);
		dw[4 + e] = be + tb.minv_sym[4] * (R[a] + R[b]) + tb.minv_sym[5] * R[4 + e] + tb.minv_sym[6] * (ev[a] + ev[b]);
	}
}

// r[k][i] = sum_j D_k[i][j] w[j] for the three reference directions, with the
// structural zeros skipped at compile time.
template <typename T, bool SPARSE>
__device__ __forceinline__ void ref_derivatives(const Tables<T> &tb, const T w[10], T r[3][10])
{
#pragma unroll
	for (int k = 0; k < 3; k++)
#pragma unroll
		for (int i = 0; i < 10; i++) {
			T acc = T(0);
#pragma unroll
			for (int j = 0; j < 10; j++)
				if (!SPARSE || (dmask(k, i) >> j & 1))
					acc += tb.D[k][i][j] * w[j];
			r[k][i] = acc;
		}
}

// dw = Minv R (dense 10 x 10)
template <typename T>
__device__ __forceinline__ void lift_minv(const Tables<T> &tb, const T R[10], T dw[10])
{
#pragma unroll
	for (int i = 0; i < 10; i++) {
		T acc = T(0);
#pragma unroll
		for (int j = 0; j < 10; j++)
			acc += tb.Minv[i][j] * R[j];
		dw[i] = acc;
	}
}

template <>
__device__ __forceinline__ void lift_minv<float>(const Tables<float> &tb, const float R[10], float dw[10])
{
	float2 acc[5];
#pragma unroll
	for (int m = 0; m < 5; m++)
		acc[m] = make_float2(0.f, 0.f);
#pragma unroll
	for (int j = 0; j < 10; j++) {
		const float2 rd = make_float2(R[j], R[j]);
#pragma unroll
		for (int m = 0; m < 5; m++)
			acc[m] = __ffma2_rn(tb.MinvP[m][j], rd, acc[m]);
	}
#pragma unroll
	for (int m = 0; m < 5; m++) {
		dw[2 * m] = acc[m].x;
		dw[2 * m + 1] = acc[m].y;
	}
}

constexpr int kRk3Threads = 192; // 6 warps, one 32-element tile

__device__ __forceinline__ unsigned smem_u32(const void *p)
{
	return (unsigned)__cvta_generic_to_shared(p);
}
// six values global -> shared, asynchronously: dst[cc * DS] = src[cc * SS]
// for cc < 6.  The strides are compile-time, so the six copies address off
// one shared and one global base register with immediate offsets (separate
// asm statements would each materialise both addresses).
template <typename T, int DS, int SS>
__device__ __forceinline__ void cp_async_6(T *dst, const T *src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n\t"
				 "cp.async.ca.shared.global [%0+%3], [%1+%4], %2;\n\t"
				 "cp.async.ca.shared.global [%0+%5], [%1+%6], %2;\n\t"
				 "cp.async.ca.shared.global [%0+%7], [%1+%8], %2;\n\t"
				 "cp.async.ca.shared.global [%0+%9], [%1+%10], %2;\n\t"
				 "cp.async.ca.shared.global [%0+%11], [%1+%12], %2;" ::"r"(smem_u32(dst)),
				 "l"(src), "n"(sizeof(T)), "n"(1 * DS * (int)sizeof(T)), "n"(1 * SS * (int)sizeof(T)),
				 "n"(2 * DS * (int)sizeof(T)), "n"(2 * SS * (int)sizeof(T)), "n"(3 * DS * (int)sizeof(T)),
				 "n"(3 * SS * (int)sizeof(T)), "n"(4 * DS * (int)sizeof(T)), "n"(4 * SS * (int)sizeof(T)),
				 "n"(5 * DS * (int)sizeof(T)), "n"(5 * SS * (int)sizeof(T))
				 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all()
{
	asm volatile("cp.async.wait_all;" ::: "memory");
}
// three 8-byte values dst[i * DS] = src[i * SS] (strides in 8-byte units)
template <int DS, int SS>
__device__ __forceinline__ void cp_async_3x8(unsigned dst, const void *src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n\t"
				 "cp.async.ca.shared.global [%0+%2], [%1+%3], 8;\n\t"
				 "cp.async.ca.shared.global [%0+%4], [%1+%5], 8;" ::"r"(dst),
				 "l"(src), "n"(8 * DS), "n"(8 * SS), "n"(16 * DS), "n"(16 * SS)
				 : "memory");
}
__device__ __forceinline__ void cp_async_commit()
{
	asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait_group()
{
	asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// bring [p, p + bytes) into L2 (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void prefetch_l2(const void *p, unsigned bytes)
{
	asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Programmatic dependent launch: let the next stage's CTAs start; wait for the
// previous stage (and everything before it) to be complete.
__device__ __forceinline__ void pdl_launch_dependents()
{
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Boundary traces of the three stages of a step, in the stage kernels' precision:
// value rk3_btrace_off(c) of out[((stage * nbf + bf) * 6 + jj) * 6 ..] = w_exact(
// x_{bf,jj}, t + C_stage dt)_c (dg_update_boundary, dg.c:101-104), with the data,
// time and time step of the face's instance.  t is t_in, or with `advance` the next
// step's time t_in + dt, which block 0 keeps in t_out (explicit.c:103).  Times are
// formed with the host's rounding (no fused multiply-add), so every stage sees
// the reference's time bits.  A thread takes the three stages of a face node: the
// trace CTAs have the stage kernel's footprint, so they are to be few (a stage
// per thread: 96^3 FP32 2.39 against 2.33 ms per step).
template <typename T>
__device__ __forceinline__ void rk3_trace_block(const Rk3Trace<T> &tr, int blk)
{
	pdl_wait();
	if (blk == 0 && tr.advance)
		for (int i = threadIdx.x; i < tr.b.ninst; i += blockDim.x)
			tr.t_out[i] = __dadd_rn(tr.t_in[i], tr.b.dt[i]);
	const long long q = blk * (long long)blockDim.x + threadIdx.x, per = tr.nbf * 6;
	if (q >= per)
		return;
	const int inst = tr.b.bfinst ? tr.b.bfinst[q / 6] : 0;
	const double dt = tr.b.dt[inst];
	const double t0 = tr.advance ? __dadd_rn(tr.t_in[inst], dt) : tr.t_in[inst];
	const double x[3] = {tr.bxyz[3 * q], tr.bxyz[3 * q + 1], tr.bxyz[3 * q + 2]};
	const Data d = tr.b.data[inst];
#pragma unroll
	for (int stage = 0; stage < 3; stage++) {
		const double c = stage == 0 ? 0. : (stage == 1 ? 1. / 3. : 3. / 4.);
		double we[6];
		exact_w(d, x, __dadd_rn(t0, __dmul_rn(c, dt)), we);
#pragma unroll
		for (int k = 0; k < 6; k++)
			tr.out[(stage * per + q) * 6 + rk3_btrace_off<T>(k)] = (T)we[k];
	}
}
constexpr int kTraceThreads = 256;
template <typename T>
__global__ void rk3_trace_kernel(Rk3Trace<T> tr)
{
	rk3_trace_block<T>(tr, blockIdx.x);
}
template <typename T>
static int trace_blocks(const Rk3Trace<T> &tr, int threads)
{
	return (int)((tr.nbf * 6 + threads - 1) / threads) + (tr.nbf == 0);
}
template <typename T>
int launch_rk3_traces(const Rk3Trace<T> &tr, cudaStream_t s)
{
	rk3_trace_kernel<T><<<trace_blocks(tr, kTraceThreads), kTraceThreads, 0, s>>>(tr);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}
template int launch_rk3_traces<double>(const Rk3Trace<double> &, cudaStream_t);
template int launch_rk3_traces<float>(const Rk3Trace<float> &, cudaStream_t);

// a stage launch: nblk tile CTAs and, on the last stage of a step, the trace CTAs
template <typename T>
static int launch_stage(void (*kernel)(Rk3Params<T>), Rk3Params<T> p, unsigned nblk, int threads, int smem,
						cudaStream_t s)
{
	p.tile_blocks = (int)nblk;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(nblk + (p.traces ? trace_blocks(p.tr, threads) : 0));
	cfg.blockDim = dim3(threads);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	GDN_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p));
	return GDN_CUDA_OK;
}

template <typename T>
struct Rk3Smem {
	static constexpr int P = 33;
	// sX: (field*2 + which)*10 + node, 120 rows (table-product path only);
	// sF: (face*6 + jj)*6 + c, 144 rows
	static constexpr int bytes = (120 + 144) * P * (int)sizeof(T);
	static constexpr int bytes_fact = 144 * P * (int)sizeof(T);
};

// The two variants of rk3_stage_kernel: register cap (minimum
// resident CTAs per SM) and how the neighbour traces are prefetched (rk3_tile).
// FP32 runs it only for tables without the P2 symmetry.
template <typename T>
struct Rk3Variants;
template <>
struct Rk3Variants<float> {
	static constexpr int lo = 4, hi = 5;
	// PF_NONE: with PF_ASYNC and the flux in packed pairs the best variant is no faster
	// (ms per step, so / with them: 11^3 0.0217 / 0.0221, 27^3 0.125 / 0.129, 48^3
	// 0.633 / 0.637; every table entry used: 0.0230 / 0.0230, 0.134 / 0.136, 0.682 / 0.676)
	static constexpr int pf_lo = 0, pf_hi = 0;
};
template <>
struct Rk3Variants<double> {
	static constexpr int lo = 2, hi = 3;
	static constexpr int pf_lo = 1, pf_hi = 2; // PF_REG at 2 CTAs per SM, PF_ASYNC at 3
};

// Upwind flux with the halving folded into the face quantities: with
// s = wR + wL, d = wR - wL, n2 = n / 2 and r2 = r / 2 (r = 1 / |n|),
//   F_E = -n2 x s_H + r2 (n (n . d_E) - |n|^2 d_E),  F_H = n2 x s_E + r2 (n (n . d_H) - |n|^2 d_H),
// the flux of maxwell_num_flux_upwind (src/models/maxwell.c:152-192) up to rounding.
template <typename T>
__device__ __forceinline__ void upwind_flux_h(const T wL[6], const T wR[6], const T n[3], T F[6])
{
	const T nn = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
	const T r2 = T(0.5) * inv_norm_eps(nn);
	const T h[3] = {T(0.5) * n[0], T(0.5) * n[1], T(0.5) * n[2]};
	T sE[3], sH[3], dE[3], dH[3];
#pragma unroll
	for (int k = 0; k < 3; k++) {
		sE[k] = wR[k] + wL[k];
		sH[k] = wR[3 + k] + wL[3 + k];
		dE[k] = wR[k] - wL[k];
		dH[k] = wR[3 + k] - wL[3 + k];
	}
	const T nE = n[0] * dE[0] + n[1] * dE[1] + n[2] * dE[2];
	const T nH = n[0] * dH[0] + n[1] * dH[1] + n[2] * dH[2];
	F[0] = -(h[1] * sH[2] - h[2] * sH[1]) + r2 * (n[0] * nE - nn * dE[0]);
	F[1] = -(h[2] * sH[0] - h[0] * sH[2]) + r2 * (n[1] * nE - nn * dE[1]);
	F[2] = -(h[0] * sH[1] - h[1] * sH[0]) + r2 * (n[2] * nE - nn * dE[2]);
	F[3] = (h[1] * sE[2] - h[2] * sE[1]) + r2 * (n[0] * nH - nn * dH[0]);
	F[4] = (h[2] * sE[0] - h[0] * sE[2]) + r2 * (n[1] * nH - nn * dH[1]);
	F[5] = (h[0] * sE[1] - h[1] * sE[0]) + r2 * (n[2] * nH - nn * dH[2]);
}

// One tile of 32 elements, phases 1-3 (all threads of the CTA call it: it
// holds the barrier between phases 2 and 3).  Wt[k * 32] is value k of this
// lane's element (global memory or a shared-memory copy of the tile), Gt[q *
// 32] its geometry value q, Kin[k * 32] its k2 value k; nbp / pmp point at its
// neighbour and face-node permutation rows.
// Neighbour-trace prefetch: none (loaded in the flux phase), into registers
// at the start, or copied asynchronously into shared memory at the start.
enum { PF_NONE = 0, PF_REG = 1, PF_ASYNC = 2 };

template <typename T, bool SPARSE, bool FACT, int PF, bool METAL>
__device__ __forceinline__ void rk3_tile(const Rk3Params<T> &p, long long tile, const T *Wt, const T *Gt,
										 const T *Kin, const int4 *nbp, const int4 *pmp, T *sX, T *sF)
{
	constexpr int P = Rk3Smem<T>::P;
	const Tables<T> &tb = tab<T>();
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const long long e = tile * 32 + lane;
	const bool live = e < p.ne;

	int nbk[4] = {0, 0, 0, 0}, pmk[4] = {0, 0, 0, 0};
	T cod[3][3], det = T(1);
	// neighbour traces of this thread's flux slot (face node jj = warp) of face f.
	// Plain loads: the stage before may still be writing w_in and btrace when this
	// grid starts, which the read-only path (__ldg) does not allow.
	auto load_wR = [&](int f, T out[6]) {
		const int nbv = nbk[f];
		const int jj = warp;
		if (nbv >= 0) {
			const int qn = (pmk[f] >> (4 * jj)) & 15;
			const T *g = p.w_in + rk3_tix<T>(nbv, qn * 6);
#pragma unroll
			for (int c = 0; c < 6; c++)
				out[c] = g[rk3_off<T>(0, c)];
		} else {
			const T *g = p.btrace + ((long long)(-nbv - 1) * 6 + jj) * 6;
#pragma unroll
			for (int c = 0; c < 6; c++)
				out[c] = g[rk3_btrace_off<T>(c)];
		}
	};
	// Prefetched at the start so that the volume phase hides their latency:
	// PF_REG into registers, PF_ASYNC into this thread's own flux slots of sF
	// ((f * 6 + jj) * 6 + c, the slots its flux later overwrites).
	T wR[PF == PF_REG ? 4 : 1][6];
	if (live) {
		const int4 nb4 = *nbp;
		const int4 pm4 = *pmp;
		nbk[0] = nb4.x, nbk[1] = nb4.y, nbk[2] = nb4.z, nbk[3] = nb4.w;
		pmk[0] = pm4.x, pmk[1] = pm4.y, pmk[2] = pm4.z, pmk[3] = pm4.w;
		if (PF == PF_REG) {
#pragma unroll
			for (int f = 0; f < 4; f++)
				load_wR(f, wR[PF == PF_REG ? f : 0]);
		}
		if (PF == PF_ASYNC) {
#pragma unroll
			for (int f = 0; f < 4; f++) {
				const int nbv = nbk[f];
				T *d = sF + ((f * 6 + warp) * 6) * P + lane;
				// constant strides in each branch, so the six copies use
				// immediate offsets; 32-bit tile offsets when the state fits
				if (nbv >= 0) {
					const unsigned qn = ((unsigned)pmk[f] >> (4 * warp)) & 15u;
					const T *g = p.idx32 ? p.w_in + (((unsigned)nbv >> 5) * 1920u + qn * 192u + ((unsigned)nbv & 31u))
										 : p.w_in + rk3_tix<T>(nbv, (int)qn * 6);
					cp_async_6<T, P, 32>(d, g);
				} else {
					const T *g = p.btrace + ((long long)(-nbv - 1) * 6 + warp) * 6;
					cp_async_6<T, P, 1>(d, g);
				}
			}
		}
#pragma unroll
		for (int r = 0; r < 3; r++)
#pragma unroll
			for (int q = 0; q < 3; q++)
				cod[r][q] = Gt[(3 * r + q) * 32];
		det = Gt[9 * 32];
	}

	// ---- 1: field c = warp in registers (kept for the RK update); the
	// table-product path also computes its two physical derivatives for the
	// curl into sX (FACT computes the curl's derivatives in phase 3) ----
	const int c = warp;
	const int a = c % 3;
	T w[10];
	if (live) {
#pragma unroll
		for (int j = 0; j < 10; j++)
			w[j] = Wt[rk3_off<T>(j, c)];
	}
	if (!FACT && live) {
		const int d1 = (a + 1) % 3, d2 = (a + 2) % 3;
		T cd1[3], cd2[3];
#pragma unroll
		for (int k = 0; k < 3; k++) {
			cd1[k] = d1 == 0 ? cod[0][k] : (d1 == 1 ? cod[1][k] : cod[2][k]);
			cd2[k] = d2 == 0 ? cod[0][k] : (d2 == 1 ? cod[1][k] : cod[2][k]);
		}
		{
			T r[3][10];
			ref_derivatives<T, SPARSE>(tb, w, r);
#pragma unroll
			for (int i = 0; i < 10; i++) {
				sX[((c * 2 + 0) * 10 + i) * P + lane] = cd1[0] * r[0][i] + cd1[1] * r[1][i] + cd1[2] * r[2][i];
				sX[((c * 2 + 1) * 10 + i) * P + lane] = cd2[0] * r[0][i] + cd2[1] * r[1][i] + cd2[2] * r[2][i];
			}
		}
	}

	// ---- 2: upwind flux at face node jj = warp of the 4 faces ----
	if (live) {
		const int jj = warp;
#pragma unroll
		for (int f = 0; f < 4; f++) {
			const int qo = tb.f2n[f][jj]; // warp-uniform: constant-cache broadcast
			T wL[6], vn[3], F[6];
#pragma unroll
			for (int cc = 0; cc < 6; cc++)
				wL[cc] = Wt[rk3_off<T>(qo, cc)];
			// own scaled outward normal codtau . n_ref(f): the reference
			// normals are -e_0, -e_1, -e_2 and (1,1,1)/sqrt(3), face 3 scaled by
			// sqrt(3) (simulation.c:377-395; checked at attach)
#pragma unroll
			for (int a2 = 0; a2 < 3; a2++)
				vn[a2] = f < 3 ? -cod[a2][f] : (cod[a2][0] + cod[a2][1] + cod[a2][2]) * tb.n3scale;
			if (PF == PF_ASYNC) {
				if (f == 0)
					cp_async_wait_all();
#pragma unroll
				for (int cc = 0; cc < 6; cc++)
					wR[0][cc] = sF[((f * 6 + jj) * 6 + cc) * P + lane];
			} else if (PF == PF_NONE) {
				load_wR(f, wR[0]);
			}
			if (METAL && nbk[f] < 0) {
				// maxwell_num_flux_boundary_metal (maxwell.c:205-223)
				F[0] = vn[2] * wL[4] - vn[1] * wL[5];
				F[1] = -vn[2] * wL[3] + vn[0] * wL[5];
				F[2] = -vn[0] * wL[4] + vn[1] * wL[3];
				F[3] = F[4] = F[5] = T(0);
			} else {
				upwind_flux_h<T>(wL, wR[PF == PF_REG ? f : 0], vn, F);
			}
#pragma unroll
			for (int cc = 0; cc < 6; cc++)
				sF[((f * 6 + jj) * 6 + cc) * P + lane] = F[cc];
		}
	}
	T k2o[10];
	T *Kt = p.k2 + tile * 60 * 32 + rk3_lane<T>(lane);
	if (live && !p.stage0) {
#pragma unroll
		for (int i = 0; i < 10; i++)
			k2o[i] = Kin[rk3_off<T>(i, c)];
	}

	__syncthreads();

	// ---- 3: residual of field c, lift, RK update ----
	if (!live)
		return;
	// R_E,b = dH_{b+2}/dx_{b+1} - dH_{b+1}/dx_{b+2};  R_H,b = -(same with E)
	const int X = c / 3, b = a;
	const int fa = 3 * (1 - X) + (b + 2) % 3; // field whose "d2" slot holds d_{b+1}
	const int fb = 3 * (1 - X) + (b + 1) % 3; // field whose "d1" slot holds d_{b+2}
	T R[10];
	if (FACT) {
		// d_{b+1} of field fa and d_{b+2} of field fb through the P1 basis
		// (p1_weak_derivative), their rows read back from the tile (L1)
		T o[2][10];
#pragma unroll
		for (int h = 0; h < 2; h++) {
			const int fld = h ? fb : fa;
			const int d = (b + 1 + h) % 3;
			T wf[10], v[4], t[4], cd[3];
#pragma unroll
			for (int j = 0; j < 10; j++)
				wf[j] = Wt[rk3_off<T>(j, fld)];
			q4_apply_sym<T>(tb, wf, v, t);
#pragma unroll
			for (int k = 0; k < 3; k++)
				cd[k] = d == 0 ? cod[0][k] : (d == 1 ? cod[1][k] : cod[2][k]);
			p1_weak_derivative<T>(cd, v, t, o[h]);
		}
#pragma unroll
		for (int i = 0; i < 10; i++)
			R[i] = X == 0 ? o[0][i] - o[1][i] : o[1][i] - o[0][i];
	} else {
		const T sgn = X == 0 ? T(1) : T(-1);
#pragma unroll
		for (int i = 0; i < 10; i++)
			R[i] = sgn * (sX[((fa * 2 + 1) * 10 + i) * P + lane] - sX[((fb * 2 + 0) * 10 + i) * P + lane]);
	}
#pragma unroll
	for (int f = 0; f < 4; f++) {
		T Fc[6];
#pragma unroll
		for (int jj = 0; jj < 6; jj++)
			Fc[jj] = sF[((f * 6 + jj) * 6 + c) * P + lane];
		if (FACT) {
			// S Fc through the triangle's symmetry (s_sym)
			const T bv = tb.s_sym[1] * ((Fc[0] + Fc[1]) + Fc[2]);
			const T be = tb.s_sym[4] * ((Fc[3] + Fc[4]) + Fc[5]);
#pragma unroll
			for (int ii = 0; ii < 3; ii++)
				R[f2n(f, ii)] += bv + tb.s_sym[0] * Fc[ii] + tb.s_sym[2] * Fc[3 + (ii + 1) % 3];
#pragma unroll
			for (int k = 0; k < 3; k++)
				R[f2n(f, 3 + k)] += be + tb.s_sym[3] * Fc[3 + k] + tb.s_sym[2] * Fc[(k + 2) % 3];
		} else {
#pragma unroll
			for (int ii = 0; ii < 6; ii++) {
				T acc = T(0);
#pragma unroll
				for (int jj = 0; jj < 6; jj++)
					if (!SPARSE || (smask(ii) >> jj & 1))
						acc += tb.S[ii][jj] * Fc[jj];
				R[f2n(f, ii)] += acc;
			}
		}
	}
	const T A = (T)p.A, B = (T)p.B;
	const T dt = p.einst ? (T)p.dt_tab[p.einst[e]] : (T)p.dt;
	const T scale = dt / det;
	T dwv[10];
	if (FACT)
		lift_minv_sym<T>(tb, R, dwv);
	else
		lift_minv<T>(tb, R, dwv);
	T *Wo = p.w_out + tile * 60 * 32 + rk3_lane<T>(lane);
#pragma unroll
	for (int i = 0; i < 10; i++) {
		const T k2 = p.stage0 ? -(scale * dwv[i]) : A * k2o[i] - scale * dwv[i];
		Wo[rk3_off<T>(i, c)] = w[i] + B * k2;
		if (p.write_k2)
			Kt[rk3_off<T>(i, c)] = k2;
	}
}

// One CTA per tile, everything read from global memory.
// MINB resident CTAs per SM: ptxas derives the register cap, including the
// split of the register file between the SM's four schedulers (18 warps of 3
// CTAs leave 5 warps on one scheduler: 96 registers, not 65536 / 576)
template <typename T, bool SPARSE, bool FACT, int MINB, int PF, bool METAL>
__global__ void __launch_bounds__(kRk3Threads, MINB) rk3_stage_kernel(Rk3Params<T> p)
{
	pdl_launch_dependents();
	if ((int)blockIdx.x >= p.tile_blocks) {
		rk3_trace_block<T>(p.tr, blockIdx.x - p.tile_blocks);
		return;
	}
	extern __shared__ __align__(16) unsigned char smem_raw[];
	T *sX = reinterpret_cast<T *>(smem_raw); // [120][P]
	T *sF = FACT ? sX : sX + 120 * Rk3Smem<T>::P; // [144][P] (FACT: no sX)
	const long long tile = blockIdx.x;
	const int lane = threadIdx.x & 31;
	const long long e = tile * 32 + lane;
	const long long ec = e < p.ne ? e : p.ne - 1;
	// the tile that starts on this SM about one CTA lifetime from now (l2_ahead
	// = resident CTAs on the GPU): its state, k2, geometry and neighbour rows
	// into L2, so that its first loads are L2 hits
	if (threadIdx.x == 0 && p.l2_ahead > 0) {
		const long long tn = tile + p.l2_ahead;
		const long long nt = (p.ne + 31) / 32;
		if (tn < nt) {
			const unsigned wb = 60 * 32 * sizeof(T);
			prefetch_l2(p.w_in + tn * 60 * 32, wb);
			if (!p.stage0)
				prefetch_l2(p.k2 + tn * 60 * 32, wb);
			prefetch_l2(p.geom + tn * 10 * 32, 10 * 32 * sizeof(T));
			const unsigned nbb = (unsigned)((p.ne - tn * 32 < 32 ? p.ne - tn * 32 : 32) * 16);
			prefetch_l2(p.nb + tn * 32 * 4, nbb);
			prefetch_l2(p.perm + tn * 32 * 4, nbb);
		}
	}
	const T *Wt = p.w_in + tile * 60 * 32 + rk3_lane<T>(lane);
	pdl_wait();
	rk3_tile<T, SPARSE, FACT, PF, METAL>(p, tile, Wt, p.geom + tile * 10 * 32 + lane, p.k2 + tile * 60 * 32 + rk3_lane<T>(lane),
										 reinterpret_cast<const int4 *>(p.nb) + ec,
										 reinterpret_cast<const int4 *>(p.perm) + ec, sX, sF);
}

// FP32 stage kernel: a thread per element, a warp per tile, no barrier.
// With the same symmetric products the stage kernel above was bound by L1
// wavefronts and instruction issue: its six warps per tile exchange the fluxes through shared memory (432 rows) and
// read the geometry six and the own state three times.  One thread that holds
// all six fields of its element reads every value once, and the (E_c, H_c) pairs
// of the layout make every step of the residual, which treats E and H alike,
// packed FP32x2 arithmetic (the flux, the face mass, the derivatives, the lift
// and the update): 64-bit rows instead of 32-bit ones, 2,100 instead of 6,670
// warp instructions and 720 instead of 1,784 L1 wavefronts per tile and stage.
// The neighbour traces (72 pairs) are copied into the lane's own slots of shared
// memory asynchronously, a group per face: they are in flight while the curl is
// computed and hold no register.  k2 stays in registers (copying it too: 2.64 ms
// per 96^3 step against 2.34).  It is bound by DRAM: 8 warps per SM at 182
// registers reach 90 % of the copy bandwidth at 96^3 by the bytes of its own
// (600 values, 30 of the geometry and 96 bytes of connectivity per element and
// step); 12 warps at 168 registers spill.  ms per step, rk3_stage_kernel at 7 launches / this kernel
// at 3: 27^3 0.125 / 0.074, 48^3 0.556 / 0.306, 96^3 4.27 / 2.33.
constexpr int kElemThreads = 128;
struct Rk3Elem {
	static constexpr int lo = 2, hi = 3; // CTAs per SM: 182 / 168 registers
	static constexpr int smem = kElemThreads / 32 * 72 * 256;
};

__device__ __forceinline__ float2 dup2(float a)
{
	return make_float2(a, a);
}

template <bool METAL, int MINB>
__global__ void __launch_bounds__(kElemThreads, MINB) rk3_elem_kernel(Rk3Params<float> p)
{
	pdl_launch_dependents();
	if ((int)blockIdx.x >= p.tile_blocks) {
		rk3_trace_block<float>(p.tr, blockIdx.x - p.tile_blocks);
		return;
	}
	const Tables<float> &tb = tab<float>();
	const int lane = threadIdx.x & 31;
	const long long tile = blockIdx.x * (long long)(kElemThreads / 32) + (threadIdx.x >> 5);
	const long long e = tile * 32 + lane;
	if (e >= p.ne)
		return;
	if (lane == 0 && p.l2_ahead > 0) {
		const long long tn = tile + p.l2_ahead;
		if (tn * 32 < p.ne) {
			prefetch_l2(p.w_in + tn * 1920, 7680);
			if (!p.stage0)
				prefetch_l2(p.k2 + tn * 1920, 7680);
			prefetch_l2(p.geom + tn * 320, 1280);
			const unsigned nbb = (unsigned)((p.ne - tn * 32 < 32 ? p.ne - tn * 32 : 32) * 16);
			prefetch_l2(p.nb + tn * 128, nbb);
			prefetch_l2(p.perm + tn * 128, nbb);
		}
	}
	const float2 *W = reinterpret_cast<const float2 *>(p.w_in) + tile * 960 + lane;
	const int4 nb4 = reinterpret_cast<const int4 *>(p.nb)[e];
	const int4 pm4 = reinterpret_cast<const int4 *>(p.perm)[e];
	float2 w[10][3], R[10][3];
	float cod[3][3];
	const float *Gt = p.geom + tile * 320 + lane;
#pragma unroll
	for (int r = 0; r < 3; r++)
#pragma unroll
		for (int q = 0; q < 3; q++)
			cod[r][q] = Gt[(3 * r + q) * 32];

	const float det = Gt[9 * 32];
	const float dt = p.einst ? (float)p.dt_tab[p.einst[e]] : (float)p.dt;
	pdl_wait();
#pragma unroll
	for (int i = 0; i < 10; i++)
#pragma unroll
		for (int a = 0; a < 3; a++)
			w[i][a] = W[(i * 3 + a) * 32];
	// neighbour traces: pair a of node jj of face f at tr[(f * 18 + jj * 3 + a) * 32]
	const int nbk[4] = {nb4.x, nb4.y, nb4.z, nb4.w}, pmk[4] = {pm4.x, pm4.y, pm4.z, pm4.w};
	extern __shared__ __align__(16) float2 shf[];
	float2 *tr = shf + (threadIdx.x >> 5) * 72 * 32 + lane;
	{
		const unsigned dst = smem_u32(tr);
#pragma unroll
		for (int f = 0; f < 4; f++) {
			const int nbv = nbk[f];
			if (nbv >= 0) {
				const float2 *g = reinterpret_cast<const float2 *>(p.w_in) + (long long)(nbv >> 5) * 960 + (nbv & 31);
#pragma unroll
				for (int jj = 0; jj < 6; jj++)
					cp_async_3x8<32, 32>(dst + (f * 18 + jj * 3) * 256, g + ((pmk[f] >> (4 * jj)) & 15) * 96);
			} else {
				const float2 *g = reinterpret_cast<const float2 *>(p.btrace) + (long long)(-nbv - 1) * 18;
#pragma unroll
				for (int jj = 0; jj < 6; jj++)
					cp_async_3x8<32, 1>(dst + (f * 18 + jj * 3) * 256, g + 3 * jj);
			}
			cp_async_commit();
		}
	}

	// ---- curl: R_E += curl H, R_H -= curl E.  Component a of (H, -E) goes along
	// direction a + 2 to component a + 1 and along a + 1, negated, to a + 2 ----
#pragma unroll
	for (int a = 0; a < 3; a++) {
		// v = Q4 x, t = v - sum(v) / 4 (q4_apply_sym) of the pairs (E_a, H_a)
		const float2 sv = __fadd2_rn(__fadd2_rn(w[0][a], w[1][a]), __fadd2_rn(w[2][a], w[3][a]));
		const float2 se = __fadd2_rn(__fadd2_rn(__fadd2_rn(w[4][a], w[5][a]), __fadd2_rn(w[6][a], w[7][a])),
									 __fadd2_rn(w[8][a], w[9][a]));
		const float2 base = __ffma2_rn(dup2(tb.q4_sym[0]), sv, __fmul2_rn(dup2(tb.q4_sym[1]), se));
		const float2 s = __ffma2_rn(dup2(tb.q4_sym[4]), sv, __fmul2_rn(dup2(tb.q4_sym[5]), se));
		float2 v[4], t[4];
#pragma unroll
		for (int l = 0; l < 4; l++) {
			float2 ev = make_float2(0.f, 0.f);
			bool first = true;
#pragma unroll
			for (int ed = 0; ed < 6; ed++)
				if (edge_end(ed, 0) == l || edge_end(ed, 1) == l) {
					ev = first ? w[4 + ed][a] : __fadd2_rn(ev, w[4 + ed][a]);
					first = false;
				}
			const float2 x =
				__ffma2_rn(dup2(tb.q4_sym[3]), ev, __ffma2_rn(dup2(tb.q4_sym[2]), w[l][a], base));
			v[l] = make_float2(x.y, -x.x); // (H, -E)
			t[l] = make_float2(x.y - s.y, s.x - x.x);
		}
#pragma unroll
		for (int h = 0; h < 2; h++) {
			const int d = (a + 2 - h) % 3, to = (a + 1 + h) % 3; // direction, component of R
			const float sg = h ? -1.f : 1.f;
			const float g1 = sg * cod[d][0], g2 = sg * cod[d][1], g3 = sg * cod[d][2];
			const float2 g[4] = {dup2(-(g1 + g2 + g3)), dup2(g1), dup2(g2), dup2(g3)};
			// the first contribution to a component of R sets it: component 1 from
			// a = 0 (h = 0), 2 from a = 0 (h = 1), 0 from a = 1 (h = 1)
			const bool set = a == 0 || (a == 1 && h == 1);
#pragma unroll
			for (int i = 0; i < 4; i++)
				R[i][to] = set ? __fmul2_rn(g[i], t[i]) : __ffma2_rn(g[i], t[i], R[i][to]);
#pragma unroll
			for (int ed = 0; ed < 6; ed++) {
				const int i = edge_end(ed, 0), j = edge_end(ed, 1);
				R[4 + ed][to] =
					__ffma2_rn(g[i], v[j], set ? __fmul2_rn(g[j], v[i]) : __ffma2_rn(g[j], v[i], R[4 + ed][to]));
			}
		}
	}

	// ---- faces: R += S F, vertices then edges of the face ----
	const float2 m1 = dup2(-1.f);
#pragma unroll
	for (int f = 0; f < 4; f++) {
		const bool inner = nbk[f] >= 0;
		if (f == 0)
			cp_async_wait_group<3>();
		else if (f == 1)
			cp_async_wait_group<2>();
		else if (f == 2)
			cp_async_wait_group<1>();
		else
			cp_async_wait_group<0>();
		float n[3];
#pragma unroll
		for (int a = 0; a < 3; a++)
			n[a] = f < 3 ? -cod[a][f] : (cod[a][0] + cod[a][1] + cod[a][2]) * tb.n3scale;
		const float rn = inv_norm_eps(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
		// F = h x u, u = m x d + (-s_H, s_E) with h = n / 2, m = n / |n|, d = wR - wL,
		// s = wR + wL: upwind_flux_h with the double cross product factored
#pragma unroll
		for (int half = 0; half < 2; half++) {
			float2 F[3][3];
#pragma unroll
			for (int j = 0; j < 3; j++) {
				const int qo = f2n(f, 3 * half + j);
				float2 d[3], q[3];
#pragma unroll
				for (int a = 0; a < 3; a++) {
					float2 r = tr[(f * 18 + (3 * half + j) * 3 + a) * 32];
					if (METAL && !inner)
						r = w[qo][a]; // no jump: F_E = -n x H_L, F_H set to zero below
					d[a] = __ffma2_rn(w[qo][a], m1, r);
					q[a] = make_float2(-(r.y + w[qo][a].y), r.x + w[qo][a].x);
				}
				float2 u[3];
#pragma unroll
				for (int a = 0; a < 3; a++) {
					const int b = (a + 1) % 3, c = (a + 2) % 3;
					u[a] = __ffma2_rn(dup2(n[b] * rn), d[c], __ffma2_rn(dup2(-n[c] * rn), d[b], q[a]));
				}
#pragma unroll
				for (int a = 0; a < 3; a++) {
					const int b = (a + 1) % 3, c = (a + 2) % 3;
					F[j][a] = __ffma2_rn(dup2(0.5f * n[b]), u[c], __fmul2_rn(dup2(-0.5f * n[c]), u[b]));
					if (METAL && !inner)
						F[j][a].y = 0.f;
				}
			}
			const float2 s_own = dup2(tb.s_sym[half ? 3 : 0]), s_all = dup2(tb.s_sym[half ? 4 : 1]),
						 s_opp = dup2(tb.s_sym[2]);
#pragma unroll
			for (int a = 0; a < 3; a++) {
				const float2 sum = __fmul2_rn(s_all, __fadd2_rn(__fadd2_rn(F[0][a], F[1][a]), F[2][a]));
#pragma unroll
				for (int j = 0; j < 3; j++) {
					// face-local vertex j is opposite the edge 3 + (j + 1) % 3
					const int own = f2n(f, 3 * half + j), opp = f2n(f, half ? (j + 2) % 3 : 3 + (j + 1) % 3);
					R[own][a] = __fadd2_rn(R[own][a], __ffma2_rn(s_own, F[j][a], sum));
					R[opp][a] = __ffma2_rn(s_opp, F[j][a], R[opp][a]);
				}
			}
		}
	}

	// ---- lift (lift_minv_sym) and RK update ----
	const float2 A = dup2((float)p.A), B = dup2((float)p.B), scale = dup2(-(dt / det));
	float2 *K = reinterpret_cast<float2 *>(p.k2) + tile * 960 + lane;
	float2 *Wo = reinterpret_cast<float2 *>(p.w_out) + tile * 960 + lane;
	// k2 of a component is read before the stores of the one before it: the
	// compiler moves no load over a store, and 30 loads behind one another cost
	// as much as the rest of the stage
	float2 ko[10];
	if (!p.stage0) {
#pragma unroll
		for (int i = 0; i < 10; i++)
			ko[i] = K[i * 96];
	}
#pragma unroll
	for (int a = 0; a < 3; a++) {
		const float2 sv = __fadd2_rn(__fadd2_rn(R[0][a], R[1][a]), __fadd2_rn(R[2][a], R[3][a]));
		const float2 se = __fadd2_rn(__fadd2_rn(__fadd2_rn(R[4][a], R[5][a]), __fadd2_rn(R[6][a], R[7][a])),
									 __fadd2_rn(R[8][a], R[9][a]));
		const float2 bv = __ffma2_rn(dup2(tb.minv_sym[0]), sv, __fmul2_rn(dup2(tb.minv_sym[1]), se));
		const float2 be = __ffma2_rn(dup2(tb.minv_sym[1]), sv, __fmul2_rn(dup2(tb.minv_sym[2]), se));
		float2 ev[4];
#pragma unroll
		for (int l = 0; l < 4; l++) {
			bool first = true;
#pragma unroll
			for (int ed = 0; ed < 6; ed++)
				if (edge_end(ed, 0) == l || edge_end(ed, 1) == l) {
					ev[l] = first ? R[4 + ed][a] : __fadd2_rn(ev[l], R[4 + ed][a]);
					first = false;
				}
		}
		float2 kn[10];
#pragma unroll
		for (int i = 0; i < 10; i++) {
			float2 dw;
			if (i < 4) {
				dw = __ffma2_rn(dup2(tb.minv_sym[4]), ev[i], __ffma2_rn(dup2(tb.minv_sym[3]), R[i][a], bv));
			} else {
				const int l = edge_end(i - 4, 0), m = edge_end(i - 4, 1);
				dw = __ffma2_rn(dup2(tb.minv_sym[4]), __fadd2_rn(R[l][a], R[m][a]), be);
				dw = __ffma2_rn(dup2(tb.minv_sym[5]), R[i][a], dw);
				dw = __ffma2_rn(dup2(tb.minv_sym[6]), __fadd2_rn(ev[l], ev[m]), dw);
			}
			kn[i] = __fmul2_rn(scale, dw);
			if (!p.stage0)
				kn[i] = __ffma2_rn(A, ko[i], kn[i]);
		}
		if (!p.stage0 && a < 2) {
#pragma unroll
			for (int i = 0; i < 10; i++)
				ko[i] = K[(i * 3 + a + 1) * 32];
		}
#pragma unroll
		for (int i = 0; i < 10; i++) {
			Wo[(i * 3 + a) * 32] = __ffma2_rn(B, kn[i], w[i][a]);
			if (p.write_k2)
				K[(i * 3 + a) * 32] = kn[i];
		}
	}
}

// FP64 stage kernel: two warps per tile, one holding E and one holding H of its
// 32 elements (a thread per element and half, everything of the half in
// registers).  A half X reads only its own three fields, of its element and of
// the neighbours, and computes from them what they give to both residuals:
//   to its own    Q = sum_faces S (h x (m x d_X)),
//   to the other  P = -curl X + sum_faces S (h x s_X)   (negated by the H half),
// with h = n / 2, m = n / |n|, d = xR - xL, s = xR + xL (upwind_flux_h: F_E = h x
// (m x d_E - s_H), F_H = h x (m x d_H + s_E)).  The halves exchange P through
// shared memory, then lift and update their own fields.
// The neighbour traces come by asynchronous copies into the lane's own slots of
// shared memory, as in rk3_elem_kernel; P then takes their place.
// rk3_stage_kernel is bound by L1 wavefronts (3,755 per tile and stage, 79 % of
// the pipe) with FP64 arithmetic at a third of its rate.  ms per step, it / this
// kernel, both on the reordered elements: 24^3 0.151 / 0.113, 48^3 0.93 / 0.763.
// What is left is latency: 254 registers leave 8 warps per SM.
constexpr int kHalfThreads = 64;
struct Rk3Half {
	static constexpr int ctas = 4; // per SM: 254 registers
	static constexpr int smem = 2 * 72 * 32 * (int)sizeof(double);
};

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double o[3])
{
	o[0] = a[1] * b[2] - a[2] * b[1];
	o[1] = a[2] * b[0] - a[0] * b[2];
	o[2] = a[0] * b[1] - a[1] * b[0];
}

template <bool METAL>
__global__ void __launch_bounds__(kHalfThreads, Rk3Half::ctas) rk3_half_kernel(Rk3Params<double> p)
{
	pdl_launch_dependents();
	if ((int)blockIdx.x >= p.tile_blocks) {
		rk3_trace_block<double>(p.tr, blockIdx.x - p.tile_blocks);
		return;
	}
	extern __shared__ __align__(16) double sh[];
	const Tables<double> &tb = tab<double>();
	const int lane = threadIdx.x & 31, X = threadIdx.x >> 5;
	const long long tile = blockIdx.x;
	const long long e = tile * 32 + lane;
	const bool live = e < p.ne;
	const long long ec = live ? e : p.ne - 1;
	if (threadIdx.x == 0 && p.l2_ahead > 0) {
		const long long tn = tile + p.l2_ahead;
		if (tn * 32 < p.ne) {
			prefetch_l2(p.w_in + tn * 1920, 15360);
			if (!p.stage0)
				prefetch_l2(p.k2 + tn * 1920, 15360);
			prefetch_l2(p.geom + tn * 320, 2560);
			const unsigned nbb = (unsigned)((p.ne - tn * 32 < 32 ? p.ne - tn * 32 : 32) * 16);
			prefetch_l2(p.nb + tn * 128, nbb);
			prefetch_l2(p.perm + tn * 128, nbb);
		}
	}
	const int4 nb4 = reinterpret_cast<const int4 *>(p.nb)[ec];
	const int4 pm4 = reinterpret_cast<const int4 *>(p.perm)[ec];
	const int nbk[4] = {nb4.x, nb4.y, nb4.z, nb4.w}, pmk[4] = {pm4.x, pm4.y, pm4.z, pm4.w};
	const double *W = p.w_in + tile * 1920 + X * 96 + lane;
	double w[10][3];
	double cod[3][3];
	const double *Gt = p.geom + tile * 320 + lane;
#pragma unroll
	for (int r = 0; r < 3; r++)
#pragma unroll
		for (int q = 0; q < 3; q++)
			cod[r][q] = Gt[(3 * r + q) * 32];
	pdl_wait();
#pragma unroll
	for (int i = 0; i < 10; i++)
#pragma unroll
		for (int a = 0; a < 3; a++)
			w[i][a] = W[(i * 6 + a) * 32];
	// neighbour traces: value a of node jj of face f at tr[(f * 18 + jj * 3 + a) * 32]
	double *tr = sh + X * 72 * 32 + lane;
	{
		const unsigned dst = smem_u32(tr);
#pragma unroll
		for (int f = 0; f < 4; f++) {
			const int nbv = nbk[f];
			if (nbv >= 0) {
				const double *g = p.w_in + (long long)(nbv >> 5) * 1920 + X * 96 + (nbv & 31);
#pragma unroll
				for (int jj = 0; jj < 6; jj++)
					cp_async_3x8<32, 32>(dst + (f * 18 + jj * 3) * 256, g + ((pmk[f] >> (4 * jj)) & 15) * 192);
			} else {
				const double *g = p.btrace + (long long)(-nbv - 1) * 36 + X * 3;
#pragma unroll
				for (int jj = 0; jj < 6; jj++)
					cp_async_3x8<32, 1>(dst + (f * 18 + jj * 3) * 256, g + 6 * jj);
			}
			cp_async_commit();
		}
	}

	// ---- P = -curl X: component a goes along direction a + 2, negated, to
	// component a + 1 and along a + 1 to a + 2 ----
	double P[10][3], Q[10][3];
#pragma unroll
	for (int a = 0; a < 3; a++) {
		double x[10], v[4], t[4];
#pragma unroll
		for (int i = 0; i < 10; i++)
			x[i] = w[i][a];
		q4_apply_sym<double>(tb, x, v, t);
#pragma unroll
		for (int h = 0; h < 2; h++) {
			const int d = (a + 2 - h) % 3, to = (a + 1 + h) % 3;
			const double sg = h ? 1.0 : -1.0;
			const double g1 = sg * cod[d][0], g2 = sg * cod[d][1], g3 = sg * cod[d][2];
			const double g[4] = {-(g1 + g2 + g3), g1, g2, g3};
			const bool set = a == 0 || (a == 1 && h == 1); // first contribution to the component
#pragma unroll
			for (int i = 0; i < 4; i++)
				P[i][to] = set ? g[i] * t[i] : P[i][to] + g[i] * t[i];
#pragma unroll
			for (int ed = 0; ed < 6; ed++) {
				const int i = edge_end(ed, 0), j = edge_end(ed, 1);
				P[4 + ed][to] = g[i] * v[j] + (set ? g[j] * v[i] : P[4 + ed][to] + g[j] * v[i]);
			}
		}
	}
#pragma unroll
	for (int i = 0; i < 10; i++)
#pragma unroll
		for (int a = 0; a < 3; a++)
			Q[i][a] = 0.0;

	// ---- faces: P += S (h x s), Q += S (h x (m x d)), vertices then edges ----
#pragma unroll
	for (int f = 0; f < 4; f++) {
		double h[3], m[3];
		{
			double n[3];
#pragma unroll
			for (int a = 0; a < 3; a++)
				n[a] = f < 3 ? -cod[a][f] : (cod[a][0] + cod[a][1] + cod[a][2]) * tb.n3scale;
			const double rn = inv_norm_eps(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
#pragma unroll
			for (int a = 0; a < 3; a++) {
				h[a] = 0.5 * n[a];
				m[a] = rn * n[a];
			}
		}
		const bool metal = METAL && nbk[f] < 0;
		if (f == 0)
			cp_async_wait_group<3>();
		else if (f == 1)
			cp_async_wait_group<2>();
		else if (f == 2)
			cp_async_wait_group<1>();
		else
			cp_async_wait_group<0>();
#pragma unroll
		for (int half = 0; half < 2; half++) {
			double FP[3][3], FQ[3][3];
#pragma unroll
			for (int j = 0; j < 3; j++) {
				const int qo = f2n(f, 3 * half + j);
				double sx[3], dx[3], md[3];
#pragma unroll
				for (int a = 0; a < 3; a++) {
					// metal: no jump; E gives nothing to H, H gives -n x H_L to E
					const double xr = metal ? (X == 0 ? -w[qo][a] : w[qo][a]) : tr[(f * 18 + (3 * half + j) * 3 + a) * 32];
					sx[a] = xr + w[qo][a];
					dx[a] = metal ? 0.0 : xr - w[qo][a];
				}
				cross3(h, sx, FP[j]);
				cross3(m, dx, md);
				cross3(h, md, FQ[j]);
			}
			const double s_own = tb.s_sym[half ? 3 : 0], s_all = tb.s_sym[half ? 4 : 1], s_opp = tb.s_sym[2];
#pragma unroll
			for (int a = 0; a < 3; a++) {
				const double sp = s_all * ((FP[0][a] + FP[1][a]) + FP[2][a]);
				const double sq = s_all * ((FQ[0][a] + FQ[1][a]) + FQ[2][a]);
#pragma unroll
				for (int j = 0; j < 3; j++) {
					// face-local vertex j is opposite the edge 3 + (j + 1) % 3
					const int own = f2n(f, 3 * half + j), opp = f2n(f, half ? (j + 2) % 3 : 3 + (j + 1) % 3);
					P[own][a] += sp + s_own * FP[j][a];
					P[opp][a] += s_opp * FP[j][a];
					Q[own][a] += sq + s_own * FQ[j][a];
					Q[opp][a] += s_opp * FQ[j][a];
				}
			}
		}
	}

	// ---- exchange P (the lane's traces are used up); k2 is on its way meanwhile ----
#pragma unroll
	for (int i = 0; i < 10; i++)
#pragma unroll
		for (int a = 0; a < 3; a++)
			tr[(i * 3 + a) * 32] = P[i][a];
	const double scale = (p.einst ? p.dt_tab[p.einst[ec]] : p.dt) / Gt[9 * 32];
	double *K = p.k2 + tile * 1920 + X * 96 + lane;
	double ko[10][3];
	if (!p.stage0) {
#pragma unroll
		for (int i = 0; i < 10; i++)
#pragma unroll
			for (int a = 0; a < 3; a++)
				ko[i][a] = K[(i * 6 + a) * 32];
	}
	__syncthreads();
	if (!live)
		return;
	const double *oth = sh + (1 - X) * 72 * 32 + lane;
	const double sgn = X == 0 ? -1.0 : 1.0;
	double *Wo = p.w_out + tile * 1920 + X * 96 + lane;
#pragma unroll
	for (int a = 0; a < 3; a++) {
		double R[10], dw[10];
#pragma unroll
		for (int i = 0; i < 10; i++)
			R[i] = Q[i][a] + sgn * oth[(i * 3 + a) * 32];
		lift_minv_sym<double>(tb, R, dw);
#pragma unroll
		for (int i = 0; i < 10; i++) {
			const double k2 = p.stage0 ? -(scale * dw[i]) : p.A * ko[i][a] - scale * dw[i];
			Wo[(i * 6 + a) * 32] = w[i][a] + p.B * k2;
			if (p.write_k2)
				K[(i * 6 + a) * 32] = k2;
		}
	}
}

// P2 structural-zero pattern check for the tables handed to attach.
bool rk3_tables_sparse(const gdn_cuda_tables *t)
{
	for (int k = 0; k < 3; k++)
		for (int i = 0; i < 10; i++)
			for (int j = 0; j < 10; j++)
				if (!(dmask(k, i) >> j & 1) && !(t->internal[i][j][k] < 1e-15 && t->internal[i][j][k] > -1e-15))
					return false;
	for (int i = 0; i < 6; i++)
		for (int j = 0; j < 6; j++)
			if (!(smask(i) >> j & 1) && t->face_scal[i][j] != 0.0)
				return false;
	return true;
}

// Q4[l][j] = 4 int lambda_l phi_j = 4 sum_m lambda_l(x_m) M[m][j] (lambda_l is
// linear, so its P2 interpolant is exact); the vertex diagonal is zero for
// the P2 basis and is set to zero (rk3_tables_factor checks the whole
// product).
void rk3_q4(const gdn_cuda_tables *t, double q4[4][10])
{
	for (int l = 0; l < 4; l++)
		for (int j = 0; j < 10; j++) {
			double acc = t->mass[l][j];
			for (int e = 0; e < 6; e++)
				if (edge_end(e, 0) == l || edge_end(e, 1) == l)
					acc += 0.5 * t->mass[4 + e][j];
			q4[l][j] = j == l ? 0.0 : 4.0 * acc;
		}
}

// How nodes i and j of the P2 tetrahedron sit relative to each other: 0 same
// vertex, 1 two vertices, 2 vertex on the edge, 3 vertex off the edge, 4 same
// edge, 5 edges sharing a vertex, 6 opposite edges.
static int node_pair_kind(int i, int j)
{
	if (i < 4 && j < 4)
		return i == j ? 0 : 1;
	if (i < 4 || j < 4) {
		const int v = i < 4 ? i : j, e = (i < 4 ? j : i) - 4;
		return (edge_end(e, 0) == v || edge_end(e, 1) == v) ? 2 : 3;
	}
	if (i == j)
		return 4;
	const int a0 = edge_end(i - 4, 0), a1 = edge_end(i - 4, 1), b0 = edge_end(j - 4, 0), b1 = edge_end(j - 4, 1);
	return (a0 == b0 || a0 == b1 || a1 == b0 || a1 == b1) ? 5 : 6;
}

// Coefficients of q4_apply_sym and lift_minv_sym from one representative
// entry per kind (rk3_tables_factor checks that every entry equals its kind's).
void rk3_sym_coeffs(const gdn_cuda_tables *t, double q4_sym[6], double minv_sym[7], double s_sym[5])
{
	const double(*S)[6] = t->face_scal; // face nodes: vertices 0-2, edges 01, 12, 20
	s_sym[0] = S[0][0] - S[0][1];
	s_sym[1] = S[0][1];
	s_sym[2] = S[0][4]; // vertex 0 and its opposite edge 12
	s_sym[3] = S[3][3] - S[3][4];
	s_sym[4] = S[3][4];
	double q4[4][10];
	rk3_q4(t, q4);
	const double qa = q4[0][1], qb = q4[0][4], qc = q4[0][5]; // edge 4 = 0-1, edge 5 = 1-2
	q4_sym[0] = qa;
	q4_sym[1] = qc;
	q4_sym[2] = -qa;
	q4_sym[3] = qb - qc;
	q4_sym[4] = 0.75 * qa; // sum_l v_l = 3 qa sv + 2 (qb + qc) se
	q4_sym[5] = 0.5 * (qb + qc);
	const double(*M)[10] = t->inv_mass;
	const double vv0 = M[0][0], vv1 = M[0][1], vin = M[0][4], vout = M[0][5];
	const double ee0 = M[4][4], ee1 = M[4][5], ee2 = M[4][9]; // edges 0-1 / 1-2 / 2-3
	minv_sym[0] = vv1;
	minv_sym[1] = vout;
	minv_sym[2] = ee2;
	minv_sym[3] = vv0 - vv1;
	minv_sym[4] = vin - vout;
	minv_sym[5] = ee0 - 2.0 * ee1 + ee2;
	minv_sym[6] = ee1 - ee2;
}

// The symmetric forms: every entry of Q4 and Minv equals its kind's
// representative (to 1e-15 of the largest entry).
static bool rk3_tables_symmetric(const gdn_cuda_tables *t)
{
	double q4[4][10], qmax = 0.0, mmax = 0.0;
	rk3_q4(t, q4);
	for (int l = 0; l < 4; l++)
		for (int j = 0; j < 10; j++)
			qmax = std::fmax(qmax, std::fabs(q4[l][j]));
	for (int i = 0; i < 10; i++)
		for (int j = 0; j < 10; j++)
			mmax = std::fmax(mmax, std::fabs(t->inv_mass[i][j]));
	const double qrep[4] = {0.0, q4[0][1], q4[0][4], q4[0][5]};
	for (int l = 0; l < 4; l++)
		for (int j = 0; j < 10; j++)
			if (!(std::fabs(q4[l][j] - qrep[node_pair_kind(l, j)]) <= 1e-15 * qmax))
				return false;
	const double(*M)[10] = t->inv_mass;
	const double mrep[7] = {M[0][0], M[0][1], M[0][4], M[0][5], M[4][4], M[4][5], M[4][9]};
	for (int i = 0; i < 10; i++)
		for (int j = 0; j < 10; j++)
			if (!(std::fabs(M[i][j] - mrep[node_pair_kind(i, j)]) <= 1e-15 * mmax))
				return false;
	// face mass: kinds on the P2 triangle (face-local vertex i is opposite the
	// edge 3 + (i + 1) % 3); a vertex and an edge through it: structural zero
	const double(*S)[6] = t->face_scal;
	double smax = 0.0;
	for (int i = 0; i < 6; i++)
		for (int j = 0; j < 6; j++)
			smax = std::fmax(smax, std::fabs(S[i][j]));
	for (int i = 0; i < 6; i++)
		for (int j = 0; j < 6; j++) {
			double rep;
			if (i < 3 && j < 3)
				rep = i == j ? S[0][0] : S[0][1];
			else if (i >= 3 && j >= 3)
				rep = i == j ? S[3][3] : S[3][4];
			else {
				const int v = i < 3 ? i : j, ed = i < 3 ? j : i;
				rep = ed == 3 + (v + 1) % 3 ? S[0][4] : 0.0;
			}
			if (!(std::fabs(S[i][j] - rep) <= 1e-15 * smax))
				return false;
		}
	return true;
}

// D_k[i][j] = sum_l G_k[i][l] Q4[l][j] / 4 with G_k the P1 coefficients of
// d_k(phi_i) (reference vertices 0, e_0, e_1, e_2), to 1e-15; and Q4 and Minv
// have the tetrahedral symmetry the factored kernel uses.
bool rk3_tables_factor(const gdn_cuda_tables *t)
{
	if (!rk3_tables_symmetric(t))
		return false;
	double q4[4][10];
	rk3_q4(t, q4);
	for (int k = 0; k < 3; k++) {
		double dl[4] = {-1.0, 0.0, 0.0, 0.0}; // d_k lambda_l
		dl[k + 1] = 1.0;
		for (int i = 0; i < 10; i++) {
			double G[4] = {0.0, 0.0, 0.0, 0.0};
			if (i < 4) {
				for (int l = 0; l < 4; l++)
					G[l] = dl[i] * (l == i ? 3.0 : -1.0);
			} else {
				const int a = edge_end(i - 4, 0), b = edge_end(i - 4, 1);
				G[a] += 4.0 * dl[b];
				G[b] += 4.0 * dl[a];
			}
			for (int j = 0; j < 10; j++) {
				double d = 0.0;
				for (int l = 0; l < 4; l++)
					d += G[l] * 0.25 * q4[l][j];
				if (!(std::fabs(d - t->internal[i][j][k]) <= 1e-15))
					return false;
			}
		}
	}
	return true;
}

bool rk3_tables_standard_faces(const gdn_cuda_tables *t)
{
	for (int f = 0; f < 4; f++)
		for (int j = 0; j < 6; j++)
			if (t->face2node[f][j] != f2n(f, j))
				return false;
	// reference normals -e_0, -e_1, -e_2, (1, 1, 1)/sqrt(3)
	for (int f = 0; f < 3; f++)
		for (int k = 0; k < 3; k++)
			if (t->ref_normal[f][k] != (k == f ? -1.0 : 0.0))
				return false;
	for (int k = 0; k < 3; k++)
		if (!(std::fabs(t->ref_normal[3][k] - 0.57735026918962576) < 1e-15))
			return false;
	return true;
}

#define GDN_RK3_TRY(expr)                                                                                         \
	do {                                                                                                           \
		int _rc = (expr);                                                                                          \
		if (_rc != GDN_CUDA_OK)                                                                                    \
			return _rc;                                                                                            \
	} while (0)

template <typename T, bool FA>
constexpr int rk3_smem_bytes()
{
	return FA ? Rk3Smem<T>::bytes_fact : Rk3Smem<T>::bytes;
}

template <typename T, bool SP, bool FA, bool METAL>
static int prepare_rk3_one()
{
	typedef Rk3Variants<T> V;
	GDN_CUDA_TRY(cudaFuncSetAttribute(rk3_stage_kernel<T, SP, FA, V::lo, V::pf_lo, METAL>,
									  cudaFuncAttributeMaxDynamicSharedMemorySize, rk3_smem_bytes<T, FA>()));
	GDN_CUDA_TRY(cudaFuncSetAttribute(rk3_stage_kernel<T, SP, FA, V::hi, V::pf_hi, METAL>,
									  cudaFuncAttributeMaxDynamicSharedMemorySize, rk3_smem_bytes<T, FA>()));
	return GDN_CUDA_OK;
}

template <typename K>
static int prepare_rk3_smem(K kernel, int bytes)
{
	GDN_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	return GDN_CUDA_OK;
}

template <typename T>
int prepare_rk3()
{
	if constexpr (sizeof(T) == 8) {
		typedef Rk3Variants<double> V;
		GDN_RK3_TRY(prepare_rk3_smem(rk3_half_kernel<false>, Rk3Half::smem));
		GDN_RK3_TRY(prepare_rk3_smem(rk3_half_kernel<true>, Rk3Half::smem));
		GDN_RK3_TRY(prepare_rk3_smem(rk3_stage_kernel<double, true, true, V::lo, V::pf_lo, false>, rk3_smem_bytes<double, true>()));
		GDN_RK3_TRY(prepare_rk3_smem(rk3_stage_kernel<double, true, true, V::lo, V::pf_lo, true>, rk3_smem_bytes<double, true>()));
	} else {
		GDN_RK3_TRY(prepare_rk3_smem(rk3_elem_kernel<false, Rk3Elem::lo>, Rk3Elem::smem));
		GDN_RK3_TRY(prepare_rk3_smem(rk3_elem_kernel<false, Rk3Elem::hi>, Rk3Elem::smem));
		GDN_RK3_TRY(prepare_rk3_smem(rk3_elem_kernel<true, Rk3Elem::lo>, Rk3Elem::smem));
		GDN_RK3_TRY(prepare_rk3_smem(rk3_elem_kernel<true, Rk3Elem::hi>, Rk3Elem::smem));
	}
	GDN_RK3_TRY((prepare_rk3_one<T, true, false, false>()));
	GDN_RK3_TRY((prepare_rk3_one<T, false, false, false>()));
	GDN_RK3_TRY((prepare_rk3_one<T, true, false, true>()));
	GDN_RK3_TRY((prepare_rk3_one<T, false, false, true>()));
	return GDN_CUDA_OK;
}

template <typename T, bool SP, bool FA, bool METAL>
static int launch_rk3_one(const Rk3Params<T> &pin, int variant, cudaStream_t s)
{
	typedef Rk3Variants<T> V;
	Rk3Params<T> p = pin;
	// L2 prefetch distance: the CTAs resident on the GPU at this variant's cap
	// (FP32), half of them (FP64).  Chosen when this kernel ran the P2 tables in both
	// precisions, in the mesh's own order: 96^3 ms per step, FP32 / FP64, for none,
	// half, one and two times the resident CTAs: 4.35 / 9.45, 4.25 / 9.03, 4.24 /
	// 9.14, 4.32 / 9.67.
	const int resident = p.num_sms * (variant == 0 ? V::lo : V::hi);
	p.l2_ahead = p.l2_ahead ? (sizeof(T) == 8 ? resident / 2 : resident) : 0;
	const unsigned nblk = (unsigned)((p.ne + 31) / 32);
	const int sm = rk3_smem_bytes<T, FA>();
	if constexpr (!FA) // with the P2 symmetry the other variant is rk3_half_kernel
		if (variant != 0)
			return launch_stage<T>(rk3_stage_kernel<T, SP, FA, V::hi, V::pf_hi, METAL>, p, nblk, kRk3Threads, sm, s);
	return launch_stage<T>(rk3_stage_kernel<T, SP, FA, V::lo, V::pf_lo, METAL>, p, nblk, kRk3Threads, sm, s);
}

template <bool METAL>
static int launch_rk3_elem(const Rk3Params<float> &pin, int variant, cudaStream_t s)
{
	Rk3Params<float> p = pin;
	constexpr int tiles = kElemThreads / 32;
	// a quarter of the resident tiles ahead (ms per step for 1/8, 1/4 and 1/2: 48^3
	// 0.328, 0.329, 0.339; 96^3 2.35, 2.34, 2.42; none, before the traces were
	// copied asynchronously: 48^3 0.405 against 0.354)
	p.l2_ahead = p.l2_ahead ? p.num_sms * (variant == 0 ? Rk3Elem::lo : Rk3Elem::hi) : 0;
	const unsigned nblk = (unsigned)(((p.ne + 31) / 32 + tiles - 1) / tiles);
	return launch_stage<float>(variant == 0 ? rk3_elem_kernel<METAL, Rk3Elem::lo> : rk3_elem_kernel<METAL, Rk3Elem::hi>,
							   p, nblk, kElemThreads, Rk3Elem::smem, s);
}

// FP64 with the P2 tables: variant 0 the stage kernel at 2 CTAs of 6 warps per SM,
// variant 1 the half kernel
template <bool METAL>
static int launch_rk3_fp64(const Rk3Params<double> &pin, int variant, cudaStream_t s)
{
	if (variant == 0)
		return launch_rk3_one<double, true, true, METAL>(pin, 0, s);
	Rk3Params<double> p = pin;
	p.l2_ahead = p.l2_ahead ? p.num_sms * Rk3Half::ctas / 2 : 0; // tiles: half of the resident ones
	return launch_stage<double>(rk3_half_kernel<METAL>, p, (unsigned)((p.ne + 31) / 32), kHalfThreads, Rk3Half::smem, s);
}

template <typename T, bool METAL>
static int launch_rk3_tables(const Rk3Params<T> &p, int variant, cudaStream_t s)
{
	if (p.sparse && p.fact) {
		if constexpr (sizeof(T) == 4)
			return launch_rk3_elem<METAL>(p, variant, s);
		else
			return launch_rk3_fp64<METAL>(p, variant, s);
	} else if (p.sparse)
		return launch_rk3_one<T, true, false, METAL>(p, variant, s);
	else
		return launch_rk3_one<T, false, false, METAL>(p, variant, s);
}

// variant 0: register cap for Rk3Variants::lo CTAs per SM, 1: for ::hi
template <typename T>
int launch_rk3_stage(const Rk3Params<T> &p, int variant, cudaStream_t s)
{
	return p.bc_metal ? launch_rk3_tables<T, true>(p, variant, s) : launch_rk3_tables<T, false>(p, variant, s);
}

int rk3_min_blocks(int precision_fp64, int fact, int variant)
{
	if (precision_fp64 && fact)
		return variant == 0 ? Rk3Variants<double>::lo : Rk3Half::ctas;
	if (precision_fp64)
		return variant == 0 ? Rk3Variants<double>::lo : Rk3Variants<double>::hi;
	if (fact)
		return variant == 0 ? Rk3Elem::lo : Rk3Elem::hi;
	return variant == 0 ? Rk3Variants<float>::lo : Rk3Variants<float>::hi;
}

// The variant by the mesh and the device alone: FP64 has two kernels with the P2
// tables, whose sums round differently (1e-15), so that a timing would make equal
// calls give different bits; and a timing of small stages measures their launches
// (FP32 16^3 took variant 1: 0.0266 ms per step against 0.0219).
// Figures are ms per step of variant 0 / 1; "sectors" a gather's (rk3_sectors_kernel).
//   FP32, P2 tables: 0.  3^3 0.0146 / 0.0155, 16^3 0.0219 / 0.0266, 27^3 0.0739 / 0.0782,
//     96^3 2.64 / 2.73; gmsh 14 k elements 0.0246 / 0.0342, 97 k points triangulated
//     0.70 / 1.58, 48^3 numbered at random 1.92 / 4.06 (12 warps per SM crowd one
//     another out of L1 where their gathers touch many sectors).
//   FP64, P2 tables: 1, but 0 while its CTAs are resident at once, for its three times
//     as many warps (4^3 0.0158 / 0.0185, 11^3, 250 tiles, 0.0205 / 0.0246, 12^3, 324,
//     0.0297 / 0.0267, 24^3 0.151 / 0.113; gmsh 452 tiles 0.0369 / 0.0322), and 0 where
//     the gathers go to memory scattered, i.e. over more than 24 sectors of 32 with the
//     state read and the one written beyond L2 (numbered at random, 31.5 sectors: 24^3
//     0.250 / 0.232, 28^3 0.453 / 0.461, 48^3 4.83 / 4.95; 48^3 in blocks of 4 at
//     random, 22.4, 3.42 / 3.51, of 16, 16.1, 1.92 / 1.86; 97 k points triangulated,
//     19.7, 1.69 / 1.61).
//   Other tables: 1, but 0 while its CTAs are resident at once and where a gather takes
//     more than 10 sectors.  FP64 11^3 0.0237 / 0.0309, 12^3 0.0366 / 0.0328, 27^3, 8.4
//     sectors, 0.237 / 0.205, 48^3 in blocks of 64 at random, 10.6, 1.45 / 1.69, at
//     random 4.95 / 8.97; FP32 14^3, 515 tiles, 0.0261 / 0.0299, 16^3, 768, 0.0361 /
//     0.0360, 27^3 0.134 / 0.127, at random 28^3 0.233 / 0.261.
int rk3_default_variant(int precision_fp64, int fact, long long ne, int num_sms, long long l2_bytes,
						unsigned long long sectors)
{
	const long long tiles = (ne + 31) / 32;
	const unsigned long long gathers = 4ull * (unsigned long long)tiles;
	if (!precision_fp64 && fact)
		return 0;
	if (tiles <= (long long)(precision_fp64 ? Rk3Variants<double>::lo : Rk3Variants<float>::lo) * num_sms)
		return 0;
	if (!fact)
		return sectors > 10 * gathers ? 0 : 1;
	return sectors > 24 * gathers && 2 * tiles * 1920 * (long long)sizeof(double) > l2_bytes ? 0 : 1;
}

// Device element order.  The neighbour traces of a warp are one access to the
// same face node of 32 elements' neighbours: coalesced when the 32 elements
// have the same local picture (their neighbours then are of one kind too, side by
// side in the same rows, and the face permutations agree).  Elements whose
// vertices have the same index stencil do, wherever a mesh was built by
// repeating a cell.  Inside each aligned block of kOrderBlock elements the
// elements are grouped by stencil, groups and members in order of first
// appearance.  Elements of different instances never mix (their groups follow one
// another).  192: 32 of each of the six tetrahedra of a cut cube.
// The attach keeps the order only where it lowers the gathers' sectors
// (rk3_sectors_kernel).  An unstructured mesh has elements of one stencil too; their
// neighbours are not side by side, and the order loses the nearness of the mesh's own
// numbering: 97 k points triangulated, 19.4 sectors as numbered and 22.0 ordered, ms
// per step 1.37 against 1.53 (FP64) and 0.61 against 0.66 (FP32).
// Measured on the jittered Kuhn cubes (every element kind in each block): L1
// wavefronts per 48^3 FP32 stage 18.7 M -> 9.1 M, ms per step 96^3 FP32 3.00 ->
// 2.68, 48^3 FP64 1.06 -> 0.93 (the kernels of the time).
constexpr int kOrderBlock = 192;
__global__ void rk3_order_kernel(const int *__restrict__ e2q, const int *__restrict__ einst, long long ne,
								 int *__restrict__ pos, int *__restrict__ items)
{
	__shared__ int4 sig[kOrderBlock];
	__shared__ int first[kOrderBlock];
	const int t = threadIdx.x;
	const long long e = blockIdx.x * (long long)kOrderBlock + t;
	const int n = (int)(ne - blockIdx.x * (long long)kOrderBlock < kOrderBlock ? ne - blockIdx.x * (long long)kOrderBlock
																			   : kOrderBlock);
	int4 me = make_int4(0, 0, 0, 0);
	if (t < n) {
		const int *q = e2q + 10 * e;
		me = make_int4(q[1] - q[0], q[2] - q[0], q[3] - q[0], einst ? einst[e] : 0);
		sig[t] = me;
	}
	__syncthreads();
	int f = t;
	if (t < n) {
		for (int j = 0; j < t; j++) {
			const int4 o = sig[j];
			if (o.x == me.x && o.y == me.y && o.z == me.z && o.w == me.w) {
				f = j;
				break;
			}
		}
		first[t] = f;
	}
	__syncthreads();
	if (t >= n)
		return;
	int r = 0;
	for (int j = 0; j < n; j++)
		r += first[j] < f || (first[j] == f && j < t);
	const int k = (int)(blockIdx.x * (long long)kOrderBlock) + r;
	pos[e] = k;
	items[k] = (int)e;
}

// neighbour and permutation rows into the device order
__global__ void rk3_permute_kernel(const int4 *__restrict__ nb, const int4 *__restrict__ perm,
								   const int *__restrict__ pos, long long ne, int4 *__restrict__ nb_out,
								   int4 *__restrict__ perm_out)
{
	const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (e >= ne)
		return;
	int4 n = nb[e];
	n.x = n.x >= 0 ? pos[n.x] : n.x;
	n.y = n.y >= 0 ? pos[n.y] : n.y;
	n.z = n.z >= 0 ? pos[n.z] : n.z;
	n.w = n.w >= 0 ? pos[n.w] : n.w;
	const int k = pos[e];
	nb_out[k] = n;
	perm_out[k] = perm[e];
}

int launch_rk3_order(const int *e2q, const int *einst, const int *nb, const int *perm, long long ne, int *pos,
					 int *items, int *nb_out, int *perm_out, cudaStream_t s)
{
	rk3_order_kernel<<<(unsigned)((ne + kOrderBlock - 1) / kOrderBlock), kOrderBlock, 0, s>>>(e2q, einst, ne, pos, items);
	GDN_CUDA_TRY(cudaGetLastError());
	rk3_permute_kernel<<<(unsigned)((ne + 255) / 256), 256, 0, s>>>(
		reinterpret_cast<const int4 *>(nb), reinterpret_cast<const int4 *>(perm), pos, ne,
		reinterpret_cast<int4 *>(nb_out), reinterpret_cast<int4 *>(perm_out));
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

// the mesh's own order
__global__ void rk3_natural_order_kernel(long long ne, int *__restrict__ pos, int *__restrict__ items)
{
	const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (e < ne)
		pos[e] = items[e] = (int)e;
}

int launch_rk3_natural_order(long long ne, int *pos, int *items, cudaStream_t s)
{
	rk3_natural_order_kernel<<<(unsigned)((ne + 255) / 256), 256, 0, s>>>(ne, pos, items);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

// 32-byte sectors of the state that the gathers of one face node touch (four
// elements of a row), summed over tiles and faces: 8 of each where the neighbours
// of a tile lie side by side, up to 32 where nothing does
__global__ void rk3_sectors_kernel(const int4 *__restrict__ nb, const int4 *__restrict__ perm, long long ne,
								   unsigned long long *__restrict__ count)
{
	const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	const int lane = threadIdx.x & 31;
	const long long ec = e < ne ? e : ne - 1;
	const int4 n = nb[ec], pm = perm[ec];
	const int nbk[4] = {n.x, n.y, n.z, n.w}, pmk[4] = {pm.x, pm.y, pm.z, pm.w};
	int total = 0;
#pragma unroll
	for (int f = 0; f < 4; f++) {
		const bool in = e < ne && nbk[f] >= 0;
		const unsigned long long key = in ? (unsigned long long)(nbk[f] >> 2) * 16 + (pmk[f] & 15) : ~0ull;
		const unsigned same = __match_any_sync(0xffffffffu, key);
		total += __popc(__ballot_sync(0xffffffffu, in && __ffs(same) - 1 == lane));
	}
	if (lane == 0 && total > 0)
		atomicAdd(count, (unsigned long long)total);
}

int launch_rk3_sectors(const int *nb, const int *perm, long long ne, unsigned long long *count, cudaStream_t s)
{
	GDN_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(*count), s));
	rk3_sectors_kernel<<<(unsigned)((ne + 255) / 256), 256, 0, s>>>(reinterpret_cast<const int4 *>(nb),
																	 reinterpret_cast<const int4 *>(perm), ne, count);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

// reference layout [e][node i][field c] (FP64, ne elements of one instance) <->
// tiles, element e at position pos[e]
template <typename T>
__global__ void rk3_to_tiles_kernel(const double *__restrict__ src, T *__restrict__ dst, const int *__restrict__ pos,
									long long ne)
{
	const long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (u >= ne * 60)
		return;
	dst[rk3_tix<T>(pos[u / 60], (int)(u % 60))] = (T)src[u];
}
template <typename T>
__global__ void rk3_from_tiles_kernel(const T *__restrict__ src, double *__restrict__ dst, const int *__restrict__ pos,
									  long long ne)
{
	const long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (u >= ne * 60)
		return;
	dst[u] = (double)src[rk3_tix<T>(pos[u / 60], (int)(u % 60))];
}
// geometry [e][10] FP64 -> tiles of T
template <typename T>
__global__ void geom_to_tiles_kernel(const double *__restrict__ g, T *__restrict__ out, const int *__restrict__ pos,
									 long long ne)
{
	const long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (u >= ne * 10)
		return;
	const long long e = pos[u / 10];
	const int q = (int)(u % 10);
	out[((e >> 5) * 10 + q) * 32 + (e & 31)] = (T)g[u];
}

template <typename T>
int launch_rk3_to_tiles(const double *src, T *dst, const int *pos, long long ne, cudaStream_t s)
{
	if (ne <= 0)
		return GDN_CUDA_OK;
	rk3_to_tiles_kernel<T><<<(unsigned)((ne * 60 + 255) / 256), 256, 0, s>>>(src, dst, pos, ne);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}
template <typename T>
int launch_rk3_from_tiles(const T *src, double *dst, const int *pos, long long ne, cudaStream_t s)
{
	if (ne <= 0)
		return GDN_CUDA_OK;
	rk3_from_tiles_kernel<T><<<(unsigned)((ne * 60 + 255) / 256), 256, 0, s>>>(src, dst, pos, ne);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}
template <typename T>
int launch_geom_to_tiles(const double *g, T *out, const int *pos, long long ne, cudaStream_t s)
{
	geom_to_tiles_kernel<T><<<(unsigned)((ne * 10 + 255) / 256), 256, 0, s>>>(g, out, pos, ne);
	GDN_CUDA_TRY(cudaGetLastError());
	return GDN_CUDA_OK;
}

template int prepare_rk3<double>();
template int prepare_rk3<float>();
template int launch_rk3_stage<double>(const Rk3Params<double> &, int, cudaStream_t);
template int launch_rk3_stage<float>(const Rk3Params<float> &, int, cudaStream_t);
template int launch_rk3_to_tiles<double>(const double *, double *, const int *, long long, cudaStream_t);
template int launch_rk3_to_tiles<float>(const double *, float *, const int *, long long, cudaStream_t);
template int launch_rk3_from_tiles<double>(const double *, double *, const int *, long long, cudaStream_t);
template int launch_rk3_from_tiles<float>(const float *, double *, const int *, long long, cudaStream_t);
template int launch_geom_to_tiles<double>(const double *, double *, const int *, long long, cudaStream_t);
template int launch_geom_to_tiles<float>(const double *, float *, const int *, long long, cudaStream_t);

} // namespace gdn
