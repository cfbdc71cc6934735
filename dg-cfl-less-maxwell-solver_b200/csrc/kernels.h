// Kernel parameter blocks and launchers shared between the translation units.
#pragma once

#include <vector>

#include "common.cuh"

namespace gdn {

// Device memory of handles and of their setup, from one stream-ordered pool per
// device.  A program that attaches one simulation after another spent more time
// in cudaMalloc and cudaFree (each maps memory and waits for the device) than in
// the solve: a whole 17^3 CFL-less run of 20 steps, 25 ms, had 10 to 15 ms of
// them.  The pool keeps at most kPoolKeep bytes of free memory between handles;
// what is above goes back to the device at the next synchronisation.  It orders
// reuse between streams itself.
// A block of more than a quarter of that is cudaMalloc's: a pool grows and shrinks
// at ~7 ms per GiB (1536 MiB: 10.4 ms to take, 10.4 to give back; cudaMalloc 1.3
// and 1.5), and a handle with several such blocks outgrows what is kept.  ms of
// attach + detach, all cudaMalloc / all in the pool / so: kinetic 64^3 FP32 165 + 16
// / 187 + 50 / 146 + 10, 40^3 FP64 59 + 10 / 51 + 17 / 43 + 9; RK3 48^3 FP64 with two
// others alive, detach 4.9 / 9.1 / 2.2.
// The current device is the block's in both calls.  Where memory runs out, the pool
// gives back what it keeps before the call fails; dev_malloc is cudaMalloc with that.
constexpr size_t kPoolKeep = (size_t)1 << 30;
constexpr size_t kPoolBlock = kPoolKeep / 4;
cudaError_t dev_alloc(void **p, size_t bytes, cudaStream_t s);
void dev_free(void *p, cudaStream_t s);
cudaError_t dev_malloc(void **p, size_t bytes);

// A handle holds a batch of independent solves (one or more instances): their
// meshes are concatenated (elements, faces, boundary faces and P2 nodes of
// instance i follow those of instance i - 1), and each instance keeps its
// own time step, analytic data and time.
struct Batch {
	const int *einst; // [ne] instance of each element (nullptr: one instance)
	const int *bfinst; // [nbf] instance of each boundary face (nullptr: one instance)
	const Data *data; // [ninst] analytic data
	const double *dt; // [ninst] time step
	double *t; // [ninst] device time
	int ninst;
};

// The boundary traces of a step's three stages (rk3_trace_block).
template <typename T>
struct Rk3Trace {
	const double *bxyz; // [nbf][6][3]
	long long nbf;
	Batch b; // instances: data, dt, bfinst
	const double *t_in; // [ninst] time
	double *t_out; // [ninst] t_in + dt (advance)
	T *out; // [3][nbf][6][6]
	int advance; // 1: the traces of the next step
};

template <typename T>
struct Rk3Params {
	const T *w_in; // state read this stage, tiled (rk3_tix)
	T *w_out; // state written this stage (ping-pong), tiled
	T *k2; // low-storage register, in place, tiled
	const T *geom; // codtau (row-major 3x3) and det, tiles of 32 elements x 10 values
	const int *nb; // [ne][4] neighbour element (all rows in the device order), or -(boundary face + 1)
	const int *perm; // [ne][4] neighbour local node of face node jj, 4 bits each
	const T *btrace; // [nbf][6][6] boundary data at t_stage
	const int *einst; // [ne] instance of each element, nullptr for one instance
	const double *dt_tab; // [ninst] time step of each instance (used with einst)
	long long ne;
	double dt, A, B;
	int stage0; // k2 = -dt dw (no k2 read)
	int write_k2; // 0 on the last stage: k2 is dead until the next stage 0
	int sparse; // tables follow the P2 structural-zero pattern
	int fact; // the derivative tables factor through the P1 basis (rk3_tables_factor)
	int bc_metal; // boundary faces take the metal flux (-n x H_L, 0)
	int num_sms; // SMs of the device
	int traces; // the launch also writes tr (the last stage of a step)
	int tile_blocks; // CTAs of the tiles, before those of tr (set at launch)
	Rk3Trace<T> tr;
	int idx32; // every tiled state offset fits 32 bits (ntiles * 1920 < 2^32)
	int l2_ahead; // nonzero: prefetch into L2 the tile this many tiles ahead (set per variant at launch)
};

bool rk3_tables_sparse(const gdn_cuda_tables *t);
bool rk3_tables_factor(const gdn_cuda_tables *t);
void rk3_q4(const gdn_cuda_tables *t, double q4[4][10]);
void rk3_sym_coeffs(const gdn_cuda_tables *t, double q4_sym[6], double minv_sym[7], double s_sym[5]);
bool rk3_tables_standard_faces(const gdn_cuda_tables *t);

// variant 0 / 1: one kernel compiled for fewer / more resident CTAs per SM
// (rk3_min_blocks), i.e. more / fewer registers per thread: rk3_elem_kernel (FP32
// with the P2 tables) or rk3_stage_kernel (other tables).  FP64 with the P2 tables:
// rk3_stage_kernel / rk3_half_kernel, whose sums round differently
template <typename T>
int launch_rk3_stage(const Rk3Params<T> &p, int variant, cudaStream_t s);
template <typename T>
int prepare_rk3();

int rk3_min_blocks(int precision_fp64, int fact, int variant);
// the variant for a mesh (sectors: launch_rk3_sectors of the order in use) on a device
int rk3_default_variant(int precision_fp64, int fact, long long ne, int num_sms, long long l2_bytes,
						unsigned long long sectors);
// the mesh's own order, and the gather sectors of an order (rk3_sectors_kernel) into
// *count (device)
int launch_rk3_natural_order(long long ne, int *pos, int *items, cudaStream_t s);
int launch_rk3_sectors(const int *nb, const int *perm, long long ne, unsigned long long *count, cudaStream_t s);
// device element order: pos[e] (elements of one vertex-index stencil side by
// side inside blocks, rk3_order_kernel), its inverse items[k], and the neighbour
// / permutation rows in
// that order (nb_out, perm_out [pos[e]][4])
int launch_rk3_order(const int *e2q, const int *einst, const int *nb, const int *perm, long long ne, int *pos,
					 int *items, int *nb_out, int *perm_out, cudaStream_t s);
// reference layout [e][node][field] (FP64, ne elements) <-> tiled layout,
// element e at position pos[e]
template <typename T>
int launch_rk3_to_tiles(const double *src, T *dst, const int *pos, long long ne, cudaStream_t s);
template <typename T>
int launch_rk3_from_tiles(const T *src, double *dst, const int *pos, long long ne, cudaStream_t s);
template <typename T>
int launch_geom_to_tiles(const double *g, T *out, const int *pos, long long ne, cudaStream_t s);
template <typename T>
int launch_rk3_traces(const Rk3Trace<T> &tr, cudaStream_t s);
int launch_set_time(const Batch &b, double value, cudaStream_t s);
int launch_advance_time(const Batch &b, cudaStream_t s);

// Kinetic (CFL-less) path.  The kinetic state is stored in sweep order: item
// k (its position in the level-sorted list of (element, velocity) pairs)
// owns f[k*60 .. +60], y[k*60 ..], G[k*100 ..]; within an item the layout is
// [field c][node i].
struct KinSweepParams {
	const void *f; // right-hand side of M1 y = f (F)
	void *y; // solution, written level by level; read back as the inflow traces (Y)
	double *yacc; // refinement: FP64 solution, = y (ACC 1) or += y (ACC 2)
	const void *G; // [k][10][10] inverse of the M1 diagonal block, by columns (T)
	const void *rs; // [k][4] own-side v.vn per face (T)
	const void *rcoef; // [k] theta dt / det (T)
	const int4 *rnb; // [k] per face: inflow neighbour item, -(bf + 1) inflow boundary face, INT_MIN none
	const int4 *rpm; // [k] per face: neighbour local node of face node jj, 4 bits each
	const int *items; // [k] e * nv + v
	const double *bt; // [bf][v][c][jj] f_eq of the boundary data at t + dt/2
	int nv;
	int item_begin, item_end;
};

// f: F, y: Y, arithmetic and G: T.  acc: 0 none, 1 yacc = y, 2 yacc += y.
// bdata: inflow boundary faces take bt (0: zero boundary data, for
// correction solves).
template <typename F, typename Y, typename T>
int launch_kin_sweep(const KinSweepParams &p, int acc, int bdata, int sparse, cudaStream_t s);

// The same solve as one cooperative launch walking all levels with a grid
// barrier between them (grid = CTAs resident at once, kin_levels_grid); a
// barrier that times out sets *err.
template <typename F, typename Y, typename T>
int launch_kin_levels(const KinSweepParams &p, const int *level_off, int nlevels, int grid, unsigned *bar, int *err,
					  long long spin_limit, int acc, int bdata, int sparse, cudaStream_t s);
template <typename F, typename Y, typename T>
int kin_levels_grid(int device, int acc, int sparse, int *grid);

// items a CTA of the sweeps takes at once (five per warp); the groups of the
// row-driven sweep hold at most as many
int kin_group_items(int fp64);

// The same solve in one cooperative launch driven by the solution rows
// themselves: every word of y is marked unwritten (all bits set) first, then
// CTAs walk level-aligned
// groups of items (groups[g] = first item, end item) in sweep order, and a
// warp waits until the traces of its items are written.  CTA b takes the groups
// b, b + grid, ..., or with `group_off` those of its own spatial part (positions in
// list[]).  A wait that gives up after spin_limit polls sets *err.
template <typename F, typename Y, typename T>
int launch_kin_flow(const KinSweepParams &p, const int2 *groups, int ngroups, const int *list, const int *group_off,
					int grid, long long nitems, int *err, long long spin_limit, int acc, int bdata, int sparse,
					cudaStream_t s);
template <typename F, typename Y, typename T>
int kin_flow_grid(int device, int acc, int sparse, int *grid);
// the parts: elements split into nparts equal ranges along a Morton curve of
// their centroids (bounding box lo, hi); plist (device) and its host copy,
// the part of every list entry (host)
int kin_build_parts(const int *e2q, const double *node, long long ne, const double lo[3], const double hi[3],
					const int *items, long long nitems, int nv, int nparts, int *plist,
					std::vector<int> &plist_host, std::vector<int> &pkey_host, cudaStream_t s);

// Level schedule of the upwind item graph on the device (Kahn's algorithm by
// levels, one cooperative launch): items[k] (e * nv + v in level order,
// ascending within a level), pos (its inverse), level_off (host, first item of
// each level, then the item count); GDN_CUDA_ERR_CYCLE when the graph has a
// cycle, GDN_CUDA_ERR_TIMEOUT when a grid barrier waited spin_limit polls.
int kin_device_schedule(const unsigned char *mask, const int *nb, const double *sown64, long long ne, int nv,
						int *items, int *pos, std::vector<int> &level_off, long long spin_limit, cudaStream_t s);

// f_eq of the analytic data at the boundary face nodes, t + dt/2 (FP64)
int launch_kin_boundary_trace(const double *bxyz, long long nbf, const Batch &b, int nv, const double *vi,
							  double feq_c, double *bt, cudaStream_t s);

// FP64 residual r = f - b - M1 yacc of every item (b: inflow boundary data)
struct KinResidualParams {
	const double *f;
	const double *yacc;
	float *r;
	const int4 *rnb, *rpm;
	const int *items;
	const double4 *ru64; // [k] u_0, u_1, u_2 (u_q = v . codtau[:, q]), theta dt / det
	const double4 *rs64; // [k] own-side v.vn per face
	const double *bt;
	int nv;
	long long nitems;
};
int launch_kin_residual(const KinResidualParams &p, int sparse, cudaStream_t s);

struct KinRelaxParams {
	void *f; // in: f^n, out: f^{n+1} (F, sweep order)
	const void *y; // (Y)
	const int *pos; // [e * nv + v] item index k of (e, v)
	long long ne;
	int nv;
	double vi[3 * NV_MAX];
	double feq_c, omega;
	double a_y, a_f; // x = a_y y + a_f f  (2, -1 for theta = 1/2)
};
template <typename F, typename Y, typename T>
int launch_kin_relax(const KinRelaxParams &p, cudaStream_t s);

} // namespace gdn
