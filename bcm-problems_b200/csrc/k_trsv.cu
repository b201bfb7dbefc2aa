// Triangular solves with an IC2 / ILU2 factor (CSMatrixR::SolveL,
// Bslib/mvm.cpp:3042 -- L by columns, inverse pivot first; SolveU, :3343 --
// U by rows, inverse pivot first).
//
// The column-stored L is turned into rows (gather form) once per factor, so
// both solves read their factor rows contiguously:
//   forward  y_i = dinv_l[i] * (x_i - sum_{k<i} L(i,k) y_k)
//   backward y_i = dinv_u[i] * (x_i - sum_{k>i} U(i,k) y_k)
//
// mode 0 -- exact, sync-free: a warp solves one row, in level order within the
//   block of consecutive rows its CTA owns (or, where that does not pay, among all
//   rows), and each lane waits on the entry it needs.  "Solved" is encoded in the value itself: y is pre-filled with a NaN
//   bit pattern no arithmetic produces, and a 64-bit store publishes the result
//   in one transaction.  A wait gives up (BSG_ERR_TIMEOUT) when globaltimer runs
//   on for the limit without a row solved anywhere.
// mode 1 -- Jacobi sweeps: y <- D^{-1}(x - N y) repeated nsweeps times from
//   y = D^{-1} x; every sweep is a fully parallel pass over the factor (HBM
//   bound: 4 B value (FP32) or 8 B (FP64) + 4 B column per entry).  It applies
//   a fixed polynomial in the factor, so it is a valid flexible (FGMRES)
//   preconditioner and, applied symmetrically, a valid PCG preconditioner.
#include "bsg_internal.cuh"
#include "k_stream.cuh"
#include <cub/device/device_radix_sort.cuh>

#ifndef SELL_SIGMA
#define SELL_SIGMA 128 // rows per length-sorting window of the factor's sliced copies
#endif

namespace {

// One Jacobi sweep y_out = D^{-1}(x - N y_in) by row-chunk streaming; with
// IN == IN_SCALED the input is the first iterate D^{-1} x, formed on the fly
// (the first two sweeps in one pass).
template <typename VT, int IN>
__global__ void __launch_bounds__(256) k_trsv_sweep(int n, const int *__restrict__ rp, const int *__restrict__ ci,
                                                    const VT *__restrict__ v, int skip,
                                                    const double *__restrict__ dinv, const double *__restrict__ x,
                                                    const double *__restrict__ yin, double *__restrict__ yout) {
	__shared__ double prod[8][STREAM_CAP];
	stream_rows<VT, IN, OUT_SWEEP>(n, rp, ci, v, skip, IN == IN_VEC ? yin : x, dinv, x, dinv, yout,
	                               prod[threadIdx.x >> 5]);
}

__global__ void k_scale_vec(int n, const double *x, const double *d, double *y) {
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = x[i] * d[i];
}

// ---- exact solve ------------------------------------------------------------
// Bound: the longest chain of dependent rows times the latency of one link, so
// the kernel is laid out for short links.
//  - Every CTA owns a block of consecutive rows and solves them in level order,
//    its warps taking the rows in turn.  In natural order most dependencies lie
//    close by, so most links stay inside a CTA and pass through shared memory
//    (ys); only links between blocks go through L2.
//  - A row's columns, values, right-hand side and inverse pivot are in registers
//    before its wait; the next row's load during it.
//  - With one entry of the row still unsolved, the warp has already added up
//    the rest: the waiting lane holds the five partial sums that the butterfly
//    of warp_sum() would add to its own and adds them in that order, so the
//    result has the bits of the plain reduction, without its shuffles after
//    the wait.
// Blocks are claimed from a counter in solve order (ascending for L, descending
// for U).  A block's rows depend on rows of its own and of blocks claimed before,
// whose CTAs run already or are done; within a block, the unsolved row that comes
// first by (level, place in its list) waits for solved rows or other blocks only,
// and its warp has no earlier row left.  So the solve always progresses, with any
// number of CTAs resident: on a part of the GPU, beside other kernels, or with more
// blocks than SMs.
// Measured against one warp per row claimed in global level order with every
// link through L2 (us per forward solve, before / after, FP64 IC2 tau 1e-3 of the
// 7-point heat operator): 12^3 553 / 145, 32^3 1668 / 309, 47x40x33 3537 / 514,
// 128^3 18690 / 5470; IC(0) 128^3 2075 / 1170; 2-D 500^2 22752 / 1836; a chain of
// 100000 rows 437 / 21 ms (0.21 us a link).  Factors without locality go by rows
// (k_trsv_rows, see trsv_scattered).
#define TRSV_WARPS 32 // 24 warps: 47x40x33 580, 128^3 5520; 16: 760, 6600
#define TRSV_M 2 // entries of a row each lane holds (32 TRSV_M a row; longer rows walk their head first)
#define TRSV_ROWS_MAX 28000 // rows of a block: 8 bytes each in shared memory
// fewest rows of a block: smaller blocks spread a small system over more SMs,
// larger ones keep more links inside (us, 12^3 / 47x40x33: 128 rows 144 / 521,
// 256 146 / 516, 512 152 / 566, 1024 158 / 634)
#define TRSV_ROWS_MIN 256

// The spin limit of a wait.  A block waits from the launch on for all the blocks
// that come before it, so the limit counts from the last progress of the whole
// solve: a warp adds to *solved after every 32 rows of its own and after its last,
// and a wait that sees *solved move starts again.  (An add every eight rows, in the
// row loop, costs 1.5 to 3 %.)
struct TrsvLimit {
	unsigned t0 = 0, seen = 0; // in units of 1024 ns (registers are short here)
	// whether to give up: another warp failed, or the limit has passed
	__device__ __forceinline__ bool over(const unsigned *solved, int row, bsg_devstat *st) {
		const int code = *(volatile int *)&st->code; // (one round trip for both)
		const unsigned cnt = *(const volatile unsigned *)solved, now = (unsigned)(globaltimer_ns() >> 10) | 1u;
		if (code != 0) return true;
		if (t0 == 0 || cnt != seen) {
			t0 = now;
			seen = cnt;
		} else if (now - t0 > (unsigned)(BSG_SPIN_LIMIT_NS >> 10)) {
			devstat_fail(st, BSG_ERR_TIMEOUT, row);
			return true;
		}
		return false;
	}
};

// The solved entry at p (shared or global), waiting for it; the spin limit or
// another warp's failure gives 0.
__device__ __forceinline__ unsigned long long trsv_wait(const double *p, int row, const unsigned *solved,
                                                        bsg_devstat *st) {
	unsigned long long raw = ld_volatile_generic_u64(p);
	if (raw != BSG_PENDING) return raw;
	TrsvLimit limit;
	for (unsigned it = 1;; it++) {
		raw = ld_volatile_generic_u64(p);
		if (raw != BSG_PENDING) return raw;
		if ((it & 127) == 0 && limit.over(solved, row, st)) return 0;
	}
}

template <typename VT>
__global__ void __launch_bounds__(TRSV_WARPS * 32, 1)
k_trsv_blocks(int n, int lower, int rows, const int *__restrict__ perm, const int *__restrict__ rp,
              const int *__restrict__ ci, const VT *__restrict__ v, int skip_first, const double *__restrict__ dinv,
              const double *__restrict__ x, double *y, unsigned *claim, unsigned *solved,
              bsg_devstat *st) {
	extern __shared__ double ys[]; // the block's solved rows, BSG_PENDING before
	__shared__ unsigned block;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	if (threadIdx.x == 0) block = atomicAdd(claim, 1u);
	for (int k = threadIdx.x; k < rows; k += blockDim.x) ys[k] = __longlong_as_double((long long)BSG_PENDING);
	__syncthreads();
	const int r0 = (int)(lower ? block : gridDim.x - 1 - block) * rows, cnt = min(rows, n - r0);
	// item k of this warp: place warp + k TRSV_WARPS of the block's list (read backwards for U)
	auto item = [&](int k) {
		const int o = warp + k * TRSV_WARPS;
		return o < cnt ? perm[r0 + (lower ? o : cnt - 1 - o)] : -1;
	};
	struct Meta {
		int row, b, e;
		double x, d;
	};
	auto meta = [&](int row) {
		Meta m = {row, 0, 0, 0.0, 0.0};
		if (row >= 0) {
			m.b = rp[row] + skip_first;
			m.e = rp[row + 1];
			m.x = x[row];
			m.d = dinv[row];
		}
		return m;
	};
	int row1 = item(lane);
	Meta cur = meta(row1);
	row1 = item(32 + lane);
	int nc[TRSV_M];
	VT nv[TRSV_M];
	auto load = [&](int b, int e) { // the last 32 TRSV_M entries of a row at most
		const int tail = max(b, b + ((e - b - 1) / 32 - (TRSV_M - 1)) * 32);
#pragma unroll
		for (int u = 0; u < TRSV_M; u++) {
			const int k = tail + u * 32 + lane;
			nc[u] = -1;
			nv[u] = VT(0);
			if (k < e) {
				nc[u] = ci[k];
				nv[u] = v[k];
			}
		}
	};
	load(__shfl_sync(0xffffffffu, cur.b, 0), __shfl_sync(0xffffffffu, cur.e, 0));
	for (int k0 = 0; warp + k0 * TRSV_WARPS < cnt; k0 += 32) {
		const Meta nxt = meta(row1); // 32 rows ahead
		row1 = item(k0 + 64 + lane);
		for (int j = 0; j < 32 && warp + (k0 + j) * TRSV_WARPS < cnt; j++) {
			const int row = __shfl_sync(0xffffffffu, cur.row, j);
			const int b = __shfl_sync(0xffffffffu, cur.b, j), e = __shfl_sync(0xffffffffu, cur.e, j);
			const double xr = __shfl_sync(0xffffffffu, cur.x, j), dr = __shfl_sync(0xffffffffu, cur.d, j);
			int c[TRSV_M];
			double a[TRSV_M];
#pragma unroll
			for (int u = 0; u < TRSV_M; u++) {
				c[u] = nc[u];
				a[u] = (double)nv[u];
			}
			load(__shfl_sync(0xffffffffu, j < 31 ? cur.b : nxt.b, (j + 1) & 31),
			     __shfl_sync(0xffffffffu, j < 31 ? cur.e : nxt.e, (j + 1) & 31));
			auto entry = [&](int col) -> const double * {
				const unsigned s = (unsigned)(col - r0);
				return s < (unsigned)cnt ? ys + s : y + col;
			};
			double s = 0.0;
			if (e - b > 32 * TRSV_M) { // head of a long row, in order
				const int tail = b + ((e - b - 1) / 32 - (TRSV_M - 1)) * 32;
				for (int k = b + lane; k < tail; k += 32) {
					const int col = ci[k];
					s = fma((double)v[k], __longlong_as_double((long long)trsv_wait(entry(col), row, solved, st)), s);
				}
				__syncwarp();
			}
			const double *src[TRSV_M];
			unsigned long long raw[TRSV_M];
#pragma unroll
			for (int u = 0; u < TRSV_M; u++) {
				src[u] = c[u] >= 0 ? entry(c[u]) : nullptr;
				raw[u] = src[u] ? BSG_PENDING : 0ull;
			}
			// poll until at most one lane waits
			unsigned wait;
			TrsvLimit limit;
			for (unsigned it = 1;; it++) {
				bool mine = false;
#pragma unroll
				for (int u = 0; u < TRSV_M; u++) {
					if (raw[u] == BSG_PENDING) raw[u] = ld_volatile_generic_u64(src[u]);
					mine = mine || raw[u] == BSG_PENDING;
				}
				wait = __ballot_sync(0xffffffffu, mine);
				if ((wait & (wait - 1)) == 0) break;
				if ((it & 127) == 0 && __any_sync(0xffffffffu, limit.over(solved, row, st))) { // leave the rest at 0
#pragma unroll
					for (int u = 0; u < TRSV_M; u++)
						if (raw[u] == BSG_PENDING) raw[u] = 0;
					wait = 0;
					break;
				}
			}
			const int last = wait ? __ffs(wait) - 1 : 0; // the lane that finishes the row
			double t = s;
			if (wait == 0 || lane != last) {
#pragma unroll
				for (int u = 0; u < TRSV_M; u++)
					if (c[u] >= 0) t = fma(a[u], __longlong_as_double((long long)raw[u]), t);
			}
			double part[5];
			{
				double r = t;
#pragma unroll
				for (int k = 0; k < 5; k++) {
					part[k] = __shfl_xor_sync(0xffffffffu, r, 16 >> k);
					r += part[k];
				}
			}
			if (lane == last) {
				if (wait) {
#pragma unroll
					for (int u = 0; u < TRSV_M; u++)
						if (c[u] >= 0) {
							if (raw[u] == BSG_PENDING) raw[u] = trsv_wait(src[u], row, solved, st);
							t = fma(a[u], __longlong_as_double((long long)raw[u]), t);
						}
				}
#pragma unroll
				for (int k = 0; k < 5; k++) t += part[k];
				const double yr = (xr - t) * dr;
				st_volatile_shared_f64(ys + (row - r0), yr);
				st_volatile_f64(y + row, yr);
			}
			__syncwarp();
		}
		if (lane == 0) atomicAdd(solved, 1u);
		cur = nxt;
	}
}

// The exact solve where blocks do not pay (see trsv_scattered): a warp per row, the
// rows claimed in global level order (perm, read backwards for U), so that the
// rows in flight are those of the current wavefront, wherever they lie.  Bound: a
// link through L2, about 4 us a level, and the claims, 0.7 ns a row.
template <typename VT>
__global__ void __launch_bounds__(256) k_trsv_rows(int n, int lower, const int *__restrict__ perm,
                                                   const int *__restrict__ rp, const int *__restrict__ ci,
                                                   const VT *__restrict__ v, int skip_first,
                                                   const double *__restrict__ dinv, const double *__restrict__ x,
                                                   double *y, unsigned *claim, bsg_devstat *st) {
	const int lane = threadIdx.x & 31;
	for (;;) {
		int t = 0;
		if (lane == 0) t = (int)atomicAdd(claim, 1u);
		t = __shfl_sync(0xffffffffu, t, 0);
		if (t >= n) return;
		const int row = perm[lower ? t : n - 1 - t];
		const int b = rp[row] + skip_first, e = rp[row + 1];
		double s = 0.0;
		for (int k = b + lane; k < e; k += 32) {
			const int c = ci[k];
			unsigned long long raw = ld_volatile_u64(y + c);
			if (raw == BSG_PENDING) {
				TrsvLimit limit; // (claims are progress)
				for (unsigned it = 1;; it++) {
					__nanosleep(32);
					raw = ld_volatile_u64(y + c);
					if (raw != BSG_PENDING) break;
					if ((it & 127) == 0 && limit.over(claim, row, st)) {
						raw = 0;
						break;
					}
				}
			}
			s = fma((double)v[k], __longlong_as_double((long long)raw), s);
		}
		s = warp_sum(s);
		if (lane == 0) st_volatile_f64(y + row, (x[row] - s) * dinv[row]);
	}
}

// Sort keys of the solve order: the row's block (all in one for rows == 0), then
// its level; *most gets the largest level.
__global__ void k_trsv_keys(int n, int rows, const int *lev, unsigned long long *keys, int *vals) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	keys[i] = ((unsigned long long)(unsigned)(rows ? i / rows : 0) << 32) | (unsigned)lev[i];
	vals[i] = i;
}
__global__ void k_trsv_levels(int n, const int *lev, int *most) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	const int m = __reduce_max_sync(0xffffffffu, i < n ? lev[i] : 0);
	if ((threadIdx.x & 31) == 0) atomicMax(most, m);
}
// most[l] = the most rows of level l in one block (sorted keys: a run per block
// and level)
__global__ void k_trsv_crowd(int n, const unsigned long long *keys, int *most) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const unsigned long long k = keys[i];
	if (i > 0 && keys[i - 1] == k) return;
	int lo = i + 1, hi = n; // the first place with another key
	while (lo < hi) {
		const int mid = lo + (hi - lo) / 2;
		if (keys[mid] == k) lo = mid + 1;
		else hi = mid;
	}
	atomicMax(most + (unsigned)k, lo - i);
}
__global__ void k_trsv_sum(int n, const int *v, int *sum) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	const int t = __reduce_add_sync(0xffffffffu, i < n ? v[i] : 0);
	if ((threadIdx.x & 31) == 0 && t) atomicAdd(sum, t);
}

// y before an exact solve: nothing solved, no block claimed
__global__ void k_fill_u64(long long n, unsigned long long *p, unsigned long long v, unsigned *claim) {
	if (blockIdx.x == 0 && threadIdx.x == 0) *claim = 0;
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
		p[i] = v;
}

__global__ void k_diag_inv(int n, const int *iu, const double *l, const double *u, double *dl, double *du) {
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) {
		dl[i] = l[iu[i]];
		du[i] = u[iu[i]];
	}
}

__global__ void k_permute(int nk, const int *perm, const double *src, double *dst) {
	int k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k < nk) dst[k] = src[perm[k]];
}

__global__ void k_to_f32(long long nk, const double *src, float *dst) {
	for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < nk; k += (long long)gridDim.x * blockDim.x)
		dst[k] = (float)src[k];
}

inline int nb(long long n, int t) { return n > 0 ? (int)((n + t - 1) / t) : 1; }

} // namespace

int bsg_strict_transpose(bsg_ctx *c, int n, const int *ia, const int *ja, int nnz, int **it_o, int **jt_o,
                         int **perm_o, int *nnz_o);

// Whether an exact solve goes by rows in global level order instead of by blocks:
// crowd is the sum over the levels of the most rows of the level in one block.  The
// block with the most rows of a level holds the level up, 32 rows a microsecond;
// without blocks a level takes 4 us and a row 0.7 ns.  So wavefronts that stand in
// few blocks (windowed graphs) or wide ones without locality (permuted grids) go by
// rows.  Below 50000 rows blocks were never slower.  us a solve, by rows / by blocks,
// * the one taken: IC(0) of random graphs with 3 neighbours within +-w: 300000 rows,
// w 1000 8940 / 6960*, 3000 3095* / 4650, 30000 243* / 655, any 235 / 214*; 1000000
// rows, w 30000 760* / 6030, any 692 / 657*; 8 neighbours, 300000 rows, w 3000 7660 /
// 7390*, 100000 239* / 556; permuted 64^3 grid, IC2 273* / 439, IC(0) 208 / 192*;
// natural 128^3, IC(0) 2070 / 1160*.
#define TRSV_SCATTER_MIN 50000
static bool trsv_scattered(int n, int levels, double crowd) {
	const double blocks = 20.0 + 0.9 * crowd / TRSV_WARPS, rows1 = 4.0 * levels - 15.0, rows2 = 25.0 + 0.69e-3 * n;
	return blocks > (rows1 > rows2 ? rows1 : rows2);
}

// The exact solves' order of f's n rows from their levels (ascending depth in
// the forward solve's dependency graph): blocks of f->trsv_rows consecutive
// rows, by (level, index) inside a block, in f->d_perm; or, with trsv_rows 0, all
// rows by (level, index).  Sets levels_l / levels_u.
int bsg_trsv_schedule(bsg_ctx *c, bsg_fct *f, const int *lev) {
	cudaStream_t s = c->stream;
	const int n = f->n;
	f->levels_l = f->levels_u = 0;
	f->trsv_rows = TRSV_ROWS_MIN;
	BSG_CUDA(cudaMallocAsync(&f->d_perm, sizeof(int) * (n > 0 ? n : 1), s));
	if (n <= 0) return BSG_OK;
	// an equal share per SM, but no less than TRSV_ROWS_MIN (a smaller block has
	// more of its links outside) and no more than shared memory holds
	long long rows = (n + BSG_SMS - 1) / BSG_SMS;
	if (rows < TRSV_ROWS_MIN) rows = TRSV_ROWS_MIN;
	if (rows > TRSV_ROWS_MAX) {
		const long long steps = (n + (long long)BSG_SMS * TRSV_ROWS_MAX - 1) / ((long long)BSG_SMS * TRSV_ROWS_MAX);
		rows = (n + steps * BSG_SMS - 1) / (steps * BSG_SMS);
	}
	f->trsv_rows = (int)rows;
	int bits = 32;
	while ((1ll << (bits - 32)) < (n + rows - 1) / rows) bits++;
	struct Tmp { // freed on every way out
		cudaStream_t s;
		void *p = nullptr;
		~Tmp() {
			if (p) cudaFreeAsync(p, s);
		}
	} dkeys{s}, dk2{s}, dvals{s}, dmost{s}, dcrowd{s}, dtmp{s};
	int top[2] = {0, 0}; // largest level, sum of crowd
	size_t tb = 0;
	BSG_CUDA(cudaMallocAsync(&dkeys.p, sizeof(unsigned long long) * n, s));
	BSG_CUDA(cudaMallocAsync(&dk2.p, sizeof(unsigned long long) * n, s));
	BSG_CUDA(cudaMallocAsync(&dvals.p, sizeof(int) * n, s));
	BSG_CUDA(cudaMallocAsync(&dmost.p, sizeof(top), s));
	unsigned long long *keys = (unsigned long long *)dkeys.p, *k2 = (unsigned long long *)dk2.p;
	int *vals = (int *)dvals.p, *most = (int *)dmost.p;
	BSG_CUDA(cudaMemsetAsync(most, 0, sizeof(top), s));
	BSG_COUNT(2);
	k_trsv_levels<<<nb(n, 256), 256, 0, s>>>(n, lev, most);
	k_trsv_keys<<<nb(n, 256), 256, 0, s>>>(n, f->trsv_rows, lev, keys, vals);
	BSG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, keys, k2, vals, f->d_perm, n, 0, bits, s));
	BSG_CUDA(cudaMallocAsync(&dtmp.p, tb > 0 ? tb : 1, s));
	BSG_CUDA(cub::DeviceRadixSort::SortPairs(dtmp.p, tb, keys, k2, vals, f->d_perm, n, 0, bits, s));
	if (n >= TRSV_SCATTER_MIN) {
		BSG_CUDA(cudaMallocAsync(&dcrowd.p, sizeof(int) * n, s)); // (levels < n)
		int *crowd = (int *)dcrowd.p;
		BSG_CUDA(cudaMemsetAsync(crowd, 0, sizeof(int) * n, s));
		BSG_COUNT(2);
		k_trsv_crowd<<<nb(n, 256), 256, 0, s>>>(n, k2, crowd);
		k_trsv_sum<<<nb(n, 256), 256, 0, s>>>(n, crowd, most + 1);
	}
	BSG_CUDA(cudaMemcpyAsync(top, most, sizeof(top), cudaMemcpyDeviceToHost, s));
	BSG_CUDA(cudaStreamSynchronize(s));
	f->levels_l = f->levels_u = top[0] + 1;
	// more blocks than SMs run in turn
	const long long turns = ((n + rows - 1) / rows + BSG_SMS - 1) / BSG_SMS;
	if (n >= TRSV_SCATTER_MIN && trsv_scattered(n, f->levels_l, (double)top[1] * turns)) {
		f->trsv_rows = 0;
		BSG_COUNT(1);
		k_trsv_keys<<<nb(n, 256), 256, 0, s>>>(n, 0, lev, keys, vals);
		BSG_CUDA(cub::DeviceRadixSort::SortPairs(dtmp.p, tb, keys, k2, vals, f->d_perm, n, 0, bits, s));
	}
	return BSG_OK;
}

// Build the gather forms of a freshly compacted factor.
int bsg_fct_finish(bsg_ctx *c, bsg_fct *f) {
	cudaStream_t s = c->stream;
	const int n = f->n;
	BSG_CUDA(cudaMallocAsync(&f->d_dinv_l, sizeof(double) * n, s));
	BSG_CUDA(cudaMallocAsync(&f->d_dinv_u, sizeof(double) * n, s));
	BSG_COUNT(2); // diagonal inverse + value permutation
	k_diag_inv<<<nb(n, 256), 256, 0, s>>>(n, f->d_iu, f->d_l, f->d_u, f->d_dinv_l, f->d_dinv_u);
	int *perm = nullptr, nk = 0;
	int rc = bsg_strict_transpose(c, n, f->d_iu, f->d_ju, f->nnz, &f->d_lr_i, &f->d_lr_j, &perm, &nk);
	if (rc) return rc;
	f->nnz_strict = nk;
	BSG_CUDA(cudaMallocAsync(&f->d_lr_v, sizeof(double) * (nk > 0 ? nk : 1), s));
	k_permute<<<nb(nk, 256), 256, 0, s>>>(nk, perm, f->d_l, f->d_lr_v);
	BSG_CUDA(cudaFreeAsync(perm, s));
	// strict U rows are the factor rows minus their first (diagonal) entry
	f->d_ur_i = f->d_iu;
	f->d_ur_j = f->d_ju;
	f->d_ur_v = f->d_u;
	// factor rows vary in length from row to row (thresholds): sort them by
	// length inside windows of SELL_SIGMA rows so the slices need little padding
	rc = bsg_sell_build(c, n, f->d_lr_i, f->d_lr_j, f->d_lr_v, 0, 0, &f->sl, SELL_SIGMA);
	if (!rc) rc = bsg_sell_build(c, n, f->d_iu, f->d_ju, f->d_u, 1, 0, &f->su, SELL_SIGMA);
	if (rc) return rc;
	BSG_CUDA(cudaGetLastError());
	BSG_CUDA(cudaStreamSynchronize(s));
	return BSG_OK;
}

int bsg_fct_make_fp32(bsg_fct *f) {
	if (f->fp32) return BSG_OK;
	cudaStream_t s = f->ctx->stream;
	if (f->has_t && f->kind == 1) { // the transposed forms are rebuilt in FP32 on next use
		bsg_sell_free(&f->slt, s);
		bsg_sell_free(&f->sut, s);
		if (f->d_utr_v) cudaFreeAsync(f->d_utr_v, s);
		f->d_utr_v = nullptr;
		f->has_t = 0;
	}
	BSG_CUDA(cudaMallocAsync(&f->d_ur_f, sizeof(float) * (f->nnz > 0 ? f->nnz : 1), s));
	BSG_CUDA(cudaMallocAsync(&f->d_lr_f, sizeof(float) * (f->nnz_strict > 0 ? f->nnz_strict : 1), s));
	BSG_COUNT(2);
	k_to_f32<<<BSG_SMS * 4, 256, 0, s>>>(f->nnz, f->d_u, f->d_ur_f);
	k_to_f32<<<BSG_SMS * 4, 256, 0, s>>>(f->nnz_strict, f->d_lr_v, f->d_lr_f);
	BSG_CUDA(cudaGetLastError());
	// the sweeps read the SELL copies: rebuild them with FP32 values
	bsg_sell_free(&f->sl, s);
	bsg_sell_free(&f->su, s);
	int rc = bsg_sell_build(f->ctx, f->n, f->d_lr_i, f->d_lr_j, f->d_lr_v, 0, 1, &f->sl, SELL_SIGMA, 1);
	if (!rc) rc = bsg_sell_build(f->ctx, f->n, f->d_iu, f->d_ju, f->d_u, 1, 1, &f->su, SELL_SIGMA, 1);
	if (rc) return rc;
	f->fp32 = 1;
	return BSG_OK;
}

int bsg_fill_launch(cudaStream_t s, long long n, double *x, double v);

// One full Jacobi sweep y_out = D^{-1}(x - N y_in) (reads the whole factor);
// used to time the sweep kernel on its own.
int bsg_trisolve_sweep_launch(bsg_ctx *c, const bsg_fct *f, int lower, const double *x, const double *yin,
                              double *yout) {
	if (f->d_bia) return bsg_set_error(BSG_ERR_UNSUPPORTED, "single sweep timing of a block factor");
	const double *dinv = lower ? f->d_dinv_l : f->d_dinv_u;
	if (f->fp32) // the FP32-iterate pass of the mixed path; yin's bytes serve as its FP32 input
		return bsg_sell_sweep32_pass(c->stream, lower ? &f->sl : &f->su, x, dinv, reinterpret_cast<const float *>(yin),
		                             yout);
	return bsg_sell_sweep(c->stream, lower ? &f->sl : &f->su, x, dinv, yin, 0, yout);
}

namespace {
// A triangular operand: its rows (strict part, `skip` leading diagonal
// entries), FP64 / FP32 values, inverse pivots and sliced copy.
struct TriOp {
	int lower;
	const int *rp, *ci;
	int skip;
	const double *vd;
	const float *vf;
	const double *dinv;
	const bsg_sell *sell;
};

int trisolve_impl(bsg_ctx *c, const bsg_fct *f, const TriOp &t, int mode, int nsweeps, const double *x, double *y,
                  double *work) {
	cudaStream_t s = c->stream;
	const int n = f->n;
	const bool use32 = f->fp32 != 0;
	if (mode == 0) {
		if (n == 0) return BSG_OK;
		BSG_COUNT(2);
		unsigned *claim = c->d_counters + 1, *solved = c->d_counters + 2;
		const int fill = nb(n, 256) < BSG_SMS * 4 ? nb(n, 256) : BSG_SMS * 4;
		k_fill_u64<<<fill, 256, 0, s>>>(n, (unsigned long long *)y, BSG_PENDING, claim);
		const int rows = f->trsv_rows;
		if (!rows) {
			const int grid = (n + 7) / 8 < BSG_SMS * 8 ? (n + 7) / 8 : BSG_SMS * 8;
			if (use32)
				k_trsv_rows<float><<<grid, 256, 0, s>>>(n, t.lower, f->d_perm, t.rp, t.ci, t.vf, t.skip, t.dinv, x, y, claim,
				                                       c->d_stat);
			else
				k_trsv_rows<double><<<grid, 256, 0, s>>>(n, t.lower, f->d_perm, t.rp, t.ci, t.vd, t.skip, t.dinv, x, y, claim,
				                                        c->d_stat);
			return cudaGetLastError() == cudaSuccess ? BSG_OK : BSG_ERR_CUDA;
		}
		const int blocks = (n + rows - 1) / rows;
		const int smem = (int)sizeof(double) * rows, most = (int)sizeof(double) * TRSV_ROWS_MAX;
		if (use32) {
			BSG_CUDA(cudaFuncSetAttribute(k_trsv_blocks<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
			k_trsv_blocks<float><<<blocks, TRSV_WARPS * 32, smem, s>>>(n, t.lower, rows, f->d_perm, t.rp, t.ci, t.vf, t.skip,
			                                                           t.dinv, x, y, claim, solved, c->d_stat);
		} else {
			BSG_CUDA(cudaFuncSetAttribute(k_trsv_blocks<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
			k_trsv_blocks<double><<<blocks, TRSV_WARPS * 32, smem, s>>>(n, t.lower, rows, f->d_perm, t.rp, t.ci, t.vd, t.skip,
			                                                            t.dinv, x, y, claim, solved, c->d_stat);
		}
		return cudaGetLastError() == cudaSuccess ? BSG_OK : BSG_ERR_CUDA;
	}
	if (nsweeps < 1) nsweeps = 1;
	if (nsweeps > 2 && !work) return BSG_ERR_ARG;
	if (nsweeps == 1) { // the first iterate only: y = D^{-1} x
		BSG_COUNT(1);
		k_scale_vec<<<BSG_SMS * 8, 256, 0, s>>>(n, x, t.dinv, y);
		return cudaGetLastError() == cudaSuccess ? BSG_OK : BSG_ERR_CUDA;
	}
	if (use32) {
		// FP32 factor: FP32 iterates, ping-ponged in work (2 n floats)
		if (!work) return BSG_ERR_ARG;
		return bsg_sell_sweeps32(s, t.sell, x, t.dinv, nsweeps, reinterpret_cast<float *>(work), y);
	}
	// nsweeps - 1 passes (the first two iterates share one), ping-pong so
	// that the last pass lands in y
	const int passes = nsweeps - 1;
	double *bufs[2] = {y, work};
	int cur = (passes + 1) % 2;
	const double *yin = nullptr;
	for (int p = 0; p < passes; p++) {
		double *out = bufs[cur];
		int rc = bsg_sell_sweep(s, t.sell, x, t.dinv, yin, p == 0, out);
		if (rc) return rc;
		yin = out;
		cur ^= 1;
	}
	return BSG_OK;
}
} // namespace

// Solve with L (lower != 0) or U.  x and y must not alias.  `work` (n
// doubles) is needed for mode 1 with nsweeps > 2, and with nsweeps > 1 for an
// FP32 factor, whose sweeps keep their intermediate iterates in FP32 there.
int bsg_trisolve_launch(bsg_ctx *c, const bsg_fct *f, int lower, int mode, int nsweeps, const double *x, double *y,
                        double *work) {
	if (f->d_bia) return bsg_btrisolve_launch(c, f, lower, mode, nsweeps, x, y, work);
	TriOp t;
	t.lower = lower ? 1 : 0;
	t.rp = lower ? f->d_lr_i : f->d_ur_i;
	t.ci = lower ? f->d_lr_j : f->d_ur_j;
	t.skip = lower ? 0 : 1;
	t.vd = lower ? f->d_lr_v : f->d_ur_v;
	t.vf = lower ? f->d_lr_f : f->d_ur_f;
	t.dinv = lower ? f->d_dinv_l : f->d_dinv_u;
	t.sell = lower ? &f->sl : &f->su;
	return trisolve_impl(c, f, t, mode, nsweeps, x, y, work);
}

// nr solves with one factor, vectors at stride n; work holds n nr doubles
// (needed for sweeps).  Sweeps read the untiled sliced copy once per 8
// vectors and give every vector the bits of a single solve (the tiled FP32
// sweeps sum in the same order); exact solves run one vector at a time.
int bsg_trisolve_multi(bsg_ctx *c, const bsg_fct *f, int lower, int mode, int nsweeps, int nr, const double *x,
                       double *y, double *work) {
	if (f->d_bia) return bsg_btrisolve_multi(c, f, lower, mode, nsweeps, nr, x, y, work);
	const int n = f->n;
	if (nr > 1 && mode != 0 && nsweeps >= 2) {
		if (!work) return bsg_set_error(BSG_ERR_ARG, "sweeps of several vectors: work vector missing");
		const bsg_sell *sl = lower ? &f->sl : &f->su;
		const double *dinv = lower ? f->d_dinv_l : f->d_dinv_u;
		if (f->fp32) return bsg_sell_sweeps32_multi(c->stream, sl, nr, x, dinv, nsweeps, reinterpret_cast<float *>(work), y);
		// FP64: nsweeps - 1 passes, ping-pong so that the last lands in y
		const int passes = nsweeps - 1;
		double *bufs[2] = {y, work};
		int cur = (passes + 1) % 2;
		const double *yin = nullptr;
		for (int p = 0; p < passes; p++) {
			int rc = bsg_sell_sweep_multi(c->stream, sl, nr, x, dinv, yin, p == 0, bufs[cur]);
			if (rc) return rc;
			yin = bufs[cur];
			cur ^= 1;
		}
		return BSG_OK;
	}
	for (int q = 0; q < nr; q++) {
		const size_t o = (size_t)q * n;
		int rc = bsg_trisolve_launch(c, f, lower, mode, nsweeps, x + o, y + o, work ? work + o : nullptr);
		if (rc) return rc;
	}
	return BSG_OK;
}

// The transposed forms of an ILU2 factor: U^T rows are the L-row pattern
// with U's values (the transposition that built the L rows, applied to U),
// L^T rows are U's own pattern with L's values.  IC2 factors need none
// (U^T = L, L^T = U).
static int fct_build_transposes(bsg_ctx *c, bsg_fct *f) {
	if (f->has_t || f->kind == 0) { f->has_t = 1; return BSG_OK; }
	cudaStream_t s = c->stream;
	const int n = f->n;
	int *perm = nullptr, nk = 0, *ti = nullptr, *tj = nullptr;
	int rc = bsg_strict_transpose(c, n, f->d_iu, f->d_ju, f->nnz, &ti, &tj, &perm, &nk);
	if (rc) return rc;
	cudaFreeAsync(ti, s);
	cudaFreeAsync(tj, s);
	BSG_CUDA(cudaMallocAsync(&f->d_utr_v, sizeof(double) * (nk > 0 ? nk : 1), s));
	BSG_COUNT(1);
	k_permute<<<nb(nk, 256), 256, 0, s>>>(nk, perm, f->d_u, f->d_utr_v);
	BSG_CUDA(cudaFreeAsync(perm, s));
	const int fp32 = f->fp32 ? 1 : 0;
	if (fp32) {
		BSG_CUDA(cudaMallocAsync(&f->d_utr_f, sizeof(float) * (nk > 0 ? nk : 1), s));
		BSG_CUDA(cudaMallocAsync(&f->d_l_f, sizeof(float) * (f->nnz > 0 ? f->nnz : 1), s));
		BSG_COUNT(2);
		k_to_f32<<<BSG_SMS * 4, 256, 0, s>>>(nk, f->d_utr_v, f->d_utr_f);
		k_to_f32<<<BSG_SMS * 4, 256, 0, s>>>(f->nnz, f->d_l, f->d_l_f);
	}
	rc = bsg_sell_build(c, n, f->d_lr_i, f->d_lr_j, f->d_utr_v, 0, fp32, &f->slt, SELL_SIGMA, fp32);
	if (!rc) rc = bsg_sell_build(c, n, f->d_iu, f->d_ju, f->d_l, 1, fp32, &f->sut, SELL_SIGMA, fp32);
	if (rc) return rc;
	BSG_CUDA(cudaGetLastError());
	f->has_t = 1;
	return BSG_OK;
}

int bsg_trisolve_t_launch(bsg_ctx *c, bsg_fct *f, int which, int mode, int nsweeps, const double *x, double *y,
                          double *work) {
	if (f->kind == 0) return bsg_trisolve_launch(c, f, which == 0 ? 1 : 0, mode, nsweeps, x, y, work);
	if (f->d_bia) return bsg_set_error(BSG_ERR_UNSUPPORTED, "transposed solves of a block factor");
	int rc = fct_build_transposes(c, f);
	if (rc) return rc;
	TriOp t;
	if (which == 0) { // U^T: lower, L-row pattern, U's values, U's inverse pivots
		t.lower = 1; t.rp = f->d_lr_i; t.ci = f->d_lr_j; t.skip = 0;
		t.vd = f->d_utr_v; t.vf = f->d_utr_f; t.dinv = f->d_dinv_u; t.sell = &f->slt;
	} else {          // L^T: upper, U's pattern, L's values, L's inverse pivots
		t.lower = 0; t.rp = f->d_iu; t.ci = f->d_ju; t.skip = 1;
		t.vd = f->d_l; t.vf = f->d_l_f; t.dinv = f->d_dinv_l; t.sell = &f->sut;
	}
	return trisolve_impl(c, f, t, mode, nsweeps, x, y, work);
}

// this unit's copy of the spin-wait bound (bsg_set_spin_limit_ns)
int bsg_spin_limit_set_trsv(unsigned long long ns) {
	return bsg_spin_limit_set_here(ns) == cudaSuccess ? BSG_OK : BSG_ERR_CUDA;
}
