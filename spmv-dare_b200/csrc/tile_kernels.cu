// Row tiles: one execution layout and one kernel for every format whose rows are summed in
// order (csr_naive, csr_vec, sell, sell_sorted, SELL-C-sigma; FP64, and FP32 with Dot2 rows).
//
// Layout.  The rows of a matrix are sorted by their number of stored entries inside windows of
// 1,024 rows (longest first, stable) and cut into slices of 32, so the rows of a slice have
// nearly the same length and padding is a few percent at most.  A slice of width W holds its
// values column-major (32 W entries) and its column indices row-major in tiles of 8 slice
// columns (entry (r, k) at k8 * 32 + r * tw + k - k8, k8 = k & ~7, tw = min(8, W - k8)): 32
// consecutive lanes then read x for 4 rows x 8 neighbouring columns.  Beside it, the y index
// and the entry count of every slot.  The format's own arrays are untouched (they are what
// spmv_export returns); the layout is built once at conversion.
//
// Kernel.  One warp per range of consecutive slices, which it takes tile by tile without a
// break between slices.  A lane owns a row.  Per tile it reads 8 column indices (two 16-byte
// loads) and its row's 8 values (16-byte loads), copies x asynchronously into the warp's shared
// buffer in gather order (4 rows x 8 neighbouring columns an instruction) and takes it from
// there in row order, adding to its row in the format's own operation order: y is bit-identical
// to the reference's.  Columns run two tiles ahead, x and values one, so no load's latency is
// waited for in turn; there is no barrier above the warp, and no state is written but y.
//
// What bounds it: under continuous load the chip's power limit holds the SMs near 1.67 GHz and
// the gather's L1 wavefronts (one per line and row segment) share the L1 pipe with the stream;
// alone, DRAM (csr_naive on 4M rows 174 us, 6.0 TB/s).  Measured in a loop over three matrices,
// before (warp-specialised CTAs staging blocks in shared memory, where row threads met in banks;
// SELL-C-sigma: a queue of register tiles with 16 warps an SM) and now: csr_naive 4M rows
// 213 -> 191 us, SELL-C-sigma 4M rows 224 -> 202, csr_vec 1M rows 150 -> 93, SELL 2M rows
// 160 -> 132, sell_sorted 700k rows 101 -> 62.  Tried on csr_naive when it took 198: x transposed between
// lanes by shuffles (16 warps of 114 registers an SM: 255 us), CTAs of 256 threads (202) and 128
// (199), bulk prefetches into L2 (1-10% slower), columns and x one tile further ahead (209),
// four threads a row straight from CSR (csr_vec 143: a wavefront per row and request).
//
// Rows too long for that (a lane would walk them for tens of microseconds) stay in the
// format's arrays: the first warp of a CTA takes one, its 32 lanes load and gather 256 entries
// ahead and one lane (csr_vec: one per lane of its order) sums them from shared memory.
#include <algorithm>

#include "internal.h"
#include "primitives.cuh"
#include "tile.h"

namespace spmv {

namespace {

constexpr int TILE_THREADS = 64;        // small CTAs: a finished pair of warps makes room at once
constexpr int TILE_WARPS = TILE_THREADS / 32;

constexpr int TILE_WINDOW = 1024;       // rows sorted together
constexpr int LONG_STEP = 256;          // entries a warp stages at a time of a long row
constexpr int64_t SLICE_COST = 128;     // entries' worth of a slice's bookkeeping
// csr_naive rows of fewer entries run kernel 4 at any size: it multiplies in its gather and adds from
// consecutive shared memory, and tiles spend their time on slices (4 M rows of 6 86 us and 104, 2 M of 5
// 38 and 45, 1 M of 9 28-36 and 31-40; 4 M of 13 136-182 and 130-177, 400,000 of 16 25 and 23).
constexpr int64_t NAIVE_MEAN = 12;
constexpr int64_t RANGE_COST = 2048;

// ------------------------------------------------------------------ arithmetic of a row
enum class Sum { NAIVE, FMA, LANES4, LANES8, DOT2, MIXED };

// One row's running state.  step<J, FULL>() adds the row's entry k (k % 8 == J), entries in
// order; FULL: k is known to be below the row's count n.  Past the count an operand that
// changes nothing takes the entry's place (adding -0.0 leaves every number as it is), so that
// the dependent chain is the bare additions.
template <Sum S>
struct RowSum;

struct SplitSum {                               // product and sum rounded separately (csr.cpp:167-182)
	using T = double;
	double s = 0.0;
	template <int J, bool FULL>
	__device__ __forceinline__ void step(int k, int n, double v, double x)
	{
		const double p = __dmul_rn(v, x);
		s = __dadd_rn(s, FULL || k < n ? p : -0.0);
	}
	__device__ __forceinline__ double total(int) const { return s; }
};
template <>
struct RowSum<Sum::NAIVE> : SplitSum {};

struct FusedSum {                               // one fused multiply-add per slice column
	using T = double;
	double s = 0.0, last = 0.0;                 // and the x of the last one
	template <int J, bool FULL>
	__device__ __forceinline__ void step(int k, int n, double v, double x)
	{
		s = __fma_rn(FULL || k < n ? v : -0.0, FULL || k < n ? x : 1.0, s);
		last = FULL || k < n ? x : last;
	}
	__device__ __forceinline__ double total(int) const { return s; }
};
template <>
struct RowSum<Sum::FMA> : FusedSum {};

template <>
struct RowSum<Sum::MIXED> : FusedSum {          // batches: either of the two, by slice
	bool split = false;
};

template <int L>
struct LaneSum {                                // csr_vec.cpp:183-211: L fused lanes, then the tail
	using T = double;
	double s[L], tail[L];
	__device__ __forceinline__ LaneSum()
	{
		#pragma unroll
		for (int l = 0; l < L; l++)
			s[l] = tail[l] = 0.0;
	}
	template <int J, bool FULL>                     // FULL: in a lane's part, not in the tail
	__device__ __forceinline__ void step(int k, int n, double v, double x)
	{
		constexpr int l = J % L;                    // k % L
		if (FULL || k < (n & ~(L - 1)))
			s[l] = __fma_rn(v, x, s[l]);
		else if (k < n)
			tail[l] = __dmul_rn(v, x);
	}
	__device__ __forceinline__ double total(int n) const
	{
		double t = (s[0] + s[2]) + (s[1] + s[3]);
		if (L == 8)
			t = (0.0 + t) + ((s[4] + s[6]) + (s[5] + s[7]));
		#pragma unroll
		for (int i = 0; i < L - 1; i++)
			if ((n & ~(L - 1)) + i < n)
				t = __dadd_rn(t, tail[i]);
		return t;
	}
};
template <>
struct RowSum<Sum::LANES4> : LaneSum<4> {};
template <>
struct RowSum<Sum::LANES8> : LaneSum<8> {};

template <>
struct RowSum<Sum::DOT2> {                      // FP32 values, compensated (Ogita, Rump, Oishi 2005)
	using T = float;
	float s = 0.0f, c = 0.0f;
	__device__ __forceinline__ void add(float v, float x)
	{
		const float p = __fmul_rn(v, x), pe = __fmaf_rn(v, x, -p);
		const float t = __fadd_rn(s, p), z = __fsub_rn(t, s);
		const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(p, z));
		s = t;
		c = __fadd_rn(c, __fadd_rn(e, pe));
	}
	template <int J, bool FULL>
	__device__ __forceinline__ void step(int k, int n, float v, float x)
	{
		if (FULL || k < n)
			add(v, x);
	}
	__device__ __forceinline__ float total(int) const { return __fadd_rn(s, c); }
};

// The 8 values of a lane's row in one tile: stored so that lanes read 16 bytes at a time,
// columns in pairs (double) or fours (float) per row, then what is left in pairs and singles.
template <typename T>
__host__ __device__ __forceinline__ int value_place(int j, int tw, int r)
{
	if (sizeof(T) == 4 && (j | 3) < tw)
		return (j & ~3) * 32 + r * 4 + (j & 3);
	if ((j | 1) < tw)
		return (j & ~1) * 32 + r * 2 + (j & 1);
	return j * 32 + r;
}

__device__ __forceinline__ void load_values(const double * tv, int tw, int lane, double (&v)[8])
{
	if (tw == 8) {
		const double2 * p = reinterpret_cast<const double2 *>(tv) + lane;
		#pragma unroll
		for (int i = 0; i < 4; i++) {
			const double2 d = __ldcs(p + i * 32);
			v[2 * i] = d.x;
			v[2 * i + 1] = d.y;
		}
		return;
	}
	#pragma unroll
	for (int p = 0; p < 8; p += 2) {
		if (p + 1 < tw) {
			const double2 d = __ldcs(reinterpret_cast<const double2 *>(tv + p * 32) + lane);
			v[p] = d.x;
			v[p + 1] = d.y;
		} else if (p < tw) {
			v[p] = __ldcs(tv + p * 32 + lane);
		}
	}
}

__device__ __forceinline__ void load_values(const float * tv, int tw, int lane, float (&v)[8])
{
	if (tw == 8) {
		const float4 * p = reinterpret_cast<const float4 *>(tv) + lane;
		#pragma unroll
		for (int i = 0; i < 2; i++) {
			const float4 d = __ldcs(p + i * 32);
			v[4 * i] = d.x;
			v[4 * i + 1] = d.y;
			v[4 * i + 2] = d.z;
			v[4 * i + 3] = d.w;
		}
		return;
	}
	#pragma unroll
	for (int p = 0; p < 8; p += 4) {
		if (p + 3 < tw) {
			const float4 d = __ldcs(reinterpret_cast<const float4 *>(tv + p * 32) + lane);
			v[p] = d.x;
			v[p + 1] = d.y;
			v[p + 2] = d.z;
			v[p + 3] = d.w;
		} else {
			if (p + 1 < tw) {
				const float2 d = __ldcs(reinterpret_cast<const float2 *>(tv + p * 32) + lane);
				v[p] = d.x;
				v[p + 1] = d.y;
				if (p + 2 < tw)
					v[p + 2] = __ldcs(tv + (p + 2) * 32 + lane);
			} else if (p < tw) {
				v[p] = __ldcs(tv + p * 32 + lane);
			}
		}
	}
}

// Column indices of a tile: row r = 4 q + r0 and column j belong to lane 8 r0 + j, which
// reads its eight (q = 0 .. 7) as two 16-byte words; a narrower tile leaves out the lanes of
// the columns it has not.
__host__ __device__ __forceinline__ int column_place(int j, int tw, int r)
{
	const int q = r >> 2, r0 = r & 3;
	return (q >> 2) * 16 * tw + (r0 * tw + j) * 4 + (q & 3);
}

// A warp's x buffer holds a tile row-major, 8 entries a row, in 16-byte units exchanged
// inside a row so that the 16-byte reads of 8 neighbouring rows meet in no bank: double,
// unit j / 2 ^ (r / 2) % 4; float, unit j / 4 ^ (r / 4) % 2.  gather_place: byte of a lane's
// entry of row r0 (q = 0); rows 4 q + r0 follow at q times four rows, FLIPped for odd q.
template <typename T>
struct XPlace;
template <>
struct XPlace<double> {
	static constexpr uint32_t FLIP = 32;
	static __device__ __forceinline__ uint32_t gather_place(int lane)
	{
		const int j = lane & 7, r0 = lane >> 3;
		return (uint32_t) (r0 * 64 + ((j >> 1) ^ (r0 >> 1)) * 16 + (j & 1) * 8);
	}
	static __device__ __forceinline__ uint32_t row_place(int r) { return (uint32_t) (r * 64 + ((r >> 1) & 3) * 16); }
	template <int J>
	static __device__ __forceinline__ void read(uint32_t row, double (&X)[4])     // entries J .. J + 3
	{
		asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(X[0]), "=d"(X[1]) : "r"(row ^ (J * 8)));
		asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(X[2]), "=d"(X[3]) : "r"(row ^ (J * 8 + 16)));
	}
};
template <>
struct XPlace<float> {
	static constexpr uint32_t FLIP = 16;
	static __device__ __forceinline__ uint32_t gather_place(int lane)
	{
		const int j = lane & 7, r0 = lane >> 3;
		return (uint32_t) (r0 * 32 + (j >> 2) * 16 + (j & 3) * 4);
	}
	static __device__ __forceinline__ uint32_t row_place(int r) { return (uint32_t) (r * 32 + ((r >> 2) & 1) * 16); }
	template <int J>
	static __device__ __forceinline__ void read(uint32_t row, float (&X)[4])
	{
		asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(X[0]), "=f"(X[1]), "=f"(X[2]), "=f"(X[3])
		             : "r"(row ^ (J * 4)));
	}
};

// The row's entries k0 .. k0 + 7 in order; the row has n.
template <bool FULL, typename A, typename T>
__device__ __forceinline__ void tile_steps(A & acc, int k0, int n, const T (&v)[8], uint32_t xrow)
{
	T X[4], Y[4];
	XPlace<T>::template read<0>(xrow, X);
	XPlace<T>::template read<4>(xrow, Y);
	acc.template step<0, FULL>(k0 + 0, n, v[0], X[0]);
	acc.template step<1, FULL>(k0 + 1, n, v[1], X[1]);
	acc.template step<2, FULL>(k0 + 2, n, v[2], X[2]);
	acc.template step<3, FULL>(k0 + 3, n, v[3], X[3]);
	acc.template step<4, FULL>(k0 + 4, n, v[4], Y[0]);
	acc.template step<5, FULL>(k0 + 5, n, v[5], Y[1]);
	acc.template step<6, FULL>(k0 + 6, n, v[6], Y[2]);
	acc.template step<7, FULL>(k0 + 7, n, v[7], Y[3]);
}

// tile_steps for the warp's tile, without masks where no row of it ends.
template <Sum S, typename A, typename T>
__device__ __forceinline__ void add_tile(A & acc, bool full, int k0, int n, const T (&v)[8], uint32_t xrow)
{
	if constexpr (S == Sum::MIXED) {
		if (acc.split) {
			SplitSum t;
			t.s = acc.s;
			add_tile<Sum::NAIVE>(t, full, k0, n, v, xrow);
			acc.s = t.s;
			return;
		}
	}
	if (full)
		tile_steps<true>(acc, k0, n, v, xrow);
	else
		tile_steps<false>(acc, k0, n, v, xrow);
}

// Asynchronous copy of one x entry into shared memory.
__device__ __forceinline__ void gather_async(uint32_t dst, const double * src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void gather_async(uint32_t dst, const float * src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void store_shared(uint32_t p, double v)
{
	asm volatile("st.shared.f64 [%0], %1;" ::"r"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void store_shared(uint32_t p, float v)
{
	asm volatile("st.shared.f32 [%0], %1;" ::"r"(p), "f"(v) : "memory");
}

struct TileArgs {
	const int32_t * sptr;     // first stored entry of each slice
	const int32_t * tcols;
	const void * vals;
	const int32_t * slot_row; // y index of each slot, -1: none
	const int32_t * slot_cnt; // entries of each slot
	const int32_t * pad;      // MIXED: each slice's pad column or arithmetic
	const void * x;
	void * y;
	int32_t pad_col;          // column that ends a padded row, PAD_OWN: its last one's
	const int4 * ranges;      // per warp: first slice, end, first entry, end of the first slice
	int nranges;
	const LongUnit * longs;
	int nlong;
};

// ------------------------------------------------------------------ long units
template <Sum S>
__device__ void long_unit(const TileArgs & a, const LongUnit & u, int lane, typename RowSum<S>::T * sv,
		typename RowSum<S>::T * sx)
{
	using T = typename RowSum<S>::T;
	constexpr int PER = LONG_STEP / 32;
	const T * __restrict__ x = static_cast<const T *>(a.x) + u.x_off;
	const T * __restrict__ vals = static_cast<const T *>(u.vals);
	const bool split = S == Sum::NAIVE || (S == Sum::MIXED && u.split);
	constexpr int L = S == Sum::LANES8 ? 8 : S == Sum::LANES4 ? 4 : 1;      // chains of the row
	const int nl = L > 1 ? u.n & ~(L - 1) : u.n;          // entries of the chains (the rest is csr_vec's tail)
	int32_t c[PER];
	T v[PER], vn[PER];
	auto at = [&](int e) { return (int64_t) e * u.stride; };
	auto load = [&](int e0) {
		#pragma unroll
		for (int i = 0; i < PER; i++) {
			const int e = e0 + i * 32 + lane;
			c[i] = e < u.n ? __ldcs(u.cols + at(e)) : 0;
			vn[i] = e < u.n ? __ldcs(vals + at(e)) : T(0);
		}
	};
	load(0);
	wait_previous();
	RowSum<S> acc;
	T s = T(0);
	for (int e0 = 0; e0 < u.n; e0 += LONG_STEP) {
		T xv[PER];
		#pragma unroll
		for (int i = 0; i < PER; i++) {
			const int e = e0 + i * 32 + lane;
			xv[i] = e < u.n ? load_x(x + c[i]) : T(0);
			v[i] = vn[i];
		}
		load(e0 + LONG_STEP);
		#pragma unroll
		for (int i = 0; i < PER; i++) {
			if (split) {
				sv[i * 32 + lane] = v[i] * xv[i];
			} else {
				sv[i * 32 + lane] = v[i];
				sx[i * 32 + lane] = xv[i];
			}
		}
		__syncwarp();
		const int cnt = nl - e0 < LONG_STEP ? nl - e0 : LONG_STEP;
		if (lane < L) {
			if constexpr (S == Sum::DOT2) {
				#pragma unroll 4
				for (int e = 0; e < cnt; e++)
					acc.add(sv[e], sx[e]);
			} else if (split) {
				#pragma unroll 8
				for (int e = 0; e < cnt; e++)
					s = __dadd_rn(s, sv[e]);
			} else {
				#pragma unroll 8
				for (int e = lane; e < cnt; e += L)
					s = __fma_rn(sv[e], sx[e], s);
			}
		}
		if (e0 + LONG_STEP < u.n)
			__syncwarp();
	}
	T * y = static_cast<T *>(a.y);
	if constexpr (L > 1) {
		T t = s + __shfl_down_sync(0xffffffffu, s, 2);
		t = t + __shfl_down_sync(0xffffffffu, t, 1);          // lane 0: (s0 + s2) + (s1 + s3)
		if (L == 8)
			t = (T(0) + t) + __shfl_down_sync(0xffffffffu, t, 4);
		if (lane == 0) {
			for (int e = nl; e < u.n; e++) {                  // the tail lies in the last step
				const int i = e % LONG_STEP;
				t = __dadd_rn(t, __dmul_rn(sv[i], sx[i]));
			}
			y[u.row] = t;
		}
	} else if constexpr (S == Sum::DOT2) {
		if (lane == 0)
			y[u.row] = acc.total(u.n);
	} else {
		if (lane == 0) {
			if (!split && u.padded)
				s = __fma_rn(0.0, load_x(x + (u.pad_col == PAD_OWN ? u.cols[at(u.n - 1)] : u.pad_col)), s);
			y[u.row] = s;
		}
	}
}

// ------------------------------------------------------------------ the kernel
// A slot's count; PADDED: the row's slice is wider than the row.  Any number of padding entries
// (value 0, one column) adds what one does: 0 * x is a zero, or NaN, and adding it again changes
// nothing.  So padding is not stored: one fused multiply-add with the pad column's x ends the row.
// SELL on 2M rows of 26 +- 3 in slices of 4: 137 -> 132 us, 500,000 rows of 50 +- 35 in slices of 8:
// 169 (kernel 4) -> 76, the 48-matrix batch 113 -> 98.
constexpr int PADDED = 1 << 30, COUNT = PADDED - 1;

// The tiles of a range in order.  next() gives the tile's width (0 .. 8) with TILE_LAST on the
// last one of a slice, and 0 past the end of the range; t0 is the tile's first entry.
constexpr uint32_t TILE_LAST = 16, TILE_BITS = 5, TILE_MASK = 31;

struct TileCursor {
	int t0 = 0, t1;           // this tile and the next
	int e, en;                // end of the next tile's slice, and of the slice after it
	int sl, sl_end;           // the next tile's slice
	__device__ __forceinline__ TileCursor(const int32_t * sptr, int4 range)
	{
		sl = range.x;
		sl_end = range.y;
		t1 = range.z;
		e = range.w;
		en = __ldg(sptr + (sl + 2 <= sl_end ? sl + 2 : sl_end));
	}
	__device__ __forceinline__ uint32_t next(const int32_t * sptr)
	{
		if (sl >= sl_end)
			return 0;
		t0 = t1;
		const int left = e - t0;
		if (left > 256) {
			t1 = t0 + 256;
			return 8;
		}
		t1 = e;                                              // slices of a range are contiguous
		sl++;
		e = en;
		en = __ldg(sptr + (sl + 2 <= sl_end ? sl + 2 : sl_end));
		return (uint32_t) left >> 5 | TILE_LAST;
	}
};

template <Sum S, int MINB, bool AHEAD, bool STAGED = false>
__global__ void __launch_bounds__(TILE_THREADS, MINB) tile_kernel(TileArgs a)
{
	using T = typename RowSum<S>::T;
	__shared__ __align__(128) T xs[TILE_WARPS][2][256];
	constexpr int WHOLE = S == Sum::LANES8 ? ~7 : S == Sum::LANES4 ? ~3 : ~0;   // csr_vec: the lanes' part of a row
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const int cta = (int) blockIdx.x;
	int w;
	release_next();
	if (cta < a.nlong) {
		if (wid == 0) {
			long_unit<S>(a, a.longs[cta], lane, xs[0][0], xs[0][1]);
			return;
		}
		w = cta * (TILE_WARPS - 1) + wid - 1;
	} else {
		w = cta * TILE_WARPS + wid - a.nlong;
	}
	const int4 range = w < a.nranges ? __ldg(a.ranges + w) : make_int4(0, 0, 0, 0);
	int sl = range.x;
	if (sl >= range.y) {
		wait_previous();
		return;
	}
	const T * __restrict__ x = static_cast<const T *>(a.x);
	const T * __restrict__ vals = static_cast<const T *>(a.vals);
	T * __restrict__ y = static_cast<T *>(a.y);
	constexpr uint32_t BUF = 256 * sizeof(T);                 // bytes of one x buffer
	const int col = lane & 7, r0 = lane >> 3;
	const uint32_t xbase = smem_u32(&xs[wid][0][0]);
	const uint32_t xdst = xbase + XPlace<T>::gather_place(lane), xrow = xbase + XPlace<T>::row_place(lane);
	int4 c0, c1;
	T v[AHEAD ? 2 : 1][8];
	auto load_cols = [&](int t0, int tw) {
		const int4 * __restrict__ tc = reinterpret_cast<const int4 *>(a.tcols + t0) + r0 * tw + col;
		if (col < tw) {
			c0 = __ldcs(tc);
			c1 = __ldcs(tc + 4 * tw);
		}
	};
	// x of the tile whose columns are held: copied into `buf`, or (STAGED) loaded into
	// registers that store_x() copies there
	T X[8];
	auto gather = [&](uint32_t buf, int tw) {
		if constexpr (STAGED) {
			if (col < tw) {
				X[0] = load_x(x + c0.x);
				X[1] = load_x(x + c0.y);
				X[2] = load_x(x + c0.z);
				X[3] = load_x(x + c0.w);
				X[4] = load_x(x + c1.x);
				X[5] = load_x(x + c1.y);
				X[6] = load_x(x + c1.z);
				X[7] = load_x(x + c1.w);
			}
			return;
		}
		if (col < tw) {
			const uint32_t d = xdst + buf, f = d ^ XPlace<T>::FLIP;
			constexpr uint32_t Q = 32 * sizeof(T);             // rows 4 q .. 4 q + 3
			gather_async(d + 0 * Q, x + c0.x);
			gather_async(f + 1 * Q, x + c0.y);
			gather_async(d + 2 * Q, x + c0.z);
			gather_async(f + 3 * Q, x + c0.w);
			gather_async(d + 4 * Q, x + c1.x);
			gather_async(f + 5 * Q, x + c1.y);
			gather_async(d + 6 * Q, x + c1.z);
			gather_async(f + 7 * Q, x + c1.w);
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	auto store_x = [&](uint32_t buf, int tw) {
		if (col < tw) {
			const uint32_t d = xdst + buf, f = d ^ XPlace<T>::FLIP;
			#pragma unroll
			for (int i = 0; i < 8; i++)
				store_shared((i & 1 ? f : d) + i * (uint32_t) (32 * sizeof(T)), X[i]);
		}
	};
	// tile 0: columns, x and values under way; tile 1: columns.  q holds the widths of the tile
	// being summed and the two after it, 5 bits each.
	TileCursor cu(a.sptr, range);
	int t0 = cu.t1, b = t0;                                  // the tile being summed, its slice
	uint32_t q = cu.next(a.sptr);
	load_cols(t0, q & 15);
	load_values(vals + t0, q & 15, lane, v[0]);
	int n = __ldg(a.slot_cnt + (int64_t) sl * 32 + lane), row = __ldg(a.slot_row + (int64_t) sl * 32 + lane);
	const uint32_t d1 = cu.next(a.sptr);
	wait_previous();
	gather(0, q & 15);
	if constexpr (STAGED)
		store_x(0, q & 15);
	load_cols(cu.t0, d1 & 15);
	q |= d1 << TILE_BITS;
	int nn = 0, rown = -1;                                   // the next slice's counts and rows, loaded ahead
	if (sl + 1 < range.y) {
		nn = __ldg(a.slot_cnt + (int64_t) (sl + 1) * 32 + lane);
		rown = __ldg(a.slot_row + (int64_t) (sl + 1) * 32 + lane);
	}
	RowSum<S> acc;
	int pad = a.pad_col;
	if constexpr (S == Sum::MIXED) {
		pad = a.pad[sl];
		acc.split = pad == PAD_SPLIT;
	}
	uint32_t buf = 0;
	// one tile, its values in vt; the next tile's go to vn.  Returns false after the last.
	auto tile = [&](T (&vt)[8], T (&vn)[8]) -> bool {
		const int t1 = t0 + (int) (q & 15) * 32;
		gather(buf ^ BUF, q >> TILE_BITS & 15);
		if (AHEAD)
			load_values(vals + t1, q >> TILE_BITS & 15, lane, vn);
		const uint32_t dn = cu.next(a.sptr);
		load_cols(cu.t0, dn & 15);
		q |= dn << (2 * TILE_BITS);
		if constexpr (!STAGED)
			asm volatile("cp.async.wait_group 1;" ::: "memory");
		__syncwarp();
		const int k0 = (t0 - b) >> 5;
		const int cnt = n & COUNT;
		const bool full = __all_sync(0xffffffffu, k0 + 8 <= (cnt & WHOLE));
		add_tile<S>(acc, full, k0, cnt, vt, xrow + buf);
		if (!AHEAD)
			load_values(vals + t1, q >> TILE_BITS & 15, lane, vn);
		if constexpr (STAGED)
			store_x(buf ^ BUF, q >> TILE_BITS & 15);
		__syncwarp();                                        // every lane has read the buffer that is gathered into next
		const bool last = (q & TILE_LAST) != 0;
		q >>= TILE_BITS;
		t0 = t1;
		buf ^= BUF;
		if (last) {
			if constexpr (S == Sum::FMA || S == Sum::MIXED)
				if (n & PADDED)
					acc.s = __fma_rn(0.0, pad == PAD_OWN ? acc.last : load_x(x + pad), acc.s);
			if (row >= 0)
				y[row] = acc.total(n);
			if ((q & TILE_MASK) == 0)
				return false;
			acc = RowSum<S>();
			sl++;
			if constexpr (S == Sum::MIXED) {
				pad = a.pad[sl];
				acc.split = pad == PAD_SPLIT;
			}
			b = t1;
			n = nn;
			row = rown;
			if (sl + 1 < range.y) {
				nn = __ldg(a.slot_cnt + (int64_t) (sl + 1) * 32 + lane);
				rown = __ldg(a.slot_row + (int64_t) (sl + 1) * 32 + lane);
			}
		}
		return true;
	};
	if constexpr (AHEAD) {
		while (tile(v[0], v[1]) && tile(v[1], v[0])) {
		}
	} else {
		while (tile(v[0], v[0])) {
		}
	}
}

// ------------------------------------------------------------------ building the layout
// Entries of row i of a source: start and stride in its arrays, count, and whether padding
// follows them (a row that is all padding keeps one entry of it).
__device__ __forceinline__ bool source_row(const TileSource & s, int64_t i, int64_t & start, int & stride, int & cnt)
{
	if (s.V == 1) {
		start = s.P[i];
		stride = 1;
		cnt = (int) ((int64_t) s.P[i + 1] - start);
	} else {
		const int64_t sl = i / s.V, p = s.P[sl];
		start = p + i % s.V;
		stride = s.V;
		cnt = (int) (((int64_t) s.P[sl + 1] - p) / s.V);
	}
	if (!s.rp)
		return false;
	const int64_t r = s.ymap ? s.ymap[i] : i;
	const int len = s.rp[r + 1] - s.rp[r];
	if (len == 0)
		cnt = cnt > 0 ? 1 : 0;
	const bool padded = len > 0 && len < cnt;
	if (padded)
		cnt = len;
	return padded;
}

// What the sort notes about the rows, beside the number of long ones: the next long row's place, the
// longest row, the widest slice, and lines of x in the first entries of every eighth window's rows.
enum { NEXT = 1, LONGEST, WIDEST, LINES, LINES_OF, STATS };

// One CTA per window: its rows sorted by count (descending, stable; long rows and the places
// past the matrix last), their slots written, and the width of every slice.  A bitonic sort of
// 1,024 keys in shared memory; key = (max - count) << 10 | place.
__global__ void __launch_bounds__(TILE_WINDOW / 2) tile_sort_kernel(TileSource s, int long_min, int64_t slot0,
		int64_t nslots, int32_t * slot_src, int32_t * slot_row, int32_t * slot_cnt, int64_t * width, int * stat)
{
	__shared__ uint32_t key[TILE_WINDOW];
	const int64_t base = (int64_t) blockIdx.x * TILE_WINDOW;
	constexpr uint32_t MOST = (1u << 21) - 1;
	for (int i = threadIdx.x; i < TILE_WINDOW; i += blockDim.x) {
		uint32_t rank = MOST;                         // nothing to sum here
		int64_t start;
		int stride, cnt = 0;
		if (base + i < s.m) {
			source_row(s, base + i, start, stride, cnt);
			if (cnt >= long_min) {
				atomicAdd(&stat[0], 1);
			} else {
				rank = MOST - 1 - (uint32_t) cnt;
			}
		}
		key[i] = rank << 10 | (uint32_t) i;
		const int most = __reduce_max_sync(0xffffffffu, cnt);        // TILE_WINDOW: whole warps
		if ((i & 31) == 0 && most > *(volatile int *) &stat[LONGEST])
			atomicMax(&stat[LONGEST], most);
		// lines of x at the start of some rows
		if (blockIdx.x % 8 == 0) {
			const int seen = cnt < 8 ? cnt : 8;
			int lines = seen > 0, line = seen > 0 ? s.cols[start] >> 4 : 0;
			for (int k = 1; k < seen; k++) {
				const int at = s.cols[start + (int64_t) k * stride] >> 4;
				lines += at != line;
				line = at;
			}
			lines = __reduce_add_sync(0xffffffffu, lines);
			const int of = __reduce_add_sync(0xffffffffu, seen);
			if ((i & 31) == 0) {
				atomicAdd(&stat[LINES], lines);
				atomicAdd(&stat[LINES_OF], of);
			}
		}
	}
	for (int size = 2; size <= TILE_WINDOW; size <<= 1)
		for (int step = size >> 1; step > 0; step >>= 1) {
			__syncthreads();
			const int t = threadIdx.x;
			const int lo = 2 * step * (t / step) + t % step, hi = lo + step;
			const bool up = (lo & size) == 0;
			const uint32_t p = key[lo], q = key[hi];
			if ((p > q) == up) {
				key[lo] = q;
				key[hi] = p;
			}
		}
	__syncthreads();
	for (int i = threadIdx.x; i < TILE_WINDOW; i += blockDim.x) {
		if (base + i >= nslots)
			break;
		const uint32_t rank = key[i] >> 10;
		const int64_t r = base + (key[i] & (TILE_WINDOW - 1));
		const int cnt = rank == MOST ? 0 : (int) (MOST - 1 - rank);
		const int64_t slot = slot0 + base + i;
		slot_src[slot] = rank == MOST ? -1 : (int32_t) r;
		slot_row[slot] = rank == MOST ? -1 : (int32_t) (s.y_off + (s.ymap ? s.ymap[r] : r));
		int64_t start;
		int stride, own;
		slot_cnt[slot] = rank != MOST && source_row(s, r, start, stride, own) ? cnt | PADDED : cnt;
		if (i % 32 == 0)
			width[slot / 32] = (int64_t) cnt * 32;
		if (i == 0)
			atomicMax(&stat[WIDEST], cnt);
	}
}

// Rows of at least so many entries, among the source's.
constexpr int CENSUS = 6;
struct Census {
	int64_t length[CENSUS];
};
__global__ void long_census_kernel(TileSource s, Census c, int * count)
{
	const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
	int64_t start;
	int stride, cnt = 0;
	if (i < s.m)
		source_row(s, i, start, stride, cnt);
	#pragma unroll
	for (int k = 0; k < CENSUS; k++) {
		const unsigned b = __ballot_sync(0xffffffffu, i < s.m && cnt >= c.length[k]);
		if ((threadIdx.x & 31) == 0 && b)
			atomicAdd(count + k, __popc(b));
	}
}

__global__ void tile_sptr_kernel(const int64_t * in, int64_t n, int32_t * out)
{
	const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n)
		out[i] = (int32_t) in[i];
}

// One warp per slice, a lane per row: the entries into the tiled layout.
template <typename T>
__global__ void tile_fill_kernel(TileSource s, int64_t slice0, int64_t nslices, const int32_t * slot_src,
		const int32_t * sptr, int32_t * tcols, T * tvals, int32_t * pad_of)
{
	const int64_t i = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int r = threadIdx.x & 31;
	if (i >= nslices)
		return;
	const int64_t sl = slice0 + i;
	const int64_t b = sptr[sl];
	const int W = (int) ((sptr[sl + 1] - b) >> 5);
	const int src = slot_src[sl * 32 + r];
	int64_t start = 0;
	int stride = 1, cnt = 0;
	if (src >= 0)
		source_row(s, src, start, stride, cnt);
	if (pad_of && r == 0)
		pad_of[sl] = s.split ? PAD_SPLIT : s.pad_col == PAD_OWN ? PAD_OWN : (int32_t) (s.pad_col + s.x_off);
	int32_t pad = cnt > 0 ? s.cols[start] : 0;      // columns of the padding: read, never summed
	for (int k8 = 0; k8 < W; k8 += 8) {
		const int tw = W - k8 < 8 ? W - k8 : 8;
		#pragma unroll
		for (int j = 0; j < 8; j++) {
			if (j >= tw)
				break;
			const int k = k8 + j;
			T v = T(0);
			if (k < cnt) {
				pad = s.cols[start + (int64_t) k * stride];
				v = (T) s.vals[start + (int64_t) k * stride];
			}
			tcols[b + (int64_t) k8 * 32 + column_place(j, tw, r)] = pad + (int32_t) s.x_off;
			tvals[b + (int64_t) k8 * 32 + value_place<T>(j, tw, r)] = v;
		}
	}
}

// First slice whose cost prefix (entries and SLICE_COST a slice) reaches `target`.
__device__ __forceinline__ int64_t cost_slice(const int32_t * sptr, int64_t ns, int64_t target)
{
	int64_t lo = 0, hi = ns;
	while (lo < hi) {
		const int64_t mid = (lo + hi) >> 1;
		if ((int64_t) sptr[mid] + mid * SLICE_COST < target)
			lo = mid + 1;
		else
			hi = mid;
	}
	return lo;
}

__global__ void tile_ranges_kernel(const int32_t * sptr, int64_t ns, int64_t share, int64_t nranges, int4 * ranges)
{
	const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= nranges)
		return;
	const int64_t s0 = cost_slice(sptr, ns, i * share);
	const int64_t s1 = i + 1 == nranges ? ns : cost_slice(sptr, ns, (i + 1) * share);
	ranges[i] = make_int4((int) s0, (int) s1, sptr[s0], s0 < s1 ? sptr[s0 + 1] : sptr[s0]);
}

// Over evenly spaced slices (a warp each): the lines of x that rows of one gather instruction
// share (lines[0]: counted row by row less counted once) and the stored entries (lines[1]).
__global__ void gather_lines_kernel(const int32_t * sptr, const int32_t * tcols, int64_t ns, int64_t step,
		unsigned long long * lines)
{
	const int64_t sl = (((int64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 5) * step;
	if (sl >= ns)
		return;
	const int lane = threadIdx.x & 31, col = lane & 7, r0 = lane >> 3;
	unsigned once = 0, rows = 0;
	for (int t0 = sptr[sl]; t0 < sptr[sl + 1]; t0 += 256) {
		const int left = (sptr[sl + 1] - t0) >> 5, tw = left < 8 ? left : 8;
		for (int q = 0; q < 8; q++) {
			const int line = col < tw ? tcols[t0 + column_place(col, tw, 4 * q + r0)] >> 4 : -1;
			const unsigned m = __match_any_sync(0xffffffffu, line);
			const unsigned mine = m & (0xffu << (8 * r0));
			once += __popc(__ballot_sync(0xffffffffu, line >= 0 && __ffs(m) - 1 == lane));
			rows += __popc(__ballot_sync(0xffffffffu, line >= 0 && __ffs(mine) - 1 == lane));
		}
	}
	if (lane == 0) {
		atomicAdd(&lines[0], rows - once);
		atomicAdd(&lines[1], sptr[sl + 1] - sptr[sl]);
	}
}

template <typename T>
__global__ void long_units_kernel(TileSource s, const T * vals, int long_min, int * next, LongUnit * out)
{
	const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= s.m)
		return;
	int64_t start;
	int stride, cnt;
	const bool padded = source_row(s, i, start, stride, cnt);
	if (cnt < long_min)
		return;
	LongUnit u;
	u.padded = padded;
	u.pad_col = s.pad_col;
	u.cols = s.cols + start;
	u.vals = vals + start;
	u.n = cnt;
	u.stride = stride;
	u.x_off = (int32_t) s.x_off;
	u.split = s.split;
	u.row = (int32_t) (s.y_off + (s.ymap ? s.ymap[i] : i));
	out[atomicAdd(next, 1)] = u;
}

using TileFn = void (*)(TileArgs);

// STAGED: the gather's asynchronous copies fetch a line once for every row of the instruction
// that reads it; plain loads fetch it once, but x then passes through registers to the shared
// buffer.  Rows that share columns decide: 1.5M rows of 40, no neighbours, pairs of equal rows
// 170 us copied and 154 staged (0.29 lines an entry saved), a third in such pairs 177 and 174
// (0.13), none 192 and 199; csr_naive on 4M rows (0.06) 196 and 206; SELL 2M rows (0.17) 140 and
// 134.  Measured on a sample of the slices at conversion, for the sums in order of a single
// FP64 matrix: csr_vec's lanes, FP32 and mixed batches have no such build.
//
// Two builds of the plain sums.  WIDE (12 CTAs an SM, 80 registers a thread, a tile's values
// loaded after the tile before it is summed) for matrices of many ranges a warp: csr_naive on
// 4M rows 200 us against 206.  DEEP (10 CTAs, values a whole tile ahead) below: 0.31 us a tile of
// a lone slice against 0.40, csr_naive on 60,000 equal rows of 19 5.25 us against 5.65.
constexpr int WIDE_CTAS = 12, DEEP_CTAS = 10, LANES_CTAS = 9;

// The arithmetic first, its builds after: a build stands for one order of operations.
TileFn tile_fn(const TilePlan & p)
{
	if (p.mixed)
		return p.wide ? tile_kernel<Sum::MIXED, WIDE_CTAS, false> : tile_kernel<Sum::MIXED, DEEP_CTAS, true>;
	if (p.f32)
		return p.wide ? tile_kernel<Sum::DOT2, WIDE_CTAS, false> : tile_kernel<Sum::DOT2, DEEP_CTAS, true>;
	if (p.lanes)
		return p.lanes == 8 ? tile_kernel<Sum::LANES8, LANES_CTAS, false> : tile_kernel<Sum::LANES4, LANES_CTAS, false>;
	if (p.split)
		return p.staged ? tile_kernel<Sum::NAIVE, WIDE_CTAS, false, true>
		     : p.wide   ? tile_kernel<Sum::NAIVE, WIDE_CTAS, false>
		                : tile_kernel<Sum::NAIVE, DEEP_CTAS, true>;
	return p.staged ? tile_kernel<Sum::FMA, WIDE_CTAS, false, true>
	     : p.wide   ? tile_kernel<Sum::FMA, WIDE_CTAS, false>
	                : tile_kernel<Sum::FMA, DEEP_CTAS, true>;
}

// The kernel that takes less time than row tiles, or 0.  Row tiles give a slice of 32 rows to a warp, which
// waits for x tile by tile; below two slices a resident warp (190,000 rows on 148 SMs) the widest
// slices are their time, and matrices of few long rows took up to eight times as long as on kernel 4
// (2,000 rows of 2,000, SELL 35 us and 282; csr_naive 6,000 rows of 600 39 and 94, 40,000 of 100 18
// and 26).  us an entry of the mean and of the widest slice by the slices an SM has: measured 0.14,
// 0.19 and 0.25 with 1, 4 and 12 or more of even rows of 0.4 lines an entry, half of that with
// consecutive columns; 0.08 to 0.14 where a few are widest.
//
// Slices of 32 even rows of 100 entries and more have kernel 10 besides, whose warps take a slice at a
// time at any size: 60,000 rows of 200 35 us (tiles 57, kernel 4 50), 120,000 of 100 37 (43, 49), 200,000
// of 200 92 (103, 147); shorter or uneven rows are the tiles' (700,000 of 30 62 and 60).
int faster_kernel(const StagedTime & k, int V, bool f32, int64_t entries, int64_t rows, int64_t stored, int64_t slices,
		const int * stat, int num_sms)
{
	const int longest = stat[LONGEST], widest = stat[WIDEST];
	const double mean = (double) entries / rows, slice = (double) stored / (32 * slices), an_sm = (double) slices / num_sms;
	const bool enough = slices >= (int64_t) num_sms * 2 * DEEP_CTAS * TILE_WARPS;
	const bool ten = V == 32 && mean >= 96 && longest < 2 * mean;
	if (enough && !ten)
		return 0;
	const double lines = std::min(1.0, 0.35 + 1.66 * stat[LINES] / std::max(stat[LINES_OF], 1));
	const double even = lines * std::min(0.15 + 0.009 * an_sm, 0.25), few = lines * std::min(0.08 + 0.004 * an_sm, 0.13);
	double tiles = stored * (f32 ? 1.6e-6 : 2.7e-6);
	if (!enough)
		tiles = std::max(tiles, std::max(slice * even, widest * few));
	tiles = std::max(tiles, longest * 0.005);
	double staged = entries * 1e-6 * std::min(k.base + mean / k.per_length, k.most);
	if (widest > 2 * slice)
		staged *= k.uneven;
	const double chain = longest > k.chain_from ? longest * k.chain * 1e-3 : 0.0;
	// far longer rows than the rest come together and wait for each other
	staged = longest > 8 * mean ? staged + chain : std::max(staged, chain);
	if (ten) {
		const double t = std::max(std::max(30.0, 7 + entries * 1.8e-6), widest * 0.09);
		if (t < staged)
			return t < 0.95 * tiles ? 10 : 0;
	}
	return staged < 0.95 * tiles && !enough ? 4 : 0;
}

int lay_out(TilePlan & p, const std::vector<TileSource> & src, int lanes, bool f32, bool mixed, const StagedTime * staged,
		int num_sms, cudaStream_t s, const std::function<int(void **, size_t)> & alloc)
{
	p.f32 = f32;
	p.mixed = mixed;
	p.lanes = lanes;
	int64_t nslots = 0, entries = 0, rows = 0;
	std::vector<int64_t> slot0;
	for (const TileSource & t : src) {
		slot0.push_back(nslots);
		nslots += ceil_div(t.m, 32) * 32;
		entries += t.entries;
		rows += t.m;
	}
	const int64_t ns = nslots / 32;
	if (rows == 0) {
		p.built = true;
		return SPMV_OK;
	}
	const int64_t mean = entries / rows;
	if (staged && src[0].split && !f32 && mean < NAIVE_MEAN) {
		p.faster = 4;
		return SPMV_OK;
	}
	// From how many entries a row gets a warp of its own.  A lane adds 8 entries of its row in
	// 0.3 us at best (2 us with every SM full), a warp of its own a row in 3 us and 5 ns an entry.
	// Launches of 10 us and more (12 bytes an entry at 6 TB/s): rows that would take a lane about
	// a fifth of the launch, and four times the mean (sell_sorted, 700k rows with rows up to
	// 1,830: 112 us with 192 entries and four rows a unit, 66 so).  Shorter ones wait for their
	// longest rows alone: as many long rows as the chip holds warps beside the slices.
	DevBuf cnt;
	SPMV_TRY(cnt.alloc((STATS + CENSUS) * sizeof(int), s));
	const int64_t us = 4 + entries * 12 / 6000000;
	int64_t lm = 2 * us < 512 ? 2 * us : 512;
	lm = lm > 4 * mean ? lm : 4 * mean;
	lm = lm > 32 ? lm : 32;
	const bool brief = us < 10;
	auto count_rows = [&](const Census & c, int (&rows_of)[CENSUS]) -> int {
		SPMV_CUDA_TRY(cudaMemsetAsync(cnt.as<int>() + STATS, 0, sizeof(rows_of), s));
		for (const TileSource & t : src) {
			if (t.m > 0)
				long_census_kernel<<<(unsigned) ceil_div(t.m, 256), 256, 0, s>>>(t, c, cnt.as<int>() + STATS);
			SPMV_CUDA_TRY(cudaGetLastError());
		}
		SPMV_CUDA_TRY(cudaMemcpyAsync(rows_of, cnt.as<int>() + STATS, sizeof(rows_of), cudaMemcpyDeviceToHost, s));
		SPMV_CUDA_TRY(cudaStreamSynchronize(s));
		return SPMV_OK;
	};
	Census c;
	int census[CENSUS];
	if (brief) {
		for (int i = 0; i < CENSUS; i++)
			c.length[i] = std::max((i + 2) * mean / 2, (int64_t) 32);
		SPMV_TRY(count_rows(c, census));
		for (int i = 0; i < CENSUS; i++)
			if (census[i] + ns <= (int64_t) num_sms * DEEP_CTAS * TILE_WARPS) {
				lm = c.length[i];
				break;
			}
	}
	std::vector<int> long_min;                  // a batch's matrices: four times their own mean at least
	for (const TileSource & t : src) {
		const int64_t own = src.size() > 1 && t.m > 0 ? 4 * (t.entries / t.m) : 0;
		lm = lm > (1 << 21) - 3 ? (1 << 21) - 3 : lm;
		long_min.push_back((int) (own > lm && own < (1 << 21) - 3 ? own : lm));
	}
	if (4 * mean >= (1 << 21) - 3 || nslots > INT32_MAX - 64)
		return SPMV_OK;
	DevBuf d_src, width, sptr64;
	SPMV_TRY(d_src.alloc(nslots * sizeof(int32_t), s));
	SPMV_TRY(width.alloc(ns * sizeof(int64_t), s));
	SPMV_TRY(sptr64.alloc((ns + 1) * sizeof(int64_t), s));
	SPMV_TRY(alloc((void **) &p.slot_row, nslots * sizeof(int32_t)));
	SPMV_TRY(alloc((void **) &p.slot_cnt, nslots * sizeof(int32_t)));
	int64_t total = 0;
	int stat[STATS];
	for (int pass = 0;; pass++) {
		SPMV_CUDA_TRY(cudaMemsetAsync(cnt.p, 0, STATS * sizeof(int), s));
		for (size_t i = 0; i < src.size(); i++) {
			if (src[i].m == 0)
				continue;
			tile_sort_kernel<<<(unsigned) ceil_div(src[i].m, TILE_WINDOW), TILE_WINDOW / 2, 0, s>>>(src[i], long_min[i], slot0[i],
					ceil_div(src[i].m, 32) * 32, d_src.as<int32_t>(), p.slot_row, p.slot_cnt, width.as<int64_t>(), cnt.as<int>());
			SPMV_CUDA_TRY(cudaGetLastError());
		}
		SPMV_TRY(scan_exclusive(width.as<int64_t>(), sptr64.as<int64_t>(), ns, s));
		SPMV_CUDA_TRY(cudaMemcpyAsync(&total, sptr64.as<int64_t>() + ns, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
		SPMV_CUDA_TRY(cudaMemcpyAsync(stat, cnt.p, sizeof(stat), cudaMemcpyDeviceToHost, s));
		SPMV_CUDA_TRY(cudaStreamSynchronize(s));
		// Many long rows in a longer launch of one matrix: once more with the length from which the warps
		// of the long ones (3.2 us each) and the wait for the widest slice take least (csr_vec, 1 M rows of 12,
		// exponential lengths: 9,400 rows from 56 entries on 67 us, 900 from 84 on 54).
		const double warps_us = 3.2 / (num_sms * DEEP_CTAS), entry_us = 0.13;
		if (pass > 0 || brief || src.size() > 1 || stat[0] * warps_us < lm / 2 * entry_us)
			break;
		for (int i = 0; i < CENSUS; i++)
			c.length[i] = (i + 3) * lm / 2;
		SPMV_TRY(count_rows(c, census));
		double least = stat[0] * warps_us + lm * entry_us;
		for (int i = 0; i < CENSUS; i++)
			if (census[i] * warps_us + c.length[i] * entry_us < least) {
				least = census[i] * warps_us + c.length[i] * entry_us;
				long_min[0] = (int) std::min(c.length[i], (int64_t) ((1 << 21) - 3));
			}
		if (long_min[0] == lm)
			break;
	}
	const int nlong = stat[0];
	if (total > INT32_MAX - 4096 || total > entries + entries / 3 + 65536)
		return SPMV_OK;
	if (staged)
		p.faster = faster_kernel(*staged, src[0].V, f32, entries, rows, total, ns, stat, num_sms);
	if (p.faster)
		return SPMV_OK;
	const size_t vs = f32 ? sizeof(float) : sizeof(double);
	SPMV_TRY(alloc((void **) &p.sptr, (ns + 1) * sizeof(int32_t)));
	SPMV_TRY(alloc((void **) &p.tcols, total * sizeof(int32_t)));
	SPMV_TRY(alloc((void **) &p.vals, total * vs));
	if (mixed)
		SPMV_TRY(alloc((void **) &p.pad, ns * sizeof(int32_t)));
	SPMV_TRY(alloc((void **) &p.longs, nlong * sizeof(LongUnit)));
	tile_sptr_kernel<<<(unsigned) ceil_div(ns + 1, 256), 256, 0, s>>>(sptr64.as<int64_t>(), ns + 1, p.sptr);
	SPMV_CUDA_TRY(cudaGetLastError());
	for (size_t i = 0; i < src.size(); i++) {
		const int64_t n = ceil_div(src[i].m, 32);
		if (n == 0)
			continue;
		const unsigned g = (unsigned) ceil_div(n * 32, 256);
		const unsigned gl = (unsigned) ceil_div(src[i].m, 256);
		if (f32) {
			tile_fill_kernel<float><<<g, 256, 0, s>>>(src[i], slot0[i] / 32, n, d_src.as<int32_t>(), p.sptr, p.tcols,
					(float *) p.vals, p.pad);
			if (nlong > 0)
				long_units_kernel<float><<<gl, 256, 0, s>>>(src[i], src[i].vals_f, long_min[i], cnt.as<int>() + NEXT, p.longs);
		} else {
			tile_fill_kernel<double><<<g, 256, 0, s>>>(src[i], slot0[i] / 32, n, d_src.as<int32_t>(), p.sptr, p.tcols,
					(double *) p.vals, p.pad);
			if (nlong > 0)
				long_units_kernel<double><<<gl, 256, 0, s>>>(src[i], src[i].vals, long_min[i], cnt.as<int>() + NEXT, p.longs);
		}
		SPMV_CUDA_TRY(cudaGetLastError());
	}
	const int64_t cost = total + ns * SLICE_COST;
	// ranges of at most RANGE_COST entries, as many as fill the resident warps a whole number of
	// times, none smaller than a slice: csr_naive on 4M rows takes 195-199 us with 1,536 to 3,072
	// and 209 with 1,024, SELL on 2M rows 144 and 148 (each range starts with a chain of four
	// dependent loads); one long range a warp takes 230 and 184 (with 256-thread CTAs)
	const int64_t warps = (int64_t) num_sms * WIDE_CTAS * TILE_WARPS;
	int64_t share = ceil_div(cost, warps * ceil_div(cost, warps * RANGE_COST));
	share = share > cost / ns ? share : cost / ns;
	share = share > 1 ? share : 1;
	p.nranges = ceil_div(cost, share);
	p.wide = cost > 4 * warps * RANGE_COST;
	p.staged = false;
	if (p.wide && !f32 && !mixed && lanes == 0) {
		DevBuf lines;
		unsigned long long l[2];
		SPMV_TRY(lines.alloc(sizeof(l), s));
		SPMV_CUDA_TRY(cudaMemsetAsync(lines.p, 0, sizeof(l), s));
		gather_lines_kernel<<<256, 128, 0, s>>>(p.sptr, p.tcols, ns, ceil_div(ns, 1024), lines.as<unsigned long long>());
		SPMV_CUDA_TRY(cudaGetLastError());
		SPMV_CUDA_TRY(cudaMemcpyAsync(l, lines.p, sizeof(l), cudaMemcpyDeviceToHost, s));
		SPMV_CUDA_TRY(cudaStreamSynchronize(s));
		p.staged = (double) l[0] >= 0.13 * (double) l[1];
	}
	p.nlong = nlong;
	SPMV_TRY(alloc((void **) &p.ranges, p.nranges * sizeof(int4)));
	tile_ranges_kernel<<<(unsigned) ceil_div(p.nranges, 256), 256, 0, s>>>(p.sptr, ns, share, p.nranges, p.ranges);
	SPMV_CUDA_TRY(cudaGetLastError());
	p.grid = ceil_div(p.nranges + nlong, TILE_WARPS);
	if (p.grid < nlong)
		p.grid = nlong;
	p.split = src[0].split;
	p.pad_col = src[0].pad_col;
	p.built = true;
	return SPMV_OK;
}

}  // namespace

int build_tiles(TilePlan & p, const std::vector<TileSource> & src, int lanes, bool f32, bool mixed,
		const StagedTime * staged, int num_sms, cudaStream_t s, const TileMemory & memory)
{
	std::vector<void *> taken;
	p = TilePlan();
	const int st = lay_out(p, src, lanes, f32, mixed, staged, num_sms, s, [&](void ** a, size_t bytes) {
		const int got = memory.take(a, bytes);
		if (got == SPMV_OK)
			taken.push_back(*a);
		return got;
	});
	if (!p.built) {
		for (void * a : taken)
			memory.drop(a);
		const int faster = p.faster;
		p = TilePlan();
		p.faster = faster;
	}
	if (st == SPMV_ERR_NOMEM) {
		clear_error();
		return SPMV_OK;
	}
	return st;
}

int launch_tiles(const TilePlan & p, const void * x, void * y, cudaStream_t s)
{
	if (p.grid == 0)
		return SPMV_OK;
	TileArgs a{};
	a.sptr = p.sptr;
	a.tcols = p.tcols;
	a.vals = p.vals;
	a.slot_row = p.slot_row;
	a.slot_cnt = p.slot_cnt;
	a.pad = p.pad;
	a.pad_col = p.pad_col;
	a.x = x;
	a.y = y;
	a.ranges = p.ranges;
	a.nranges = (int) p.nranges;
	a.longs = p.longs;
	a.nlong = (int) p.nlong;
	SPMV_CUDA_TRY(launch_overlapped(tile_fn(p), (unsigned) p.grid, TILE_THREADS, 0, s, a));
	return SPMV_OK;
}

}  // namespace spmv
