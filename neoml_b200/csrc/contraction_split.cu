// The large dense contractions at fp32 accuracy on fp16 tensor cores (tcgen05.mma kind::f16, fp32 accumulators in TMEM).
//
//   C[M x N] = act( A[M x K] * B[N x K]^T + bias + residual ),   A, C fp32, B in the split form split_rows_kernel makes
//
// Arithmetic.  Every fp32 operand x is scaled by a power of two s (one per row of A, one per row of B), and
//   hi = fp16( s x ),  lo = fp16( 2^11 (s x - hi) )
// keep 22 significant bits of it (both steps round to nearest, s x - hi is exact).  Three products per multiply:
// hi*hi into the main accumulator, lo*hi and hi*lo into a second one; the epilogue forms
// (main + 2^-11 cross) / (s_row s_col).  lo*lo lies below fp32's resolution.
// Against three TF32 products of the same operands (contraction_tc.cu) a K block of 32 takes half the tensor time (the
// fp16 rate is twice the TF32 rate), half the instructions (K = 16 each), half the bytes of B and half the tensor memory
// of A; the split keeps one bit more and rounds instead of truncating, and the tensor core's truncating accumulate is
// applied to half as many partial sums.
//
// Range.  fp16 reaches from 2^-24 to 65504, fp32 much further; the scales close the gap.  B's are exact (one pass over
// its rows when it is prepared).  A's rows are seen block by block: the first block of a row that holds anything puts
// its largest element between 2^9 and 2^10; from there elements may grow 2^5-fold at least before the scale has to
// change.  When a later block does exceed that, the converter warp waits for the products issued so far and divides its
// rows of the accumulators by the (power of two) change of scale before it goes on: exact, rare on ordinary data, right
// on any.
// Small elements: from 2^-14 up in scaled units an element keeps its 22 bits; below, it is held to 2^-36, and both operands'
// together put an error of at most 2^-20 on each of a result's products (the other factor is below 2^15).  With
// S = sum |a||b| in scaled units, K * 2^-20 <= K * 2^-25 * S wherever S >= 2^5, as much as the accumulation of three TF32
// products may take.  S >= 2^5 follows from a sum of 2^5 or more, and from a main part of 2^5 + K * 2^-8 or more (an element's hi half
// is larger than the element by 2^-11 of it or by 2^-25 at most).  The sums of which neither holds -- of ordinary operands
// one in 10^8 -- the epilogue looks into (coarse_rows, sums_anew): where the row of A or the row of B holds such elements the sum is
// formed anew from the fp32 operands.  That serves rows whose large elements meet small or no ones on the other side
// (1e6 and 1e-6 by weights of 1e-6 and 1e6: 5e-3 of sum |a||b| without it).  A launch
// of nothing but such sums takes far longer (20000 x 1152 x 128: 2.3 ms for 53 us, 4096 x 4096 x 1024 7.8 ms for 0.12), one of
// operands so sparse that most sums are zero, whose rows are only looked through, up to twice as long as three TF32
// products (zeros in 99 % of both: 171 us for 89; 80 % and 95 %: 87 for 90).  The look at every sum costs 1 to 4 % of an ordinary launch; marks of A's rows from the converters, which
// every block would pay for, cost 10 to 18 %.
// A row of subnormal numbers alone counts where its first K block holds one.
//
// Pipeline: as in contraction_tc.cu, a persistent CTA per SM (24 warps) walks the 128 x BN tiles:
//   warps 0, 1   copy by TMA into a ring of raw slots: A (128 rows x 32 floats; plain rows, im2col or row windows) and B
//                (BN rows x 128 bytes: 32 hi halves, 32 lo halves), a warp each: a wait, an announcement and two copies took
//                one warp about as long (640 cycles) as the block's conversion (3x3 64 -> 64, 32 x 56 x 56: 54.5 us with one
//                copy warp and tile coordinates by division, 50.9 now)
//   warps 4-15   convert, three groups of four warps that take the K blocks in turn, each with a stage of its own in tensor
//                memory (32 columns); thread = row of the tile.  The row scales go from group to group in shared memory:
//                a group looks at its block's maxima, waits for the scales after the block before, publishes its own and
//                converts.  One group alone takes 577 ns per K block on 4096^3 (the latency of a block's chain of waits,
//                reads, stores and arrivals, not its arithmetic), two 404, three 382, four 415 (registers).
//   warp 2       allocates TMEM, issues 6 products per K block
//   warps 16-23  epilogue, as in contraction_tc.cu.
// The roles' registers are split by setmaxnreg (without it the epilogue spills and takes three times as long).
// Every wait is bounded as in contraction_tc.cu.
//
// What bounds it: at BN = 128 a K block's products take 384 cycles and a period 660 (converters), at a clock that the
// power cap has brought to 1.5 GHz by then.  4096^3: 385 us = 357 TFLOP/s (TF32 kernel: 650 us); ResNet-50's 3x3 layers of
// stages 2 to 4 at batch 256: 183-197 us (270-284).  A tile costs about 3000 cycles beyond its K blocks (fold of the
// single cross accumulator at BN = 128, transposed stores), so up to four K blocks the TF32 kernel's short-K variant is
// the faster one: 64 -> 256 with residual 355 us against 430, 128 -> 512 197 against 239, 256 -> 1024 158 against 150.
#include "contraction.cuh"
#include <cuda.h>
#include <cuda_fp16.h>
#include <string.h>
#include <atomic>

namespace nb200 {

namespace {

constexpr int BM = 128;
constexpr int BK = 32;                     // floats of A per K block = one 128-byte swizzle row
constexpr int MMA_WARP = 2;
constexpr int CVT_WARP0 = 4, CVT_GROUPS = 3, CVT_WARPS = 4; // groups of four warps that take the K blocks in turn
constexpr int EPI_WARP0 = CVT_WARP0 + CVT_GROUPS * CVT_WARPS, EPI_WARPS = 8;
constexpr int THREADS = (EPI_WARP0 + EPI_WARPS) * 32;
// Registers per thread once the roles have parted.  The block is launched with THREADS x 80 = 61440 of the SM's 65536;
// 4 warps x 32 x 56 + 12 x 32 x 72 + 8 x 32 x 104 = 61440.
constexpr int REGS_LAUNCH = 80, REGS_ISSUE = 56, REGS_CVT = 72, REGS_EPI = 104;
static_assert(4 * REGS_ISSUE + CVT_GROUPS * CVT_WARPS * REGS_CVT + EPI_WARPS * REGS_EPI <= THREADS / 32 * REGS_LAUNCH, "register split");
constexpr int A_TILE_BYTES = BM * BK * 4;  // 16 KB
constexpr int B_ROW_BYTES = 128;           // 32 hi halves + 32 lo halves
constexpr int STAGING_BYTES_PER_WARP = 32 * 64;
constexpr int STAGES = CVT_GROUPS;         // A stages in tensor memory, one per group
constexpr uint32_t STAGE_COLS = 32;        // per 16 elements of K: 8 columns of hi pairs, 8 of lo pairs
constexpr int MAX_RAW_SLOTS = 8;
// Row scales travel from the converters to the epilogue through a ring of tiles.  The converters write tile t when they
// have passed the stage wait of its last K block, so the products of K block (last - STAGES) are done; with one K block
// per tile that is tile t - STAGES, whose start waited for the epilogue to empty tile t - STAGES - 2 at the latest.
constexpr int SCALE_RING = STAGES + 4;
constexpr float LO_SCALE = 2048.f;
constexpr int TARGET_EXP = 9;              // log2 of where a row's first maximum is put
constexpr int SCALE_EXP_MAX = 254 - 11;    // biased exponent of the largest scale: LO_SCALE (2^11) times it is still finite
constexpr float FULL_BITS = 0x1p-14f;      // a scaled element below this has fewer than 22 bits
constexpr float SMALL_SUM = 32.f;          // see Range: sums that are smaller (scaled), and their main parts, are looked into
constexpr float RAISE_AT = 32768.f;        // a scaled element beyond this moves the row's scale (fp16 ends at 65504)

enum {
	SITE_RAW_EMPTY = 0x201, SITE_RAW_FULL = 0x202, SITE_CVT_FULL = 0x203, SITE_STAGE_EMPTY = 0x204,
	SITE_ACC_FULL = 0x205, SITE_ACC_EMPTY = 0x206, SITE_RAISE = 0x207, SITE_SCALES = 0x208, SITE_CHAIN = 0x209
};

__device__ __forceinline__ uint32_t swz(int row, int chunk)
{
	return static_cast<uint32_t>(row) * 128u + (static_cast<uint32_t>(chunk ^ (row & 7)) << 4);
}

// The power of two that puts `largest` into [2^TARGET_EXP, 2^(TARGET_EXP + 1)), kept where its inverse and LO_SCALE times it
// are normal numbers: at most 2^116, which leaves even the smallest normal element at 2^-10 (an infinite element keeps being
// infinite).  With 2^126 as the limit t = LO_SCALE * s below was infinite from maxima of 2^-107 down, and with it the lo halves.
__device__ __forceinline__ float scale_for(float largest)
{
	const int e = static_cast<int>(__float_as_uint(largest) >> 23) & 0xff;
	int se = 254 + TARGET_EXP - e;
	se = se < 1 ? 1 : (se > SCALE_EXP_MAX ? SCALE_EXP_MAX : se);
	return __uint_as_float(static_cast<uint32_t>(se) << 23);
}
// 1 / s of such a power of two
__device__ __forceinline__ float inverse_scale(float s)
{
	return __uint_as_float((254u << 23) - __float_as_uint(s));
}

// Order-preserving key of |x|, zero last: the smallest key of a set is its smallest element that is not zero.
__device__ __forceinline__ uint32_t small_key(float x)
{
	return 2u * __float_as_uint(x) - 1u;
}
// The key below which the elements of a row with this inverse scale have fewer than 22 bits (subnormal ones among them).
__device__ __forceinline__ uint32_t coarse_below(float inv)
{
	return small_key(fmaxf(FULL_BITS * inv, 0x1p-126f));
}
__device__ __forceinline__ uint32_t smallest_key(uint32_t m, const float4& v)
{
	return min(min(min(m, small_key(v.x)), min(small_key(v.y), small_key(v.z))), small_key(v.w));
}

// v * rowInv * colInv for powers of two whose product with v may leave fp32's range although all three together do not (rows of
// 1e34 by columns of 1e-30): the exponents are added and applied in two halves of one sign, so that a step overflows or
// vanishes only where the result does.
__device__ __forceinline__ float unscale(float v, float rowInv, float colInv)
{
	const int e = static_cast<int>(__float_as_uint(rowInv) >> 23) + static_cast<int>(__float_as_uint(colInv) >> 23) - 254;
	const int half = e >> 1;
	return v * __uint_as_float(static_cast<uint32_t>(127 + half) << 23) * __uint_as_float(static_cast<uint32_t>(127 + e - half) << 23);
}
// The accumulators stay below 2^50 or so and sums of any weight above 2^-40: within these limits v * rowInv is safe by itself.
constexpr float ROW_INV_MIN = 0x1p-64f, ROW_INV_MAX = 0x1p64f;

// hi and lo halves of two scaled neighbours, the first in the low half; t = LO_SCALE * s.  (x0, x1) as packed pairs: the
// converters are bound by instruction issue.
__device__ __forceinline__ void split_pair(float x0, float x1, float s, float t, uint32_t& hi, uint32_t& lo)
{
	float a, b, c, d;
	asm("{\n\t.reg .b64 x, s, t, a, c;\n\t"
		"mov.b64 x, {%4, %5};\n\tmov.b64 s, {%6, %6};\n\tmov.b64 t, {%7, %7};\n\t"
		"mul.rn.f32x2 a, x, s;\n\tmul.rn.f32x2 c, x, t;\n\t" // subnormal elements count, too
		"mov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, c;\n\t}"
		: "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "f"(x0), "f"(x1), "f"(s), "f"(t));
	const __half2 h = __floats2half2_rn(a, b);
	const float2 back = __half22float2(h);
	asm("{\n\t.reg .b64 h, m, a;\n\t"
		"mov.b64 h, {%2, %3};\n\tmov.b64 m, {%4, %4};\n\tmov.b64 a, {%0, %1};\n\t"
		"fma.rn.ftz.f32x2 a, h, m, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
		: "+f"(c), "+f"(d) : "f"(back.x), "f"(back.y), "f"(-LO_SCALE));
	const __half2 l = __floats2half2_rn(c, d);
	hi = *reinterpret_cast<const uint32_t*>(&h);
	lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ float max_abs(float m, const float4& v)
{
	float r;
	asm("{\n\t.reg .f32 a, b, c, d;\n\tabs.ftz.f32 a, %2;\n\tabs.ftz.f32 b, %3;\n\tabs.ftz.f32 c, %4;\n\tabs.ftz.f32 d, %5;\n\t"
		"max.ftz.f32 a, a, b, c;\n\tmax.ftz.f32 %0, a, d, %1;\n\t}"
		: "=f"(r) : "f"(m), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
	return r;
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
	asm("min.ftz.f32 %0, %0, %1, %2;" : "+f"(a) : "f"(b), "f"(c));
	return a;
}

// The 32 floats of K block kb in row m of the first operand (`at`: conv_row of m), or null where they are a convolution's padding.
__device__ __forceinline__ const float* row_block(const ContractionParams& p, const float* A, const ConvRow& at, int m, int kb)
{
	if(p.a_mode == A_ROWS) return A + static_cast<size_t>(m) * p.lda + kb * BK;
	int iy = at.iy0 + kb, ix = at.ix0, c = 0; // windows: a block per image row, the padding is in the copy
	if(p.a_mode == A_CONV_TAP) {
		const int tap = kb * BK / p.Cin, fr = tap / p.S;
		c = kb * BK - tap * p.Cin;
		iy = at.iy0 + fr * p.dilH;
		ix = at.ix0 + (tap - fr * p.S) * p.dilW;
		if(static_cast<unsigned>(iy) >= static_cast<unsigned>(p.H) || static_cast<unsigned>(ix) >= static_cast<unsigned>(p.W)) return nullptr;
	}
	return A + at.base + (iy * p.W + ix) * p.Cin + c;
}

// How many of a K block's 32 floats belong to the sum: the last block's remainder; windows: the filter's taps.
__device__ __forceinline__ int floats_in_block(const ContractionParams& p, int kb)
{
	return p.a_mode == A_CONV_WINDOW ? p.filterS * p.Cin : min(BK, p.K - kb * BK);
}
// Floats 4c .. 4c + 3 of a block at src (16-byte aligned; null: zeros) of which `count` belong to the sum: those that are whole
// quads.  No branch, so that several are in flight; the others by last_floats().
__device__ __forceinline__ float4 whole_quad(const float* src, int c, int count)
{
	return src != nullptr && 4 * c + 4 <= count ? __ldg(reinterpret_cast<const float4*>(src) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ float4 last_floats(const float* src, int count)
{
	float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
	src += count & ~3;
	if((count & 3) > 0) v.x = __ldg(src);
	if((count & 3) > 1) v.y = __ldg(src + 1);
	if((count & 3) > 2) v.z = __ldg(src + 2);
	return v;
}

// Which of a warp's rows (bits of `rows`, from row m0 on) hold elements of fewer than 22 bits; lane r has row r's inverse scale.
// A warp takes four K blocks of a row at a time, four loads ahead: sums that are zero are what sparse operands are full of,
// and their rows are looked through to no avail.
__device__ __forceinline__ uint32_t coarse_rows(const ContractionParams& p, uint32_t rows, float inv, int batch, int m0, int kbBegin,
	int kbEnd)
{
	const int lane = threadIdx.x & 31, c = lane & 7;
	const float* A = p.A + batch * p.strideA;
	uint32_t coarse = 0;
#pragma unroll 1
	for(; rows != 0; rows &= rows - 1) {
		const int r = __ffs(rows) - 1;
		const uint32_t below = coarse_below(__shfl_sync(0xffffffffu, inv, r));
		const ConvRow at = p.a_mode == A_ROWS ? ConvRow{} : conv_row(p, m0 + r);
		uint32_t smallest = 0xffffffffu;
#pragma unroll 1
		for(int first = kbBegin + (lane >> 3); first < kbEnd; first += 16) {
			float4 v[4];
#pragma unroll
			for(int i = 0; i < 4; ++i) {
				const int kb = min(first + 4 * i, kbEnd - 1);
				v[i] = whole_quad(row_block(p, A, at, m0 + r, kb), c, floats_in_block(p, kb));
			}
#pragma unroll
			for(int i = 0; i < 4; ++i) smallest = smallest_key(smallest, v[i]);
		}
		if(p.a_mode == A_ROWS && (p.K & 3) != 0 && kbEnd * BK >= p.K) {
			smallest = smallest_key(smallest, last_floats(A + static_cast<size_t>(m0 + r) * p.lda, p.K));
		}
		if(__any_sync(0xffffffffu, smallest < below)) coarse |= 1u << r;
	}
	return coarse;
}

__device__ __forceinline__ void fma_full(float& sum, float a, float b) // subnormal numbers included
{
	asm("fma.rn.f32 %0, %1, %2, %0;" : "+f"(sum) : "f"(a), "f"(b));
}
__device__ __forceinline__ float add_full(float a, float b)
{
	asm("add.rn.f32 %0, %0, %1;" : "+f"(a) : "f"(b));
	return a;
}

// Forms sums anew from the fp32 operands: those of row m (one per lane) and of the columns n0 + t with bit t in `wanted`.  They
// replace mine[t].  A lane holds its row's floats of a K block; the columns of B that any lane wants are fetched four at
// a time, a float per lane, and handed round by shuffles: whole tiles of such sums occur in data that is made for it.
__device__ __forceinline__ void sums_anew(const ContractionParams& p, uint32_t wanted, int batch, int m, int n0, int kbBegin, int kbEnd,
	float* mine)
{
	const uint32_t columns = __reduce_or_sync(0xffffffffu, wanted);
	if(columns == 0) return;
	const int lane = threadIdx.x & 31;
	const float* A = p.A + batch * p.strideA;
	const float* B = p.B + batch * p.strideB;
	const ConvRow at = p.a_mode == A_ROWS || wanted == 0 ? ConvRow{} : conv_row(p, m);
	// where this lane's float of a K block lies in a row of B, and how far it is to the next block's and the next row's
	int inBlock = lane, block = BK;
	long long row = p.ldb;
	bool there = true;
	if(p.a_mode == A_CONV_WINDOW) {
		// the filter as the caller has it: channels and taps that are not there count nothing
		const int tap = lane / p.Cin, ch = lane - tap * p.Cin;
		there = tap < p.filterS && ch < p.filterC;
		inBlock = tap * p.filterC + ch;
		block = p.filterS * p.filterC;
		row = static_cast<long long>(p.K / BK) * block;
	}
#pragma unroll 1
	for(uint32_t w = wanted; w != 0; w &= w - 1) mine[__ffs(w) - 1] = 0.f;
#pragma unroll 1
	for(int kb = kbBegin; kb < kbEnd; ++kb) {
		const float* src = wanted != 0 ? row_block(p, A, at, m, kb) : nullptr;
		const int count = floats_in_block(p, kb);
		float x[BK];
#pragma unroll
		for(int c = 0; c < 8; ++c) {
			float4 v = whole_quad(src, c, count);
			if((count & 3) != 0 && c == count >> 2 && src != nullptr) v = last_floats(src, count);
			x[4 * c] = v.x; x[4 * c + 1] = v.y; x[4 * c + 2] = v.z; x[4 * c + 3] = v.w;
		}
		const bool real = there && kb * BK + lane < p.K;
		const float* b = B + n0 * row + static_cast<long long>(kb) * block + inBlock;
#pragma unroll 1
		for(int q = 0; q < 16; q += 4) {
			const uint32_t four = (columns >> q) & 15u;
			if(four == 0) continue;
			float w[4];
#pragma unroll
			for(int t = 0; t < 4; ++t) w[t] = real && ((four >> t) & 1u) ? __ldg(b + (q + t) * row) : 0.f;
			// (not unrolled: with four copies of the loop below the 128- and 96-column kernels spilled)
#pragma unroll 1
			for(int t = 0; t < 4; ++t) {
				float sum[4] = { 0.f, 0.f, 0.f, 0.f };
#pragma unroll
				for(int i = 0; i < BK; ++i) fma_full(sum[i & 3], x[i], __shfl_sync(0xffffffffu, w[0], i));
				w[0] = w[1]; w[1] = w[2]; w[2] = w[3];
				if((wanted >> (q + t)) & 1u) mine[q + t] = add_full(mine[q + t], add_full(add_full(sum[0], sum[1]), add_full(sum[2], sum[3])));
			}
		}
	}
}

template<int BN>
__global__ void __maxnreg__(REGS_LAUNCH) contraction_split_kernel(const ContractionParams p, int numTiles, int nTiles,
	int tilesPerBatch, int rawSlots, const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB)
{
	extern __shared__ uint8_t smem_raw[];
	if(*reinterpret_cast<volatile int*>(p.status) != 0) return;
	uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));

	constexpr int B_TILE_BYTES = BN * B_ROW_BYTES;
	// Two main accumulators (the epilogue of tile i overlaps the products of tile i + 1) and as many cross accumulators
	// as fit beside the stages; the epilogue first folds a tile's into its main accumulator, and where there is but one
	// (BN = 128) hands it back.
	constexpr bool FOLD = BN > 96;
	constexpr uint32_t CROSS_BASE = 2 * BN;
	constexpr uint32_t A_BASE = (FOLD ? 3 : 4) * BN;
	static_assert(A_BASE + STAGES * STAGE_COLS <= 512, "tensor memory budget");
	constexpr uint32_t TMEM_USED = A_BASE + STAGES * STAGE_COLS;
	constexpr uint32_t TMEM_COLS = TMEM_USED <= 256 ? 256 : 512;
	constexpr int HALF_COLS = BN / 2;
	constexpr int CHUNKS = HALF_COLS / 16;

	// with split K the unit of work is (tile, K part): `numTiles` counts those, each covers numKb K blocks
	const int kSplits = p.kSplits;
	const int numKb = ((p.K + BK - 1) / BK) / kSplits;
	constexpr int SLOT_BYTES = A_TILE_BYTES + B_TILE_BYTES;

	uint8_t* rawRing = smem;
	uint8_t* staging = rawRing + static_cast<size_t>(rawSlots) * SLOT_BYTES;
	float* strips = reinterpret_cast<float*>(staging + EPI_WARPS * STAGING_BYTES_PER_WARP); // per warp: bias, column scale, large for columns that are not there or zero
	float* rowInv = strips + EPI_WARPS * 3 * HALF_COLS;
	float* rowScale = rowInv + SCALE_RING * BM; // the scale of each row of the tile being converted
	uint64_t* rawFullBar = reinterpret_cast<uint64_t*>(rowScale + BM);
	uint64_t* rawEmptyBar = rawFullBar + MAX_RAW_SLOTS;
	uint64_t* cvtFullBar = rawEmptyBar + MAX_RAW_SLOTS;
	uint64_t* accFullBar = cvtFullBar + STAGES;
	uint64_t* accEmptyBar = accFullBar + 2;
	uint64_t* crossEmptyBar = accEmptyBar + 2; // FOLD: the one cross accumulator is free again
	uint64_t* scalesBar = crossEmptyBar + 1; // a tile's row scales are in the ring (one arrival per converter warp)
	uint64_t* chainBar = scalesBar + SCALE_RING; // [quad][group]: the row scales after a K block of that group are in rowScale
	uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(chainBar + CVT_WARPS * CVT_GROUPS);
	volatile int* abortFlag = reinterpret_cast<volatile int*>(tmemSlot + 1);

	const int tid = threadIdx.x;
	const int warp = tid >> 5;
	const int lane = tid & 31;
	const int myTiles = static_cast<int>(blockIdx.x) < numTiles ? (numTiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;

	if(tid == 0) {
		for(int s = 0; s < MAX_RAW_SLOTS; ++s) {
			mbar_init(&rawFullBar[s], 2); // one announcement per copy warp
			mbar_init(&rawEmptyBar[s], 1);
		}
		for(int s = 0; s < STAGES; ++s) mbar_init(&cvtFullBar[s], CVT_WARPS);
		for(int b = 0; b < 2; ++b) {
			mbar_init(&accFullBar[b], 1);
			mbar_init(&accEmptyBar[b], EPI_WARPS);
		}
		for(int t = 0; t < SCALE_RING; ++t) mbar_init(&scalesBar[t], CVT_WARPS);
		for(int c = 0; c < CVT_WARPS * CVT_GROUPS; ++c) mbar_init(&chainBar[c], 1);
		mbar_init(crossEmptyBar, EPI_WARPS);
		*abortFlag = 0;
		mbar_init_fence();
	}
	if(warp == MMA_WARP) {
		tmem_alloc(tmemSlot, TMEM_COLS);
		tmem_relinquish();
	}
	if(tid == 0) {
		tma_prefetch_descriptor(&mapA);
		tma_prefetch_descriptor(&mapB);
	}
	tc_fence_before_sync();
	__syncthreads();
	tc_fence_after_sync();
	const uint32_t tmemBase = *tmemSlot;
	// everything above touched only this CTA's own state and ran while the previous kernel was finishing
	dependent_wait();
	dependents_may_start();

	if(warp < CVT_WARP0) {
		registers_down<REGS_ISSUE>();
		if(warp == 0) {
		// ------------------------------------------------------------------ copy A
		int tile = blockIdx.x;
		int slot = 0;
		uint32_t parity = 1; // the first pass over the ring finds every slot free
		bool ok = true;
		const int hw = p.Ho * p.Wo;
		for(int local = 0; local < myTiles && ok; ++local, tile += gridDim.x) {
			const int tileIdx = p.div.splits(tile);
			const int kbBegin = (tile - tileIdx * kSplits) * numKb;
			const TileCoord tc = tile_coord(p, tileIdx, nTiles, tilesPerBatch, BN);
			int w0 = 0, h0 = 0, img = 0;
			if(p.a_tma == 3) {
				img = p.div.ho(tc.mTile); // the tile is output row image * Ho + oy
				h0 = tc.mTile - img * p.Ho;
			} else if(p.a_tma == 2) {
				img = p.div.hw(tc.m0);
				const int rem = tc.m0 - img * hw;
				const int oy = p.div.wo(rem);
				w0 = (rem - oy * p.Wo) * p.strW - p.padW;
				h0 = oy * p.strH - p.padH;
			}
			int c0 = 0, fs = 0, fr = 0; // channel offset inside the filter tap, tap column, tap row
			if(p.a_tma == 2 && kbBegin > 0) {
				const int tap = kbBegin * BK / p.Cin;
				c0 = kbBegin * BK - tap * p.Cin;
				fr = tap / p.S;
				fs = tap - fr * p.S;
			}
			for(int kb = kbBegin; kb < kbBegin + numKb; ++kb) {
				if(!mbar_wait_bounded_warp(&rawEmptyBar[slot], parity, abortFlag, p.status, SITE_RAW_EMPTY)) { ok = false; break; }
				const uint32_t aTile = smem_u32(rawRing + static_cast<size_t>(slot) * SLOT_BYTES);
				if(elect_one()) {
					mbar_arrive_expect_tx(&rawFullBar[slot], A_TILE_BYTES);
					if(p.a_tma == 1) {
						tma_load_3d(aTile, &mapA, &rawFullBar[slot], kb * BK, tc.m0, tc.batch);
					} else if(p.a_tma == 3) {
						tma_load_5d(aTile, &mapA, &rawFullBar[slot], 0, 0, kb, h0, img);
					} else {
						tma_load_im2col_4d(aTile, &mapA, &rawFullBar[slot], c0, w0, h0, img,
							static_cast<uint16_t>(fs * p.dilW), static_cast<uint16_t>(fr * p.dilH));
					}
				}
				__syncwarp();
				if(p.a_tma == 2) {
					c0 += BK;
					if(c0 >= p.Cin) { c0 = 0; if(++fs == p.S) { fs = 0; ++fr; } }
				}
				if(++slot == rawSlots) { slot = 0; parity ^= 1; }
			}
		}
		} else if(warp == 1) {
		// ------------------------------------------------------------------ copy B
		int slot = 0;
		uint32_t parity = 1;
		bool ok = true;
		for(int local = 0, tile = blockIdx.x; local < myTiles && ok; ++local, tile += gridDim.x) {
			const int tileIdx = p.div.splits(tile);
			const int kbBegin = (tile - tileIdx * kSplits) * numKb;
			const TileCoord tc = tile_coord(p, tileIdx, nTiles, tilesPerBatch, BN);
			for(int kb = kbBegin; kb < kbBegin + numKb; ++kb) {
				if(!mbar_wait_bounded_warp(&rawEmptyBar[slot], parity, abortFlag, p.status, SITE_RAW_EMPTY)) { ok = false; break; }
				if(elect_one()) {
					mbar_arrive_expect_tx(&rawFullBar[slot], B_TILE_BYTES);
					tma_load_3d(smem_u32(rawRing + static_cast<size_t>(slot) * SLOT_BYTES) + A_TILE_BYTES, &mapB, &rawFullBar[slot],
						kb * BK, tc.n0, tc.batch);
				}
				__syncwarp();
				if(++slot == rawSlots) { slot = 0; parity ^= 1; }
			}
		}
		} else if(warp == MMA_WARP) {
		// ------------------------------------------------------------------ MMA issuer
		constexpr uint32_t idesc = umma_idesc_f16(BM, BN);
		bool ok = true;
		int slot = 0, stage = 0;
		uint32_t stageParity = 0;
		for(int local = 0; local < myTiles && ok; ++local) {
			const int set = local & 1;
			if(!mbar_wait_bounded_warp(&accEmptyBar[set], ((local >> 1) & 1) ^ 1, abortFlag, p.status, SITE_ACC_EMPTY)) { ok = false; break; }
			if(FOLD && !mbar_wait_bounded_warp(crossEmptyBar, (local & 1) ^ 1, abortFlag, p.status, SITE_ACC_EMPTY)) { ok = false; break; }
			tc_fence_after_sync();
			const uint32_t accMain = tmemBase + set * BN;
			const uint32_t accCross = tmemBase + CROSS_BASE + (FOLD ? 0 : set * BN);
			uint32_t acc = 0u; // the first products of a tile overwrite the accumulators
			const int work = blockIdx.x + local * gridDim.x;
			const int kbBegin = kSplits == 1 ? 0 : (work - p.div.splits(work) * kSplits) * numKb;
			for(int kb = 0; kb < numKb; ++kb) {
				if(!mbar_wait_bounded_warp(&cvtFullBar[stage], stageParity, abortFlag, p.status, SITE_CVT_FULL)) { ok = false; break; }
				tc_fence_after_sync();
				const uint32_t aHi = tmemBase + A_BASE + stage * STAGE_COLS, aLo = aHi + 8;
				const uint32_t bTile = smem_u32(rawRing + static_cast<size_t>(slot) * SLOT_BYTES) + A_TILE_BYTES;
				const uint64_t dB = umma_desc_k128(bTile); // 16 halves = 32 bytes = +2; the lo halves start 64 bytes in
				const bool both = p.K - (kbBegin + kb) * BK > 16;
				if(elect_one()) {
					umma_f16_ts(accCross, aLo, dB, idesc, acc);
					umma_f16_ts(accMain, aHi, dB, idesc, acc);
					umma_f16_ts(accCross, aHi, dB + 4, idesc, 1u);
					if(both) {
						umma_f16_ts(accMain, aHi + 16, dB + 2, idesc, 1u);
						umma_f16_ts(accCross, aLo + 16, dB + 2, idesc, 1u);
						umma_f16_ts(accCross, aHi + 16, dB + 6, idesc, 1u);
					}
					umma_commit(&rawEmptyBar[slot]); // the slot and the stage
					if(kb == numKb - 1) umma_commit(&accFullBar[set]);
				}
				acc = 1u;
				__syncwarp();
				if(++slot == rawSlots) slot = 0;
				if(++stage == STAGES) { stage = 0; stageParity ^= 1; }
			}
		}
		if(!ok && lane == 0) {
			// something timed out: give whatever was issued time to finish before TMEM is freed
			const uint64_t t0 = global_timer_ns();
			while(global_timer_ns() - t0 < 1000000ull) {
			}
		}
		__syncwarp();
		}
	} else if(warp < EPI_WARP0) {
		registers_down<REGS_CVT>();
		// ------------------------------------------------------------------ convert
		const int quad = warp & 3, group = (warp - CVT_WARP0) >> 2;
		const int row = quad * 32 + lane; // tile row = tensor-memory lane of this thread
		const uint32_t laneBase = tmemBase + (static_cast<uint32_t>(quad * 32) << 16);
		const int totalSteps = myTiles * numKb;
		uint64_t* const chainOwn = &chainBar[quad * CVT_GROUPS + group];
		uint64_t* const chainBefore = &chainBar[quad * CVT_GROUPS + (group + CVT_GROUPS - 1) % CVT_GROUPS];
		int slot = group, kb = group, local = 0, ring = 0, n = 0; // n: this group's K blocks so far
		uint32_t rawParity = 0;
		int freeSlot = 0;        // the slot and phase of the group's K block before: its products also empty the stage
		uint32_t freeParity = 0;
		while(slot >= rawSlots) { slot -= rawSlots; rawParity ^= 1; }
		while(kb >= numKb) { kb -= numKb; ++local; ++ring; }
		for(int step = group; step < totalSteps; step += CVT_GROUPS, ++n) {
			if(!mbar_wait_bounded_warp(&rawFullBar[slot], rawParity, abortFlag, p.status, SITE_RAW_FULL)) break;
			const uint8_t* raw = rawRing + static_cast<size_t>(slot) * SLOT_BYTES;
			float4 x[8];
#pragma unroll
			for(int c = 0; c < 8; ++c) x[c] = *reinterpret_cast<const float4*>(raw + swz(row, c));
			float largest = 0.f;
#pragma unroll
			for(int c = 0; c < 8; ++c) largest = max_abs(largest, x[c]);
			// the scale after the K block before, which the group before has looked at
			if(step > 0 && !mbar_wait_bounded_warp(chainBefore, (group > 0 ? n : n - 1) & 1, abortFlag, p.status, SITE_CHAIN)) break;
			float s = kb > 0 ? rowScale[row] : 0.f; // 0: nothing but zeros so far
			bool move = s == 0.f ? largest > 0.f : largest * s > RAISE_AT;
			if(kb == 0 || __any_sync(0xffffffffu, move)) {
				// of a row that holds zeros or subnormal numbers, which max_abs takes for zeros, the latter count as the smallest
				// normal number (no branch: its code would be fetched anew by every launch)
				uint32_t bits = 0;
#pragma unroll
				for(int c = 0; c < 8; ++c) {
					bits |= __float_as_uint(x[c].x) | __float_as_uint(x[c].y) | __float_as_uint(x[c].z) | __float_as_uint(x[c].w);
				}
				const bool subnormal = s == 0.f && largest == 0.f && (bits << 1) != 0;
				largest = subnormal ? 0x1p-126f : largest;
				move = move || subnormal;
				const float next = move ? scale_for(largest) : s;
				if(__any_sync(0xffffffffu, move && s != 0.f)) {
					// rare: rows whose accumulated sums are in the old scale.  The products issued so far must have
					// completed (those of this K block cannot start: this warp has not handed over its rows)
					if(!mbar_wait_bounded_warp(&rawEmptyBar[(step - 1) % rawSlots], ((step - 1) / rawSlots) & 1, abortFlag, p.status, SITE_RAISE)) break;
					tc_fence_after_sync();
					const float factor = move && s != 0.f ? next * inverse_scale(s) : 1.f;
					const uint32_t main = laneBase + (local & 1) * BN, cross = laneBase + CROSS_BASE + (FOLD ? 0 : (local & 1) * BN);
#pragma unroll 1
					for(int c = 0; c < 2 * BN; c += 8) {
						const uint32_t at = c < BN ? main + c : cross + (c - BN);
						uint32_t r[8];
						tmem_ld8_issue(at, r);
						tmem_ld_wait();
#pragma unroll
						for(int i = 0; i < 8; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * factor);
						tmem_st8(at, r);
					}
					tmem_st_wait();
				}
				s = next;
				rowScale[row] = s;
				__syncwarp();
			}
			if(lane == 0) mbar_arrive(chainOwn);
			// the stage is free once the products of the group's K block before have completed
			if(n > 0 && !mbar_wait_bounded_warp(&rawEmptyBar[freeSlot], freeParity, abortFlag, p.status, SITE_STAGE_EMPTY)) break;
			freeSlot = slot;
			freeParity = rawParity;
			tc_fence_after_sync();
			const float t = s * LO_SCALE;
#pragma unroll
			for(int half = 0; half < 2; ++half) {
				uint32_t r[16]; // 8 columns of hi pairs, 8 of lo pairs
#pragma unroll
				for(int c = 0; c < 4; ++c) {
					split_pair(x[4 * half + c].x, x[4 * half + c].y, s, t, r[2 * c], r[8 + 2 * c]);
					split_pair(x[4 * half + c].z, x[4 * half + c].w, s, t, r[2 * c + 1], r[8 + 2 * c + 1]);
				}
				tmem_st16(laneBase + A_BASE + group * STAGE_COLS + 16 * half, r);
			}
			const bool last = kb == numKb - 1;
			if(last) rowInv[ring * BM + row] = s == 0.f ? 0.f : inverse_scale(s); // 0: a row of zeros
			slot += CVT_GROUPS;
			while(slot >= rawSlots) { slot -= rawSlots; rawParity ^= 1; }
			tmem_st_wait();
			tc_fence_before_sync();
			__syncwarp();
			if(lane == 0) {
				mbar_arrive(&cvtFullBar[group]);
				if(last) mbar_arrive(&scalesBar[ring]);
			}
			kb += CVT_GROUPS;
			while(kb >= numKb) {
				kb -= numKb;
				++local;
				if(++ring == SCALE_RING) ring = 0;
			}
		}
	} else {
		registers_up<REGS_EPI>();
		// ------------------------------------------------------------------ epilogue
		const int ew = warp - EPI_WARP0;
		const int quad = warp & 3;  // the TMEM lane quarter this warp may read
		const int half = ew >> 2;   // which half of the tile's columns
		uint8_t* stg = staging + ew * STAGING_BYTES_PER_WARP;
		const int rowInGroup = lane >> 2;  // 0..7: which of the 8 rows a warp-wide 16-byte access covers
		const int c4 = lane & 3;           // which 16-byte piece of the 64-byte row slice
		const bool vec = p.c_vec != 0;
		float* biasStrip = strips + ew * 3 * HALF_COLS;
		float* scaleStrip = biasStrip + HALF_COLS;
		float* skipStrip = scaleStrip + HALF_COLS;
		int stripCol = -1, stripBatch = -1;
		const bool fastStore = vec && p.accumulate == 0 && p.act != NB200_ACT_HSWISH && p.act != NB200_ACT_SIGMOID_GATE;
		const bool gateStore = vec && p.accumulate == 0 && p.act == NB200_ACT_SIGMOID_GATE;
		const bool hswishStore = vec && p.accumulate == 0 && p.act == NB200_ACT_HSWISH;
		const bool clampOn = p.act == NB200_ACT_RELU;
		const float actParam = p.act_param_device != nullptr ? __ldg(p.act_param_device) : p.act_param;
		const float clampHi = actParam > 0.f ? actParam : __int_as_float(0x7f800000);
		const float small = 2.f * (SMALL_SUM + numKb * (BK / 256.f));
		bool ok = true;
		int ring = 0;
		for(int local = 0; local < myTiles && ok; ++local) {
			const int work = blockIdx.x + local * gridDim.x;
			const int tileIdx = p.div.splits(work);
			const TileCoord tc = tile_coord(p, tileIdx, nTiles, tilesPerBatch, BN);
			// a K part of a split launch stores its partial sums in its own slab
			float* __restrict__ C = p.C + tc.batch * p.strideC + static_cast<size_t>(work - tileIdx * kSplits) * p.M * p.ldc;
			const float* __restrict__ R = p.residual != nullptr ? p.residual + tc.batch * p.strideC : nullptr;
			const int set = local & 1;
			const uint32_t accParity = (local >> 1) & 1;
			const int rowBase = tc.m0 + quad * 32;
			const int colBase = tc.n0 + half * HALF_COLS;
			const bool useRes = vec && R != nullptr;
			const int mEnd = min(p.M, tc.m0 + p.tileM); // rows of this tile that exist and belong to it

			auto load_res = [&](int ch, float4* dst) {
				const int n = colBase + ch * 16 + c4 * 4;
#pragma unroll
				for(int i = 0; i < 4; ++i) {
					const int m = rowBase + 8 * i + rowInGroup;
					dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
					if(m < mEnd && n + 4 <= p.N) dst[i] = *reinterpret_cast<const float4*>(R + static_cast<size_t>(m) * p.ldr + n);
				}
			};

			// bias and column scales of this warp's columns, reloaded only when the columns change
			if(colBase != stripCol || tc.batch != stripBatch) {
				__syncwarp();
				for(int j = lane; j < HALF_COLS; j += 32) {
					const int n = colBase + j;
					biasStrip[j] = (p.bias != nullptr && n < p.N) ? __ldg(p.bias + n) : 0.f;
					const float scale = n < p.N ? __ldg(p.bScale + static_cast<size_t>(tc.batch) * p.N + n) : 0.f;
					scaleStrip[j] = scale;
					skipStrip[j] = scale == 0.f ? 1e30f : 0.f;
				}
				stripCol = colBase;
				stripBatch = tc.batch;
				__syncwarp();
			}
			if(useRes) {
				// pull this warp's residual rows towards L2 while the main loop of the tile runs
				const int m = rowBase + lane;
				if(m < p.M && colBase < p.N) {
					const char* line = reinterpret_cast<const char*>(R + static_cast<size_t>(m) * p.ldr + colBase);
					const int bytes = min(HALF_COLS, p.N - colBase) * 4;
					for(int off = 0; off < bytes; off += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(line + off));
				}
			}

			if(!mbar_wait_bounded_warp(&scalesBar[ring], (local / SCALE_RING) & 1, abortFlag, p.status, SITE_SCALES)
				|| !mbar_wait_bounded_warp(&accFullBar[set], accParity, abortFlag, p.status, SITE_ACC_FULL)) { ok = false; break; }
			tc_fence_after_sync();
			const uint32_t laneCol = (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(half * HALF_COLS);
			const uint32_t accMain = tmemBase + set * BN + laneCol;
			const uint32_t accCross = tmemBase + CROSS_BASE + (FOLD ? 0 : set * BN) + laneCol;
			// The cross terms are folded into the main accumulator in place, with a look at how small the sums are (not unrolled: with
			// that the 128-column kernel spilled, a 28 x 28, 512 -> 128 layer at batch 21 took 13.4 us for 12.8).
			float inv = rowInv[ring * BM + quad * 32 + lane];
			const bool alive = inv != 0.f && rowBase + lane < mEnd; // a row that exists and is not all zeros
			float least = __int_as_float(0x7f800000);
#pragma unroll 1
			for(int g = 0; g < HALF_COLS; g += 16) {
				uint32_t a[16], b[16];
				tmem_ld16_issue(accMain + g, a);
				tmem_ld16_issue(accCross + g, b);
				tmem_ld_wait();
#pragma unroll
				for(int i = 0; i < 16; i += 2) {
					const float x = __uint_as_float(a[i]), y = __uint_as_float(a[i + 1]);
					const float v = fmaf(__uint_as_float(b[i]), 1.f / LO_SCALE, x), w = fmaf(__uint_as_float(b[i + 1]), 1.f / LO_SCALE, y);
					const float2 skip = *reinterpret_cast<const float2*>(skipStrip + g + i);
					least = min3(least, fabsf(v) + (fabsf(x) + skip.x), fabsf(w) + (fabsf(y) + skip.y));
					a[i] = __float_as_uint(v);
					a[i + 1] = __float_as_uint(w);
				}
				tmem_st16(accMain + g, a);
			}
			tmem_st_wait();
			if(FOLD) {
				tc_fence_before_sync();
				__syncwarp();
				if(lane == 0) mbar_arrive(crossEmptyBar);
			}
			if(++ring == SCALE_RING) ring = 0;
			// Where the row's scale alone might take a sum out of range both scales are applied at once, and small sums are looked
			// into, ahead of the loop below: rare, and a branch per warp and tile.
			const bool careful = __any_sync(0xffffffffu, (alive && least < small) || (inv < ROW_INV_MIN && inv != 0.f) || inv > ROW_INV_MAX) != 0;
			if(__builtin_expect(careful, 0)) {
				float* mine = reinterpret_cast<float*>(stg + lane * 64);
				const int kbBegin = (work - tileIdx * kSplits) * numKb;
				// (rows this tiny may have lost subnormal elements in blocks before the scale was set)
				const bool tiny = inv < 0x1p-90f;
				const uint32_t suspects = __ballot_sync(0xffffffffu, alive && (least < small || tiny));
				const uint32_t coarse = coarse_rows(p, suspects, inv, tc.batch, rowBase, kbBegin, kbBegin + numKb);
				const bool coarseRow = (coarse >> lane & 1u) != 0;
#pragma unroll 1
				for(int g = 0; g < HALF_COLS; g += 16) {
					uint32_t a[16], wanted = 0;
					tmem_ld16_issue(accMain + g, a);
					tmem_ld_wait();
#pragma unroll
					for(int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(mine)[q] = make_uint4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
#pragma unroll 1
					for(int i = 0; i < 16; ++i) {
						const float v = mine[i], scale = scaleStrip[g + i]; // 0: a row of B that is all zeros, or none
						if(alive && scale != 0.f && (coarseRow || scale < 0.f) && (fabsf(v) < small || tiny)) wanted |= 1u << i;
						mine[i] = unscale(v, inv, fabsf(scale));
					}
					sums_anew(p, wanted, tc.batch, rowBase + lane, colBase + g, kbBegin, kbBegin + numKb, mine);
					__syncwarp();
#pragma unroll
					for(int q = 0; q < 4; ++q) {
						const uint4 o = reinterpret_cast<const uint4*>(mine)[q];
						a[4 * q] = o.x; a[4 * q + 1] = o.y; a[4 * q + 2] = o.z; a[4 * q + 3] = o.w;
					}
					__syncwarp();
					tmem_st16(accMain + g, a);
				}
				tmem_st_wait();
				inv = 1.f;
			}

			float4 res[4], resNext[4];
			if(useRes) load_res(0, res);
			// 16 columns at a time; the tensor-memory loads of chunk ch + 1 run while chunk ch is transposed and stored
			uint32_t vm[16];
			tmem_ld16_issue(accMain, vm);
#pragma unroll
			for(int ch = 0; ch < CHUNKS; ++ch) {
				tmem_ld_wait();
				float v[16];
#pragma unroll
				for(int i = 0; i < 16; ++i) v[i] = __uint_as_float(vm[i]) * inv;
				const int n = colBase + ch * 16 + c4 * 4; // first of this lane's four columns in the transposed phase
				const bool colsFull = n + 4 <= p.N;
				if(useRes && ch + 1 < CHUNKS) load_res(ch + 1, resNext);
				// transpose through shared memory: row-per-lane -> 8 rows x 64 B per warp access
#pragma unroll
				for(int q = 0; q < 4; ++q) {
					*reinterpret_cast<float4*>(stg + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) =
						make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
				}
				if(ch + 1 < CHUNKS) {
					tmem_ld16_issue(accMain + (ch + 1) * 16, vm);
				} else {
					// last read of this tile's accumulators: hand them back
					tc_fence_before_sync();
					__syncwarp();
					if(lane == 0) mbar_arrive(&accEmptyBar[set]);
				}
				__syncwarp();
				const float4 bias4 = *reinterpret_cast<const float4*>(biasStrip + ch * 16 + c4 * 4);
				float4 scale4 = make_float4(1.f, 1.f, 1.f, 1.f);
				if(!careful) {
					scale4 = *reinterpret_cast<const float4*>(scaleStrip + ch * 16 + c4 * 4);
					scale4 = make_float4(fabsf(scale4.x), fabsf(scale4.y), fabsf(scale4.z), fabsf(scale4.w)); // the sign is a mark
				}
				float4 ov[4];
#pragma unroll
				for(int i = 0; i < 4; ++i) {
					const int r = 8 * i + rowInGroup;
					ov[i] = *reinterpret_cast<const float4*>(stg + r * 64 + ((c4 ^ ((r >> 1) & 3)) << 4));
				}
#pragma unroll
				for(int i = 0; i < 4; ++i) {
					ov[i].x = fmaf(ov[i].x, scale4.x, bias4.x); ov[i].y = fmaf(ov[i].y, scale4.y, bias4.y);
					ov[i].z = fmaf(ov[i].z, scale4.z, bias4.z); ov[i].w = fmaf(ov[i].w, scale4.w, bias4.w);
				}
				if(fastStore && colsFull) {
					// the common case, free of branches: bias, optional residual, clamp by select, predicated 16-byte store
#pragma unroll
					for(int i = 0; i < 4; ++i) {
						const int m = rowBase + 8 * i + rowInGroup;
						float4 o = ov[i];
						if(useRes) { o.x += res[i].x; o.y += res[i].y; o.z += res[i].z; o.w += res[i].w; }
						o.x = clampOn ? fminf(fmaxf(o.x, 0.f), clampHi) : o.x;
						o.y = clampOn ? fminf(fmaxf(o.y, 0.f), clampHi) : o.y;
						o.z = clampOn ? fminf(fmaxf(o.z, 0.f), clampHi) : o.z;
						o.w = clampOn ? fminf(fmaxf(o.w, 0.f), clampHi) : o.w;
						float* dst = C + static_cast<size_t>(m) * p.ldc + n;
						if(m < mEnd) {
							asm volatile("st.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(o.x), "f"(o.y), "f"(o.z), "f"(o.w) : "memory");
						}
					}
				} else if(gateStore && colsFull) {
					// the same with the sigmoid gate, in a loop of its own so that the common one carries none of its code
#pragma unroll
					for(int i = 0; i < 4; ++i) {
						const int m = rowBase + 8 * i + rowInGroup;
						float4 o = ov[i];
						if(useRes) { o.x += res[i].x; o.y += res[i].y; o.z += res[i].z; o.w += res[i].w; }
						o.x = apply_act(o.x, NB200_ACT_SIGMOID_GATE, actParam); o.y = apply_act(o.y, NB200_ACT_SIGMOID_GATE, actParam);
						o.z = apply_act(o.z, NB200_ACT_SIGMOID_GATE, actParam); o.w = apply_act(o.w, NB200_ACT_SIGMOID_GATE, actParam);
						float* dst = C + static_cast<size_t>(m) * p.ldc + n;
						if(m < mEnd) {
							asm volatile("st.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(o.x), "f"(o.y), "f"(o.z), "f"(o.w) : "memory");
						}
					}
				} else if(hswishStore && colsFull) {
					// and with the hard swish (the element-wise path below takes twice as long: an expand layer of 24 -> 144 channels)
#pragma unroll
					for(int i = 0; i < 4; ++i) {
						const int m = rowBase + 8 * i + rowInGroup;
						float4 o = ov[i];
						if(useRes) { o.x += res[i].x; o.y += res[i].y; o.z += res[i].z; o.w += res[i].w; }
						o.x = apply_act(o.x, NB200_ACT_HSWISH, actParam); o.y = apply_act(o.y, NB200_ACT_HSWISH, actParam);
						o.z = apply_act(o.z, NB200_ACT_HSWISH, actParam); o.w = apply_act(o.w, NB200_ACT_HSWISH, actParam);
						float* dst = C + static_cast<size_t>(m) * p.ldc + n;
						if(m < mEnd) {
							asm volatile("st.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(o.x), "f"(o.y), "f"(o.z), "f"(o.w) : "memory");
						}
					}
				} else {
#pragma unroll
					for(int i = 0; i < 4; ++i) {
						const int m = rowBase + 8 * i + rowInGroup;
						if(m >= mEnd || n >= p.N) continue;
						const float e[4] = { ov[i].x, ov[i].y, ov[i].z, ov[i].w };
						float* dst = C + static_cast<size_t>(m) * p.ldc + n;
#pragma unroll
						for(int t = 0; t < 4; ++t) {
							if(n + t < p.N) {
								float y = e[t];
								if(R != nullptr) y += R[static_cast<size_t>(m) * p.ldr + n + t];
								y = apply_act(y, p.act, actParam);
								if(p.accumulate) y += dst[t];
								dst[t] = y;
							}
						}
					}
				}
#pragma unroll
				for(int i = 0; i < 4; ++i) res[i] = resNext[i];
				__syncwarp(); // the staging slice is rewritten by the next column chunk
			}
		}
	}

	tc_fence_before_sync();
	__syncthreads();
	if(warp == MMA_WARP) {
		tc_fence_after_sync();
		tmem_dealloc(tmemBase, TMEM_COLS);
	}
}

// B in split form: row n of `rows` becomes numKb blocks of 128 bytes (32 hi halves, 32 lo halves; zeros beyond K) at
// packed[n * numKb * 32 floats], and scales[n] = 1 / s_n, negative where the row has elements of fewer than 22 bits, 0 where it
// has nothing but zeros.  A row is held in registers between the search for its maximum
// and the split (up to 8 x 16 bytes per thread; the rest of a longer row is read again): by one warp where that suffices
// (K <= 1024), four rows to a block, else by the block.  Bound: memory, and for a layer's filter the launch itself.
// (4096 x 4096 took 60 us as two passes of dependent loads, one quad of a thread after the other.)
// WINDOW: the row is a convolution filter of r rows x s taps x c channels, and each filter row is widened to 32 floats
// (tap j / c4, channel j % c4), the row-window form of a few-channel layer.
struct RowWindow {
	int s, c, c4;
};
constexpr int ROW_THREADS = 128, ROW_QUADS = 8;

template<bool WINDOW, bool WARP_ROW>
__global__ void __launch_bounds__(ROW_THREADS) split_rows_kernel(const float* __restrict__ x, long long rows, long long ld, int k,
	int numKb, RowWindow w, uint2* __restrict__ packed, float* __restrict__ scales)
{
	// the scratch this writes may still be read by the contraction before it in the stream
	dependent_wait();
	dependents_may_start();
	constexpr int LANES = WARP_ROW ? 32 : ROW_THREADS;
	__shared__ float warpMax[ROW_THREADS / 32];
	__shared__ uint32_t warpMin[ROW_THREADS / 32];
	const int lane = WARP_ROW ? threadIdx.x & 31 : threadIdx.x;
	const long long row = WARP_ROW ? static_cast<long long>(blockIdx.x) * (ROW_THREADS / 32) + (threadIdx.x >> 5) : blockIdx.x;
	if(row >= rows) return; // whole warps (WARP_ROW) or none
	const float* src = x + row * ld;
	auto quad_at = [&](int q) { // floats 4q .. 4q + 3 of the row
		float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
		if(WINDOW) {
			const int fr = q >> 3, j = (q & 7) * 4;
			const int tap = j / w.c4, ch = j - tap * w.c4; // c4 is a multiple of four: one tap per quad
			if(tap < w.s) {
				const float* f = src + (fr * w.s + tap) * w.c;
				if(ch < w.c) v.x = __ldg(f + ch);
				if(ch + 1 < w.c) v.y = __ldg(f + ch + 1);
				if(ch + 2 < w.c) v.z = __ldg(f + ch + 2);
				if(ch + 3 < w.c) v.w = __ldg(f + ch + 3);
			}
		} else if(4 * q + 4 <= k) { // rows are 16-byte aligned
			v = __ldg(reinterpret_cast<const float4*>(src) + q);
		} else {
			if(4 * q < k) v.x = __ldg(src + 4 * q);
			if(4 * q + 1 < k) v.y = __ldg(src + 4 * q + 1);
			if(4 * q + 2 < k) v.z = __ldg(src + 4 * q + 2);
		}
		return v;
	};
	const int quads = numKb * 8;
	float4 held[ROW_QUADS];
	float largest = 0.f;
	uint32_t smallest = 0xffffffffu;
#pragma unroll
	for(int i = 0; i < ROW_QUADS; ++i) {
		const int q = lane + i * LANES;
		held[i] = q < quads ? quad_at(q) : make_float4(0.f, 0.f, 0.f, 0.f);
	}
#pragma unroll
	for(int i = 0; i < ROW_QUADS; ++i) {
		largest = max_abs(largest, held[i]);
		smallest = smallest_key(smallest, held[i]);
	}
	for(int q = lane + ROW_QUADS * LANES; q < quads; q += LANES) {
		const float4 v = quad_at(q);
		largest = max_abs(largest, v);
		smallest = smallest_key(smallest, v);
	}
#pragma unroll
	for(int o = 16; o > 0; o >>= 1) largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, o));
	smallest = __reduce_min_sync(0xffffffffu, smallest);
	if(!WARP_ROW) {
		if((threadIdx.x & 31) == 0) {
			warpMax[threadIdx.x >> 5] = largest;
			warpMin[threadIdx.x >> 5] = smallest;
		}
		__syncthreads();
		largest = fmaxf(fmaxf(warpMax[0], warpMax[1]), fmaxf(warpMax[2], warpMax[3]));
		smallest = min(min(warpMin[0], warpMin[1]), min(warpMin[2], warpMin[3]));
	}
	// 2^5 times the target of A's rows: nothing larger follows, so the whole range is used (subnormal maxima: the largest scale)
	const bool zeros = smallest == 0xffffffffu;
	const float s = zeros ? 1.f : scale_for(largest * (1.f / 32.f)), inv = inverse_scale(s);
	if(lane == 0) scales[row] = zeros ? 0.f : (smallest < coarse_below(inv) ? -inv : inv);
	uint2* out = packed + row * numKb * 16;
	auto put = [&](int q, const float4& v) {
		uint2 hi, lo;
		split_pair(v.x, v.y, s, s * LO_SCALE, hi.x, lo.x);
		split_pair(v.z, v.w, s, s * LO_SCALE, hi.y, lo.y);
		out[(q >> 3) * 16 + (q & 7)] = hi;
		out[(q >> 3) * 16 + 8 + (q & 7)] = lo;
	};
#pragma unroll
	for(int i = 0; i < ROW_QUADS; ++i) {
		const int q = lane + i * LANES;
		if(q < quads) put(q, held[i]);
	}
	for(int q = lane + ROW_QUADS * LANES; q < quads; q += LANES) put(q, quad_at(q));
}

template<bool WINDOW>
int launch_split_rows(const float* x, long long rows, long long ld, int k, int numKb, RowWindow w, float* out, cudaStream_t stream)
{
	float* scales = out + rows * numKb * BK;
	if(numKb * 8 <= 32 * ROW_QUADS) {
		const long long blocks = (rows + ROW_THREADS / 32 - 1) / (ROW_THREADS / 32);
		launch_dependent(overlap_launches(), split_rows_kernel<WINDOW, true>, dim3(static_cast<unsigned>(blocks)), dim3(ROW_THREADS), 0,
			stream, x, rows, ld, k, numKb, w, reinterpret_cast<uint2*>(out), scales);
	} else {
		launch_dependent(overlap_launches(), split_rows_kernel<WINDOW, false>, dim3(static_cast<unsigned>(rows)), dim3(ROW_THREADS), 0,
			stream, x, rows, ld, k, numKb, w, reinterpret_cast<uint2*>(out), scales);
	}
	count_launch();
	return check_launch();
}

template<int BN>
int launch_bn(const ContractionParams& p0, int batch, cudaStream_t stream)
{
	ContractionParams p = p0;
	static std::atomic<bool> attrSet[64];
	int dev = 0;
	if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NB200_ENODEVICE;
	if(!attrSet[dev].load()) {
		const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
		if(cudaFuncSetAttribute(contraction_split_kernel<BN>, attr, 227 * 1024) != cudaSuccess) {
			cudaGetLastError();
			return NB200_ENODEVICE;
		}
		attrSet[dev].store(true);
	}
	if(p.tileM <= 0 || p.tileM > BM || p.a_mode != A_CONV_WINDOW) p.tileM = BM;
	const long long mTiles = (static_cast<long long>(p.M) + p.tileM - 1) / p.tileM;
	const long long nTiles = (p.N + BN - 1) / BN;
	const long long tilesPerBatch = mTiles * nTiles;
	const long long numTiles = tilesPerBatch * batch;
	const int numKb = (p.K + BK - 1) / BK;
	if(numTiles > 0x7fffffffLL || numTiles * numKb > 0x7fffffffLL) return NB200_ETOOBIG;
	const int sms = sm_count();
	alignas(64) CUtensorMap mapA, mapB;
	memset(&mapA, 0, sizeof(mapA));
	memset(&mapB, 0, sizeof(mapB));
	p.a_tma = make_operand_map(&mapA, p, batch, BM);
	const int packedRow = numKb * BK; // in floats
	if(p.a_tma == 0 || !make_rows_map(&mapB, reinterpret_cast<const float*>(p.bSplit), packedRow, p.N, packedRow, batch,
		static_cast<long long>(p.N) * packedRow, BN)) {
		return NB200_EINVAL;
	}
	const SplitFinish finish = split_k(p, numTiles, numKb, batch);
	const long long numWork = numTiles * p.kSplits;
	const int grid = numWork < sms ? static_cast<int>(numWork) : sms;
	// as many raw slots as fit the 227 KB a CTA may use: the copies run that many K blocks ahead
	constexpr int fixedBytes = EPI_WARPS * STAGING_BYTES_PER_WARP + EPI_WARPS * BN * 6 /*strips*/ + (SCALE_RING + 1) * BM * 4
		+ 512 /*barriers*/ + 1024 /*alignment slack*/;
	constexpr int slotBytes = A_TILE_BYTES + BN * B_ROW_BYTES;
	constexpr int fitting = (227 * 1024 - fixedBytes) / slotBytes;
	constexpr int rawSlots = fitting < MAX_RAW_SLOTS ? fitting : MAX_RAW_SLOTS;
	constexpr size_t smemBytes = static_cast<size_t>(rawSlots) * slotBytes + fixedBytes;
	p.div = tile_divs(p, nTiles, tilesPerBatch);
	const int nt = static_cast<int>(numWork), nn = static_cast<int>(nTiles), tpb = static_cast<int>(tilesPerBatch);
	cudaEvent_t timedStart = nullptr, timedStop = nullptr;
	const bool timed = timing_events(&timedStart, &timedStop);
	if(timed) cudaEventRecord(timedStart, stream);
	const bool overlap = overlap_launches();
	launch_dependent(overlap, contraction_split_kernel<BN>, dim3(grid), dim3(THREADS), smemBytes, stream, p, nt, nn, tpb, rawSlots, mapA, mapB);
	count_launch();
	if(p.kSplits > 1) launch_split_finish(p, finish, stream);
	if(timed) cudaEventRecord(timedStop, stream);
	return check_launch();
}

} // namespace

size_t split_operand_floats(long long rows, long long k)
{
	return static_cast<size_t>(rows * ((k + BK - 1) / BK * BK) + (rows + 3) / 4 * 4);
}

int split_operand(const float* x, long long rows, long long ld, int k, float* out, cudaStream_t stream)
{
	return launch_split_rows<false>(x, rows, ld, k, (k + BK - 1) / BK, RowWindow{}, out, stream);
}

int split_window_filter(const float* f, int rows, int r, int s, int c, int c4, float* out, cudaStream_t stream)
{
	return launch_split_rows<true>(f, rows, static_cast<long long>(r) * s * c, r * BK, r, RowWindow{ s, c, c4 }, out, stream);
}

int launch_contraction_split(const ContractionParams& p, int batch, cudaStream_t stream)
{
	if(p.M <= 0 || p.N <= 0 || batch <= 0) return NB200_OK;
	const int tileM = p.a_mode == A_CONV_WINDOW && p.tileM > 0 && p.tileM <= BM ? p.tileM : BM;
	const bool maySplit = p.splitScratch != nullptr && batch == 1 && p.K >= 8 * BK;
	switch(maySplit ? contraction_tile_width(p.N) : balanced_tile_width(p, (p.M + tileM - 1LL) / tileM, batch)) {
		case 32: return launch_bn<32>(p, batch, stream);
		case 64: return launch_bn<64>(p, batch, stream);
		case 96: return launch_bn<96>(p, batch, stream);
		default: return launch_bn<128>(p, batch, stream);
	}
}

} // namespace nb200
