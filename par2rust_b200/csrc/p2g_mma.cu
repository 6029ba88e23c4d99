// p2g_mma.cu -- the Reed-Solomon accumulator on the tensor cores (tcgen05,
// kind::mxf4), as a bit-sliced GF(2) product.
//
// recovery[r] = XOR_s c(r,s) * source[s] over GF(2^16) (src/reedsolomon.rs:
// 87-126, src/creator.rs:934-1007).  Multiplication by a constant c is
// GF(2)-linear on the 16 bits of a symbol: bit i of c * x is the parity of
// sum_j M_c[i][j] bit_j(x), where M_c[i][j] is bit i of c * a^j (a = 2).  So
//
//     bit_i(rec[r][n]) = parity of  sum_s sum_j M_c(r,s)[i][j] * bit_j(src[s][n]) ,
//
// an integer matrix product D = A * B^T with 0/1 entries:
//     A[n, (s,j)]     = bit j of src[s][n]           (M = symbols)
//     B[(r,i), (s,j)] = M_c(r,s)[i][j]               (N = 16 rows per recovery row)
// summed over K = 16 S, of which only the parity is kept.  0 and 1 are exact
// e2m1 values (1.0 = 0x2), all scale factors are 1.0 (UE8M0 127), and the
// fp32 accumulator holds the sums exactly (at most 16 * 32768 < 2^24).
//
// Bit i of z is Tr(d_i z) for the basis d_0..d_15 dual to 1, a, .., a^15 under
// the trace, so row i of M_c is 16 consecutive terms of the sequence Tr(a^k)
// from k = log c + log d_i: one table lookup (d_trace_bits) per 16 entries.
//
// Tile: 256 symbols (two M = 128 MMAs) x up to 13 recovery rows (N = 16 a
// row), accumulated in TMEM over all input slices, K-step = 4 slices (K = 64
// e2m1 values = 32 bytes per operand row).  The R rows are dealt to the fewest
// row tiles of at most 13, evenly (mma_rows).  a_image_kernel first writes B of
// the whole job to global memory (R x S x 128 bytes, built once instead of
// once per symbol tile).  Warp roles:
//   warp 0       TMA producer: per 16 input slices, one bulk copy of their B
//                rows and one 2-D tensor copy of the tile's source symbols
//   warp 1       TMEM allocation; issues the MMAs and commits
//   warps 4..15  spread the source symbols to e2m1 into A stages in TMEM, then
//                run the epilogue: tcgen05.ld of the sums, parity, store
// The tile pipeline itself is p2g_mma_tile.cuh, shared with the persistent
// batch kernel's tensor-core items.
// Every mbarrier wait is bounded; a wait that gives up sets the error flag,
// stops all roles, drains copies and MMAs in flight and frees TMEM.
#include <mutex>

#include "p2g_internal.h"
#include "p2g_mma_tile.cuh"

namespace p2g {

// d_trace_bits[k] = sum_{j<16} Tr(a^(k+j)) 2^j, k < 65535; d_dual_log[i] = log d_i.
__device__ uint16_t d_trace_bits[65536];
__device__ uint16_t d_dual_log[16];

namespace {

using namespace mma;
constexpr int kThreads = 512;
constexpr int kImageThreads = 224;  // a K-step of 13 rows has 416 units, of 7 224
constexpr int kInStages = 6;  // 4 K-steps each: the MMAs of 20 in reserve, 4,200 cycles

// shared memory layout (bytes): the ring, barriers, misc
constexpr uint32_t kOffBars = kInStages * kInStageBytes;
constexpr uint32_t kOffMisc = kOffBars + bar_bytes(kInStages);
constexpr uint32_t kOffNext = kOffMisc + 32;  // two tiles: the one at work and the next
constexpr uint32_t kSmemBytes = kOffNext + 2 * sizeof(Tile);
static_assert(kSmemBytes > 116 * 1024, "one CTA per SM: TMEM is allocated whole");
static_assert(kSmemBytes <= 227 * 1024, "shared memory per CTA");
static_assert(mma_image_steps(1027) == image_steps(1027) && mma_image_steps(32) == image_steps(32) &&
                  kMmaTileSymbols == kTileSyms && kMmaMaxRows == kMaxRows,
              "host and device agree on the tile and the image layout");

}  // namespace

// The coefficient image of one job (layout: image_steps in p2g_mma_tile.cuh):
// K-steps b0, b0 + step, .. of its row tiles, one CTA a K-step at a time, a
// thread per 16-byte K half of a B row, so that the only divisions are one a
// K-step.  Rows of recovery row r >= R and slices s >= S are 0.  c(r,s) =
// base_s ^ (first_exp + r) = 2^(logbase_s * (first_exp + r) mod 65535)
// (RsEncoder::coefficient, src/reedsolomon.rs:56-60; gf_pow
// src/galois.rs:74-87).  Bound by the writes: 512 MB (2,000 rows x 2,000
// slices) took 181 us with an index division a unit, 136 now.
__device__ __forceinline__ void fill_a_image(uint8_t* __restrict__ aimg, uint32_t S, uint32_t R, uint32_t first_exp,
                                             const uint16_t* __restrict__ logbase, uint32_t b0, uint32_t step) {
    const uint32_t rows = mma_rows(R), ksteps = image_steps(S), n_row = (R + rows - 1) / rows;
    const uint32_t units = rows * (kRowStepBytes / 16);  // 16-byte units of a K-step
    for (uint32_t q = b0; q < n_row * ksteps; q += step) {  // < 2^13 row tiles x 2^13 K-steps
        const uint32_t rt = q / ksteps, k = q - rt * ksteps;
        uint4* out = reinterpret_cast<uint4*>(aimg) + (size_t)q * units;
        for (uint32_t c = threadIdx.x; c < units; c += blockDim.x) {  // byte c*16 = grp*256 + kh*128 + m8*16
            const uint32_t n = (c >> 4) * 8 + (c & 7u), kh = (c >> 3) & 1u;
            const uint32_t r = rt * rows + (n >> 4), s0 = k * kKSlices + 2 * kh;
            const uint32_t e = (first_exp + r) % kFieldLimit, d = d_dual_log[n & 15u];
            auto bits = [&](uint32_t s) -> uint32_t {  // row n & 15 of M_c(r,s)
                if (r >= R || s >= S) return 0u;
                uint32_t x = (uint32_t)logbase[s] * e;  // < 2^32
                x = (x & 0xFFFFu) + (x >> 16);
                x = (x & 0xFFFFu) + (x >> 16);
                if (x >= kFieldLimit) x -= kFieldLimit;
                x += d;
                if (x >= kFieldLimit) x -= kFieldLimit;
                return d_trace_bits[x];
            };
            const uint2 v0 = spread16(bits(s0)), v1 = spread16(bits(s0 + 1));
            out[c] = make_uint4(v0.x, v0.y, v1.x, v1.y);
        }
    }
}

__global__ void a_image_kernel(uint8_t* __restrict__ aimg, const uint16_t* __restrict__ logbase, uint32_t S, uint32_t R,
                               uint32_t first_exp) {
    fill_a_image(aimg, S, R, first_exp, logbase, blockIdx.x, gridDim.x);
}

struct EncodeArgs {
    CUtensorMap src_map;
    const uint8_t* aimg;
    uint8_t* rec;
    uint64_t rec_stride;
    uint32_t S, Np, R, rows, row_tiles, sym_tiles;
};

// Tile `at` of the grid's order: blocks of kMmaRowBlock row tiles, symbol tile
// by symbol tile, row tiles fastest, so the CTAs at work share both their
// source symbols (up to 8 ways) and their coefficients (19 ways) in L2,
// whichever is larger.
__device__ __forceinline__ Tile tile_of(const EncodeArgs& A, uint32_t at) {
    const uint32_t rb = at / (kMmaRowBlock * A.sym_tiles);
    at -= rb * kMmaRowBlock * A.sym_tiles;
    const uint32_t wide = min(kMmaRowBlock, A.row_tiles - rb * kMmaRowBlock);
    const uint32_t rt = rb * kMmaRowBlock + at % wide;
    Tile T;
    T.src_map = &A.src_map;
    T.aimg = A.aimg + (size_t)rt * image_steps(A.S) * A.rows * kRowStepBytes;
    T.rec = A.rec;
    T.rec_stride = A.rec_stride;
    T.s0 = 0;
    T.sn = A.S;
    T.rows = A.rows;
    T.R = A.R;
    T.r0 = rt * A.rows;
    T.n0 = at / wide * kTileSyms;
    T.syms = min(kTileSyms, A.Np - T.n0);
    T.accumulate = 0;
    return T;
}

// One tile, out of line as in the batch kernel: inlined into the tile loop the
// compiler keeps the MMA warp's operands out of uniform registers, and a
// K-step takes 300 cycles.  The pipeline's state stays in registers from tile
// to tile (shared memory and a second CTA barrier cost 1-2 % on short tiles).
// The tile is in shared memory, worked out by one thread: its divisions by
// every thread ahead of the roles cost 3 us of 56 at 64 slices.
// misc: [0] TMEM base, [1] abort flag, [5] input stages issued.
struct PipeState {
    uint32_t gi, tcount, pre, ok;
};
template <uint32_t POLLS, uint32_t DROP>
__device__ __noinline__ PipeState encode_mma_tile(const EncodeArgs& A, uint32_t next, uint32_t gi, uint32_t tcount,
                                                  uint32_t pre) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + kOffMisc);
    mma::Pipe P;
    P.ring = smem_addr(smem);
    P.bars = smem_addr(smem + kOffBars);
    P.tmem = misc[0];
    P.abort_flag = misc + 1;
    P.gi = gi;
    P.tcount = tcount;
    P.pre = pre;
    P.issued = misc + 5;
    // the helper warp works out the next tile while this one runs
    Tile* const slots = reinterpret_cast<Tile*>(smem + kOffNext);
    Tile* const slot = slots + ((P.tcount & 1u) ^ 1u);
    P.next = slot;
    const bool ok = run_tile<kInStages, false, true, POLLS, DROP>(P, slots[P.tcount & 1u], [&] {
        if ((threadIdx.x & 31) == 0) {
            if (next < A.row_tiles * A.sym_tiles)
                *slot = tile_of(A, next);
            else
                slot->rows = 0;
        }
    });  // ends with a CTA barrier
    return {P.gi, P.tcount, P.pre, ok};
}

template <uint32_t POLLS, uint32_t DROP>
__global__ void __launch_bounds__(kThreads, 1) encode_mma_kernel(const __grid_constant__ EncodeArgs A,
                                                                 int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5;
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + kOffMisc);
    if (tid == 0) {
        init_bars<kInStages>(smem_addr(smem + kOffBars));
        misc[1] = misc[5] = 0;
        *reinterpret_cast<Tile*>(smem + kOffNext) = tile_of(A, blockIdx.x);
    }
    if (warp == 1) tmem_alloc(smem_addr(misc));  // the whole of TMEM: two accumulators, A stages, scale factors
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = misc[0];
    if (warp >= 4 && warp < 8) sf_fill(tmem, (uint32_t)warp & 3u);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    PipeState st = {0, 0, 0, 1};
    for (uint32_t tile = blockIdx.x; st.ok && tile < A.row_tiles * A.sym_tiles; tile += gridDim.x)
        st = encode_mma_tile<POLLS, DROP>(A, tile + gridDim.x, st.gi, st.tcount, st.pre);
    if (tid == 0 && !st.ok) atomicOr(err, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (!st.ok) mma_drain(Bars<kInStages>(smem_addr(smem + kOffBars)).drain);
        __syncwarp();
        tc_fence_after();
        tmem_free(tmem);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {
// The kernel of every encode, and the one that checks the give-up path: a tile's
// third stage never arrives and a wait is 4,096 polls.
constexpr auto encode_kernel = encode_mma_kernel<kTilePolls, kDropNone>;
constexpr auto giveup_kernel = encode_mma_kernel<4096, 2>;
// The trace sequence and the dual basis from the field itself (polynomial
// 0x1100B, generator 2).  Returns false if the trace form were singular (it
// never is).
bool build_trace_tables(std::vector<uint16_t>& bits, uint16_t dual_log[16]) {
    std::vector<uint32_t> al(65536), lg(65536);
    uint32_t b = 1;
    for (uint32_t l = 0; l < kFieldLimit; ++l) {
        al[l] = b;
        lg[b] = l;
        b <<= 1;
        if (b & 0x10000u) b ^= kFieldGenerator;
    }
    auto mul = [&](uint32_t x, uint32_t y) -> uint32_t {
        return (x && y) ? al[(lg[x] + lg[y]) % kFieldLimit] : 0u;
    };
    auto trace = [&](uint32_t y) {  // y + y^2 + ... + y^(2^15), in {0, 1}
        uint32_t acc = y, z = y;
        for (int i = 0; i < 15; ++i) {
            z = mul(z, z);
            acc ^= z;
        }
        return acc & 1u;
    };
    std::vector<uint8_t> tr(kFieldLimit + 16);
    for (uint32_t k = 0; k < kFieldLimit; ++k) tr[k] = (uint8_t)trace(al[k]);
    for (uint32_t k = 0; k < 16; ++k) tr[kFieldLimit + k] = tr[k];
    bits.assign(65536, 0);
    for (uint32_t k = 0; k < kFieldLimit; ++k)
        for (uint32_t j = 0; j < 16; ++j) bits[k] |= (uint16_t)(tr[k + j] << j);
    // G[i][j] = Tr(a^(i+j)); invert over GF(2): rows as 32-bit [G | I].  The
    // dual basis is d_i = sum_j G^-1[i][j] a^j.
    uint32_t rows[16];
    for (uint32_t i = 0; i < 16; ++i) {
        rows[i] = 1u << (16 + i);
        for (uint32_t j = 0; j < 16; ++j) rows[i] |= (uint32_t)tr[i + j] << j;
    }
    for (uint32_t c = 0; c < 16; ++c) {
        uint32_t p = c;
        while (p < 16 && !((rows[p] >> c) & 1u)) ++p;
        if (p == 16) return false;
        std::swap(rows[c], rows[p]);
        for (uint32_t r = 0; r < 16; ++r)
            if (r != c && ((rows[r] >> c) & 1u)) rows[r] ^= rows[c];
    }
    for (uint32_t i = 0; i < 16; ++i) dual_log[i] = (uint16_t)lg[rows[i] >> 16];
    return true;
}
}  // namespace

cudaError_t mma_prepare() {
    static std::mutex mu;
    static bool done[256] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 0 && dev < 256 && done[dev]) return cudaSuccess;
    std::vector<uint16_t> bits;
    uint16_t dual[16];
    if (!build_trace_tables(bits, dual)) return cudaErrorInvalidValue;
    if ((e = cudaMemcpyToSymbol(d_trace_bits, bits.data(), 2 * bits.size())) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(d_dual_log, dual, sizeof dual)) != cudaSuccess) return e;
    for (auto k : {encode_kernel, giveup_kernel})
        if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes)) != cudaSuccess)
            return e;
    if (dev >= 0 && dev < 256) done[dev] = true;
    return cudaSuccess;
}

// The coefficient images of every tensor-core job of a batch (blockIdx.y = job).
__global__ void a_image_batch_kernel(const BatchJob* __restrict__ jobs, const uint16_t* __restrict__ logbase) {
    const BatchJob& J = jobs[blockIdx.y];
    if (!J.mma || !J.R || !J.aimg) return;
    fill_a_image(J.aimg, J.S, J.R, J.first_exp, logbase, blockIdx.x, gridDim.x);
}

cudaError_t launch_a_image_batch(const BatchJob* jobs, uint32_t n_jobs, uint64_t max_bytes, cudaStream_t st) {
    if (!n_jobs || !max_bytes) return cudaSuccess;
    cudaError_t e = mma_prepare();
    if (e != cudaSuccess) return e;
    const uint16_t *antilog = nullptr, *logbase = nullptr;
    if ((e = gf_device_tables(&antilog, &logbase)) != cudaSuccess) return e;
    const uint64_t want = max_bytes / kRowStepBytes;  // K-steps of the largest image, at most
    const unsigned bx = (unsigned)std::min<uint64_t>(want, (uint64_t)device_sm_count() * 8);
    a_image_batch_kernel<<<dim3(bx, n_jobs), kImageThreads, 0, st>>>(jobs, logbase);
    add_launches(1);
    return cudaGetLastError();
}

size_t mma_aimg_bytes(uint32_t S, uint32_t R) {
    const uint32_t rows = mma_rows(R);
    return (size_t)((R + rows - 1) / rows * rows) * image_steps(S) * kRowStepBytes;
}

// The source as a 2-D tensor of u16 symbols: Np symbols per input slice, S
// slices `stride` bytes apart (16-byte aligned base and stride), read in
// boxes of 256 symbols x 16 slices, zeros past either extent.
cudaError_t make_src_map(CUtensorMap* map, const void* src, uint64_t stride, uint32_t S, uint32_t Np) {
    using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                     const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeTiled encode = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<EncodeTiled>(fn);
    });
    if (!encode) return cudaErrorNotSupported;
    if ((uintptr_t)src % 16 || stride % 16 || !S || !Np) return cudaErrorInvalidValue;
    const cuuint64_t dims[2] = {Np, S};
    const cuuint64_t strides[1] = {stride};
    const cuuint32_t box[2] = {kTileSyms, kInSlices};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(src), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_encode_mma(const uint8_t* src, uint64_t src_stride, uint32_t S, uint64_t slice_size, uint32_t R,
                              uint32_t first_exp, uint8_t* aimg, uint8_t* rec, uint64_t rec_stride, int* err,
                              cudaStream_t st, bool give_up) {
    if (!S || !R) return cudaSuccess;
    cudaError_t e = mma_prepare();
    if (e != cudaSuccess) return e;
    const uint16_t *antilog = nullptr, *logbase = nullptr;
    if ((e = gf_device_tables(&antilog, &logbase)) != cudaSuccess) return e;
    const uint32_t Np = (uint32_t)(((slice_size + 15) & ~15ull) / 2);
    EncodeArgs A;
    if ((e = make_src_map(&A.src_map, src, src_stride, S, Np)) != cudaSuccess) return e;
    A.aimg = aimg;
    A.rec = rec;
    A.rec_stride = rec_stride;
    A.S = S;
    A.Np = Np;
    A.R = R;
    A.rows = mma_rows(R);
    A.row_tiles = mma_row_tiles(R);
    A.sym_tiles = (Np + kTileSyms - 1) / kTileSyms;
    const int sms = device_sm_count();
    const unsigned cb = (unsigned)std::min<uint64_t>((uint64_t)A.row_tiles * image_steps(S), (uint64_t)sms * 8);
    a_image_kernel<<<cb, kImageThreads, 0, st>>>(aimg, logbase, S, R, first_exp);
    add_launches(1);
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)A.row_tiles * A.sym_tiles, (uint64_t)sms);
    (give_up ? giveup_kernel : encode_kernel)<<<grid, kThreads, kSmemBytes, st>>>(A, err);
    add_launches(1);
    return cudaGetLastError();
}

}  // namespace p2g
