// p2g_mma_tile.cuh -- device code of the tensor-core (tcgen05, kind::mxf4)
// encode shared by its standalone kernel (p2g_mma.cu) and the persistent
// batch kernel (p2g_kernels.cu).
//
// The arithmetic (a recovery row as a GF(2) matrix product) is explained at
// the top of p2g_mma.cu.  Here: the shared-memory and TMEM layout of one CTA
// and the work of one tile, 256 symbols x up to 13 recovery rows, over a range
// of input slices.
//
// The symbols are the M side: lane m of the two M = 128 accumulators holds
// symbols 2m and 2m+1 of the tile, and the 16 columns of a recovery row are its
// 16 bits, so a lane ends up with whole recovery symbols and the epilogue needs
// no exchange between lanes.  The symbols' bits (A) go from registers straight
// to TMEM (tcgen05.st) and are read from there by the MMAs; the coefficients'
// bit matrices (B, N = 16 x rows) are built once per job in global memory (the
// coefficient image, image_steps below) and copied in per 16 slices.
//
// What bounds the tile is shared memory, which feeds the MMAs 64 B/clk (B, 32 N
// bytes per N/2 cycles) of its 128.  With A there too (128 rows x 32 B an MMA,
// stored by the builders, read by the MMAs) a 4-slice K-step of two N = 240
// MMAs took 430 cycles where the MMAs alone take 240; with A in TMEM a K-step
// of two N = 208 MMAs takes 230 where they alone take 208 (538 MB, 200 rows:
// 5.33 -> 3.93 ms with the tile's start and epilogue; under a steady load the
// clock falls to 1.83-1.95 GHz at the 1,000 W limit).  13 rows: two accumulators of 208 columns,
// 8 for the scale factors and four K-steps of A of 16 fit TMEM's 512.
//
// Shared memory (from `ring`, 1024-aligned): input stages of 34,816 B, each
// covering 4 K-steps (16 input slices): their coefficient rows (4 x 512 B a
// recovery row, one bulk copy) and, 26,624 B in, the tile's symbols of those
// slices ([slice][256 symbols], 8 KiB, one 2-D tensor copy).  B is K-major
// without swizzle: core matrices of 8 rows x 16 B, K halves 128 B apart, 8-row
// groups 256 B apart.
#pragma once
#include <stdint.h>

namespace p2g {
namespace mma {

constexpr uint32_t kTileSyms = 256;  // symbols per tile: two M = 128 MMAs
constexpr uint32_t kMaxRows = 13;    // recovery rows per tile (MMA N = 16 x rows)
constexpr uint32_t kKSlices = 4;     // input slices per K-step (K = 64 e2m1 values)
constexpr uint32_t kInSteps = 4;                     // K-steps per input stage
constexpr uint32_t kInSlices = kInSteps * kKSlices;  // 16 input slices per input stage
constexpr uint32_t kRowStepBytes = 16 * 32;          // B rows of one recovery row and K-step
constexpr uint32_t kSrcSliceBytes = kTileSyms * 2;
constexpr uint32_t kInBBytes = kInSteps * kMaxRows * kRowStepBytes;  // 26,624 B at most
constexpr uint32_t kInSrcBytes = kInSlices * kSrcSliceBytes;         // 8 KiB
constexpr uint32_t kInStageBytes = kInBBytes + kInSrcBytes;
constexpr uint32_t kAStages = 2;                      // halves of an input stage (2 K-steps each) in TMEM
constexpr uint32_t kAccCol1 = 16 * kMaxRows;          // TMEM column of the second accumulator
constexpr uint32_t kSfCol = 2 * kAccCol1;             // scale factors (all 1.0, read as both operands')
constexpr uint32_t kACol = kSfCol + 8;                // A, 16 columns a K-step: 8 a M = 128 half
constexpr uint32_t kEpilogueWarps = 12;               // three to a TMEM lane quadrant
static_assert(kACol + 16 * kInSteps <= 512, "TMEM columns");
static_assert(kInStageBytes % 1024 == 0 && kInBBytes % 128 == 0, "tensor copies land 128-byte aligned");
// barriers: in_full/in_empty per input stage, a_full/a_empty per A stage, acc_full, acc_empty, next_full, drain
__host__ __device__ constexpr uint32_t bar_bytes(int in_stages) { return (2 * in_stages + 2 * (int)kAStages + 4) * 8; }

// The coefficient image in global memory: for row tile rt (`rows` recovery
// rows) and K-step k (slices 4k .. 4k+3), rows x 512 B laid out as in shared
// memory -- byte
//   (rt * ksteps + k) * rows * 512 + grp * 256 + kh * 128 + m8 * 16
// holds B row n = 8 grp + m8 (recovery row rt * rows + n / 16, bit n % 16), K
// half kh (slices 4k + 2kh, 4k + 2kh + 1): 8 e2m1 bytes per slice.  ksteps =
// image_steps(S): whole input stages, zero past S and R.
__host__ __device__ constexpr uint32_t image_steps(uint32_t S) {
    return (S + kInSlices - 1) / kInSlices * kInSteps;
}

// Instruction descriptor of kind::mxf4 with UE8M0 block scales: A and B
// e2m1 (format 1 at bits 7 and 10), K-major, N >> 3 at bit 17, scale format
// UE8M0 at bit 23, M >> 4 at bit 24, scale-factor ids 0, dense K = 64.
__device__ __forceinline__ uint32_t idesc(uint32_t n) {
    return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (1u << 23) | ((128u >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Polls of one wait before it gives up.
constexpr uint32_t kTilePolls = 1u << 22;
// Waits (bounded) for a phase without looking at the abort flag: for
// copies and MMAs in flight, which land whatever happened elsewhere.
__device__ __forceinline__ void bar_drain(uint32_t bar, uint32_t parity, uint32_t polls = kTilePolls) {
    for (uint32_t it = 0; it < polls && !bar_try_wait(bar, parity); ++it) {
    }
}
__device__ __forceinline__ void tma_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// 2-D tiled tensor copy: the box at (x, y) of the tensor map `map` (a generic
// address of a CUtensorMap in kernel-parameter or global memory).  x times
// the element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_2d(uint32_t dst, const void* map, int32_t x, int32_t y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
// Before the first copy through a tensor map that ordinary stores wrote to
// global memory (the batch job descriptors).
__device__ __forceinline__ void tensormap_acquire(const void* map) {
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Shared-memory matrix descriptor, K-major, no swizzle: start >> 4, leading
// (K-half) byte offset >> 4 at bit 16, stride (8-row group) byte offset >> 4
// at bit 32, version 1 at bit 46.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// A in TMEM (8 columns: lane = row, 8 nibbles a column), one scale-factor
// address for both operands.
__device__ __forceinline__ void mma_mxf4(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t id, uint32_t sf,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %5, 0;\n"
        " tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], [%1], %2, %3, [%4], [%4], p;\n}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(id), "r"(sf), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(v)
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Two runs of 16 columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld16x2(uint32_t ta, uint32_t tb, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, "
        "%29, %30, %31}, [%33];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(ta), "r"(tb)
        : "memory");
}
// 16 bits -> 16 e2m1 values (0 or 1.0 = 0x2), 8 bytes.  Bit pairs (4q, 4q+1)
// go to byte q of the low word, pairs (4q+2, 4q+3) to byte q of the high
// word, each pair through a 4-entry byte table (PRMT).  A and B go through
// the same map, so K positions pair bit j with bit j.
constexpr uint32_t kPairs = 0x22200200u;  // byte g = e2m1 pair of bits (g & 1, g >> 1)
__device__ __forceinline__ uint2 spread16(uint32_t x) {
    return make_uint2(__byte_perm(kPairs, 0u, x & 0x3333u), __byte_perm(kPairs, 0u, (x >> 2) & 0x3333u));
}
// 4 slices' words (symbols 2m low, 2m+1 high) -> 8 e2m1 words of either half
__device__ __forceinline__ void spread4(const uint32_t* x, uint32_t (&v)[16]) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        // spread16 of both symbols: pairs (4q, 4q+1) from x & 0x3333, pairs (4q+2, 4q+3) from (x >> 2) & 0x3333
        const uint32_t e = x[s] & 0x33333333u, o = (x[s] >> 2) & 0x33333333u;
        v[2 * s] = __byte_perm(kPairs, 0u, e & 0xFFFFu);
        v[2 * s + 1] = __byte_perm(kPairs, 0u, o & 0xFFFFu);
        v[8 + 2 * s] = __byte_perm(kPairs, 0u, e >> 16);
        v[8 + 2 * s + 1] = __byte_perm(kPairs, 0u, o >> 16);
    }
}
__device__ __forceinline__ uint32_t lds_b32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// The values of tmem_ld16x2 are there (they pass through, so that nothing
// reads them before; an asm statement takes 30 in-out operands, the last two
// pass through a second one, which stays behind the first).
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.wait::ld.sync.aligned;"
        : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
          "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
          "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]),
          "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29])
        :
        : "memory");
    asm volatile("" : "+r"(v[30]), "+r"(v[31]));
}

// Barrier block of a pipeline with IN input stages.
template <int IN>
struct Bars {
    uint32_t in_full, in_empty, a_full, a_empty, acc_full, acc_empty, next_full, drain;
    __device__ explicit Bars(uint32_t b)
        : in_full(b), in_empty(b + 8 * IN), a_full(b + 16 * IN), a_empty(b + 16 * IN + 8 * kAStages),
          acc_full(b + 16 * IN + 16 * kAStages), acc_empty(acc_full + 8), next_full(acc_full + 16),
          drain(acc_full + 24) {}
};
// One thread.  An input stage is released by the MMA warp's commit after its
// last K-step (the builders have read it by then: the MMAs waited for their A).
template <int IN>
__device__ __forceinline__ void init_bars(uint32_t b) {
    const Bars<IN> B(b);
    for (int i = 0; i < IN; ++i) {
        bar_init(B.in_full + 8 * i, 1);
        bar_init(B.in_empty + 8 * i, 1);
    }
    for (uint32_t i = 0; i < kAStages; ++i) {
        bar_init(B.a_full + 8 * i, 8);  // the builder warps
        bar_init(B.a_empty + 8 * i, 1);
    }
    bar_init(B.acc_full, 1);
    bar_init(B.acc_empty, kEpilogueWarps);
    bar_init(B.next_full, 1);
    bar_init(B.drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// The whole of TMEM (one warp; the slot receives the base address), and
// given up again at the end by the same warp.
__device__ __forceinline__ void tmem_alloc(uint32_t slot) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(slot) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}
// The lane that issues a warp's asynchronous instructions.
__device__ __forceinline__ bool elect_one(uint32_t& leader) {
    uint32_t p;
    asm volatile("{\n .reg .pred P;\n elect.sync %0|P, 0xFFFFFFFF;\n selp.u32 %1, 1, 0, P;\n}" : "=r"(leader), "=r"(p));
    return p != 0;
}
// Every MMA that this warp issued has completed (all lanes of the MMA warp, once
// per launch: the barrier's first phase).
__device__ __forceinline__ void mma_drain(uint32_t drain) {
    uint32_t leader;
    if (elect_one(leader)) mma_commit(drain);
    bar_drain(drain, 0);
    __syncwarp();
}
// Scale factors 1.0 (UE8M0 127) over the 32 lanes of warp quadrant q
// (called by four warps with distinct quadrants).
__device__ __forceinline__ void sf_fill(uint32_t tmem, uint32_t q) {
    tmem_st8(tmem + ((32 * q) << 16) + kSfCol, 0x7F7F7F7Fu);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// One tile: recovery rows [r0, r0+rows) x symbols [n0, n0+syms) over input
// slices [s0, s0+sn), s0 a multiple of 16 and s0+sn a multiple of 4 or S.
// src_map: 2-D tensor map over the source (u16 symbols x input slices, the
// slice stride a multiple of 16 bytes; symbols and slices past its extent
// read 0); n0 and syms are multiples of 8.  aimg: the row tile's part of the
// job's coefficient image (`rows` is the image's, also where R ends inside
// the tile).  accumulate: XOR the tile into the rows (the caller zeroed them)
// instead of storing it.
struct Tile {
    const void* src_map;
    const uint8_t* aimg;
    uint8_t* rec;
    uint64_t rec_stride;
    uint32_t s0, sn, rows, R, r0, n0, syms, accumulate;
};

// Per-CTA pipeline state, the same in every thread: input stages and tiles so
// far (ring positions and barrier parities follow from them; every A stage
// takes part once per input stage).
struct Pipe {
    uint32_t ring, bars, tmem;
    volatile uint32_t* abort_flag;
    uint32_t gi, tcount;
    uint32_t pre;  // input stages of the coming tile already issued by the previous call
    volatile uint32_t* issued;  // shared: input stages issued so far, for the helper warp
    const Tile* next;           // shared: the tile that follows, written by the helper warp (rows 0: none)
};

__device__ __forceinline__ uint32_t uni(uint32_t v) { return __shfl_sync(0xFFFFFFFFu, v, 0); }
__device__ __forceinline__ uint64_t uni(uint64_t v) { return __shfl_sync(0xFFFFFFFFu, (unsigned long long)v, 0); }
// Bounded wait by a whole warp: false when it gave up (it then sets the abort
// flag) or when another role has given up.  The lanes vote on every poll, so
// that the loop's branch is one for the warp.  A failed poll takes ~8 us (the
// instruction waits by itself), a pipeline without faults sees one or two in a
// row: the flag is looked at after every 16th, so that a role which runs on after
// giving up is through an unsatisfied wait in 0.13 ms instead of the 2 ms of 256
// (a tile of 32,768 slices has 6,000 waits), and never before (after the first,
// the 538 MB job took 1.2 % longer; after the 16th of 256, 0.4 %, and a batch of
// 48 mixed jobs 0.8 %, by the loop's code alone).
template <uint32_t POLLS>
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag) {
    for (uint32_t it = 0; it < POLLS; ++it) {
        if (__all_sync(0xFFFFFFFFu, bar_try_wait(bar, parity))) return true;
        if ((it & 15u) == 15u && __any_sync(0xFFFFFFFFu, *abort_flag != 0)) return false;
    }
    *abort_flag = 1u;
    __threadfence_block();  // before anything this role still commits or arrives at
    return false;
}

// All threads of the CTA (16 warps) call this.  Warp 0 streams the inputs,
// warp 1 issues the MMAs, warp 2 finds the next tile, warps 4..11 build A (warp w its lane quadrant w % 4
// of every other K-step), and warps 4..15 run the epilogue (every third row of
// their quadrant).  Returns false (uniformly, after a CTA barrier) when a
// bounded wait gave up; copies in flight have then landed.
// helper: run by warp 2 when warp 0 has kHelperLead stages of this tile left to
// issue; it writes the tile this CTA runs next to *P.next.  Warp 0 then issues
// that tile's first input stages while this tile's last K-steps and epilogue
// run, so the next tile starts without a copy round trip.  Only warp 0's P.pre
// counts (the stages it issued ahead); the next call must be for that same
// tile.  When any role's wait gives up, warp 0 issues nothing more and waits for
// every copy it issued, the next tile's included, before this returns.  MMAs may
// then still run where only another role gave up: mma_drain stands before TMEM
// is freed (a wait for them here, after the roles, made the 538 MB job 2 % slower).
//
// Every role runs whole warps on values the compiler knows to be the same in
// every lane (uni), with only the asynchronous instructions under the elected
// lane: these take their operands from uniform registers.  It matters: with
// one lane in the loop, an MMA warp's iteration (wait, two MMAs, commit) took
// 580 cycles where the MMAs take 208, and one early return on a per-lane value
// ahead of the roles (a tile field read from memory) made a K-step 340-680;
// this way the warp keeps up with the MMAs.  For
// the same reason the MMA and builder loops have no branch beside the waits'
// own: K-steps past the tile's last multiply the builders' zeros, and a role
// whose wait gave up runs on to its end (the tile is dropped, its memory is the
// CTA's own and nothing is stored).
constexpr uint32_t kHelperLead = 4;  // with 5 more in flight, about 8,000 cycles before the tile's end
// ACQUIRE: the tensor maps were written by ordinary stores or copies (the
// batch job descriptors); the warp that issues the copies acquires each.
// LOAD_AHEAD: the epilogue loads a row's sums while it folds the row before;
// 94 registers instead of 63.  Together with the pipeline's state kept in
// registers between tiles, the standalone encode of 64 slices x 256 KiB and 32
// rows went from 53.2 to 49.1 us and 331 x 100,004 B x 53 from 96.2 to 94.2;
// large ones, which the board's power limit holds, stay within 0.6 %.  In the
// batch kernel the registers spill in its other items, and a 16 MiB job took
// 682 us instead of 672.
// POLLS, DROP: for the check of the give-up path alone (encode_mma_kernel's
// other form); it waits POLLS polls and leaves out the copies of a tile's stage
// DROP, so that every wait behind them runs out.
constexpr uint32_t kDropNone = 0xFFFFFFFFu;
template <int IN, bool ACQUIRE, bool LOAD_AHEAD, uint32_t POLLS = kTilePolls, uint32_t DROP = kDropNone, class Helper>
__device__ __forceinline__ bool run_tile(Pipe& P, const Tile& T, Helper&& helper) {
    const uint32_t warp = uni(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const Bars<IN> B(uni(P.bars));
    const uint32_t in0 = uni(P.ring), tmem = uni(P.tmem), rows = uni(T.rows);
    const uint32_t n0 = uni(T.n0), s0 = uni(T.s0), sn = uni(T.sn);
    const uint32_t NI = (sn + kInSlices - 1) / kInSlices;  // input stages
    const uint32_t gi0 = uni(P.gi), tc = uni(P.tcount);
    // a tensor copy's x offset must be 16-byte aligned, the image is cut in
    // whole input stages (the same in every thread)
    if ((n0 & 7u) || (s0 % kInSlices) || rows > kMaxRows) return false;
    // warp 0: the input-stage position after the last copy it issued and
    // has not drained (0: none), the next tile's first stages included
    uint32_t issued_end = 0;
    bool ok = true;
    if (warp == 0) {
        uint32_t leader;
        const bool lead = elect_one(leader);
        // stages [0, P.pre) of this tile went out with the previous tile
        const uint32_t pre = uni(P.pre);
        uint32_t gi = gi0 + pre;
        uint32_t st = gi % IN, par = ((gi / IN) & 1u) ^ 1u;
        // stages [k0, k1) of a tile; slices past its range (up to 15) are
        // copied too: the builders mask their A words
        auto issue = [&](uint64_t map, uint64_t aimg, uint32_t x, uint32_t first, uint32_t tile_rows, uint32_t k0,
                         uint32_t k1) {
            const uint32_t bytes = kInSteps * tile_rows * kRowStepBytes;
            const uint8_t* a = reinterpret_cast<const uint8_t*>(aimg) + (uint64_t)(first / kInSlices + k0) * bytes;
            uint32_t sa = first + k0 * kInSlices;
            for (uint32_t k = k0; k < k1; ++k, ++gi, sa += kInSlices, a += bytes) {
                // A role that gave up on a stage runs on and gives the stage
                // back with its copies perhaps in flight: none may follow them
                // into it, nor its barrier be armed a second time.  The flag
                // was set before the stage was given back.
                ok = warp_wait<POLLS>(B.in_empty + 8 * st, par, P.abort_flag) &&
                     !__any_sync(0xFFFFFFFFu, *P.abort_flag != 0);
                if (!ok) return;
                const uint32_t dst = in0 + st * kInStageBytes, full = B.in_full + 8 * st;
                if (lead && k != DROP) {
                    bar_expect_tx(full, bytes + kInSrcBytes);
                    tma_1d(dst, a, bytes, full);
                    tma_2d(dst + kInBBytes, reinterpret_cast<const void*>(map), (int32_t)x, (int32_t)sa, full);
                    *P.issued = gi + 1;
                }
                if (++st == IN) {
                    st = 0;
                    par ^= 1u;
                }
            }
        };
        if (ACQUIRE && pre == 0) tensormap_acquire(T.src_map);
        issue(uni((uint64_t)(uintptr_t)T.src_map), uni((uint64_t)(uintptr_t)T.aimg), n0, s0, rows, pre, NI);
        if (ok) ok = warp_wait<POLLS>(B.next_full, tc & 1u, P.abort_flag);
        if (ok) {
            const uint32_t n_rows = uni(P.next->rows), nx = uni(P.next->n0), ns = uni(P.next->s0);
            const uint32_t ni = (uni(P.next->sn) + kInSlices - 1) / kInSlices;
            if (n_rows && n_rows <= kMaxRows && !(nx & 7u) && !(ns % kInSlices)) {
                if (ACQUIRE) tensormap_acquire(P.next->src_map);
                issue(uni((uint64_t)(uintptr_t)P.next->src_map), uni((uint64_t)(uintptr_t)P.next->aimg), nx, ns, n_rows, 0,
                      ni < (uint32_t)IN ? ni : (uint32_t)IN);
            }
        }
        if (!ok) {  // copies issued but maybe not consumed land before the stages are reused
            for (uint32_t q = gi > gi0 + IN ? gi - IN : gi0; q < gi; ++q)
                bar_drain(B.in_full + 8 * (q % IN), (q / IN) & 1u, POLLS);
        } else {
            issued_end = gi;  // >= gi0 + NI: this tile's stages all went out
        }
    } else if (warp == 1) {
        uint32_t leader;
        const bool lead = elect_one(leader);
        const uint32_t id = idesc(16 * rows), step = rows * kRowStepBytes, sf = tmem + kSfCol;
        ok = warp_wait<POLLS>(B.acc_empty, (tc & 1u) ^ 1u, P.abort_flag);
        tc_fence_after();
        uint32_t si = gi0 % IN, pi = (gi0 / IN) & 1u, pa = gi0 & 1u;
        for (uint32_t k = 0; k < NI; ++k) {
            ok &= warp_wait<POLLS>(B.in_full + 8 * si, pi, P.abort_flag);
            const uint32_t b0 = in0 + si * kInStageBytes;
#pragma unroll
            for (uint32_t u = 0; u < kAStages; ++u) {
                ok &= warp_wait<POLLS>(B.a_full + 8 * u, pa, P.abort_flag);
                tc_fence_after();
                if (lead) {
#pragma unroll
                    for (uint32_t ks = 2 * u; ks < 2 * u + 2; ++ks) {
                        const uint64_t bdesc = smem_desc(b0 + ks * step, 128, 256);
                        const uint32_t a = tmem + kACol + 16 * ks;
                        mma_mxf4(tmem, a, bdesc, id, sf, k + ks);
                        mma_mxf4(tmem + kAccCol1, a + 8, bdesc, id, sf, k + ks);
                    }
                    mma_commit(B.a_empty + 8 * u);
                    if (u == kAStages - 1) mma_commit(B.in_empty + 8 * si);
                }
            }
            pa ^= 1u;
            if (++si == IN) {
                si = 0;
                pi ^= 1u;
            }
        }
        if (lead) mma_commit(B.acc_full);
        // every MMA issued completes before its stages or TMEM are reused
        if (!ok) bar_drain(B.acc_full, tc & 1u, POLLS);
    } else if (warp == 2) {
        const uint32_t at = NI > kHelperLead ? gi0 + NI - kHelperLead : gi0;
        for (uint32_t it = 0; it < (1u << 20) && (int32_t)(*P.issued - at) < 0 && !*P.abort_flag; ++it) __nanosleep(64);
        helper();
        __syncwarp();
        if (lane == 0) bar_arrive(B.next_full);
    } else if (warp >= 4) {
        const uint32_t q = warp & 3u, j = (warp >> 2) - 1u;
        const uint32_t lanes = tmem + ((32 * q) << 16);
        if (j < 2) {  // builders: K-steps j and j + 2 of every input stage
            uint32_t si = gi0 % IN, pi = (gi0 / IN) & 1u, pa = (gi0 & 1u) ^ 1u, left = sn;
            for (uint32_t k = 0; k < NI; ++k, left -= kInSlices) {
                ok &= warp_wait<POLLS>(B.in_full + 8 * si, pi, P.abort_flag);
                // one word: symbols 2m (low) and 2m+1 of a slice; past the range 0
                const uint32_t a = in0 + kInBBytes + (32 * q + lane) * 4 + si * kInStageBytes;
                uint32_t x[2 * kKSlices];
#pragma unroll
                for (uint32_t s = 0; s < 2 * kKSlices; ++s) {
                    const uint32_t at = (s / kKSlices * 2 + j) * kKSlices + s % kKSlices;
                    x[s] = lds_b32(a + at * kSrcSliceBytes);
                    if (at >= left) x[s] = 0;
                }
// the second K-step is spread while the first is stored
                uint32_t v[16], w[16];
                spread4(x, v);
                ok &= warp_wait<POLLS>(B.a_empty + 8 * 0, pa, P.abort_flag);
                tc_fence_after();
                tmem_st16(lanes + kACol + 16 * j, v);
                spread4(x + kKSlices, w);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) bar_arrive(B.a_full + 8 * 0);
                ok &= warp_wait<POLLS>(B.a_empty + 8 * 1, pa, P.abort_flag);
                tc_fence_after();
                tmem_st16(lanes + kACol + 16 * (j + 2), w);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) bar_arrive(B.a_full + 8 * 1);
                pa ^= 1u;
                if (++si == IN) {
                    si = 0;
                    pi ^= 1u;
                }
            }
        }
        ok &= warp_wait<POLLS>(B.acc_full, tc & 1u, P.abort_flag);
        tc_fence_after();
        const uint32_t m = 2 * (32 * q + lane);  // this lane's symbols m, m+1
        const uint32_t r0 = uni(T.r0), left = uni(T.R) - r0, live = left < rows ? left : rows;
        const uint64_t stride = uni(T.rec_stride);
        const bool accumulate = uni(T.accumulate) != 0, inside = ok && m < T.syms;
        uint8_t* out = T.rec + r0 * stride + (size_t)(n0 + m) * 2;
        // Parity of each count: the counts are integers below 16 * 32768 = 2^19,
        // so in count + 2^23 the mantissa's lowest bit is the count's; it is
        // shifted in from the top (one add and one funnel shift a value, a chain
        // for each of the two symbols).
        auto finish = [&](uint32_t r, const uint32_t (&v)[32]) {
            uint32_t w0 = 0, w1 = 0;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                w0 = __funnelshift_r(w0, __float_as_uint(__uint_as_float(v[i]) + 8388608.0f), 1);
                w1 = __funnelshift_r(w1, __float_as_uint(__uint_as_float(v[16 + i]) + 8388608.0f), 1);
            }
            const uint32_t w = __byte_perm(w0, w1, 0x7632);
            if (inside) {
                uint32_t* p = reinterpret_cast<uint32_t*>(out + r * stride);
                if (accumulate)
                    atomicXor(p, w);
                else
                    *p = w;
            }
        };
        auto load = [&](uint32_t r, uint32_t (&v)[32]) { tmem_ld16x2(lanes + 16 * r, lanes + kAccCol1 + 16 * r, v); };
        uint32_t va[32];
        if constexpr (LOAD_AHEAD) {
            uint32_t vb[32];
            if (j < live) load(j, va);
            for (uint32_t r = j; r < live; r += 6) {
                tmem_ld_wait(va);
                if (r + 3 < live) load(r + 3, vb);
                finish(r, va);
                if (r + 3 < live) {
                    tmem_ld_wait(vb);
                    if (r + 6 < live) load(r + 6, va);
                    finish(r + 3, vb);
                }
            }
        } else {
            for (uint32_t r = j; r < live; r += 3) {
                load(r, va);
                tmem_ld_wait(va);
                finish(r, va);
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) bar_arrive(B.acc_empty);
    }
    const bool bad = __syncthreads_or(!ok) != 0;
    if (bad && issued_end) {
        // another role gave up: the copies the producer issued (this tile's
        // last stages, the next tile's first) land before the stages are
        // reused or the CTA exits
        for (uint32_t q = issued_end > gi0 + IN ? issued_end - IN : gi0; q < issued_end; ++q)
            bar_drain(B.in_full + 8 * (q % IN), (q / IN) & 1u, POLLS);
    }
    P.gi += NI;
    P.pre = bad || !issued_end ? 0u : issued_end - gi0 - NI;
    P.tcount += 1;
    return !bad;
}

}  // namespace mma
}  // namespace p2g
