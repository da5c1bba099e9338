// Multiply-XOR on the tensor cores (tcgen05, block-scaled e2m1 operands).
//
// A stripe's job out[j] = XOR_i c[i][j] * in[i] is a matrix product over
// GF(2): bit t of an output byte is the parity of the number of input bits s
// with bit t of c * x^s set.  The tensor cores count exactly: with operands
// that are 0 or a power of two every product is 0 or 1 and every partial sum an
// integer below 4096 (2304, where the accumulators start, and at most 1791
// counts), so nothing is ever rounded and the parity is a fixed bit of the
// accumulator.
//
//   A  (128 x K)  the input bits of 128 columns, K = 8 bits of each field byte,
//                 in tensor memory (one lane per column)
//   B  (N x K)    the coefficients' 8x8 bit matrices, N = 8 bits of each output
//                 field byte, in shared memory
//   D  (128 x N)  2304 + the counts, in tensor memory
//
// A GF((2^8)^2) symbol counts as two field bytes (a, b) with the 2x2 block
// [[c0, 0x20 c1], [c1, c0 + c1]] of GF(256) constants per coefficient, so
// both fields run the same code.
//
// Why e2m1 (4-bit) operands: a byte's bits become operand elements by masking
// alone.  (w >> 0) & 0x11111111 of a word holds bits 0 and 4 of its four bytes
// as the element 0001 = 0.5, & 0x22222222 bits 1 and 5 as 0010 = 1, and
// & 0x44444444 bits 2 and 6 as 0100 = 2 (bits 3 and 7 shifted down by one); the
// coefficient elements 2, 1, 0.5 bring every product to 1.  That is five
// operations per input word for four operand words, against the XOR
// networks' work per (input, output) pair.
//
// One persistent CTA per SM, 25 warps: a publisher (claims work items), two MMA
// issuers (one for each tile of a block), two builders of B, two epilogue groups of
// four warps (counts -> parities -> bytes -> rows, alternate blocks), two expander
// groups of four warps (staged rows -> A, alternate units; they also write decode's
// present rows through) and four loaders (rows -> shared memory).  A block is 256
// columns, two tiles of 128: a thread holds two neighbouring columns, one of each
// tile, so it reads and writes both at once, and its results stay in its own
// tensor-memory lane.  Rows flow through a ring of staged units, A through a ring
// of units and D through a ring of tiles, so loads, expansion, MMAs and epilogue
// overlap.
//
// What bounds it: no pipe alone.  At 64 inputs and 16 outputs a block takes about
// 2000 cycles, of which the tensor pipe works 56 % (1150 are the least for 18 MMAs),
// the ALU pipe 59 %, shared memory 57 % and the issue slots 62 % (4850
// instructions); the rest is latency between the roles.
// Drains by CUDA events, whole batches with their plan, half encodes and half decodes
// of random losses: GF(256) 64 + 16, 4096-byte rows 276 us for 872 MB of rows
// (346 with one issuer, loads in the expanders and 128 separate columns a tile); 32 +
// 8, 1400-byte rows 231 us for 596 MB (389); tower 32 + 8, 64 KiB rows 258 us
// for 872 MB (319).
//
// Choices, with what the alternatives took.  A lane's two columns neighbours instead
// of 128 apart, and staging of one's own warp instead of the group's in the
// epilogue: 346 -> 286 us (64 + 16).  Loader warps instead of copies issued by the
// expanders: 356 -> 273 us (1400-byte rows).  An issuer per tile, and epilogue groups
// that alternate blocks instead of sharing each: 274 -> 244 us (1400), 286 -> 276
// (64 + 16), 363 -> 331 (32 + 8 of 4096 bytes).  Eight staged units instead of six:
// 244 -> 238 us (1400).  Sleeps between the polls of the roles that are ahead: no
// difference.  Of the first form (377 us for 64 + 16): units of two steps 424, of
// three 404, against four; polls with a time hint 401 against 384 without; A in
// shared memory and the columns on the N side 437 against 401.

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "kernels.cuh"
#include "mxk_device.cuh"

namespace scrs {

namespace {

constexpr int kEpiWarp = 4, kExpWarp = 12, kExpGroups = 2;
constexpr int kLoadWarp = kExpWarp + 4 * kExpGroups;
constexpr int kMma1Warp = kLoadWarp + 4;  // the second tile's issuer; the first tile's is warp 1
constexpr int kMxtThreads = 32 * (kMma1Warp + 1);
constexpr uint32_t kStepCols = 16;                    // tensor-memory columns of a step's A operand (two tiles)
constexpr uint32_t kUnitSteps = 4;                    // K = 64 steps handed over at once (a block's last unit may hold fewer)
constexpr uint32_t kUnitCols = kUnitSteps * kStepCols;
constexpr uint32_t kGroupBytes = 16;                  // output field bytes per pass (N <= 128)
constexpr uint32_t kScaleCol = 496;                   // tensor-memory columns of the unit scale factors
// Each accumulator starts at 2304: a product of constant operands, 64 times
// 6 * 6.  With at most 1791 counts on top the float's exponent stays put and its
// bit 12 is the parity.
constexpr uint32_t kSixes = 0x77777777u;              // eight elements of 6
constexpr uint32_t kBiasCol = 488;                    // tensor-memory columns of the constant A operand
constexpr uint32_t kStages = 8;      // units of rows loaded or in flight
constexpr uint32_t kUnit = 32 * 320 + 32;  // a unit's staged rows (32 of 320 or 16 of 528), their leads
constexpr uint32_t kLeads = kUnit - 32;
constexpr uint32_t kEpiStage = 64 * kGroupBytes + 16;  // an epilogue warp's staging: 64 columns, and a word past them
constexpr uint32_t kAhead = kStages + 6;  // the loads' lead over the last warp's work, in units
constexpr uint32_t kItemSlots = kAhead + 4;
constexpr uint32_t kBiasBytes = 128 * 32;  // the constant B operand
constexpr uint32_t kMaxRows = 256;
constexpr uint32_t kMaxBytes = 223;  // input field bytes of a task: at most 1791 counts
constexpr uint8_t kNoPass = 255;      // no output row (data rows end at 254)
constexpr uint32_t kMaxRing = 16;
constexpr uint32_t kDBars = 4;  // accumulator tiles' barriers: two blocks', one for each epilogue group

// A work item as the roles read it: rows [in + row[i] * in_stride, + len).
struct ItemSlot {
    const uint8_t* in;         // at the item's first column
    uint8_t* out;
    const void* coef;
    uint32_t in_stride, out_stride;
    uint32_t len, rest;        // bytes of the item; and to the end of the rows, up to 16 bytes past the item's
    uint32_t n_in, n_out, ld;
    uint32_t steps, units, passes, per, blocks;
    uint32_t valid, copies;
    uint8_t row[kMaxRows];     // input row numbers (row[0] past the end, where coefficients are zero)
    uint8_t pass[kMaxRows];    // output row of a verbatim copy, or kNoPass
    uint8_t to[kMaxRows];      // output row numbers
};

struct Bars {
    uint64_t raw_full[kStages], raw_empty[kStages];
    uint64_t exp_full[kMaxRing], exp_empty[kMaxRing];
    uint64_t d_full[kDBars], d_empty[kDBars];
    uint64_t b_full[2], b_empty[2];
    uint64_t item_full[kItemSlots], item_empty[kItemSlots];
    uint64_t fin[2];
    uint32_t tmem, abort;
};

struct Head {
    Bars bar;
    uint64_t rows_of[256];  // byte t of entry c, bit s: bit t of c * x^s
    uint8_t mul20[256];     // 0x20 * c
    uint32_t task[32];      // the publisher's descriptor
    ItemSlot item[kItemSlots];
};

// Shared memory after Head: the constant B operand, the B slots, the expanders'
// units, output staging.
struct MxtParams {
    const MxkTask* tasks;
    const uint32_t* item_task;
    uint32_t item_lo, item_end;
    uint32_t* counter;
    int32_t* status;
    uint32_t chunk;             // bytes of a row per item: whole blocks
    uint32_t n_b, b_bytes;      // B slots
    uint32_t d_cols, n_d;       // accumulator tiles: columns each, how many
    uint32_t ring;              // A units, after the accumulators
    uint32_t smem;              // bytes of shared memory
};

__host__ __device__ constexpr uint32_t up(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }

struct Ring {
    uint32_t i = 0, ph = 0;
    __device__ __forceinline__ void next(uint32_t n) {
        if (++i == n) i = 0, ph ^= 1u;
    }
};

// The tensor instructions take their operands from uniform registers.  Where
// the control flow around them, or an operand, could differ between the lanes of
// a warp as far as the compiler can tell, it serves the lanes one by one, about a
// hundred cycles each time.  So the roles' loops run on values made uniform by
// uni() (the same in all lanes), and a wait never branches away: one that runs
// out raises the abort flag, at which every later wait returns at once and the
// roles stop at their next item.
__device__ __forceinline__ uint32_t uni(uint32_t x) { return __reduce_or_sync(0xFFFFFFFFu, x); }

// A poll whose suspension the hardware limits by itself: with the time hint of
// mbar_try_wait the wake-ups came later and a drain took 7 % longer.
__device__ __forceinline__ bool poll(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ void warp_wait(uint64_t* bar, uint32_t parity, Bars* B, int32_t* status) {
    if (!poll(bar, parity)) {
        const uint64_t t0 = global_ns();
        bool done = false;
        while (!done) {
            for (int i = 0; i < 64 && !done; i++) done = poll(bar, parity);
            if (done || *reinterpret_cast<volatile uint32_t*>(&B->abort)) break;
            if (global_ns() - t0 > kWaitLimitNs) {
                *reinterpret_cast<volatile uint32_t*>(&B->abort) = 1u;
                report_status(status, SCRS_ERR_DEVICE_TIMEOUT);
                break;
            }
        }
    }
    __syncwarp();
}
__device__ __forceinline__ bool aborted(const Bars* B) {
    return uni(*reinterpret_cast<const volatile uint32_t*>(&B->abort)) != 0;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Arrival of a whole warp (count 1) after all its lanes' accesses.
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// ---- tcgen05 ------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
// tcgen05.commit and .mma take their operands from uniform registers: issued by
// an elected lane of a converged warp on warp-uniform values they cost a few
// cycles, in a divergent branch about a hundred (the compiler loops over the
// branch's lanes).  The same lane is elected every time.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_addr(bar))
        : "memory");
}
// K-major operand without swizzle: 8-row by 16-byte core matrices, the two of
// a K = 64 step 128 bytes apart, row groups 256 bytes apart.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)(128 >> 4) << 16 | (uint64_t)(256 >> 4) << 32 | 1ull << 46;
}
// e2m1 x e2m1 with ue8m0 scales, M = 128.
__device__ __forceinline__ uint32_t instr_desc(uint32_t n) {
    return 1u << 7 | 1u << 10 | (n >> 3) << 17 | 1u << 23 | 1u << 27;
}
// D (+)= A * B of one K = 64 step, A in tensor memory.
template <bool kAccumulate>
__device__ __forceinline__ void mma_step(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t scale) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xFFFFFFFF;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], [%4], p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(scale), "n"(kAccumulate ? 1 : 0)
        : "memory");
}
// A whole unit's steps, n2 descriptor units of B apart, then the arrival at
// `bar` when they end: one election, and one conversion of the common operands.
__device__ __forceinline__ void mma_unit(uint32_t d, uint32_t a, uint64_t b, uint32_t n2, uint32_t idesc, uint32_t scale,
                                         uint64_t* bar) {
    static_assert(kUnitSteps == 4, "four MMAs below");
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %5, %9, [%10], [%10], 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%2], %6, %9, [%10], [%10], 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%3], %7, %9, [%10], [%10], 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%4], %8, %9, [%10], [%10], 1;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%11];\n\t}" ::"r"(d),
        "r"(a), "r"(a + kStepCols), "r"(a + 2 * kStepCols), "r"(a + 3 * kStepCols), "l"(b), "l"(b + n2), "l"(b + 2 * n2),
        "l"(b + 3 * n2), "r"(idesc), "r"(scale), "r"(smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ void tmem_store8(uint32_t addr, const uint4& a, const uint4& b) {  // this lane's 8 columns
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(a.x),
                 "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}
// Low halves of this lane's 32 columns from addr on, two to a register.
__device__ __forceinline__ void tmem_load_halves(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.pack::16b.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_fill8(uint32_t addr, uint32_t x) {  // this lane's 8 columns from addr on
    tmem_store8(addr, make_uint4(x, x, x, x), make_uint4(x, x, x, x));
}
__device__ __forceinline__ void tmem_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Waits for the loads issued so far; v, their result, is not read before.
__device__ __forceinline__ void tmem_wait_load(uint32_t (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])::"memory");
}

// ---- geometry of an item ----------------------------------------------------------
template <int kGf16>
struct MxtGeom {
    static constexpr uint32_t kElem = kGf16 ? 2 : 1;         // field bytes of a symbol element
    static constexpr uint32_t kRow = 256 * kElem;            // bytes of a row per block
    // and per staged row: with a piece for its lead, and two of a GF(256) unit's
    // rows in different banks
    static constexpr uint32_t kPitch = kRow + (kGf16 ? 16 : 64);
    static constexpr uint32_t kSpan = 64 * kElem;            // of which a warp's lanes hold, two columns each
    static constexpr uint32_t kChunkRows = 4 / kElem;        // input rows of a chunk of 4 field bytes
    static constexpr uint32_t kStepRows = 2 * kChunkRows;    // and of a K = 64 step
    static constexpr uint32_t kGroup = kGroupBytes / kElem;  // output rows per pass
};

// K = 64 steps of n_in input rows: two chunks of 4 field bytes each.
template <int kGf16>
__host__ __device__ __forceinline__ uint32_t steps_of(uint32_t n_in) {
    return (n_in * MxtGeom<kGf16>::kElem + 7) / 8;
}

// MMA columns of cnt output rows: 32 for every 4 field bytes.
template <int kGf16>
__host__ __device__ __forceinline__ uint32_t columns_of(uint32_t cnt) {
    return up(cnt * MxtGeom<kGf16>::kElem, 4) * 8;
}

// The four operand words of one chunk: w holds four field bytes.
__device__ __forceinline__ uint4 spread(uint32_t w) {
    return make_uint4(w & 0x11111111u, w & 0x22222222u, w & 0x44444444u, (w >> 1) & 0x44444444u);
}

// Four output field bytes of this lane's column: z[n / 2] holds the low half of
// accumulator column n in half n & 1, the parity at its bit 12; column 4 t + j
// is bit t of byte j.
__device__ __forceinline__ uint32_t parity_word(const uint32_t (&z)[16]) {
    uint32_t y[8];
#pragma unroll
    for (int t = 0; t < 8; t++) y[t] = __byte_perm(z[2 * t], z[2 * t + 1], 0x7531);  // byte j: the parity at bit 4
    auto pick = [](uint32_t m, uint32_t a, uint32_t b) { return (a & m) | (b & ~m); };
    auto nibble = [&](const uint32_t* v) {  // v[t]'s bit 4 at bit 4 + t
        const uint32_t lo = pick(0x10101010u, v[0], v[1] << 1), hi = pick(0x40404040u, v[2] << 2, v[3] << 3);
        return pick(0x30303030u, lo, hi);
    };
    return pick(0xF0F0F0F0u, nibble(y + 4), nibble(y) >> 4);
}

// Asynchronous copy of 16 or 8 bytes into shared memory where `on`.
template <int kBytes>
__device__ __forceinline__ void copy_in(uint32_t dst, const void* src, bool on) {
    if constexpr (kBytes == 16)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(dst),
            "l"(src), "r"((uint32_t)on)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p cp.async.ca.shared.global [%0], [%1], 8;\n\t}" ::"r"(dst),
            "l"(src), "r"((uint32_t)on)
            : "memory");
}
// This thread's arrival as the copies that it has issued land.
__device__ __forceinline__ void copy_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void copy_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- the kernel ----------------------------------------------------------------
// kAlign (16, 8 or 1): every row, in and out, starts at a multiple of it and L is
// one.  Rows move in pieces of 16 or 8 bytes; of rows at any byte, the 16-byte
// pieces around them are fetched, which never leaves the 16-byte units that hold
// the row.
template <int kGf16, int kAlign>
__global__ void __launch_bounds__(kMxtThreads, 1) mxt_kernel(const __grid_constant__ MxtParams P) {
    using G = MxtGeom<kGf16>;
    constexpr bool kAligned = kAlign > 1;
    constexpr uint32_t kPiece = kAligned ? kAlign : 16;
    using Piece = typename std::conditional<kPiece == 8, uint2, uint4>::type;
    extern __shared__ __align__(128) uint8_t smem[];
    Head& H = *reinterpret_cast<Head*>(smem);
    Bars* B = &H.bar;
    uint8_t* s_bias = smem + up(sizeof(Head), 128);
    uint8_t* s_b = s_bias + kBiasBytes;
    uint8_t* s_raw = s_b + P.n_b * P.b_bytes;
    uint8_t* s_stg = s_raw + kStages * kUnit;
    const int tid = threadIdx.x, lane = tid & 31, warp = (int)uni(tid >> 5);

    // ---- set-up: barriers, tables, tensor memory
    if (tid == 0) {
        for (uint32_t i = 0; i < kMaxRing; i++) mbar_init(&B->exp_full[i], 4), mbar_init(&B->exp_empty[i], 2);
        for (uint32_t i = 0; i < kDBars; i++) mbar_init(&B->d_full[i], 1), mbar_init(&B->d_empty[i], 4);
        // a loader thread's arrival as its copies land; a loader warp's for the leads
        for (uint32_t i = 0; i < kStages; i++)
            mbar_init(&B->raw_full[i], kAligned ? 128 : 132), mbar_init(&B->raw_empty[i], 4);
        for (int i = 0; i < 2; i++) mbar_init(&B->b_full[i], 2), mbar_init(&B->b_empty[i], 2);
        // consumers: 2 MMA issuers, 2 builders, 8 epilogue warps, the expanders, 4 loaders
        for (uint32_t i = 0; i < kItemSlots; i++)
            mbar_init(&B->item_full[i], 1), mbar_init(&B->item_empty[i], 16 + 4 * kExpGroups);
        mbar_init(&B->fin[0], 1), mbar_init(&B->fin[1], 1);
        B->abort = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&B->tmem)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid >= 256 && tid < 512) {
        const int c = tid - 256;
        uint64_t rows = 0;
        uint32_t v = (uint32_t)c;
        for (int s = 0; s < 8; s++) {
            if (s == 5) H.mul20[c] = (uint8_t)v;
            for (int t = 0; t < 8; t++) rows |= (uint64_t)((v >> t) & 1u) << (8 * t + s);
            v = (v << 1) ^ ((v & 0x80u) ? 0x11Bu : 0u);
        }
        H.rows_of[c] = rows;
        reinterpret_cast<uint4*>(s_bias)[c] = make_uint4(kSixes, kSixes, kSixes, kSixes);
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uni(*reinterpret_cast<volatile uint32_t*>(&B->tmem));
    const uint32_t a_col = P.n_d * P.d_cols;  // the A ring
    if (warp >= kEpiWarp && warp < kEpiWarp + 4) {  // in all lanes: unit scale factors, the constant operand
        const uint32_t at = tmem + ((uint32_t)(warp & 3) << 21);
        tmem_fill8(at + kScaleCol, 0x7F7F7F7Fu);
        tmem_fill8(at + kScaleCol + 8, 0x7F7F7F7Fu);
        tmem_fill8(at + kBiasCol, kSixes);
        tmem_wait_store();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();

    Ring it;
    if (warp == 0) {
        // ---- publisher: claims items and lays their descriptors out
        uint32_t* task = H.task;
        auto claim = [&]() -> uint32_t {
            uint32_t v = 0;
            if (lane == 0) v = atomicAdd(P.counter, 1u);
            return P.item_lo + __shfl_sync(0xFFFFFFFFu, v, 0);
        };
        // An item is claimed while fewer than kAhead units are published after
        // the oldest one not yet released: the loads need that many ahead of the
        // last warp's work, and more would take items that another SM could start
        // sooner.
        Ring tail;
        uint32_t held = 0, after = 0;  // items not released; units of all but the oldest
        auto units_in = [&](const Ring& r) { return H.item[r.i].units * H.item[r.i].blocks * H.item[r.i].passes; };
        for (;;) {
            while (after >= kAhead) {
                warp_wait(&B->item_empty[tail.i], tail.ph, B, P.status);
                tail.next(kItemSlots);
                after -= units_in(tail);
                held--;
            }
            const uint32_t cur = uni(claim());
            const bool valid = cur < P.item_end && !aborted(B);  // an abort ends the items
            uint32_t word = 0;
            if (valid && lane < (int)kTaskWords)
                word = reinterpret_cast<const uint32_t*>(P.tasks + __ldg(P.item_task + cur))[lane];
            ItemSlot& I = H.item[it.i];  // free: at most kAhead + 2 items are held
            if (valid) {
                if (lane < (int)kTaskWords) task[lane] = word;
                __syncwarp();
                const MxkTask& T = *reinterpret_cast<const MxkTask*>(task);
                const uint32_t steps = steps_of<kGf16>(T.n_in);
                for (uint32_t i = lane; i < steps * G::kStepRows; i += 32) {
                    const bool real = i < T.n_in;
                    const uint32_t z = real ? i : 0u;
                    I.row[i] = (uint8_t)(T.in_rows ? T.in_rows[z] : z);
                    I.pass[i] = real && T.pass_rows ? (uint8_t)T.pass_rows[i] : kNoPass;  // kNoRow too
                }
                for (uint32_t i = lane; i < T.n_out; i += 32) I.to[i] = (uint8_t)(T.out_rows ? T.out_rows[i] : i);
                if (lane == 0) {
                    const uint64_t off = (uint64_t)(cur - T.item_begin) * P.chunk;
                    I.in = T.in + off;
                    I.out = T.out + off;
                    I.coef = T.coef;
                    I.in_stride = (uint32_t)T.in_stride;
                    I.out_stride = (uint32_t)T.out_stride;
                    const uint64_t rest = T.L - off;
                    I.rest = (uint32_t)(rest < P.chunk + 16 ? rest : P.chunk + 16);
                    I.len = umin32(I.rest, P.chunk);
                    I.n_in = T.n_in, I.n_out = T.n_out, I.ld = T.ld;
                    I.steps = steps;
                    I.units = (steps + kUnitSteps - 1) / kUnitSteps;
                    I.passes = (T.n_out + G::kGroup - 1) / G::kGroup;
                    I.per = (T.n_out + I.passes - 1) / I.passes;
                    I.blocks = (I.len + G::kRow - 1) / G::kRow;
                    I.copies = T.pass_rows != nullptr;
                }
                __syncwarp();  // task is rewritten for the next item
            }
            if (lane == 0) I.valid = valid;
            __syncwarp();
            if (valid && held++) after += units_in(it);
            warp_arrive(&B->item_full[it.i], lane);
            if (!valid) break;
            it.next(kItemSlots);
        }
        pdl_wait();  // this launch does not end before the one it started beside
    } else if (warp == 1 || warp == kMma1Warp) {
        // ---- MMA issuers, one for each tile of a block
        const uint32_t tile = warp == 1 ? 0u : 1u;
        // ds: this tile's barriers; es: those of the tile that last held its
        // accumulator, n_d tiles before
        Ring bs, ds, es, as;
        ds.i = tile, es.i = tile + kDBars - P.n_d;
        const uint64_t bias = operand_desc(smem_addr(s_bias));
        for (;;) {
            warp_wait(&B->item_full[it.i], it.ph, B, P.status);
            const ItemSlot& I = H.item[it.i];
            if (!uni(I.valid) || aborted(B)) break;
            const uint32_t passes = uni(I.passes), blocks = uni(I.blocks), steps = uni(I.steps), per = uni(I.per),
                           n_out = uni(I.n_out);
            for (uint32_t pass = 0; pass < passes; pass++) {
                const uint32_t N = columns_of<kGf16>(umin32(per, n_out - pass * per));
                const uint32_t idesc = instr_desc(N), N2 = N * 2;  // N * 32 bytes of B a step
                warp_wait(&B->b_full[bs.i], bs.ph, B, P.status);
                const uint64_t b0 = operand_desc(smem_addr(s_b + bs.i * P.b_bytes));
                for (uint32_t b = 0; b < blocks; b++) {
                    warp_wait(&B->d_empty[es.i], es.ph ^ 1u, B, P.status);
                    const uint32_t d = tmem + (ds.i & (P.n_d - 1)) * P.d_cols;
                    tc_fence_after();
                    mma_step<false>(d, tmem + kBiasCol, bias, idesc, tmem + kScaleCol);
                    uint64_t bd = b0;
                    for (uint32_t left = steps; left;) {
                        warp_wait(&B->exp_full[as.i], as.ph, B, P.status);
                        tc_fence_after();
                        const uint32_t a = tmem + a_col + as.i * kUnitCols + tile * (kStepCols / 2);
                        if (left >= kUnitSteps) {
                            mma_unit(d, a, bd, N2, idesc, tmem + kScaleCol, &B->exp_empty[as.i]);
                            left -= kUnitSteps;
                        } else {
#pragma unroll
                            for (uint32_t h = 0; h < kUnitSteps - 1; h++)
                                if (h < left) mma_step<true>(d, a + h * kStepCols, bd + h * N2, idesc, tmem + kScaleCol);
                            tc_commit(&B->exp_empty[as.i]);
                            left = 0;
                        }
                        bd += kUnitSteps * N2;
                        as.next(P.ring);
                    }
                    tc_commit(&B->d_full[ds.i]);
                    ds.next(kDBars), ds.next(kDBars);
                    es.next(kDBars), es.next(kDBars);
                }
                tc_commit(&B->b_empty[bs.i]);
                bs.next(P.n_b);
            }
            warp_arrive(&B->item_empty[it.i], lane);
            it.next(kItemSlots);
        }
        // the MMAs in flight end before tensor and shared memory are given up
        tc_commit(&B->fin[tile]);
        __syncwarp();
        const uint64_t t0 = global_ns();
        while (!mbar_try_wait(&B->fin[tile], 0) && global_ns() - t0 < 100000000ull) {
        }
    } else if (warp < kEpiWarp) {
        // ---- builders of the coefficient operand
        const uint32_t first = (uint32_t)(warp - 2) * 32 + lane;
        Ring bs;
        bool planned = false;
        for (;;) {
            warp_wait(&B->item_full[it.i], it.ph, B, P.status);
            const ItemSlot& I = H.item[it.i];
            if (!uni(I.valid) || aborted(B)) break;
            const uint32_t n_in = I.n_in, ld = I.ld, passes = uni(I.passes);
            if (!planned && uni(I.copies)) {  // a decode's coefficients: the plans before this launch
                pdl_wait();
                planned = true;
            }
            const void* coef = I.coef;
            for (uint32_t pass = 0; pass < passes; pass++) {
                warp_wait(&B->b_empty[bs.i], bs.ph ^ 1u, B, P.status);
                uint8_t* dst = s_b + bs.i * P.b_bytes;
                const uint32_t lo = pass * I.per, cnt = umin32(I.per, I.n_out - lo);
                const uint32_t groups = cnt * G::kElem, total = groups * I.steps * 2;
                const uint32_t step_bytes = columns_of<kGf16>(cnt) * 32;
                // coefficients of chunk c for output field byte j: four GF(256)
                // bytes, or the two GF((2^8)^2) symbols' 16 bits each
                auto fetch = [&](uint32_t idx) -> uint32_t {
                    if (idx >= total) return 0u;
                    const uint32_t c = idx / groups, j = (idx - c * groups) / G::kElem;
                    uint32_t v = 0;
#pragma unroll
                    for (uint32_t q = 0; q < G::kChunkRows; q++) {
                        const uint32_t i = c * G::kChunkRows + q;
                        if (i < n_in) {
                            const size_t at = (size_t)i * ld + lo + j;
                            if (kGf16)
                                v |= (uint32_t) reinterpret_cast<const uint16_t*>(coef)[at] << (16 * q);
                            else
                                v |= (uint32_t) reinterpret_cast<const uint8_t*>(coef)[at] << (8 * q);
                        }
                    }
                    return v;
                };
                uint32_t v = fetch(first);
                for (uint32_t idx = first; idx < total; idx += 64) {
                    const uint32_t nv = fetch(idx + 64);
                    const uint32_t c = idx / groups, g = idx - c * groups;
                    uint32_t k[4];
                    if (kGf16) {
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const uint32_t c0 = (v >> (16 * q)) & 0xFFu, c1 = (v >> (16 * q + 8)) & 0xFFu;
                            k[2 * q] = (g & 1u) ? c1 : c0;
                            k[2 * q + 1] = (g & 1u) ? (c0 ^ c1) : H.mul20[c1];
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; q++) k[q] = (v >> (8 * q)) & 0xFFu;
                    }
                    uint32_t rl[4], rh[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const uint64_t r = H.rows_of[k[q]];
                        rl[q] = (uint32_t)r, rh[q] = (uint32_t)(r >> 32);
                    }
                    // bit t of field byte g is row 32 (g / 4) + 4 t + g % 4
                    uint8_t* core = dst + (c >> 1) * step_bytes + (g >> 2) * 1024 + (g & 3u) * 16 + (c & 1u) * 128;
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        const uint32_t t = (u + (lane >> 2)) & 7u;  // eight neighbouring lanes, eight bank groups
                        const uint32_t p01 = __byte_perm(__byte_perm(rl[0], rh[0], t), __byte_perm(rl[1], rh[1], t), 0x0040);
                        const uint32_t p23 = __byte_perm(__byte_perm(rl[2], rh[2], t), __byte_perm(rl[3], rh[3], t), 0x0040);
                        const uint32_t p = __byte_perm(p01, p23, 0x5410);
                        const uint32_t w0 = p & 0x11111111u, w1 = (p >> 1) & 0x11111111u;
                        const uint32_t w2 = (p >> 2) & 0x11111111u, w3 = (p >> 3) & 0x11111111u;
                        // elements 2, 1, 0.5, 0.5
                        *reinterpret_cast<uint4*>(core + (t >> 1) * 256 + (t & 1u) * 64) = make_uint4(w0 << 2, w1 << 1, w2, w3);
                    }
                    v = nv;
                }
                fence_proxy_async_smem();
                warp_arrive(&B->b_full[bs.i], lane);
                bs.next(P.n_b);
            }
            warp_arrive(&B->item_empty[it.i], lane);
            it.next(kItemSlots);
        }
    } else if (warp < kExpWarp) {
        // ---- epilogue: counts -> parities -> bytes -> rows
        const uint32_t e = (uint32_t)warp & 3u, group = (uint32_t)(warp - kEpiWarp) >> 2;  // lane quarter; blocks
        const uint32_t acc = tmem + (e << 21);
        uint8_t* stg = s_stg + (uint32_t)(warp - kEpiWarp) * kEpiStage;
        Ring ds;
        uint32_t turn = 0;  // the groups take alternate blocks
        for (;;) {
            warp_wait(&B->item_full[it.i], it.ph, B, P.status);
            const ItemSlot& I = H.item[it.i];
            if (!uni(I.valid) || aborted(B)) break;
            const uint32_t len = uni(I.len), blocks = uni(I.blocks), passes = uni(I.passes), per = uni(I.per),
                           n_out = uni(I.n_out);
            uint8_t* const out = I.out;
            const uint64_t stride = I.out_stride;
            for (uint32_t pass = 0; pass < passes; pass++) {
                const uint32_t cnt = umin32(per, n_out - pass * per);
                const uint32_t words = columns_of<kGf16>(cnt) / 32;  // of 4 field bytes
                const uint8_t* to = I.to + pass * per;
                for (uint32_t b = 0; b < blocks; b++) {
                    const bool mine = turn == group;
                    turn ^= 1u;
                    if (!mine) {
                        ds.next(kDBars), ds.next(kDBars);
                        continue;
                    }
                    uint32_t w[4][2];  // [word][tile]
#pragma unroll
                    for (uint32_t tile = 0; tile < 2; tile++) {
                        warp_wait(&B->d_full[ds.i], ds.ph, B, P.status);
                        tc_fence_after();
                        const uint32_t d = acc + (ds.i & (P.n_d - 1)) * P.d_cols;
#pragma unroll
                        for (uint32_t q = 0; q < 4; q += 2) {  // two words' loads in flight
                            if (q >= words) break;
                            uint32_t z[2][16];
                            tmem_load_halves(d + 32 * q, z[0]);
                            if (q + 1 < words) tmem_load_halves(d + 32 * (q + 1), z[1]);
                            tmem_wait_load(z[0]);
                            tmem_wait_load(z[1]);
                            if (q + 2 >= words) {  // the tile has been read
                                tc_fence_before();
                                warp_arrive(&B->d_empty[ds.i], lane);
                            }
                            w[q][tile] = parity_word(z[0]);
                            w[q + 1][tile] = parity_word(z[1]);
                        }
                        ds.next(kDBars);
                    }
                    const uint32_t at = b * G::kRow + e * G::kSpan;
                    const uint32_t n = len > at ? umin32(G::kSpan, len - at) : 0u;  // the row's bytes of these columns
                    if (!n) continue;
                    __syncwarp();  // the last block's stores have read the staging rows
#pragma unroll
                    for (uint32_t j = 0; j < G::kGroup; j++) {
                        if (j >= cnt) break;
                        constexpr uint32_t kWordRows = 4 / G::kElem;  // output rows of a word
                        const uint32_t* v = w[j / kWordRows];
                        const uint32_t y = j % kWordRows;
                        if (kGf16)
                            *reinterpret_cast<uint32_t*>(stg + j * G::kSpan + 4 * lane) = __byte_perm(v[0], v[1], y ? 0x7632 : 0x5410);
                        else
                            *reinterpret_cast<uint16_t*>(stg + j * G::kSpan + 2 * lane) =
                                (uint16_t)__byte_perm(v[0], v[1], 0x0040 + 0x0011 * y);
                    }
                    __syncwarp();
                    if (kAligned) {
                        constexpr uint32_t kPieces = G::kSpan / kPiece, kMoves = G::kGroup * kPieces / 32;
                        // Both 16-byte pieces of a lane are read ahead of the stores (tower 32 + 8
                        // decodes 180 us, 183 one by one), not four of 8 bytes (1400-byte rows 233 and 228).
                        constexpr uint32_t kAtOnce = kPiece == 16 ? kMoves : 1;
#pragma unroll
                        for (uint32_t x0 = 0; x0 < kMoves; x0 += kAtOnce) {
                            Piece v[kAtOnce];
                            uint32_t row[kAtOnce];
#pragma unroll
                            for (uint32_t x = 0; x < kAtOnce; x++) {
                                const uint32_t q = 32 * (x0 + x) + lane, j = q / kPieces, o = kPiece * (q % kPieces);
                                v[x] = *reinterpret_cast<const Piece*>(stg + j * G::kSpan + o);
                                row[x] = j < cnt ? to[j] : 0;
                            }
#pragma unroll
                            for (uint32_t x = 0; x < kAtOnce; x++) {
                                const uint32_t q = 32 * (x0 + x) + lane, j = q / kPieces, o = kPiece * (q % kPieces);
                                if (j < cnt && o < n) *reinterpret_cast<Piece*>(out + row[x] * stride + at + o) = v[x];
                            }
                        }
                    } else {
                        // bytes up to the first whole word of a row, words, the rest
                        auto put = [&](uint32_t j, uint32_t o) {
                            out[to[j] * stride + at + o] = stg[j * G::kSpan + o];
                        };
                        auto head_of = [&](uint32_t j) {
                            return umin32((uint32_t)(-reinterpret_cast<intptr_t>(out + to[j] * stride + at)) & 3u, n);
                        };
                        for (uint32_t j = (uint32_t)lane / 4; j < cnt; j += 8) {
                            const uint32_t head = head_of(j), tail = head + ((n - head) & ~3u), y = (uint32_t)lane & 3u;
                            if (y < head) put(j, y);
                            if (y < n - tail) put(j, tail + y);
                        }
                        constexpr uint32_t kWords = G::kSpan / 4;
                        for (uint32_t x = lane; x < cnt * kWords; x += 32) {
                            const uint32_t j = x / kWords, head = head_of(j), o = head + 4 * (x % kWords);
                            if (o + 4 > n) continue;
                            const uint32_t* s = reinterpret_cast<const uint32_t*>(stg + j * G::kSpan + (o & ~3u));
                            const uint32_t v = head ? __funnelshift_r(s[0], s[1], 8 * head) : s[0];
                            *reinterpret_cast<uint32_t*>(out + to[j] * stride + at + o) = v;
                        }
                    }
                }
            }
            warp_arrive(&B->item_empty[it.i], lane);
            it.next(kItemSlots);
        }
    } else if (warp >= kLoadWarp) {
        // ---- loaders: rows -> the staging units
        const uint32_t t = (uint32_t)(warp - kLoadWarp) * 32 + lane;
        constexpr uint32_t kPieces = G::kRow / kPiece + (kAligned ? 0 : 1);  // of a row
        constexpr uint32_t kLoads = (kUnitSteps * G::kStepRows * kPieces + 127) / 128;
        Ring rs;
        for (;;) {
            warp_wait(&B->item_full[it.i], it.ph, B, P.status);
            const ItemSlot& I = H.item[it.i];
            if (!uni(I.valid) || aborted(B)) break;
            const uint32_t len = uni(I.len), passes = uni(I.passes), rows = uni(I.steps) * G::kStepRows;
            const uint32_t end = kAligned ? len : uni(I.rest);
            const uint64_t stride = I.in_stride;
            for (uint32_t pass = 0; pass < passes; pass++)
                for (uint32_t col = 0; col < len; col += G::kRow)
                    for (uint32_t row0 = 0; row0 < rows; row0 += kUnitSteps * G::kStepRows) {
                        const uint8_t* base = I.in + col;
                        const uint32_t left = umin32(kUnitSteps * G::kStepRows, rows - row0);
                        uint32_t row[kLoads];  // read ahead of the copies
#pragma unroll
                        for (uint32_t x = 0; x < kLoads; x++)
                            row[x] = I.row[row0 + umin32((128 * x + t) / kPieces, kUnitSteps * G::kStepRows - 1)];
                        warp_wait(&B->raw_empty[rs.i], rs.ph ^ 1u, B, P.status);
                        uint8_t* stage = s_raw + rs.i * kUnit;
#pragma unroll
                        for (uint32_t x = 0; x < kLoads; x++) {
                            const uint32_t q = (128 * x + t) / kPieces, o = kPiece * ((128 * x + t) % kPieces);
                            const uint8_t* p = base + row[x] * stride;
                            uint32_t lead = 0;
                            if (!kAligned) {
                                lead = (uint32_t) reinterpret_cast<uintptr_t>(p) & 15u;
                                if (q < left && o == 0) stage[kLeads + q] = (uint8_t)lead;
                            }
                            copy_in<(int)kPiece>(smem_addr(stage) + q * G::kPitch + o, p - lead + o,
                                                 q < left && col + o < end + lead);
                        }
                        copy_arrive(&B->raw_full[rs.i]);
                        if (!kAligned) warp_arrive(&B->raw_full[rs.i], lane);
                        rs.next(kStages);
                    }
            warp_arrive(&B->item_empty[it.i], lane);
            it.next(kItemSlots);
        }
        copy_wait_all();
    } else {
        // ---- expanders: rows -> the A operand
        const uint32_t e = (uint32_t)warp & 3u, group = (uint32_t)(warp - kExpWarp) >> 2;
        constexpr uint32_t kPitch = G::kPitch;
        // this warp's units, every kExpGroups-th one
        uint32_t unit = group, col = 0, pass = 0;  // col: bytes from the item's first column
        uint32_t n_steps, n_units, len, passes;
        bool open, with_copies;
        auto open_item = [&]() {  // the ring's next item, if there is one
            warp_wait(&B->item_full[it.i], it.ph, B, P.status);
            const ItemSlot& I = H.item[it.i];
            open = uni(I.valid) && !aborted(B);
            n_steps = uni(I.steps), n_units = uni(I.units), len = uni(I.len), passes = uni(I.passes);
            with_copies = uni(I.copies) != 0;
            col = pass = 0;
        };
        auto settle = [&]() {  // carries the unit into blocks, passes, items
            while (open && unit >= n_units) {
                unit -= n_units;
                col += G::kRow;
                if (col < len) continue;
                col = 0;
                if (++pass < passes) continue;
                warp_arrive(&B->item_empty[it.i], lane);
                it.next(kItemSlots);
                open_item();
            }
        };
        // operand bytes of a staged step: w[2 * tile + chunk], this lane's columns
        auto read_step = [&](const uint8_t* stage, const uint8_t* leads, uint32_t (&w)[4]) {
            uint32_t x[G::kStepRows];  // both columns' elements of each row
#pragma unroll
            for (uint32_t q = 0; q < G::kStepRows; q++) {
                const uint32_t lead = kAligned ? 0u : leads[q];
                const uint8_t* p = stage + q * kPitch + lead + e * G::kSpan + 2 * G::kElem * lane;
                if (kGf16) {
                    const uint32_t* a = reinterpret_cast<const uint32_t*>(p - (lead & 3u));
                    x[q] = kAligned ? a[0] : __funnelshift_r(a[0], a[1], 8 * (lead & 3u));
                } else {
                    x[q] = kAligned ? (uint32_t) *reinterpret_cast<const uint16_t*>(p) : p[0] | (uint32_t)p[1] << 8;
                }
            }
#pragma unroll
            for (int z = 0; z < 2; z++) {
                if (kGf16) {
                    w[z] = __byte_perm(x[2 * z], x[2 * z + 1], 0x5410);
                    w[2 + z] = __byte_perm(x[2 * z], x[2 * z + 1], 0x7632);
                } else {
                    const int q = (4 * z) % (int)G::kStepRows;
                    const uint32_t a = __byte_perm(x[q], x[q + 1], 0x5140);
                    const uint32_t b = __byte_perm(x[(q + 2) % G::kStepRows], x[(q + 3) % G::kStepRows], 0x5140);
                    w[z] = __byte_perm(a, b, 0x5410);
                    w[2 + z] = __byte_perm(a, b, 0x7632);
                }
            }
        };
        auto write_step = [&](uint32_t dst, const uint32_t (&w)[4]) {
            tmem_store8(dst, spread(w[0]), spread(w[1]));
            tmem_store8(dst + kStepCols / 2, spread(w[2]), spread(w[3]));
        };
        auto next_slot = [](uint32_t& i, uint32_t& ph, uint32_t n) {
            i += kExpGroups;
            if (i >= n) i -= n, ph ^= 1u;
        };
        uint32_t slot = group, slot_ph = 0;  // A slot of this warp's next unit
        uint32_t raw = group, raw_ph = 0;    // and its staged rows
        open_item();
        settle();
        while (open) {
            const ItemSlot& I = H.item[it.i];
            const uint32_t dst0 = tmem + (e << 21) + a_col + slot * kUnitCols;
            const bool copies = with_copies && pass == 0;  // decode's present rows go straight through
            const uint32_t step0 = kUnitSteps * unit, steps = umin32(kUnitSteps, n_steps - step0);
            const uint8_t *stage0 = s_raw + raw * kUnit, *leads = stage0 + kLeads;
            constexpr uint32_t kStep = G::kStepRows * kPitch;
            warp_wait(&B->raw_full[raw], raw_ph, B, P.status);
            if (steps == kUnitSteps) {  // read before the slot is free
                uint32_t w[kUnitSteps][4];
#pragma unroll
                for (uint32_t h = 0; h < kUnitSteps; h++) read_step(stage0 + h * kStep, leads + h * G::kStepRows, w[h]);
                warp_wait(&B->exp_empty[slot], slot_ph ^ 1u, B, P.status);
                tc_fence_after();
#pragma unroll
                for (uint32_t h = 0; h < kUnitSteps; h++) write_step(dst0 + h * kStepCols, w[h]);
            } else {
                warp_wait(&B->exp_empty[slot], slot_ph ^ 1u, B, P.status);
                tc_fence_after();
#pragma unroll 1
                for (uint32_t h = 0; h < steps; h++) {
                    uint32_t w[4];
                    read_step(stage0 + h * kStep, leads + h * G::kStepRows, w);
                    write_step(dst0 + h * kStepCols, w);
                }
            }
            tmem_wait_store();
            tc_fence_before();
            if (copies) __syncwarp();
            else warp_arrive(&B->raw_empty[raw], lane);
            warp_arrive(&B->exp_full[slot], lane);
            next_slot(slot, slot_ph, P.ring);
            if (copies) {
                const uint32_t first = col + e * G::kSpan;
                uint8_t* const out = I.out + first;
                const uint64_t stride = I.out_stride;
                // pieces of aligned rows, words of the others
                constexpr uint32_t kBy = kAligned ? kPiece : 4, kPer = G::kSpan / kBy, kMoves = G::kStepRows * kPer / 32;
                if constexpr (kAligned) {
                    uint32_t to[kUnitSteps][kMoves];  // read ahead of the stores
                    Piece v[kUnitSteps][kMoves];
#pragma unroll
                    for (uint32_t h = 0; h < kUnitSteps; h++)
#pragma unroll
                        for (uint32_t x = 0; x < kMoves; x++) {
                            const uint32_t q = (32 * x + lane) / kPer, o = kBy * ((32 * x + lane) % kPer);
                            to[h][x] = I.pass[(step0 + h) * G::kStepRows + q];
                            v[h][x] = *reinterpret_cast<const Piece*>(stage0 + h * kStep + q * kPitch + e * G::kSpan + o);
                        }
#pragma unroll
                    for (uint32_t h = 0; h < kUnitSteps; h++)
#pragma unroll
                        for (uint32_t x = 0; x < kMoves; x++) {
                            const uint32_t o = kBy * ((32 * x + lane) % kPer);
                            if (h < steps && to[h][x] != kNoPass && first + o < len)
                                *reinterpret_cast<Piece*>(out + to[h][x] * stride + o) = v[h][x];
                        }
                } else {
#pragma unroll 1
                    for (uint32_t h = 0; h < steps; h++) {
                        const uint8_t* stage = stage0 + h * kStep + e * G::kSpan;
#pragma unroll
                        for (uint32_t x = 0; x < kMoves; x++) {
                            const uint32_t q = (32 * x + lane) / kPer, o = kBy * ((32 * x + lane) % kPer), at = first + o;
                            const uint32_t to = I.pass[(step0 + h) * G::kStepRows + q];
                            if (to == kNoPass || at >= len) continue;
                            uint8_t* p = out + to * stride + o;
                            const uint32_t lead = leads[h * G::kStepRows + q];
                            const uint32_t* a = reinterpret_cast<const uint32_t*>(stage + q * kPitch + o + (lead & ~3u));
                            const uint32_t v = __funnelshift_r(a[0], a[1], 8 * (lead & 3u));
                            if ((reinterpret_cast<uintptr_t>(p) & 3u) == 0 && at + 4 <= len) {
                                *reinterpret_cast<uint32_t*>(p) = v;
                            } else {
#pragma unroll
                                for (uint32_t y = 0; y < 4; y++)
                                    if (at + y < len) p[y] = (uint8_t)(v >> (8 * y));
                            }
                        }
                    }
                }
                warp_arrive(&B->raw_empty[raw], lane);
            }
            next_slot(raw, raw_ph, kStages);
            unit += kExpGroups;
            settle();
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

constexpr size_t kMxtSmem = 227 * 1024;

// Shared- and tensor-memory split for the largest task of a launch; false when
// it does not fit.
template <int kGf16>
bool mxt_layout(uint32_t max_in, uint32_t max_out, MxtParams* P) {
    using G = MxtGeom<kGf16>;
    if (max_in == 0 || max_in * G::kElem > kMaxBytes || max_out == 0 || max_out > kMaxRows) return false;
    P->d_cols = columns_of<kGf16>(std::min<uint32_t>(max_out, G::kGroup));
    P->n_d = P->d_cols > 64 ? 2 : 4;  // one or two blocks' tiles; the rest is the A ring, three units or more
    P->ring = std::min<uint32_t>(kMaxRing, (kBiasCol - P->n_d * P->d_cols) / kUnitCols);
    P->b_bytes = steps_of<kGf16>(max_in) * P->d_cols * 32;
    const size_t fixed = up(sizeof(Head), 128) + kBiasBytes + kStages * kUnit + 8 * kEpiStage;
    for (P->n_b = 2; P->n_b >= 1; P->n_b--)
        if (const size_t bytes = fixed + (size_t)P->n_b * P->b_bytes; bytes <= kMxtSmem) {
            P->smem = (uint32_t)bytes;
            return true;
        }
    return false;
}

using MxtFn = void (*)(const MxtParams);
constexpr MxtFn kMxt[2][3] = {{mxt_kernel<0, 1>, mxt_kernel<0, 8>, mxt_kernel<0, 16>},
                              {mxt_kernel<1, 1>, mxt_kernel<1, 8>, mxt_kernel<1, 16>}};

cudaError_t set_mxt_attrs() {
    static std::atomic<uint64_t> done{0};
    return once_per_device(done, [] {
        cudaError_t e = cudaSuccess;
        for (auto& row : kMxt)
            for (auto fn : row)
                if (e == cudaSuccess)
                    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMxtSmem);
        return e;
    });
}

bool layout_for(int gf16, uint32_t max_in, uint32_t max_out, MxtParams* P) {
    return gf16 ? mxt_layout<1>(max_in, max_out, P) : mxt_layout<0>(max_in, max_out, P);
}

}  // namespace

bool mxt_fits(int gf16, uint32_t max_in, uint32_t max_out) {
    MxtParams P{};
    return layout_for(gf16, max_in, max_out, &P);
}

uint32_t mxt_block(int gf16) { return gf16 ? MxtGeom<1>::kRow : MxtGeom<0>::kRow; }

cudaError_t prepare_mxt() { return set_mxt_attrs(); }

cudaError_t launch_mxt(const MxkTask* tasks, const uint32_t* item_task, uint32_t item_lo, uint32_t item_end,
                       uint32_t* counter, int32_t* status, uint32_t max_in, uint32_t max_out, uint32_t chunk, int grid,
                       cudaStream_t stream, int align, int gf16, bool after_plans) {
    if (item_end <= item_lo) return cudaSuccess;
    MxtParams P{};
    if (!layout_for(gf16, max_in, max_out, &P) || chunk == 0 || chunk % mxt_block(gf16)) return cudaErrorInvalidValue;
    cudaError_t e = set_mxt_attrs();
    if (e != cudaSuccess) return e;
    P.tasks = tasks;
    P.item_task = item_task;
    P.item_lo = item_lo;
    P.item_end = item_end;
    P.counter = counter;
    P.status = status;
    P.chunk = chunk;
    if (grid > (int)(item_end - item_lo)) grid = (int)(item_end - item_lo);
    const MxtFn fn = kMxt[gf16 ? 1 : 0][align >= 16 ? 2 : align >= 8 ? 1 : 0];
    // Launched beside the batch's plans where they come right before it (after_plans;
    // whatever else came before has then ended, and is visible): only a
    // decode's coefficients wait for them, so set-up and encodes hide the plan kernel
    // (1024 stripes of 64 + 16, 4096-byte rows: 158 -> 143 us; 48 + 8: 142 -> 130).
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kMxtThreads);
    cfg.dynamicSmemBytes = P.smem;  // the least, so that plan blocks fit beside it
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = after_plans ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, fn, P);
}

}  // namespace scrs
