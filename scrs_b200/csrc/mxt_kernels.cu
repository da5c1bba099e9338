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
// One persistent CTA per SM, 20 warps: a publisher (claims work items), the MMA
// issuer, two builders of B, two epilogue groups of four warps (counts -> parities
// -> bytes -> rows, one per tile) and two expander groups of four warps (rows -> A,
// alternate units; they also write decode's present rows through).  A block is 256
// columns, two tiles of 128: a thread expands one column of each, and its results
// stay in its own tensor-memory lane.  A flows through a ring of units and D
// through a ring of tiles, so loads, expansion, MMAs and epilogue overlap.
//
// What bounds it: no pipe does.  At 64 inputs and 16 outputs a block of 256
// columns takes 2660 cycles: 1024 of MMAs and 1460 of issue slots (5820
// instructions, nearly half of them on the ALU pipe); the rest is latency between
// the roles, whose chain of hand-overs the A ring (three units) and the
// accumulator ring (one or two blocks) only partly hide.
// Measured against the XOR networks (drain alone, half encodes, half decodes of
// random losses): GF(256) 64 + 16, 4096-byte rows 700 -> 324 us for 872 MB of
// rows; 32 + 8, 1400-byte rows 1123 -> 386 us for 596 MB; tower 32 + 8, 64 KiB rows
// 821 -> 290 us for 872 MB.
//
// Choices, with what the alternatives took (the 64 + 16 batch): units of two
// steps 424 us and of three 404 against 377 with four; three expander groups 415
// against 400 with two; polls with a time hint 401 against 384 without; A in
// shared memory and the columns on the N side, whose epilogue needs no staging,
// 437 against 401.

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "kernels.cuh"
#include "mxk_device.cuh"

namespace scrs {

namespace {

constexpr int kEpiWarp = 4, kExpWarp = 12, kExpGroups = 2;
constexpr int kMxtThreads = 32 * (kExpWarp + 4 * kExpGroups);
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
constexpr uint32_t kDepth = 2;       // units an expander warp has loaded or in flight
constexpr uint32_t kStage = 784;     // staged bytes of a step's rows, 2 x 32 columns' worth, and 16 for their leads
constexpr uint32_t kUnit = kUnitSteps * kStage;
constexpr uint32_t kAhead = (kDepth + 1) * kExpGroups;  // the loads' lead over the last warp's work, in units
constexpr uint32_t kItemSlots = kAhead + 4;
constexpr uint32_t kBiasBytes = 128 * 32;  // the constant B operand
constexpr uint32_t kMaxRows = 256;
constexpr uint32_t kMaxBytes = 223;  // input field bytes of a task: at most 1791 counts
constexpr uint8_t kNoPass = 255;      // no output row (data rows end at 254)
constexpr uint32_t kMaxRing = 16;

// A work item as the roles read it: rows [in + row[i] * in_stride, + len).
struct ItemSlot {
    const uint8_t* in;         // at the item's first column
    uint8_t* out;
    const void* coef;
    const uint16_t* coef_rows;
    uint32_t in_stride, out_stride;
    uint32_t len, rest;        // bytes of the item; bytes to the end of the rows
    uint32_t n_in, n_out, ld;
    uint32_t steps, units, passes, per, blocks;
    uint32_t valid, accumulate, copies;
    uint8_t row[kMaxRows];     // input row numbers (row[0] past the end, where coefficients are zero)
    uint8_t pass[kMaxRows];    // output row of a verbatim copy, or kNoPass
    uint8_t to[kMaxRows];      // output row numbers
};

struct Bars {
    uint64_t exp_full[kMaxRing], exp_empty[kMaxRing];
    uint64_t d_full[kMaxRing], d_empty[kMaxRing];
    uint64_t b_full[2], b_empty[2];
    uint64_t stg_full[2], stg_empty[2];
    uint64_t item_full[kItemSlots], item_empty[kItemSlots];
    uint64_t fin;
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
    static constexpr uint32_t kTile = 128 * kElem;           // and per tile
    static constexpr uint32_t kSpan = 32 * kElem;            // of which an expander warp's lanes hold
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
    return cnt ? up(cnt * MxtGeom<kGf16>::kElem, 4) * 8 : 32u;
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

__device__ __forceinline__ void xor_into(uint4& a, const uint4& b) { a.x ^= b.x, a.y ^= b.y, a.z ^= b.z, a.w ^= b.w; }
__device__ __forceinline__ void xor_into(uint2& a, const uint2& b) { a.x ^= b.x, a.y ^= b.y; }

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
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

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
    uint8_t* s_stg = s_raw + 4 * kExpGroups * kDepth * kUnit;
    const int tid = threadIdx.x, lane = tid & 31, warp = (int)uni(tid >> 5);

    // ---- set-up: barriers, tables, tensor memory
    if (tid == 0) {
        for (uint32_t i = 0; i < kMaxRing; i++) {
            mbar_init(&B->exp_full[i], 4), mbar_init(&B->exp_empty[i], 1);
            mbar_init(&B->d_full[i], 1), mbar_init(&B->d_empty[i], 4);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&B->b_full[i], 2), mbar_init(&B->b_empty[i], 1);
            mbar_init(&B->stg_full[i], 4), mbar_init(&B->stg_empty[i], 4);
        }
        // consumers: MMA issuer, 2 builders, 8 epilogue warps, the expanders
        for (uint32_t i = 0; i < kItemSlots; i++)
            mbar_init(&B->item_full[i], 1), mbar_init(&B->item_empty[i], 11 + 4 * kExpGroups);
        mbar_init(&B->fin, 1);
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
                    I.coef_rows = T.coef_rows;
                    I.in_stride = (uint32_t)T.in_stride;
                    I.out_stride = (uint32_t)T.out_stride;
                    I.rest = (uint32_t)(T.L - off);
                    I.len = umin32(I.rest, P.chunk);
                    I.n_in = T.n_in, I.n_out = T.n_out, I.ld = T.ld;
                    I.steps = steps;
                    I.units = (steps + kUnitSteps - 1) / kUnitSteps;
                    I.passes = T.n_out ? (T.n_out + G::kGroup - 1) / G::kGroup : 1u;  // no outputs: copies alone
                    I.per = (T.n_out + I.passes - 1) / I.passes;
                    I.blocks = (I.len + G::kRow - 1) / G::kRow;
                    I.accumulate = T.accumulate;
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
    } else if (warp == 1) {
        // ---- MMA issuer
        Ring bs, ds, as;
        const uint64_t bias = operand_desc(smem_addr(s_bias));
        for (;;) {
            warp_wait(&B->item_full[it.i], it.ph, B, P.status);
            const ItemSlot& I = H.item[it.i];
            if (!uni(I.valid) || aborted(B)) break;
            const uint32_t passes = uni(I.passes), blocks = uni(I.blocks), steps = uni(I.steps), units = uni(I.units),
                           per = uni(I.per), n_out = uni(I.n_out);
            for (uint32_t pass = 0; pass < passes; pass++) {
                const uint32_t N = columns_of<kGf16>(umin32(per, n_out - pass * per));
                const uint32_t idesc = instr_desc(N), N2 = N * 2;  // N * 32 bytes of B a step
                warp_wait(&B->b_full[bs.i], bs.ph, B, P.status);
                const uint64_t b0 = operand_desc(smem_addr(s_b + bs.i * P.b_bytes));
                for (uint32_t b = 0; b < blocks; b++) {
                    // one tile after the other where the A ring holds a block's units
                    // (a tile's epilogue runs beside the other's MMAs), else both at
                    // every step
                    if (units <= P.ring) {
                        const Ring as0 = as;
#pragma unroll
                        for (uint32_t tile = 0; tile < 2; tile++) {
                            warp_wait(&B->d_empty[ds.i], ds.ph ^ 1u, B, P.status);
                            const uint32_t d = tmem + ds.i * P.d_cols;
                            tc_fence_after();
                            mma_step<false>(d, tmem + kBiasCol, bias, idesc, tmem + kScaleCol);
                            as = as0;
                            uint64_t bd = b0;
                            uint32_t left = steps;
                            for (uint32_t u = 0; u < units; u++) {
                                if (tile == 0) {
                                    warp_wait(&B->exp_full[as.i], as.ph, B, P.status);
                                    tc_fence_after();
                                }
                                const uint32_t a = tmem + a_col + as.i * kUnitCols + tile * (kStepCols / 2);
                                if (left >= kUnitSteps) {
#pragma unroll
                                    for (uint32_t h = 0; h < kUnitSteps; h++)
                                        mma_step<true>(d, a + h * kStepCols, bd + h * N2, idesc, tmem + kScaleCol);
                                } else {
#pragma unroll
                                    for (uint32_t h = 0; h < kUnitSteps - 1; h++)
                                        if (h < left) mma_step<true>(d, a + h * kStepCols, bd + h * N2, idesc, tmem + kScaleCol);
                                }
                                if (tile == 1) tc_commit(&B->exp_empty[as.i]);
                                bd += kUnitSteps * N2;
                                left -= kUnitSteps;
                                as.next(P.ring);
                            }
                            tc_commit(&B->d_full[ds.i]);
                            ds.next(P.n_d);
                        }
                        continue;
                    }
                    Ring d1 = ds;
                    d1.next(P.n_d);
                    warp_wait(&B->d_empty[ds.i], ds.ph ^ 1u, B, P.status);
                    warp_wait(&B->d_empty[d1.i], d1.ph ^ 1u, B, P.status);
                    const uint32_t t0 = tmem + ds.i * P.d_cols, t1 = tmem + d1.i * P.d_cols;
                    tc_fence_after();
                    mma_step<false>(t0, tmem + kBiasCol, bias, idesc, tmem + kScaleCol);
                    mma_step<false>(t1, tmem + kBiasCol, bias, idesc, tmem + kScaleCol);
                    uint64_t bd = b0;
                    for (uint32_t s = 0; s < steps;) {
                        warp_wait(&B->exp_full[as.i], as.ph, B, P.status);
                        tc_fence_after();
                        uint32_t a = tmem + a_col + as.i * kUnitCols;
                        const uint32_t end = umin32(steps, s + kUnitSteps);
                        for (; s < end; s++) {
                            mma_step<true>(t0, a, bd, idesc, tmem + kScaleCol);
                            mma_step<true>(t1, a + kStepCols / 2, bd, idesc, tmem + kScaleCol);
                            bd += N2;
                            a += kStepCols;
                        }
                        tc_commit(&B->exp_empty[as.i]);
                        as.next(P.ring);
                    }
                    tc_commit(&B->d_full[ds.i]);
                    tc_commit(&B->d_full[d1.i]);
                    ds = d1;
                    ds.next(P.n_d);
                }
                tc_commit(&B->b_empty[bs.i]);
                bs.next(P.n_b);
            }
            warp_arrive(&B->item_empty[it.i], lane);
            it.next(kItemSlots);
        }
        // the MMAs in flight end before tensor and shared memory are given up
        tc_commit(&B->fin);
        __syncwarp();
        const uint64_t t0 = global_ns();
        while (!mbar_try_wait(&B->fin, 0) && global_ns() - t0 < 100000000ull) {
        }
    } else if (warp < kEpiWarp) {
        // ---- builders of the coefficient operand
        const uint32_t first = (uint32_t)(warp - 2) * 32 + lane;
        Ring bs;
        for (;;) {
            warp_wait(&B->item_full[it.i], it.ph, B, P.status);
            const ItemSlot& I = H.item[it.i];
            if (!uni(I.valid) || aborted(B)) break;
            const uint32_t n_in = I.n_in, ld = I.ld, passes = uni(I.passes);
            const uint16_t* coef_rows = I.coef_rows;
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
                            const size_t at = (size_t)(coef_rows ? coef_rows[i] : i) * ld + lo + j;
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
        const uint32_t e = (uint32_t)warp & 3u, tile = (uint32_t)(warp - kEpiWarp) >> 2;  // lane quarter
        const uint32_t acc = tmem + (e << 21);
        const uint32_t pos = G::kElem * (32 * e + lane);  // where this lane's column lies in the tile
        uint8_t* stg = s_stg + tile * (kGroupBytes * 128);
        Ring ds;
        if (tile) ds.next(P.n_d);
        uint32_t used = 0;  // tiles so far
        for (;;) {
            warp_wait(&B->item_full[it.i], it.ph, B, P.status);
            const ItemSlot& I = H.item[it.i];
            if (!uni(I.valid) || aborted(B)) break;
            const uint32_t len = uni(I.len), blocks = uni(I.blocks), passes = uni(I.passes), per = uni(I.per),
                           n_out = uni(I.n_out);
            const bool into = uni(I.accumulate) != 0;
            for (uint32_t pass = 0; pass < passes; pass++) {
                const uint32_t lo = pass * per, cnt = umin32(per, n_out - lo);
                const uint32_t words = columns_of<kGf16>(cnt) / 32;  // of 4 field bytes
                for (uint32_t b = 0; b < blocks; b++) {
                    uint32_t w[4];
                    warp_wait(&B->d_full[ds.i], ds.ph, B, P.status);
                    tc_fence_after();
                    const uint32_t d = acc + ds.i * P.d_cols;
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
                        w[q] = parity_word(z[0]);
                        w[q + 1] = parity_word(z[1]);
                    }
                    ds.next(P.n_d);
                    ds.next(P.n_d);
                    const uint32_t at = b * G::kRow + tile * G::kTile;
                    const uint32_t n = len > at ? umin32(G::kTile, len - at) : 0u;  // the row's bytes in this tile
                    if (!cnt || !n) continue;
                    if (used) {  // the group's last stores have read the staging rows
                        warp_arrive(&B->stg_empty[tile], lane);
                        warp_wait(&B->stg_empty[tile], (used - 1) & 1u, B, P.status);
                    }
#pragma unroll
                    for (uint32_t j = 0; j < G::kGroup; j++) {
                        if (j >= cnt) break;
                        if (kGf16)
                            *reinterpret_cast<uint16_t*>(stg + j * G::kTile + pos) = (uint16_t)(w[j / 2] >> (16 * (j & 1u)));
                        else
                            stg[j * G::kTile + pos] = (uint8_t)(w[j / 4] >> (8 * (j & 3u)));
                    }
                    warp_arrive(&B->stg_full[tile], lane);
                    warp_wait(&B->stg_full[tile], used & 1u, B, P.status);
                    used++;
                    uint8_t* out = I.out + at;
                    const uint32_t stride = I.out_stride;
                    if (kAligned) {
                        constexpr uint32_t kPieces = G::kTile / kPiece;
                        for (uint32_t x = 32 * e + lane; x < cnt * kPieces; x += 128) {
                            const uint32_t j = x / kPieces, o = kPiece * (x % kPieces);
                            if (o >= n) continue;
                            Piece v = *reinterpret_cast<const Piece*>(stg + j * G::kTile + o);
                            Piece* p = reinterpret_cast<Piece*>(out + (uint64_t)I.to[lo + j] * stride + o);
                            if (into) xor_into(v, *p);
                            *p = v;
                        }
                    } else {
                        for (uint32_t j = e; j < cnt; j += 4) {
                            uint8_t* row = out + (uint64_t)I.to[lo + j] * stride;
                            const uint8_t* src = stg + j * G::kTile;
                            // bytes up to the first whole word of the row, words, the rest
                            const uint32_t head = umin32((uint32_t)(-reinterpret_cast<intptr_t>(row)) & 3u, n);
                            const uint32_t full = (n - head) / 4, tail = head + 4 * full;
                            if ((uint32_t)lane < head) row[lane] = into ? row[lane] ^ src[lane] : src[lane];
                            for (uint32_t x = lane; x < full; x += 32) {
                                const uint32_t* s = reinterpret_cast<const uint32_t*>(src + 4 * x);
                                const uint32_t v = head ? __funnelshift_r(s[0], s[1], 8 * head) : s[0];
                                uint32_t* p = reinterpret_cast<uint32_t*>(row + head + 4 * x);
                                *p = into ? *p ^ v : v;
                            }
                            if ((uint32_t)lane < n - tail)
                                row[tail + lane] = into ? row[tail + lane] ^ src[tail + lane] : src[tail + lane];
                        }
                    }
                }
            }
            warp_arrive(&B->item_empty[it.i], lane);
            it.next(kItemSlots);
        }
    } else {
        // ---- expanders: rows -> the A operand
        const uint32_t e = (uint32_t)warp & 3u, group = (uint32_t)(warp - kExpWarp) >> 2;
        uint8_t* units = s_raw + (uint32_t)(warp - kExpWarp) * kDepth * kUnit;
        // a row's staged bytes: this warp's 32 columns of either tile, in 16-byte
        // pieces around them when unaligned
        constexpr uint32_t kPieces = G::kSpan / kPiece + (kAligned ? 0 : 1), kHalf = kPiece * kPieces,
                           kPitch = 2 * kHalf;
        constexpr uint32_t kLeads = kStage - 16;  // unaligned: where each row starts in its first piece
        // a walk over this warp's units, every kExpGroups-th one
        struct Walk {
            Ring it;
            uint32_t unit, col, pass;  // col: bytes from the item's first column
            uint32_t steps, units, len, passes;
            bool open, copies;
        };
        auto open_item = [&](Walk& W) {  // the ring's next item, if there is one
            warp_wait(&B->item_full[W.it.i], W.it.ph, B, P.status);
            const ItemSlot& I = H.item[W.it.i];
            W.open = uni(I.valid) && !aborted(B);
            W.steps = uni(I.steps), W.units = uni(I.units), W.len = uni(I.len), W.passes = uni(I.passes);
            W.copies = uni(I.copies) != 0;
            W.col = W.pass = 0;
        };
        auto settle = [&](Walk& W, bool release) {  // carries the unit into blocks, passes, items
            while (W.open && W.unit >= W.units) {
                W.unit -= W.units;
                W.col += G::kRow;
                if (W.col < W.len) continue;
                W.col = 0;
                if (++W.pass < W.passes) continue;
                if (release) warp_arrive(&B->item_empty[W.it.i], lane);
                W.it.next(kItemSlots);
                open_item(W);
            }
        };
        Walk lw, pw;  // the loads' walk, kDepth units ahead of the work's
        // the unit's rows into staging slot u
        auto load_next = [&](uint32_t u) {
            if (lw.open) {
                const ItemSlot& I = H.item[lw.it.i];
                const uint32_t first = lw.col + e * G::kSpan;
                const uint8_t* base = I.in + first;
                const uint32_t stride = I.in_stride;
#pragma unroll
                for (uint32_t h = 0; h < kUnitSteps; h++) {
                    const uint32_t step = kUnitSteps * lw.unit + h;
                    if (step >= lw.steps) break;
                    uint8_t* stage = units + u * kUnit + h * kStage;
#pragma unroll
                    for (uint32_t x = 0; x < G::kStepRows * 2 * kPieces; x += 32) {
                        const uint32_t g = x + lane, q = g / (2 * kPieces), z = g % (2 * kPieces);
                        if (g >= G::kStepRows * 2 * kPieces) break;
                        const uint32_t tile = z / kPieces, o = kPiece * (z % kPieces), at = first + tile * G::kTile + o;
                        const uint8_t* p = base + (uint64_t)I.row[step * G::kStepRows + q] * stride;
                        bool has = at < lw.len;
                        if (!kAligned) {
                            const uint32_t lead = (uint32_t) reinterpret_cast<uintptr_t>(p) & 15u;
                            has = at < I.rest + lead;
                            p -= lead;
                            if (z == 0) stage[kLeads + q] = (uint8_t)lead;
                        }
                        copy_in<(int)kPiece>(smem_addr(stage) + q * kPitch + tile * kHalf + o, p + tile * G::kTile + o, has);
                    }
                }
                lw.unit += kExpGroups;
                settle(lw, false);
            }
            copy_commit();
        };
        uint32_t slot = group, slot_ph = 0;  // A slot of this warp's next unit
        auto work = [&](uint32_t u) {
            const ItemSlot& I = H.item[pw.it.i];
            const uint32_t dst0 = tmem + (e << 21) + a_col + slot * kUnitCols;
            const bool copies = pw.copies && pw.pass == 0;  // decode's present rows go straight through
            const uint32_t first = pw.col + e * G::kSpan;
            warp_wait(&B->exp_empty[slot], slot_ph ^ 1u, B, P.status);
            tc_fence_after();
#pragma unroll
            for (uint32_t h = 0; h < kUnitSteps; h++) {
                const uint32_t step = kUnitSteps * pw.unit + h;
                if (step >= pw.steps) break;
                const uint8_t* stage = units + u * kUnit + h * kStage;
                uint4 t[2][2];  // [tile][chunk]: the operand words of this lane's columns
#pragma unroll
                for (int tile = 0; tile < 2; tile++) {
                    uint32_t x[G::kStepRows];  // the column's element of each row
#pragma unroll
                    for (uint32_t q = 0; q < G::kStepRows; q++) {
                        const uint32_t lead = kAligned ? 0u : stage[kLeads + q];
                        const uint8_t* p = stage + q * kPitch + tile * kHalf + lead + G::kElem * lane;
                        if (!kGf16)
                            x[q] = *p;
                        else if (kAligned || !(lead & 1u))
                            x[q] = *reinterpret_cast<const uint16_t*>(p);
                        else
                            x[q] = p[0] | (uint32_t)p[1] << 8;
                    }
#pragma unroll
                    for (int z = 0; z < 2; z++) {
                        if (kGf16) {
                            t[tile][z] = spread(__byte_perm(x[2 * z], x[2 * z + 1], 0x5410));
                        } else {
                            const int q = (4 * z) % (int)G::kStepRows;
                            const uint32_t a = __byte_perm(x[q], x[q + 1], 0x0040);
                            const uint32_t b = __byte_perm(x[(q + 2) % G::kStepRows], x[(q + 3) % G::kStepRows], 0x0040);
                            t[tile][z] = spread(__byte_perm(a, b, 0x5410));
                        }
                    }
                }
                tmem_store8(dst0 + h * kStepCols, t[0][0], t[0][1]);
                tmem_store8(dst0 + h * kStepCols + kStepCols / 2, t[1][0], t[1][1]);
            }
            tmem_wait_store();
            tc_fence_before();
            warp_arrive(&B->exp_full[slot], lane);
            slot += kExpGroups;
            if (slot >= P.ring) slot -= P.ring, slot_ph ^= 1u;
            if (!copies) return;
            const uint32_t stride = I.out_stride;
#pragma unroll
            for (uint32_t h = 0; h < kUnitSteps; h++) {
                const uint32_t step = kUnitSteps * pw.unit + h;
                if (step >= pw.steps) break;
                const uint8_t* stage = units + u * kUnit + h * kStage;
                // pieces of aligned rows, words of the others
                constexpr uint32_t kBy = kAligned ? kPiece : 4, kPer = G::kSpan / kBy;
#pragma unroll
                for (uint32_t x = 0; x < G::kStepRows * 2 * kPer; x += 32) {
                    const uint32_t g = x + lane, q = g / (2 * kPer), z = g % (2 * kPer), tile = z / kPer;
                    const uint32_t o = kBy * (z % kPer), at = first + tile * G::kTile + o;
                    const uint32_t to = I.pass[step * G::kStepRows + q];
                    if (to == kNoPass || at >= pw.len) continue;
                    uint8_t* p = I.out + (uint64_t)to * stride + at;
                    const uint8_t* src = stage + q * kPitch + tile * kHalf + o;
                    if (kAligned) {
                        *reinterpret_cast<Piece*>(p) = *reinterpret_cast<const Piece*>(src);
                    } else {
                        const uint32_t lead = stage[kLeads + q];
                        const uint32_t* a = reinterpret_cast<const uint32_t*>(src + (lead & ~3u));
                        const uint32_t v = __funnelshift_r(a[0], a[1], 8 * (lead & 3u));
                        if ((reinterpret_cast<uintptr_t>(p) & 3u) == 0 && at + 4 <= pw.len) {
                            *reinterpret_cast<uint32_t*>(p) = v;
                        } else {
#pragma unroll
                            for (uint32_t y = 0; y < 4; y++)
                                if (at + y < pw.len) p[y] = (uint8_t)(v >> (8 * y));
                        }
                    }
                }
            }
        };
        lw.unit = pw.unit = group;
        open_item(lw);
        settle(lw, false);
        // the work's walk starts where the loads' did: items before its first
        // unit are passed over and released
        open_item(pw);
        settle(pw, true);
        for (uint32_t u = 0; u < kDepth; u++) load_next(u);
        for (uint32_t u = 0; pw.open; u = u + 1 == kDepth ? 0 : u + 1) {
            copy_wait<kDepth - 1>();
            __syncwarp();
            work(u);
            __syncwarp();
            load_next(u);
            pw.unit += kExpGroups;
            settle(pw, true);
        }
        copy_wait<0>();
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
    if (max_in == 0 || max_in * G::kElem > kMaxBytes || max_out > kMaxRows) return false;
    P->d_cols = columns_of<kGf16>(std::max<uint32_t>(1, std::min<uint32_t>(max_out, G::kGroup)));
    P->n_d = P->d_cols > 64 ? 2 : 4;  // one or two blocks' tiles; the rest is the A ring, three units or more
    P->ring = std::min<uint32_t>(kMaxRing, (kBiasCol - P->n_d * P->d_cols) / kUnitCols);
    P->b_bytes = steps_of<kGf16>(max_in) * P->d_cols * 32;
    const size_t fixed = up(sizeof(Head), 128) + kBiasBytes + 4 * kExpGroups * kDepth * kUnit + 2 * kGroupBytes * 128 + 16;
    for (P->n_b = 2; P->n_b >= 1; P->n_b--)
        if (fixed + (size_t)P->n_b * P->b_bytes <= kMxtSmem) return true;
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
                       cudaStream_t stream, int align, int gf16) {
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
    fn<<<grid, kMxtThreads, kMxtSmem, stream>>>(P);
    return cudaGetLastError();
}

}  // namespace scrs
