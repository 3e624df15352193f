// Non-causal flash-attention forward for head_dim 128, bf16, written for sm_100a.
//
// One CTA owns a pair of 128-row query tiles of one (batch, head) and walks every
// key/value tile of the attended sequence. Three warpgroups:
//
//   warps 0-3 / 4-7     softmax group for tile 0 / tile 1: one thread per query
//                       row (= TMEM lane). Reads S with tcgen05.ld, keeps the row in
//                       registers, exponentiates in the log2 domain, writes bf16 P_t to
//                       its 64 columns (handed to the MMA warp in halves, so P_t V_j
//                       starts before the row is finished) and accumulates the row sum
//                       from the unrounded fp32 values.
//   warp 8  (one lane)  TMA producer: Q tiles once, then K_j, V_j into a 4-slot
//                       ring of 32 KiB shared-memory slots (mbarrier full/empty).
//   warp 9  (converged) tcgen05.mma issuer:  S = Q_t K_j^T  (A, B from shared
//                       memory, K-major, 128-byte swizzle) and O_t += P_t V_j
//                       (A = P_t from tensor memory, B = V_j MN-major).
//   warps 10-11         give their registers to the softmax groups (setmaxnreg: 208 registers
//                       per softmax thread, 88 elsewhere). In head-exchange use they do the
//                       exchange: QK-norm + RoPE of this rank's raw Q, K and peer stores of every
//                       head row to the rank that attends it, while the other roles already work
//                       on what has arrived (ExchangeParams). Idle otherwise.
//
// Tensor memory (512 columns): one 128-column S buffer that the two tiles use in turn, P_0 and P_1
// (64 columns each), O_0 and O_1 (128 each, fp32). A softmax group has S in registers some 250 clk
// after it is complete; the buffer is then free for the other tile's S, and the next S of a tile is
// ready before its group has finished the present one. (With P_t written over its own S_t a tile's
// chain was S MMA -> softmax -> P V -> next S MMA, and the groups waited for S a third of the time:
// 295 us at 4608 tokens x 32 heads, 278 us with the shared S buffer.)
//
// Issue order per key/value tile j:  S1_j, PV1_{j-1}, S0_{j+1}, PV0_j.
//
// What bounds it: the issuing warp shares its scheduler with two softmax warps, and per key tile it
// needed some 3000 clk for what the tensor pipe does in 2048: 110 clk per barrier that was complete
// anyway, 30 per MMA. Hence the looks ahead at barriers, one asm block and one elected lane per run of
// MMAs, and operands the compiler knows to be uniform (278 -> 266 us). An iteration is now some 2850 clk;
// the tensor pipe and the special-function unit, which the two groups share, are both 68 % busy (2048 clk
// each per key tile), and the rest is hand-overs, tensor-memory latency and a CTA's start and epilogue.
// The power cap comes on top in calls back to back for long.
//
// Online softmax with a lazy reference maximum: the exponent reference of a row
// only moves when some row of the warp sees a tile maximum more than 2^8 above it;
// then the group rescales its O rows in TMEM itself, after the commit that says PV_t of tile j-1 is
// complete; PV_t of tile j is not issued before the group hands over P_t.
//
// Arithmetic follows the reference flash kernel (F2K_CUDA
// src/backend/cuda/attention.cu:601-757): scores scaled by `scale`, P rounded to
// bf16 for the P.V product, the row sum taken from fp32 P, one bf16 rounding of O.
//
// Every wait is bounded; when one expires the CTA sets the status word, drains its
// own copies and MMAs, frees its tensor memory and returns.

#include "attn_launch.h"
#include "barrier_look.h"
#include "ptx.cuh"
#include "row_math.cuh"
#include "softmax_row.cuh"

#include <cuda_bf16.h>

#include <cstddef>
#include <type_traits>

namespace f2k {

using namespace f2k::ptx;

namespace {

constexpr int kThreads     = 384;
constexpr int kLoaderWarp  = 8;
constexpr int kMmaWarp     = 9;
constexpr int kStages      = 4;
constexpr uint32_t kTileBytes = kTileM * kHeadDim * 2;  // 32 KiB: one Q, K or V tile
constexpr uint32_t kBoxBytes  = kTileBytes / 2;         // one 128 x 64 TMA box
constexpr uint32_t kTmemCols  = 512;
constexpr uint32_t kColS = 0, kColP0 = 128, kColP1 = 192, kColO0 = 256, kColO1 = 384;
constexpr float kLazyThreshold = 8.0f;  // log2 units
constexpr int kPParts = 2;     // P is handed to the MMA warp in halves (1, 2, 4 parts: 269, 266, 269 us at 4608 tokens x 32 heads)
constexpr int kPvSteps = 4;    // k-steps of 16 keys per part: umma_ts_x4
static_assert(kPParts * kPvSteps * 16 == kTileN, "the parts cover the key tile");

// Tuning switches (compile-time; the defaults are what ships).
#ifndef F2K_OPT_SETMAXNREG
#define F2K_OPT_SETMAXNREG 1   // softmax warpgroups take registers from the load/MMA warpgroup
#endif
#ifndef F2K_OPT_REGS_SOFTMAX
#define F2K_OPT_REGS_SOFTMAX 208
#endif
// registers per thread after setmaxnreg: softmax warpgroups / the load+MMA warpgroup;
// 2 * 128 * softmax + 128 * other must stay within the 384 * 168 the CTA is launched with
constexpr int kRegsSoftmax = F2K_OPT_REGS_SOFTMAX, kRegsOther = (384 * 168 - 256 * F2K_OPT_REGS_SOFTMAX) / 128 / 8 * 8;
static_assert(kRegsOther >= 40, "the load and MMA warps need some registers too");

struct SmemCtl {
    uint64_t q_full[2];
    uint64_t kv_full[kStages];
    uint64_t kv_empty[kStages];
    uint64_t s_full[2];
    uint64_t s_free;               // S has been read into registers: the other tile's S may be written
    uint64_t p_full[2][kPParts];   // [tile][part of the key tile]
    uint64_t pv_done[2];           // P_t V_j is complete: P_t may be rewritten, O_t may be touched
    uint64_t drain;
    uint64_t xchg_full[2][2];      // head exchange: [warp][staging buffer] loaded
    uint32_t tmem_base;
    uint32_t abort;
    uint32_t softmax_done;         // softmax warps that have finished (head exchange: the spare warps then stop)
};

constexpr uint32_t kSmemQ    = 0;
constexpr uint32_t kSmemRing = 2 * kTileBytes;
constexpr uint32_t kSmemCtl  = kSmemRing + kStages * kTileBytes;
constexpr uint32_t kSmemStage = (kSmemCtl + sizeof(SmemCtl) + 127u) & ~127u;   // head exchange staging (bulk copies)
constexpr uint32_t kSmemUsed = kSmemStage + 2 * 2 * (16 * 256 + 4 * 512);

template <int kMax>
__device__ __forceinline__ void locate_tile(const int* tile_start, const int* len, int nseg,
                                            int tile, int& seg, int& row0, int& valid) {
    seg = 0;
#pragma unroll
    for (int i = 1; i < kMax; ++i)
        if (i < nseg && tile >= tile_start[i]) seg = i;
    row0  = (tile - tile_start[seg]) * kTileN;
    valid = min(kTileN, len[seg] - row0);
}

// The MMA warp's side of barrier_look.h.
struct WarpBarriers {
    volatile uint32_t* abort_flag;
    long long limit;
    __device__ __forceinline__ bool test(uint32_t bar_a, uint32_t par_a, uint32_t bar_b, uint32_t par_b) const {
        return bar_a == bar_b ? mbar_test(bar_a, par_a) : mbar_test2(bar_a, par_a, bar_b, par_b);
    }
    __device__ __forceinline__ bool all(bool pred) const { return __all_sync(0xffffffffu, pred) != 0; }
    __device__ __forceinline__ bool wait(uint32_t bar, uint32_t par) const { return all(mbar_wait(bar, par, abort_flag, limit)); }
};

// The MMA-issuing warp shares its scheduler with two softmax warps, so every instruction it needs per
// MMA delays the tensor pipe. A block of MMAs is therefore one asm statement with one elected lane, and
// descriptors are built once and advanced by adding a compile-time constant (the start-address field
// counts 16-byte units and never carries out of its 14 bits inside the CTA's shared memory).

// S_t = Q_t K^T: 8 k-steps of 16 over head_dim; both operands K-major, 128-byte swizzle, stored as
// two 128 x 64 boxes (k-steps 0-3 in the first, 4-7 in the second).
__device__ __forceinline__ void issue_qk(uint32_t d_tmem, uint64_t q_desc, uint64_t k_desc) {
    constexpr uint32_t idesc = umma_idesc_bf16(kTileM, kTileN, /*b_mn_major=*/false);
    static_assert(kHeadDim == 128 && kBoxBytes == 16384, "the steps of umma_ss_x8");
    umma_ss_x8(d_tmem, q_desc, k_desc, idesc);
}

// O_t (+)= P_t V: 8 k-steps of 16 keys. A = P_t in TMEM (two bf16 per 32-bit column, 8 columns per
// k-step); B = V tile, MN-major: head_dim contiguous in 64-element (128-byte) swizzled rows, one
// row per key, the second 64 head-dim elements one box (16 KiB) further on; 8-key groups are
// 1024 bytes apart. kPart selects the k-steps.
template <int kPart>
__device__ __forceinline__ void issue_pv_part(uint32_t d_tmem, uint32_t p_tmem, uint64_t v_desc, uint32_t accumulate) {
    constexpr uint32_t idesc = umma_idesc_bf16(kTileM, kHeadDim, /*b_mn_major=*/true);
    constexpr int kk = kPart * kPvSteps;
    umma_ts_x4(d_tmem, p_tmem + kk * 8, v_desc + kk * (2048 >> 4), idesc, kPart > 0 ? 1u : accumulate);
}

// Head exchange by one of the CTA's two spare warps (see ExchangeParams). A chunk is 16 tokens of
// Q, or of K and V, for one destination. The queue walks the ranges of ExchangeParams::order: ring
// step i sends to rank - i (0 = this rank itself), which is the order in which the destinations
// get to this rank's segment.
//
// Two warps per CTA cannot keep enough loads in flight from registers (measured: 86 GB/s per
// GPU), so the rows travel as bulk copies through a small staging area in shared memory: one lane
// issues cp.async.bulk loads of up to 4 KiB of head rows (plus the tokens' cos/sin rows) into one
// of the warp's two buffers, the warp normalises + rotates the rows in place (a half-warp per
// row, as the prologue kernel does), and one bulk store sends them to the destination, local or
// peer. The loads of the next buffer are in flight while this one is worked on.
constexpr uint32_t kStageRowBytes = 16 * 256;                 // 16 head rows
constexpr uint32_t kStageTabBytes = 4 * 512;                  // cos + sin rows of up to 4 tokens
constexpr uint32_t kStageBufBytes = kStageRowBytes + kStageTabBytes;

// The warp stops taking chunks once its CTA's softmax groups are done (`softmax_done` reaches 8) if
// a later CTA will take the CTA's place (`may_stop`: CTAs start in index order, one per SM): that
// one brings exchange warps of its own. The CTAs of the last wave serve the queue until it is
// empty, so everything this rank owes its peers is sent. A CTA that waits for rows is running, so
// its own spare warps keep serving the queue: nothing can stall.
__device__ __forceinline__ bool exchange_role(const ExchangeParams& x, int lane, uint32_t stage_u32, uint8_t* stage_ptr,
                                              uint32_t bar0, volatile uint32_t* abort_flag, long long wait_limit,
                                              volatile uint32_t* softmax_done, bool may_stop) {
    const int hl = lane & 15, hw = lane >> 4;
    const int n_tiles = (x.s_loc + kTileM - 1) / kTileM;
    const int hpr = x.heads_per_rank, R = x.unit_rows, tpb = x.tokens_per_buf;
    const int n_hg = hpr / R;
    unsigned int fills = 0;                                    // buffers filled so far by this warp: buffer and parity
    bool ok = true;

    struct Chunk { int dst_rank, kind, tok0, tok1, n_tb, per_pass, n_fill; bool valid; };
    // Next chunk of the queue. The queue is a list of ranges (x.order): what the CTAs that run first
    // need first - their own query rows - comes first, then K/V in the order the kernel walks them.
    auto grab = [&]() {
        Chunk ch;
        unsigned int c = 0xffffffffu;
        if (lane == 0 && !(may_stop && *softmax_done >= 8u)) c = atomicAdd(x.next_chunk, 1u);
        c = __shfl_sync(0xffffffffu, c, 0);
        ch.valid = c < x.total_chunks;
        if (!ch.valid) return ch;
        int e = 0;
        unsigned int first = 0;
        while (e + 1 < x.n_ranges && c >= first + (unsigned int)x.order[e].n) { first += (unsigned int)x.order[e].n; ++e; }
        ch.kind = x.order[e].kind;                             // 0: Q rows, 1: K and V rows
        ch.dst_rank = (x.rank - (int)x.order[e].step + x.world) % x.world;
        ch.tok0 = (x.order[e].sub0 + (int)(c - first)) * kExchangeTokens;
        ch.tok1 = min(ch.tok0 + kExchangeTokens, x.s_loc);
        ch.n_tb = (ch.tok1 - ch.tok0 + tpb - 1) / tpb;
        ch.per_pass = n_hg * ch.n_tb;
        ch.n_fill = (ch.kind + 1) * ch.per_pass;
        return ch;
    };
    // fill f of a chunk: tensor, head group, token block
    auto issue = [&](const Chunk& ch, int f) {                 // lane 0 only
        const int pass = f / ch.per_pass, rem = f % ch.per_pass, hg = rem / ch.n_tb, t0 = ch.tok0 + (rem % ch.n_tb) * tpb;
        const int nt = min(tpb, ch.tok1 - t0);
        const bool rot = !(ch.kind == 1 && pass == 1);
        const __nv_bfloat16* xin = static_cast<const __nv_bfloat16*>(ch.kind == 0 ? x.q : (pass == 0 ? x.k : x.v));
        const unsigned int n = fills;
        const uint32_t buf = stage_u32 + (n & 1u) * kStageBufBytes, bar = bar0 + (n & 1u) * 8;
        bulk_wait_read<0>();                                   // the store that last used this buffer has read it
        mbar_arrive_expect_tx(bar, (uint32_t)nt * (uint32_t)(R * 256 + (rot ? 512 : 0)));
        for (int i = 0; i < nt; ++i) {
            bulk_load(buf + i * R * 256, xin + ((long long)(t0 + i) * x.n_heads_total + ch.dst_rank * hpr + hg * R) * kHeadDim,
                      R * 256, bar);
            if (rot) {
                bulk_load(buf + kStageRowBytes + i * 512, x.cos_tab + (long long)(t0 + i) * 64, 256, bar);
                bulk_load(buf + kStageRowBytes + i * 512 + 256, x.sin_tab + (long long)(t0 + i) * 64, 256, bar);
            }
        }
    };

    Chunk cur = grab();
    if (cur.valid && lane == 0) issue(cur, 0);
    while (cur.valid) {
        for (int f = 0; f < cur.n_fill; ++f) {
            const unsigned int n = fills;                      // the buffer fill f went into
            ++fills;
            if (f + 1 < cur.n_fill && lane == 0) issue(cur, f + 1);
            __syncwarp();
            ok = mbar_wait(bar0 + (n & 1u) * 8, (n >> 1) & 1u, abort_flag, wait_limit);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const int pass = f / cur.per_pass, rem = f % cur.per_pass, hg = rem / cur.n_tb;
            const int t0 = cur.tok0 + (rem % cur.n_tb) * tpb;
            const int nt = min(tpb, cur.tok1 - t0);
            const bool rot = !(cur.kind == 1 && pass == 1);
            uint8_t* buf = stage_ptr + (n & 1u) * kStageBufBytes;
            if (rot) {
                float g[8];
                unpack8(__ldg(reinterpret_cast<const uint4*>(cur.kind == 0 ? x.gamma_q : x.gamma_k) + hl), g);
                for (int row = hw; row < nt * R; row += 2) {   // a half-warp per row; both halves run the same count
                    const int ti = row / R;
                    uint4* cell = reinterpret_cast<uint4*>(buf + row * 256) + hl;
                    const float4 c4 = *(reinterpret_cast<const float4*>(buf + kStageRowBytes + ti * 512) + hl);
                    const float4 s4 = *(reinterpret_cast<const float4*>(buf + kStageRowBytes + ti * 512 + 256) + hl);
                    const float cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
                    *cell = norm_rope_row(*cell, g, cs, sn, x.eps);
                }
                fence_proxy_async_smem();                      // the rewritten rows, before the bulk store reads them
            }
            __syncwarp();
            if (lane == 0) {
                unsigned char* base = cur.kind == 0 ? x.dst_q[cur.dst_rank]
                                                    : (pass == 0 ? x.dst_k[cur.dst_rank] : x.dst_v[cur.dst_rank]);
                unsigned char* dst = base + (((long long)x.rank * x.s_loc + t0) * hpr + hg * R) * (long long)(kHeadDim * 2);
                const uint32_t src = stage_u32 + (n & 1u) * kStageBufBytes;
                if (n_hg == 1) {
                    bulk_store(dst, src, (uint32_t)(nt * R * 256));   // the tokens' rows are adjacent at the destination
                } else {
                    for (int i = 0; i < nt; ++i) bulk_store(dst + (long long)i * hpr * 256, src + i * R * 256, R * 256);
                }
                bulk_commit();
            }
        }
        if (!ok) break;
        // The first loads of the next chunk are started before this chunk's stores are waited for.
        const Chunk nxt = grab();
        if (nxt.valid && lane == 0) issue(nxt, 0);
        if (lane == 0) {
            bulk_wait<0>();                    // this chunk's rows are written, wherever they went
            fence_proxy_async_all();
            __threadfence_system();
            unsigned int* word = x.tile_words[cur.dst_rank] + cur.kind * n_tiles + cur.tok0 / kTileM;
            if (cur.kind == 1 && x.kv_walk_words[cur.dst_rank] != nullptr) {
                word = x.kv_walk_words[cur.dst_rank] +
                       kv_walk_tile(x.rank * x.s_loc + cur.tok0, cur.dst_rank * x.s_loc, x.world * x.s_loc);
            }
            atomicAdd_system(word, 1u);
        }
        __syncwarp();
        cur = nxt;
    }
    if (!ok) {
        // Leaving early: the loads of the buffer that was being filled ahead may still be on their way.
        volatile uint32_t never = 0;
        mbar_wait(bar0 + (fills & 1u) * 8, (fills >> 1) & 1u, &never, 40000000ll);
    }
    if (lane == 0) bulk_wait<0>();             // nothing of this warp reads shared memory after the kernel's exit
    return ok;
}

}  // namespace

// kWithExchange: the build of the kernel whose spare warps can run the head exchange (launches
// with p.xchg.enabled). The plain build has no code, shared memory or barriers for it.
template <bool kWithExchange>
__global__ void __launch_bounds__(kThreads, 1)
attn_fwd_sm100_kernel(const __grid_constant__ AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t smem     = (raw_addr + 1023u) & ~1023u;  // swizzle atoms need 1 KiB
    SmemCtl* ctl = reinterpret_cast<SmemCtl*>(smem_raw + (smem - raw_addr) + kSmemCtl);
    volatile uint32_t* abort_flag = &ctl->abort;

    // The shuffle tells the compiler that the role branches below are taken by whole warps: only then
    // does it keep the MMA warp's descriptors in uniform registers.
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int n_kv = p.n_kv_tiles;
    // This CTA's query tiles: qt0 and, with has_t1, qt0 + 1. A CTA with one tile leaves its second
    // softmax group, and the MMAs that would feed it, out.
    int qt0, head, bidx;
    bool has_t1;
    if (p.grid_head_fastest) {
        qt0 = 2 * blockIdx.y;
        head = blockIdx.x;
        bidx = blockIdx.z;
        has_t1 = qt0 + 1 < p.n_q_tiles;
    } else {
        const CtaWork w = cta_work(p.plan, p.n_q_tiles, (int)blockIdx.x);
        qt0 = w.tile;
        has_t1 = w.two;
        bidx = w.group / p.n_heads;
        head = w.group - bidx * p.n_heads;
    }
    const long long peer_limit = p.peer_wait_limit_clk;
    const long long wait_limit = p.wait_limit_clk;

    // Loader state: it starts its copies as soon as its barriers exist, before the CTA-wide barrier
    // below, unless a segment may still have to be waited for (the exchange's warps must run then).
    int issued = 0, q_issued = 0;
    auto load_q = [&](int t) {
        int seg, row0, valid;
        locate_tile<kMaxQSeg>(p.q_tile_start, p.q_len, p.n_qseg, qt0 + t, seg, row0, valid);
        const uint32_t bar = smem_u32(&ctl->q_full[t]);
        const uint32_t dst = smem + kSmemQ + t * kTileBytes;
        mbar_arrive_expect_tx(bar, kTileBytes);
        tma_load_4d(dst, &p.tm_q[seg], bar, 0, head, row0, bidx);
        tma_load_4d(dst + kBoxBytes, &p.tm_q[seg], bar, 64, head, row0, bidx);
        ++q_issued;
    };
    auto load_kv = [&](int seg, int row0, int kv) {          // into the next ring slot
        const int slot = issued % kStages;
        const uint32_t bar = smem_u32(&ctl->kv_full[slot]);
        const uint32_t dst = smem + kSmemRing + slot * kTileBytes;
        const CUtensorMap* tm = kv == 0 ? &p.tm_k[seg] : &p.tm_v[seg];
        mbar_arrive_expect_tx(bar, kTileBytes);
        tma_load_4d(dst, tm, bar, 0, head, row0, bidx);
        tma_load_4d(dst + kBoxBytes, tm, bar, 64, head, row0, bidx);
        ++issued;
    };
    // Once every CTA has started, the kernel behind this one may be set up on the SMs that are free. Not
    // while this one may wait for another rank: where ranks share a GPU, that rank needs those SMs.
    if (!kWithExchange && !p.waits_for_words) grid_launch_dependents();
    // A lane per barrier, then Q_0 and K_0 on their way, then the CTA-wide barrier: one lane that set up
    // all barriers and issued six tiles held the other warps back for 2400 clk.
    if (warp == kLoaderWarp) {
        constexpr int kBars = offsetof(SmemCtl, tmem_base) / sizeof(uint64_t);
        constexpr int kFree = offsetof(SmemCtl, s_free) / sizeof(uint64_t);
        constexpr int kP = offsetof(SmemCtl, p_full) / sizeof(uint64_t);
        static_assert(kBars <= 32, "a lane per barrier");
        const bool per_warp = lane == kFree || (lane >= kP && lane < kP + 2 * kPParts);   // a softmax group's four warps arrive
        if (lane < kBars) mbar_init(smem_u32(ctl) + lane * 8, per_warp ? 4 : 1);
        if (lane == 0) {
            ctl->abort = 0;
            ctl->softmax_done = 0;
        }
        fence_mbar_init();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            // Everything this kernel reads or overwrites may come from the kernel launched before it
            // (programmatic dependent launch: this one may have started while that one drained).
            grid_dependency_wait();
            if (!p.waits_for_words && n_kv > 0) {
                load_q(0);
                load_kv(0, 0, 0);
            }
        }
    }
    if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    // All 512 columns are taken, so the allocation can only start at column 0: a constant, which spares
    // every tensor-memory address a register (were it anything else, the status word would say so).
    constexpr uint32_t tmem = 0;
    if (*reinterpret_cast<volatile uint32_t*>(&ctl->tmem_base) != tmem) ctl->abort = 1;

    if (warp >= 8) {
        // ===================== warpgroup 2: TMA producer, MMA issuer, two idle warps =====================
#if F2K_OPT_SETMAXNREG
        setmaxnreg_dec<kRegsOther>();
#endif
        if (warp == kLoaderWarp) {
            // ------------------------------ TMA producer ------------------------------
            if (lane == 0) {
                bool ok = true;
                for (int t = q_issued; t < (has_t1 ? 2 : 1) && ok; ++t) {
                    int seg, row0, valid;
                    locate_tile<kMaxQSeg>(p.q_tile_start, p.q_len, p.n_qseg, qt0 + t, seg, row0, valid);
                    if (p.q_ready[seg] != nullptr) {   // the segment is written by another GPU's kernel
                        ok = p.ready_per_tile
                                 ? global_flag_wait(p.q_ready[seg] + row0 / kTileM,
                                                    p.ready_uses * (unsigned)((valid + kExchangeTokens - 1) / kExchangeTokens),
                                                    abort_flag, peer_limit)
                                 : global_flag_wait(p.q_ready[seg], p.kv_ready_value, abort_flag, peer_limit);
                        if (!ok) break;
                        asm volatile("fence.proxy.async.global;" ::: "memory");
                    }
                    load_q(t);
                }
                while (ok && issued < 2 * n_kv) {
                    const int j = issued >> 1, kv = issued & 1;
                    int seg, row0, valid;
                    locate_tile<kMaxKvSeg>(p.kv_tile_start, p.kv_len, p.n_kvseg, j, seg, row0, valid);
                    if (kv == 0 && p.ready_per_tile && p.kv_ready[seg] != nullptr) {
                        // fused head exchange: every tile has its own counter of delivered chunks
                        ok = global_flag_wait(p.kv_ready[seg] + row0 / kTileN,
                                              p.ready_uses * (unsigned)((valid + kExchangeTokens - 1) / kExchangeTokens),
                                              abort_flag, peer_limit);
                        if (!ok) break;
                        asm volatile("fence.proxy.async.global;" ::: "memory");
                    } else if (kv == 0 && row0 == 0 && p.kv_ready[seg] != nullptr) {
                        // first tile of a segment that is being copied in: wait for its arrival word,
                        // then order the copy engine's writes before this thread's TMA reads
                        const unsigned int* word = p.kv_ready[seg] + head / max(1, p.kv_ready_heads_per_group);
                        for (int i = 0; i < max(1, p.kv_ready_words) && ok; ++i)
                            ok = global_flag_wait(word + i, p.kv_ready_value, abort_flag, peer_limit);
                        if (!ok) break;
                        asm volatile("fence.proxy.async.global;" ::: "memory");
                    }
                    ok = mbar_wait(smem_u32(&ctl->kv_empty[issued % kStages]), ((issued / kStages) & 1) ^ 1u, abort_flag,
                                   wait_limit);
                    if (ok) load_kv(seg, row0, kv);
                }
                if (!ok) {
                    // Leaving early: let the copies this thread started land first.
                    const long long lim = 40000000ll;  // ~20 ms each, still bounded
                    volatile uint32_t never = 0;
                    for (int t = 0; t < q_issued; ++t) mbar_wait(smem_u32(&ctl->q_full[t]), 0, &never, lim);
                    for (int i = max(0, issued - kStages); i < issued; ++i)
                        mbar_wait(smem_u32(&ctl->kv_full[i % kStages]), (i / kStages) & 1, &never, lim);
                }
            }
        } else if (warp > kMmaWarp) {
            // ------------------------------ head exchange -----------------------------
            if constexpr (kWithExchange) if (p.xchg.enabled) {
                const int xw = warp - kMmaWarp - 1;
                const unsigned int cta_linear = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
                exchange_role(p.xchg, lane, smem + kSmemStage + xw * 2 * kStageBufBytes,
                              smem_raw + (smem - raw_addr) + kSmemStage + xw * 2 * kStageBufBytes,
                              smem_u32(&ctl->xchg_full[xw][0]), abort_flag, wait_limit, &ctl->softmax_done,
                              cta_linear + p.xchg.n_sms < gridDim.x * gridDim.y * gridDim.z);
            }
        } else if (warp == kMmaWarp) {
            // ------------------------------ MMA issuer --------------------------------
            // The whole warp runs this loop converged; umma_* elect one lane per instruction.
            {
                bool ok = true;
                // Descriptors: Q tiles (fixed for the CTA) and ring slot 0 as K (K-major) / V (MN-major).
                const uint64_t q0_desc = umma_smem_desc(smem + kSmemQ, 16, 1024);
                const uint64_t q1_desc = umma_smem_desc(smem + kSmemQ + kTileBytes, 16, 1024);
                const uint64_t k_desc0 = umma_smem_desc(smem + kSmemRing, 16, 1024);
                const uint64_t v_desc0 = umma_smem_desc(smem + kSmemRing, kBoxBytes, 1024);
                const uint32_t bar_full0 = smem_u32(&ctl->kv_full[0]), bar_empty0 = smem_u32(&ctl->kv_empty[0]);
                // Ring slot of K_j is 2j, of V_j is 2j+1.
                auto slot_off16 = [&](int n) { return (uint32_t)(n % kStages) * (kTileBytes >> 4); };
                // A barrier that is already complete still costs the round trip of a try_wait, some
                // 110 clk. Each wait is therefore looked at ahead (`peek`, before the MMAs in front of
                // it are issued) and only waited for when the look found it incomplete.
                const WarpBarriers bars{abort_flag, wait_limit};
                auto wait_uniform = [&](uint32_t bar, uint32_t par) { return bars.wait(bar, par); };
                auto peek = [&](auto... bar_and_parity) { return look_at(bars, bar_and_parity...); };
                auto finish = [&](const Look& l) { return f2k::finish(bars, l); };
                auto bar_full = [&](int n) { return bar_full0 + (n % kStages) * 8; };
                auto par_full = [&](int n) { return (uint32_t)(n / kStages) & 1u; };
                auto release = [&](int n) { umma_commit(bar_empty0 + (n % kStages) * 8); };
                const uint32_t bar_free = smem_u32(&ctl->s_free);
                auto bar_p = [&](int t, int part) { return smem_u32(&ctl->p_full[t][part]); };
                // S = Q_t K_j^T, and its commit.
                auto issue_s = [&](int t, int jj) {
                    tc_fence_after_sync();
                    issue_qk(tmem + kColS, t == 0 ? q0_desc : q1_desc, k_desc0 + slot_off16(2 * jj));
                    umma_commit(smem_u32(&ctl->s_full[t]));
                };
                // O_t (+)= P_t V_jj, issued part by part as the softmax group hands P over; `first` is
                // the look at the first part (and V). The look at the barriers behind it is taken by
                // `next`, in front of the last part's MMAs.
                auto issue_pv = [&](int t, int jj, const Look& first, auto&& next) -> bool {
                    const uint32_t d = tmem + (t == 0 ? kColO0 : kColO1);
                    const uint32_t a = tmem + (t == 0 ? kColP0 : kColP1);
                    const uint64_t v_desc = v_desc0 + slot_off16(2 * jj + 1);
                    if (!finish(first)) return false;
                    auto rest = [&](auto self, auto part) -> bool {
                        constexpr int kPart = decltype(part)::value;
                        Look look{};
                        if constexpr (kPart + 1 < kPParts) look = peek(bar_p(t, kPart + 1), jj & 1);
                        else next();
                        tc_fence_after_sync();
                        issue_pv_part<kPart>(d, a, v_desc, jj > 0 ? 1u : 0u);
                        if constexpr (kPart + 1 < kPParts) {
                            if (!finish(look)) return false;
                            return self(self, std::integral_constant<int, kPart + 1>{});
                        }
                        return true;
                    };
                    if (!rest(rest, std::integral_constant<int, 0>{})) return false;
                    umma_commit(smem_u32(&ctl->pv_done[t]));
                    return true;
                };

                // The S buffer is used in turn: use number u waits for release number u - 1. With two
                // tiles S0_j is use 2j and S1_j use 2j + 1, with one S0_j is use j.
                Look look_s{}, look_p{};
                if (n_kv > 0) {
                    ok = wait_uniform(bar_full(0), par_full(0)) && wait_uniform(smem_u32(&ctl->q_full[0]), 0);
                    if (ok) issue_s(0, 0);
                    if (ok && has_t1) ok = wait_uniform(smem_u32(&ctl->q_full[1]), 0);
                    look_s = peek(bar_free, 0);
                }
                for (int j = 0; j < n_kv && ok; ++j) {
                    if (has_t1) {
                        if (!(ok = finish(look_s))) break;                       // S0_j is in registers
                        if (j > 0) look_p = peek(bar_p(1, 0), (j - 1) & 1);
                        issue_s(1, j);
                    }
                    release(2 * j);
                    auto look_next_s0 = [&] {
                        if (j + 1 < n_kv)
                            look_s = peek(bar_full(2 * j + 2), par_full(2 * j + 2), bar_free, has_t1 ? 1u : (uint32_t)(j & 1));
                    };
                    if (has_t1 && j > 0) {
                        if (!(ok = issue_pv(1, j - 1, look_p, look_next_s0))) break;
                        release(2 * j - 1);
                    } else {
                        look_next_s0();
                    }
                    if (j + 1 < n_kv) {
                        if (!(ok = finish(look_s))) break;                       // K_{j+1}; S1_j is in registers
                    }
                    look_p = peek(bar_full(2 * j + 1), par_full(2 * j + 1), bar_p(0, 0), j & 1);
                    if (j + 1 < n_kv) issue_s(0, j + 1);
                    if (!(ok = issue_pv(0, j, look_p, [&] { if (has_t1) look_s = peek(bar_free, 0); }))) break;
                    if (!has_t1) release(2 * j + 1);
                }
                if (ok && n_kv > 0 && has_t1) {
                    ok = issue_pv(1, n_kv - 1, peek(bar_p(1, 0), (n_kv - 1) & 1), [] {});
                    if (ok) release(2 * n_kv - 1);
                }
                if (!ok) {
                    // Leaving early: wait (bounded) until the MMAs already issued retire, so
                    // tensor memory is idle when it is freed.
                    volatile uint32_t never = 0;
                    __syncwarp();
                    umma_commit(smem_u32(&ctl->drain));
                    mbar_wait(smem_u32(&ctl->drain), 0, &never, 40000000ll);
                }
            }
        }
    } else {
        // ===================== warpgroups 0 and 1: softmax for query tile 0 / 1 =====================
#if F2K_OPT_SETMAXNREG
        setmaxnreg_inc<kRegsSoftmax>();
#endif
        const int t = warp >> 2;                                       // which query tile
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;  // this warp's TMEM lanes
        const uint32_t tS = tmem + lane_base + kColS;
        const uint32_t tP = tmem + lane_base + (t == 0 ? kColP0 : kColP1);
        const uint32_t tO = tmem + lane_base + (t == 0 ? kColO0 : kColO1);
        const float c = p.scale_log2;

        float m_ref = -INFINITY;  // exponent reference, in raw score units
        float l_sum = 0.0f;
        bool ok = true;

        int kv_seg = 0, kv_row0 = 0;
        const int n_iter = (t == 0 || has_t1) ? n_kv : 0;
        for (int j = 0; j < n_iter; ++j) {
            const int valid = min(kTileN, p.kv_len[kv_seg] - kv_row0);
            kv_row0 += kTileN;
            if (kv_row0 >= p.kv_len[kv_seg]) { kv_row0 = 0; ++kv_seg; }

            ok = mbar_wait(smem_u32(&ctl->s_full[t]), j & 1, abort_flag, wait_limit);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();

            // The row is fetched in two halves: the maxima of the first 64 scores are folded while
            // the second 64 are still on their way from tensor memory.
            uint32_t s[128];
            float mx[kMaxChains];
            {
                uint32_t(&s0)[32] = *reinterpret_cast<uint32_t(*)[32]>(&s[0]);
                uint32_t(&s1)[32] = *reinterpret_cast<uint32_t(*)[32]>(&s[32]);
                uint32_t(&s2)[32] = *reinterpret_cast<uint32_t(*)[32]>(&s[64]);
                uint32_t(&s3)[32] = *reinterpret_cast<uint32_t(*)[32]>(&s[96]);
                tmem_ld_x32(tS + 0, s0);
                tmem_ld_x32(tS + 32, s1);
                tmem_wait_ld();
                tmem_ld_x32(tS + 64, s2);
                tmem_ld_x32(tS + 96, s3);
                if (valid < 64) {  // last tile of a segment: keys past its end do not exist
#pragma unroll
                    for (int i = 0; i < 64; ++i)
                        if (i >= valid) s[i] = __float_as_uint(-INFINITY);
                }
                row_max64<true>(&s[0], mx);
                tmem_wait_ld();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctl->s_free));
            }
            if (valid < kTileN) {
#pragma unroll
                for (int i = 64; i < 128; ++i)
                    if (i >= valid) s[i] = __float_as_uint(-INFINITY);
            }
            row_max64<false>(&s[64], mx);
            const float m_tile = row_max_finish(mx);
            // looked at here, needed a few hundred clocks later
            const bool pv_seen = j == 0 || mbar_test(smem_u32(&ctl->pv_done[t]), (j - 1) & 1);

            const bool need = (m_tile - m_ref) * c > kLazyThreshold;
            if (__any_sync(0xffffffffu, need)) {
                const float m_new = fmaxf(m_ref, m_tile);
                const float f = ex2_approx((m_ref - m_new) * c);
                l_sum *= f;
                m_ref = m_new;
                if (j > 0) {
                    // Rescale this row of O in place, once P V of the previous key tile is in.
                    ok = mbar_wait(smem_u32(&ctl->pv_done[t]), (j - 1) & 1, abort_flag, wait_limit);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after_sync();
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t o[32];
                        tmem_ld_x32(tO + q * 32, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                        tmem_st_x32(tO + q * 32, o);
                    }
                }
            }

            // P = 2^(c s - c m_ref), rounded to bf16 into the 64 columns of P_t (two keys per column);
            // the row sum keeps the unrounded values.
            const float neg_mc = -m_ref * c;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
            // A part of P is announced half a chunk after its last store was issued: by then the
            // store has drained, so the wait costs nothing and the special-function unit never
            // idles behind it. Only the last part has to wait for real.
            int pending = -1;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t pk[16];
                exp_chunk16(&s[q * 32], pk, c, neg_mc, sum);
                if (pending >= 0) {
                    tmem_wait_st();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&ctl->p_full[t][0]) + pending * 8);
                    pending = -1;
                }
                exp_chunk16(&s[q * 32 + 16], pk + 8, c, neg_mc, sum);
                if (q == 0 && !__all_sync(0xffffffffu, pv_seen)) {   // P_t of the previous key tile is still being read
                    ok = mbar_wait(smem_u32(&ctl->pv_done[t]), (j - 1) & 1, abort_flag, wait_limit);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                if (q == 0) tc_fence_after_sync();
                tmem_st_x16(tP + q * 16, pk);
                if ((q + 1) % (4 / kPParts) == 0) pending = (q + 1) / (4 / kPParts) - 1;
            }
            if (!ok) break;
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl->p_full[t][kPParts - 1]));
            l_sum += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        }

        // ------------------------------ epilogue ------------------------------------
        if (ok && n_iter > 0) {
            ok = mbar_wait(smem_u32(&ctl->pv_done[t]), (n_iter - 1) & 1, abort_flag, wait_limit);
            ok = __all_sync(0xffffffffu, ok);
        }
        if (ok && n_iter > 0) {
            tc_fence_after_sync();
            const int qt = qt0 + t;
            int seg = 0, row0 = 0, valid = 0;
            locate_tile<kMaxQSeg>(p.q_tile_start, p.q_len, p.n_qseg, qt, seg, row0, valid);
            const int r = (warp & 3) * 32 + lane;  // row inside the tile
            const float inv = 1.0f / (l_sum + 1e-30f);
            // The rows go out through the shared memory of this tile's Q (no MMA reads it any more:
            // the last pv_done comes after all of them). Each thread parks its row there, 16-byte
            // chunk c of row r at chunk position c ^ (r & 15), and the warp then writes its 32 rows
            // two at a time, 16 lanes on the 256 contiguous bytes of one row. To local memory this
            // saves partial-sector writes; to a peer's memory (head exchange) it turns 16-byte
            // packets into 256-byte ones.
            const uint32_t park = smem + kSmemQ + t * kTileBytes;
#pragma unroll
            for (int q = 0; q < 4; q += 2) {
                uint32_t o[64];
                tmem_ld_x32(tO + q * 32, *reinterpret_cast<uint32_t(*)[32]>(&o[0]));   // every lane takes part, valid row or not
                tmem_ld_x32(tO + q * 32 + 32, *reinterpret_cast<uint32_t(*)[32]>(&o[32]));
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 64; i += 8) {
                    uint4 v;
                    v.x = pack_bf16x2(__uint_as_float(o[i + 0]) * inv, __uint_as_float(o[i + 1]) * inv);
                    v.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
                    v.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
                    v.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
                    const int c = q * 4 + (i >> 3);
                    st_shared_v4(park + r * 256 + ((c ^ (r & 15)) << 4), v);
                }
            }
            __syncwarp();
            const int c = lane & 15, half = lane >> 4;
            const long long row_stride = p.o_tok_stride[seg];
            const int first = (warp & 3) * 32 + half;
            __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.o_ptr[seg]) + (long long)bidx * p.o_batch_stride[seg] +
                                 (long long)head * kHeadDim + (long long)(row0 + first) * row_stride + c * 8;
#pragma unroll
            for (int it = 0; it < 16; it += 8) {       // eight rows read back, then written
                uint4 v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int row = first + (it + k) * 2;
                    v[k] = ld_shared_v4(park + row * 256 + ((c ^ (row & 15)) << 4));
                }
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (first + (it + k) * 2 < valid) *reinterpret_cast<uint4*>(out + (it + k) * 2 * row_stride) = v[k];
            }
        }
    }

    if constexpr (kWithExchange)
        if (warp < 8 && lane == 0) atomicAdd(&ctl->softmax_done, 1u);   // (also when the warp left its loop early)

    // ------------------------------ common exit ---------------------------------
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag != 0u && p.status != nullptr)
        atomicOr(p.status, (int)kStatusWaitExpired);
    if (threadIdx.x == 0 && p.done_counter != nullptr)   // all output rows of this CTA are stored (barrier above)
        grid_done_publish(p.done_counter, gridDim.x * gridDim.y * gridDim.z, p.done_flag, p.fail_flag, p.n_done,
                          p.done_value, p.status);
    if (warp == kMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemCols);
    }
}

size_t attn_fwd_smem_bytes() { return kSmemStage + 1024; }                        // plain build
static size_t attn_fwd_smem_bytes_exchange() { return kSmemUsed + 1024; }         // + the exchange's staging area

// Loads the kernel on the current device and raises its shared-memory limit. Called when a
// handle is created, so that the first launch does not have to load code: loading may
// synchronise the device, which must not happen while a stream is parked on a wait that only a
// later call (or another process) can satisfy.
static cudaError_t prepare_on(int& dev) {       // dev: receives the current device
    static bool configured[64] = {};
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && configured[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(attn_fwd_sm100_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)attn_fwd_smem_bytes());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(attn_fwd_sm100_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)attn_fwd_smem_bytes_exchange());
    if (e != cudaSuccess) return e;
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, attn_fwd_sm100_kernel<false>);
    if (e != cudaSuccess) return e;
    e = cudaFuncGetAttributes(&attr, attn_fwd_sm100_kernel<true>);
    if (e != cudaSuccess) return e;
    if (dev < 64) configured[dev] = true;
    return cudaSuccess;
}

cudaError_t attn_fwd_prepare() {
    int dev = 0;
    return prepare_on(dev);
}

cudaError_t attn_fwd_launch(const AttnParams& params, cudaStream_t stream) {
    int dev = 0;
    cudaError_t e = prepare_on(dev);
    if (e != cudaSuccess) return e;
    AttnParams p = params;
    if (p.wait_limit_clk <= 0) p.wait_limit_clk = kDefaultWaitClk;
    if (p.peer_wait_limit_clk <= 0) p.peer_wait_limit_clk = kDefaultPeerWaitClk;
    // An in-CTA wait may sit behind a peer wait of the loader (a softmax group waits for S, the MMA
    // warp for K, the loader for the word), so it has to outlast it where peer words are in use.
    bool peer_words = false;
    for (int i = 0; i < kMaxKvSeg; ++i) peer_words |= p.kv_ready[i] != nullptr;
    for (int i = 0; i < kMaxQSeg; ++i) peer_words |= p.q_ready[i] != nullptr;
    if (peer_words) p.wait_limit_clk += p.peer_wait_limit_clk;
    p.waits_for_words = peer_words ? 1 : 0;
    dim3 grid(p.n_heads, (p.n_q_tiles + 1) / 2, p.batch);
    if (!p.grid_head_fastest) {
        int sms = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        p.plan = cta_plan(p.n_q_tiles, p.n_heads * p.batch, sms);
        grid = dim3(p.plan.n_ctas);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.stream = stream;
    if (p.xchg.enabled) {
        cfg.dynamicSmemBytes = attn_fwd_smem_bytes_exchange();
        return cudaLaunchKernelEx(&cfg, attn_fwd_sm100_kernel<true>, p);
    }
    // May start while the kernel in front of it (the prologue) drains: the loader waits for its end.
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = peer_words ? 0 : 1;
    cfg.dynamicSmemBytes = attn_fwd_smem_bytes();
    return cudaLaunchKernelEx(&cfg, attn_fwd_sm100_kernel<false>, p);
}

}  // namespace f2k
