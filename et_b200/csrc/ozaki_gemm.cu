// FP64-accurate GEMM on the int8 tensor cores of sm_100a (Ozaki's error-free slicing).
//
// Every row r of op(A) is scaled by 2^-ea_r (ea_r: the exponent of the power of two just above
// max_k |A_rk|) and cut into S digits of 7 bits,
//     A_rk = 2^ea_r sum_t DA_t[r,k] 2^(-7(t+1)),   DA_t integers in [-127, 127],
// exactly up to the truncation of the last digit (relative 2^-7S); the columns of op(B) the same
// with eb_c.  Then
//     C_rc = 2^(ea_r + eb_c) sum_{t,u} 2^(-7(t+u+2)) sum_k DA_t[r,k] DB_u[k,c],
// and every digit product sum_k is exact in int32: |d d'| <= 127^2, and an accumulator takes at
// most 7 products (one diagonal d = t + u) over a K chunk of at most 16384, 7 * 16384 * 127^2 < 2^31.
// Products with t + u <= S - 1 are kept; the dropped ones lie below the last digit of either
// operand.  With S = 7 the 28 products reproduce an FP64 GEMM to ~1e-14 of the largest output.
//
// Kernel: persistent, warp specialised like the split-BF16 GEMM (warp 0 issues TMA loads, warp 1
// issues tcgen05.mma.kind::i8 with int32 accumulation in TMEM, warps 2-5 drain), 128 x 128 output
// tiles, K blocks of 64 int8 (64-byte swizzled rows).  A stage holds the digit tiles of both
// operands for one K block (up to 7 + 7 tiles of 8 KB), two stages.  The diagonals of a tile are
// accumulated in passes of at most four (4 x 128 TMEM columns = all 512): pass 0 takes d = 0..3
// (digits 0..3 of both operands), pass 1 takes d = 4..S-1 (all digits).  The epilogue adds
// 2^(-7(d+2)) acc_d in FP64, scales by alpha 2^(ea_r + eb_c) and accumulates into the FP64 output;
// one CTA takes all units (K chunk, pass) of a tile in order, so the sum is deterministic.  That form
// serves operands of at most 128 rows; all others run on CTA pairs (ozaki_pair_kernel).  Every
// mbarrier wait is bounded and reports to the caller's error word, as in the split-BF16 GEMM.
#include <cuda.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "ozaki_gemm.cuh"
#include "tc_common.cuh"

namespace ccsd {

using namespace tc;

namespace {

constexpr int OBM = 128, OBN = 128, OBK = 64;            // tile; K block = one 64-byte row of int8
constexpr int SLOTS = 7;                                 // digit tiles per operand in a stage
constexpr int OSTAGES = 2;
constexpr int OTHREADS = 192, OEPI = 128;
constexpr int A_TILE = OBM * OBK, B_TILE = OBN * OBK;    // bytes
constexpr int OSTAGE_BYTES = SLOTS * (A_TILE + B_TILE);
constexpr int OSMEM = OSTAGES * OSTAGE_BYTES + 1024 + 256;
constexpr uint32_t OTMEM_COLS = 512;                     // four 128-column int32 accumulators
constexpr int MAX_DIAG_PER_PASS = 4;
constexpr int OK_CHUNK = 16384;                          // K elements per exact int32 accumulation
constexpr long long OWAIT_CYCLES = 4000000000ll;
// kind::i8 instruction descriptor: S8 x S8 -> S32, both K-major, M = 128, N = 128
constexpr uint32_t IDESC_I8 = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OBN >> 3) << 17) |
                              ((uint32_t)(OBM >> 4) << 24);
static_assert(OSMEM <= 232448, "shared memory of the Ozaki GEMM");
static_assert(7 * OK_CHUNK * 127 * 127 < 2147483647ll, "int32 accumulation must stay exact");
constexpr int ERR_PRODUCER = 1, ERR_MMA_FULL = 2, ERR_EPILOGUE = 3, ERR_MMA_ACC = 4, ERR_DONE = 5, ERR_DRAIN = 6;

__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(IDESC_I8), "r"(accumulate));
}

struct OzMap {
    int num_mt, num_nt, group_m;
    int nk_all;          // K blocks of 64
    int kc;              // K blocks per chunk
    int nchunks;
    int digits;          // S
    int npass;           // 1 (S <= 4) or 2
    int M, N;
    long long ldc;
    double alpha, beta;
    double *C;
    const int *ea, *eb;  // row exponents of op(A), column exponents of op(B)
    int *err;
    long long wait_cycles;
    int bm = OBM, bn = OBN;   // tile (256 rows and up to 256 columns for a CTA pair)
    __device__ __forceinline__ void tile(int t, int &m0, int &n0) const {
        const int per_group = group_m * num_nt;
        const int grp = t / per_group, in = t - grp * per_group;
        const int first_m = grp * group_m;
        const int gsz = min(group_m, num_mt - first_m);
        m0 = (first_m + in % gsz) * bm;
        n0 = (in / gsz) * bn;
    }
    // diagonals [d0, d1) of pass p and the digits they need
    __device__ __forceinline__ void pass(int p, int &d0, int &d1, int &nd) const {
        d0 = p == 0 ? 0 : MAX_DIAG_PER_PASS;
        d1 = p == 0 ? min(digits, MAX_DIAG_PER_PASS) : digits;
        nd = min(d1, digits);   // digits 0..nd-1 of both operands (t, u <= d1 - 1)
    }
};

// The MMAs of one K block for the diagonals [D0, D1) of S-digit operands, fully unrolled: the
// descriptors of digit q sit a constant offset from those of digit 0 (a 16-byte unit in the start
// field per 16 bytes, tiles of A_TILE / B_TILE bytes), so issuing an MMA costs a few integer adds.  An
// int8 MMA of 128 x 128 x 32 lasts ~64 tensor cycles; rebuilding descriptors per MMA had the single
// issuing thread, not the tensor pipe, set the pace.
template <int S, int D0, int D1>
__device__ __forceinline__ void issue_kblock(uint32_t tmem, uint64_t a0, uint64_t b0, bool first_kb) {
#pragma unroll
    for (int kk = 0; kk < OBK / 32; kk++) {
#pragma unroll
        for (int d = D0; d < D1; d++) {
#pragma unroll
            for (int t = (d - S + 1 > 0 ? d - S + 1 : 0); t <= (d < S - 1 ? d : S - 1); t++) {
                const int u = d - t;
                const bool first = kk == 0 && t == (d - S + 1 > 0 ? d - S + 1 : 0);
                mma_i8(tmem + (uint32_t)((d - D0) * OBN), a0 + (uint64_t)(t * (A_TILE >> 4) + kk * 2),
                       b0 + (uint64_t)(u * (B_TILE >> 4) + kk * 2), (first_kb && first) ? 0u : 1u);
            }
        }
    }
}

template <int S>
__device__ __forceinline__ void issue_pass(int p, uint32_t tmem, const uint8_t *st, bool first_kb) {
    const uint64_t a0 = smem_desc_k<64>(st, 0), b0 = smem_desc_k<64>(st + SLOTS * A_TILE, 0);
    if (p == 0)
        issue_kblock<S, 0, (S < MAX_DIAG_PER_PASS ? S : MAX_DIAG_PER_PASS)>(tmem, a0, b0, first_kb);
    else if constexpr (S > MAX_DIAG_PER_PASS)
        issue_kblock<S, MAX_DIAG_PER_PASS, S>(tmem, a0, b0, first_kb);
}

template <int S>
__global__ void __launch_bounds__(OTHREADS, 1)
ozaki_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OzMap map,
                  int num_tiles) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + OSTAGES * OSTAGE_BYTES);
    uint64_t *empty = full + OSTAGES;
    uint64_t *acc_full = empty + OSTAGES;
    uint64_t *acc_empty = acc_full + 1;
    uint64_t *done = acc_empty + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < OSTAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, OEPI);
        mbar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(OTMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // producer: for every (tile, chunk, pass) unit, the digit tiles of each K block
            int g = 0;
            int issued[OSTAGES] = {};
            for (int t = blockIdx.x; t < num_tiles && !*abort_flag; t += gridDim.x) {
                int m0, n0;
                map.tile(t, m0, n0);
                for (int c = 0; c < map.nchunks && !*abort_flag; c++) {
                    const int kb0 = c * map.kc, kb1 = min(map.nk_all, kb0 + map.kc);
                    for (int p = 0; p < map.npass && !*abort_flag; p++) {
                        int d0, d1, nd;
                        map.pass(p, d0, d1, nd);
                        for (int kb = kb0; kb < kb1; kb++, g++) {
                            const int s = g % OSTAGES;
                            if (!mbar_wait(&empty[s], ((g / OSTAGES) & 1) ^ 1, map.wait_cycles) || *abort_flag) {
                                record_error(map.err, ERR_PRODUCER);
                                *abort_flag = 1;
                                break;
                            }
                            issued[s]++;
                            uint8_t *st = smem + s * OSTAGE_BYTES;
                            mbar_expect_tx(&full[s], (uint32_t)nd * (A_TILE + B_TILE));
                            for (int q = 0; q < nd; q++) {
                                tma_load_3d(&tmA, &full[s], st + q * A_TILE, kb * OBK, m0, q);
                                tma_load_3d(&tmB, &full[s], st + SLOTS * A_TILE + q * B_TILE, kb * OBK, n0, q);
                            }
                        }
                    }
                }
            }
            for (int s = 0; s < OSTAGES; s++)
                if (issued[s] && !mbar_wait(&full[s], (issued[s] - 1) & 1, map.wait_cycles))
                    record_error(map.err, ERR_DRAIN);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // MMA issuer: one unit at a time into the (up to four) diagonal accumulators
            int g = 0, uc = 0;
            for (int t = blockIdx.x; t < num_tiles && !*abort_flag; t += gridDim.x) {
                for (int c = 0; c < map.nchunks && !*abort_flag; c++) {
                    const int kb0 = c * map.kc, kb1 = min(map.nk_all, kb0 + map.kc);
                    for (int p = 0; p < map.npass && !*abort_flag; p++, uc++) {
                        int d0, d1, nd;
                        map.pass(p, d0, d1, nd);
                        if (!mbar_wait(acc_empty, (uc & 1) ^ 1, map.wait_cycles)) {
                            record_error(map.err, ERR_MMA_ACC);
                            *abort_flag = 1;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        for (int kb = kb0; kb < kb1; kb++, g++) {
                            const int s = g % OSTAGES;
                            if (!mbar_wait(&full[s], (g / OSTAGES) & 1, map.wait_cycles) || *abort_flag) {
                                record_error(map.err, ERR_MMA_FULL);
                                *abort_flag = 1;
                                break;
                            }
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            issue_pass<S>(p, tmem, smem + s * OSTAGE_BYTES, kb == kb0);
                            mma_commit(&empty[s]);
                        }
                        mma_commit(acc_full);
                    }
                }
            }
            mma_commit(done);
        }
    } else {
        // epilogue: warp w drains TMEM lanes 32 (w % 4) .. +31, one output row per thread
        const int quarter = warp & 3;
        int uc = 0;
        bool aborted = false;
        for (int t = blockIdx.x; t < num_tiles && !aborted; t += gridDim.x) {
            int m0, n0;
            map.tile(t, m0, n0);
            const int row = m0 + quarter * 32 + lane;
            const double row_scale = row < map.M ? map.alpha * exp2((double)map.ea[row]) : 0.0;
            for (int c = 0; c < map.nchunks && !aborted; c++) {
                for (int p = 0; p < map.npass; p++, uc++) {
                    int d0, d1, nd;
                    map.pass(p, d0, d1, nd);
                    bool ok = !*abort_flag && mbar_wait(acc_full, uc & 1, map.wait_cycles);
                    __syncwarp();
                    if (!ok || *abort_flag) {
                        record_error(map.err, ERR_EPILOGUE);
                        *abort_flag = 1;
                        aborted = true;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const bool first = (c == 0 && p == 0);
                    const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
                    for (int cc = 0; cc < OBN; cc += 16) {
                        double v[16];
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = 0.0;
                        for (int d = d0; d < d1; d++) {
                            uint32_t r[16];
                            tmem_ld16u(base + (uint32_t)((d - d0) * OBN + cc), r);
                            const double w = exp2(-7.0 * (double)(d + 2));
#pragma unroll
                            for (int j = 0; j < 16; j++) v[j] += w * (double)(int)r[j];
                        }
                        if (row < map.M) {
                            double *out = map.C + (long long)(n0 + cc) * map.ldc + row;
                            double old[16];
#pragma unroll
                            for (int j = 0; j < 16; j++) {
                                const bool in = n0 + cc + j < map.N;
                                old[j] = (in && (!first || map.beta != 0.0)) ? __ldcg(out + (long long)j * map.ldc) : 0.0;
                            }
#pragma unroll
                            for (int j = 0; j < 16; j++) {
                                const int col = n0 + cc + j;
                                if (col < map.N) {
                                    const double x = row_scale * exp2((double)map.eb[col]) * v[j];
                                    out[(long long)j * map.ldc] = first ? x + map.beta * old[j] : x + old[j];
                                }
                            }
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(acc_empty)) : "memory");
                }
            }
        }
    }
    __syncthreads();
    if (!mbar_wait(done, 0, map.wait_cycles)) record_error(map.err, ERR_DONE);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OTMEM_COLS));
    }
}

// The digit GEMM on a pair of CTAs (a cluster of two) with N tiles of up to 256 columns: one cta_group::2 MMA of
// M = 256 (each CTA's 128 rows of A) and N = bn (half of B's rows staged by each CTA).
//
// What bounds it is shared memory, 128 bytes a cycle: an MMA of N = bn reads 4 KB of A and 32 bn bytes of B in
// bn / 2 cycles, so a 128-wide tile, its two passes staging ten digit tiles a K block on top, kept the int8
// pipe 67 % active.  At 256 columns the MMAs need 96 bytes a cycle and the staging 37, but TMEM then holds two
// accumulators: wide tiles (more than 128 columns) take the diagonals two at a time, each such unit staging the
// digits up to its higher diagonal (2 + 4 + 6 digit tiles a K block for six digits); narrow ones four.  What
// keeps the rate of wide tiles up at L2's latency is bytes in flight: their ring's slots hold one digit of A and
// of B, the products of a K block run from its highest digit down, and a slot is freed when its digit has taken
// part for the last time (freeing a whole K block at once left 96 of the 192 KB idle: 2.1 instead of 2.7 POPS
// at 4000^3).  Narrow tiles have too few cycles of products per digit to hide ten waits and commits a K block:
// their slots hold all its digits (4000 x 400 x 40000 1.68 ms with a slot per digit, 1.27 so).  Eight epilogue
// warps drain a unit (the accumulators are not double-buffered), old values a step ahead.
//
// The sums keep the order of the single-CTA kernel, diagonals 0..3 and then 4..S-1 per K chunk: the sum of a
// pass is exact in FP64 (four diagonals span 52 bits), so the units of a pass before its last leave their
// share in a scratch of the CTA and the last adds it, and only then the scaled sum is rounded into the output.
// With 6 digits, against 128-wide pair tiles with one K block a stage: 10240 x 10240 x 1200 2.70 ms (3.94), 4000^3
// 1.02 ms (1.27), 4000 x 400 x 40000 1.27 ms (1.36), 2304 x 256 x 16384 0.48 ms (0.51).
constexpr int WBN = 256;
constexpr int WSLOTS = 20;                                        // slots at most
constexpr int WEPI_WARPS = 8, WTHREADS = 64 + 32 * WEPI_WARPS;
// WIDE: tiles of more than 128 columns
template <bool WIDE>
struct PairRing {
    static constexpr int BYTES = WIDE ? 12 * (A_TILE + (WBN / 2) * OBK) : 18 * (A_TILE + (WBN / 4) * OBK);
    static constexpr int SMEM = BYTES + 1024 + 512 + WEPI_WARPS * (WBN / 2) * 8;
};
static_assert(PairRing<true>::SMEM <= 232448 && PairRing<false>::SMEM <= 232448, "shared memory of the pair digit GEMM");
constexpr uint32_t WIDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 4) << 24);

__device__ __forceinline__ void mma_i8_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// The digits of a K block in the order their slots are filled (and freed): the highest, 0, the second
// highest, 1, ...
__device__ __forceinline__ constexpr int digit_at(int pos, int nd) { return pos & 1 ? pos / 2 : nd - 1 - pos / 2; }

// position in the ring of slots
struct Ring {
    int n_slots;
    int slot = 0;
    uint32_t phase = 0;   // parity of the slot's present use
    __device__ __forceinline__ void advance(int n) {
        slot += n;
        if (slot >= n_slots) {
            slot -= n_slots;
            phase ^= 1;
        }
    }
    __device__ __forceinline__ Ring ahead(int n) const {
        Ring r = *this;
        r.advance(n);
        return r;
    }
};

// Waits for one K block (from ring position r) and issues its products of the NDIAG diagonals
// ND - NDIAG .. ND - 1 (accumulator d - (ND - NDIAG), each `width` columns), from the products of the highest
// digit down: step k pairs digit ND - 1 - k with the lower ones, so digit ND - 1 - k is free after step k and
// digit j after step j + NDIAG - 1.  BLOCK: the K block's digits share one slot, slot_bytes apart; else each has
// its own.  False when a wait ran out.
template <int ND, int NDIAG, bool BLOCK>
__device__ __forceinline__ bool issue_unit(uint32_t tmem, uint32_t width, uint64_t desc0, int slot_bytes, int digit_bytes,
                                           uint64_t *full, uint64_t *empty, const Ring &r, uint32_t idesc, bool first_kb,
                                           long long limit) {
    constexpr int D1 = ND - 1, D0 = ND - NDIAG, STEPS = D1 - (D0 + 1) / 2 + 1;
    uint64_t da[ND];
    bool ok = true;
    if constexpr (BLOCK) {
        ok = mbar_wait(&full[r.slot], r.phase, limit);
#pragma unroll
        for (int pos = 0; pos < ND; pos++)
            da[digit_at(pos, ND)] = desc0 + (uint64_t)((r.slot * slot_bytes + pos * digit_bytes) >> 4);
    }
#pragma unroll
    for (int step = 0; step < STEPS; step++) {
        const int hi = D1 - step;
        if constexpr (!BLOCK) {
#pragma unroll
            for (int pos = 2 * step; pos < 2 * step + 2; pos++) {
                if (pos < ND) {
                    const Ring p = r.ahead(pos);
                    ok = ok && mbar_wait(&full[p.slot], p.phase, limit);
                    da[digit_at(pos, ND)] = desc0 + (uint64_t)(p.slot * (slot_bytes >> 4));
                }
            }
        }
        if (!ok) return false;
        if (step == 0 || !BLOCK) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int d = D1; d >= D0; d--) {
            const int lo = d - hi;
            if (lo < 0 || lo > hi) continue;
            const uint32_t acc = tmem + (uint32_t)(d - D0) * width;
#pragma unroll
            for (int kk = 0; kk < OBK / 32; kk++) {
                // the first product of the unit into this accumulator overwrites it
                const uint32_t add = first_kb && kk == 0 && lo == 0 ? 0u : 1u;
                mma_i8_pair(acc, da[hi] + (uint64_t)(kk * 2), da[lo] + (uint64_t)((A_TILE >> 4) + kk * 2), idesc, add);
                if (lo < hi)
                    mma_i8_pair(acc, da[lo] + (uint64_t)(kk * 2), da[hi] + (uint64_t)((A_TILE >> 4) + kk * 2), idesc, 1u);
            }
        }
        if constexpr (!BLOCK) {
            // positions 2 step (digit ND - 1 - step) and 2 (step - NDIAG + 1) + 1 (digit step - NDIAG + 1)
            if (2 * step < ND) mma_commit_pair(&empty[r.ahead(2 * step).slot]);
            const int low = 2 * (step - NDIAG + 1) + 1;
            if (low > 0 && low < ND) mma_commit_pair(&empty[r.ahead(low).slot]);
        }
    }
    if constexpr (BLOCK) {
        mma_commit_pair(&empty[r.slot]);
    } else {
        // what the last step leaves
#pragma unroll
        for (int pos = 0; pos < ND; pos++) {
            const bool freed = pos % 2 == 0 ? pos / 2 < STEPS : pos / 2 + NDIAG - 1 < STEPS;
            if (!freed) mma_commit_pair(&empty[r.ahead(pos).slot]);
        }
    }
    return true;
}

// Units of an S-digit product: wide tiles take the diagonals two at a time, others four at a time; unit u stages
// the digits up to its highest diagonal.
template <bool WIDE>
__device__ __forceinline__ int unit_digits(int u, int digits) { return min((WIDE ? 2 : 4) * (u + 1), digits); }

template <bool WIDE>
__global__ void __launch_bounds__(WTHREADS, 1)
ozaki_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OzMap map,
                  int num_tiles, double *__restrict__ scratch) {
    constexpr int RING = PairRing<WIDE>::BYTES, WIDTH = WIDE ? WBN : WBN / 2;   // columns of an accumulator
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + RING);
    uint64_t *empty = full + WSLOTS;
    uint64_t *acc_full = empty + WSLOTS;
    uint64_t *acc_empty = acc_full + 1;   // used on CTA 0
    uint64_t *done = acc_empty + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    double *col_scales = reinterpret_cast<double *>(smem + RING + 512);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool lead = rank == 0;
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < WSLOTS; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 2 * WEPI_WARPS);   // one arrival per epilogue warp of each CTA
        mbar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(OTMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    constexpr int per = WIDE ? 2 : 4;   // diagonals of a unit
    const int half = map.bn / 2, units = (map.digits + per - 1) / per;
    // a slot holds one digit of both operands, or all digits of a K block of a narrow tile
    const int digit_bytes = A_TILE + half * OBK, slot_bytes = WIDE ? digit_bytes : map.digits * digit_bytes;
    const int n_slots = min(WSLOTS, RING / slot_bytes);

    if (warp == 0) {
        if (lane == 0) {
            // producer of this CTA: for every (tile, chunk, unit) the digits of each K block
            const uint32_t bytes = 2u * (uint32_t)digit_bytes;
            Ring r{n_slots};
            int g = 0;
            for (int t = pair; t < num_tiles && !*abort_flag; t += npairs) {
                int m0, n0;
                map.tile(t, m0, n0);
                const int ma = m0 + OBM * (int)rank, nb = n0 + half * (int)rank;
                for (int c = 0; c < map.nchunks && !*abort_flag; c++) {
                    const int kb0 = c * map.kc, kb1 = min(map.nk_all, kb0 + map.kc);
                    for (int u = 0; u < units && !*abort_flag; u++) {
                        const int nd = unit_digits<WIDE>(u, map.digits), per_slot = WIDE ? 1 : nd;
                        for (int kb = kb0; kb < kb1 && !*abort_flag; kb++) {
                            for (int pos = 0; pos < nd; pos += per_slot) {
                                if (!mbar_wait(&empty[r.slot], r.phase ^ 1, map.wait_cycles)) {
                                    record_error(map.err, ERR_PRODUCER);
                                    *abort_flag = 1;
                                    break;
                                }
                                uint8_t *st = smem + r.slot * slot_bytes;
                                if (lead) mbar_expect_tx(&full[r.slot], (uint32_t)per_slot * bytes);
                                for (int p = pos; p < pos + per_slot; p++, st += digit_bytes) {
                                    const int q = digit_at(p, nd);
                                    tma_load_3d_pair(&tmA, &full[r.slot], st, kb * OBK, ma, q);
                                    tma_load_3d_pair(&tmB, &full[r.slot], st + A_TILE, kb * OBK, nb, q);
                                }
                                r.advance(1);
                                g++;
                            }
                        }
                    }
                }
            }
            // CTA 0 waits for the last load of each slot (both CTAs' bytes land on its barrier); CTA 1 keeps its
            // shared memory until the final cluster barrier, which CTA 0 reaches after this
            if (lead)
                for (int s = 0; s < n_slots && s < g; s++)
                    if (!mbar_wait(&full[s], ((g - 1 - s) / n_slots) & 1, map.wait_cycles)) record_error(map.err, ERR_DRAIN);
        }
    } else if (warp == 1) {
        if (lane == 0 && lead) {
            const uint32_t idesc = WIDESC | ((uint32_t)(map.bn >> 3) << 17);
            const uint64_t desc0 = smem_desc_k<64>(smem, 0);
            Ring r{n_slots};
            int uc = 0;
            for (int t = pair; t < num_tiles && !*abort_flag; t += npairs) {
                for (int c = 0; c < map.nchunks && !*abort_flag; c++) {
                    const int kb0 = c * map.kc, kb1 = min(map.nk_all, kb0 + map.kc);
                    for (int u = 0; u < units && !*abort_flag; u++, uc++) {
                        const int nd = unit_digits<WIDE>(u, map.digits), diags = nd - per * u;
                        if (!mbar_wait(acc_empty, (uc & 1) ^ 1, map.wait_cycles)) {
                            record_error(map.err, ERR_MMA_ACC);
                            *abort_flag = 1;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        for (int kb = kb0; kb < kb1; kb++) {
                            const bool first = kb == kb0;
                            bool ok = false;
#define OZ_UNIT(ND, NDIAG)                                                                                        \
    case 8 * ND + NDIAG:                                                                                          \
        ok = issue_unit<ND, NDIAG, !WIDE>(tmem, WIDTH, desc0, slot_bytes, digit_bytes, full, empty, r, idesc,     \
                                          first, map.wait_cycles);                                                \
        break;
                            if constexpr (WIDE) {
                                switch (8 * nd + diags) {   // 2, 4, 6 digits, or the last diagonal of 5, 7
                                    OZ_UNIT(2, 2) OZ_UNIT(4, 2) OZ_UNIT(6, 2) OZ_UNIT(5, 1) OZ_UNIT(7, 1)
                                }
                            } else {
                                switch (8 * nd + diags) {   // four digits, then the rest of 5, 6 or 7
                                    OZ_UNIT(4, 4) OZ_UNIT(5, 1) OZ_UNIT(6, 2) OZ_UNIT(7, 3)
                                }
                            }
#undef OZ_UNIT
                            if (!ok || *abort_flag) {
                                record_error(map.err, ERR_MMA_FULL);
                                *abort_flag = 1;
                                break;
                            }
                            r.advance(WIDE ? nd : 1);
                        }
                        mma_commit_pair(acc_full);
                    }
                }
            }
            mma_commit_pair(done);
        }
    } else {
        // epilogue: this CTA's 128 rows; warp w drains TMEM lanes 32 (w % 4) .. +31, the first four warps the
        // lower half of the columns
        const int quarter = warp & 3, e = warp - 2;
        double *scale = col_scales + e * (WBN / 2);
        const int cbeg = e < 4 ? 0 : (map.bn / 32) * 16, cend = e < 4 ? (map.bn / 32) * 16 : map.bn;
        // this thread's column of the CTA's scratch, 128 rows a column
        double *part = scratch + (size_t)blockIdx.x * OBM * WBN + quarter * 32 + lane;
        int uc = 0;
        bool aborted = false;
        for (int t = pair; t < num_tiles && !aborted; t += npairs) {
            int m0, n0;
            map.tile(t, m0, n0);
            const int row = m0 + OBM * (int)rank + quarter * 32 + lane;
            const bool live = row < map.M;
            const double row_scale = live ? map.alpha * exp2((double)map.ea[row]) : 0.0;
            __syncwarp();
            for (int i = lane; i < cend - cbeg; i += 32)
                scale[i] = n0 + cbeg + i < map.N ? exp2((double)map.eb[n0 + cbeg + i]) : 0.0;
            __syncwarp();
            double *out = map.C + (long long)n0 * map.ldc + row;
            for (int c = 0; c < map.nchunks && !aborted; c++) {
                for (int u = 0; u < units; u++, uc++) {
                    bool ok = !*abort_flag && mbar_wait(acc_full, uc & 1, map.wait_cycles);
                    __syncwarp();
                    if (!ok || *abort_flag) {
                        record_error(map.err, ERR_EPILOGUE);
                        *abort_flag = 1;
                        aborted = true;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const int d_lo = per * u, diags = unit_digits<WIDE>(u, map.digits) - d_lo;
                    // of a pass of four diagonals, the first unit and the last
                    const bool opens = d_lo % MAX_DIAG_PER_PASS == 0;
                    const bool closes = !WIDE || u == units - 1 || u == 1;
                    const bool first = c == 0 && d_lo < MAX_DIAG_PER_PASS;      // beta applies to the first pass
                    const bool read_c = closes && live && (!first || map.beta != 0.0);
                    const double w0 = exp2(-7.0 * (double)(d_lo + 2));
                    const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16);
                    double ca[8], cb[8], pa[8], pb[8];   // output and scratch values of this step and the next
                    auto fetch = [&](int cc, double (&o)[8], double (&p)[8]) {
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            o[j] = read_c && cc < cend && n0 + cc + j < map.N ? __ldcg(out + (long long)(cc + j) * map.ldc) : 0.0;
                            p[j] = !opens && cc < cend ? __ldcg(part + (size_t)(cc + j) * OBM) : 0.0;
                        }
                    };
                    auto emit = [&](int cc, const double (&o)[8], const double (&p)[8]) {
                        uint32_t acc[MAX_DIAG_PER_PASS][8];
#pragma unroll
                        for (int h = 0; h < MAX_DIAG_PER_PASS; h++)   // diags is the same for every lane
                            if (h < diags) tmem_ld8u_async(base + (uint32_t)(h * WIDTH + cc), acc[h]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        double v[8], w = w0;
#pragma unroll
                        for (int j = 0; j < 8; j++) v[j] = p[j];
#pragma unroll
                        for (int h = 0; h < MAX_DIAG_PER_PASS; h++) {
                            if (h < diags) {
                                tmem_loaded8u(acc[h]);
#pragma unroll
                                for (int j = 0; j < 8; j++) v[j] += w * (double)(int)acc[h][j];
                                w *= 1.0 / 128.0;
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            if (!closes) {
                                part[(size_t)(cc + j) * OBM] = v[j];
                            } else if (live && n0 + cc + j < map.N) {
                                const double x = row_scale * scale[cc - cbeg + j] * v[j];
                                out[(long long)(cc + j) * map.ldc] = first ? x + map.beta * o[j] : x + o[j];
                            }
                        }
                    };
                    fetch(cbeg, ca, pa);
#pragma unroll 1
                    for (int cc = cbeg; cc < cend; cc += 16) {
                        fetch(cc + 8, cb, pb);
                        emit(cc, ca, pa);
                        fetch(cc + 16, ca, pa);
                        emit(cc + 8, cb, pb);
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) arrive_cta0(acc_empty);
                }
            }
        }
    }
    __syncthreads();
    if (!mbar_wait(done, 0, map.wait_cycles)) record_error(map.err, ERR_DONE);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OTMEM_COLS));
    }
}

// Row exponents of a strided FP64 view (element (r, k) at src[r sr + k sk]): e[r] = the exponent of
// the power of two just above max_k |x_rk| (frexp), by atomicMax over K slices of 32 x 32 tiles
// (e must start below any exponent: all-zero rows keep the start value).
__global__ void oz_rowexp_kernel(const double *__restrict__ src, long long sr, long long sk, int R, int K,
                                 int *__restrict__ e) {
    __shared__ double tile[32][33];
    __shared__ double red[8][33];
    const int r0 = blockIdx.x * 32, tx = threadIdx.x, ty = threadIdx.y;
    const bool k_fast = (sk == 1);
    double m = 0.0;
    for (int k0 = blockIdx.y * 32; k0 < K; k0 += gridDim.y * 32) {
        for (int i = ty; i < 32; i += 8) {
            int r, k;
            if (k_fast) {
                r = r0 + i;
                k = k0 + tx;
            } else {
                r = r0 + tx;
                k = k0 + i;
            }
            const double x = (r < R && k < K) ? src[(long long)r * sr + (long long)k * sk] : 0.0;
            if (k_fast) tile[i][tx] = x;
            else tile[tx][i] = x;
        }
        __syncthreads();
        for (int i = ty; i < 32; i += 8) m = fmax(m, fabs(tile[tx][i]));
        __syncthreads();
    }
    red[ty][tx] = m;
    __syncthreads();
    if (ty == 0 && r0 + tx < R) {
        for (int j = 1; j < 8; j++) m = fmax(m, red[j][tx]);
        if (m > 0.0) {
            int ex;
            frexp(m, &ex);
            atomicMax(&e[r0 + tx], ex);
        }
    }
}

// Digits of the scaled rows: x 2^-e = sum_t d_t 2^(-7(t+1)), d_t = trunc of the remaining fraction
// times 128 (exact in FP64), written as int8 planes [digit][Rp][Kp], K-major, zero padded.
__global__ void oz_digits_kernel(const double *__restrict__ src, long long sr, long long sk, int R, int K, int Rp,
                                 int Kp, int digits, const int *__restrict__ e, int8_t *__restrict__ out) {
    __shared__ double tile[32][33];
    const int r0 = blockIdx.x * 32, tx = threadIdx.x, ty = threadIdx.y;
    const bool k_fast = (sk == 1);
    const size_t plane = (size_t)Rp * Kp;
    for (int k0 = blockIdx.y * 32; k0 < Kp; k0 += gridDim.y * 32) {
        for (int i = ty; i < 32; i += 8) {
            int r, k;
            if (k_fast) {
                r = r0 + i;
                k = k0 + tx;
            } else {
                r = r0 + tx;
                k = k0 + i;
            }
            const double x = (r < R && k < K) ? src[(long long)r * sr + (long long)k * sk] : 0.0;
            if (k_fast) tile[i][tx] = x;
            else tile[tx][i] = x;
        }
        __syncthreads();
        for (int i = ty; i < 32; i += 8) {
            const int r = r0 + i, k = k0 + tx;
            if (r < Rp && k < Kp) {
                const int er = (r < R) ? e[r] : 0;
                double y = (r < R && er > -1100) ? ldexp(tile[i][tx], -er) : 0.0;   // |y| < 1
                const size_t o = (size_t)r * Kp + k;
                for (int t = 0; t < digits; t++) {
                    y *= 128.0;
                    const double d = trunc(y);
                    y -= d;
                    out[t * plane + o] = (int8_t)(int)d;
                }
            }
        }
        __syncthreads();
    }
}

// The same two steps for operands whose K index is contiguous (element (r, k) at src[r sr + k]):
// no transpose is needed, so the rows stream through with 16-byte loads.  One warp per (row, K
// slice) for the exponents; for the digits each thread takes 8 consecutive k of a row and writes one
// 8-byte word per digit plane.
__global__ void oz_rowexp_kfast_kernel(const double *__restrict__ src, long long sr, int R, int K, int kslices,
                                       int *__restrict__ e) {
    const int lane = threadIdx.x & 31;
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long wid = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int per = (K + kslices - 1) / kslices;
    for (long long w = wid; w < (long long)R * kslices; w += nwarps) {
        const int r = (int)(w / kslices), sl = (int)(w - (long long)r * kslices);
        const int k0 = sl * per, k1 = min(K, k0 + per);
        const double *row = src + (long long)r * sr;
        double m = 0.0;
        for (int k = k0 + lane; k < k1; k += 32) m = fmax(m, fabs(__ldg(row + k)));
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0 && m > 0.0) {
            int ex;
            frexp(m, &ex);
            atomicMax(&e[r], ex);
        }
    }
}

__global__ void oz_digits_kfast_kernel(const double *__restrict__ src, long long sr, int R, int K, int Rp, int Kp,
                                       int digits, const int *__restrict__ e, int8_t *__restrict__ out) {
    const size_t plane = (size_t)Rp * Kp;
    const int per_row = Kp / 8;
    const long long total = (long long)Rp * per_row;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(idx / per_row), k0 = (int)(idx - (long long)r * per_row) * 8;
        double y[8];
        const int er = r < R ? e[r] : 0;
        const bool live = r < R && er > -1100;
        const double *row = src + (long long)r * sr;
#pragma unroll
        for (int j = 0; j < 8; j++) y[j] = (live && k0 + j < K) ? ldexp(__ldg(row + k0 + j), -er) : 0.0;   // |y| < 1
        int8_t *o = out + (size_t)r * Kp + k0;
        for (int t = 0; t < digits; t++) {
            uint64_t word = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                y[j] *= 128.0;
                const double d = trunc(y[j]);
                y[j] -= d;
                word |= (uint64_t)(uint8_t)(int8_t)(int)d << (8 * j);
            }
            *reinterpret_cast<uint64_t *>(o + t * plane) = word;
        }
    }
}

inline int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }
inline size_t round_up(size_t x, size_t m) { return (x + m - 1) / m * m; }

// digits x rows x Kp tensor of int8, box (64, box_rows, 1), 64-byte swizzle; rows beyond `rows` read
// as zero
CUtensorMap make_i8_map(void *base, int64_t rows, int64_t Kp, int64_t plane_stride, int planes, int box_rows = 128,
                        int64_t row_stride = 0) {
    CUtensorMap m;
    if (row_stride == 0) row_stride = Kp;
    REQUIRE((reinterpret_cast<uintptr_t>(base) & 15) == 0, CCSD_GPU_EINVAL, "tensor map base must be 16-byte aligned");
    REQUIRE(Kp % 64 == 0 && row_stride % 16 == 0 && plane_stride % 16 == 0 && row_stride >= Kp, CCSD_GPU_EINVAL,
            "int8 digit planes: bad padding");
    cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)row_stride, (cuuint64_t)plane_stride};
    cuuint32_t box[3] = {OBK, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    REQUIRE(r == CUDA_SUCCESS, CCSD_GPU_ECUDA, "cuTensorMapEncodeTiled (int8) failed: " + std::to_string((int)r));
    return m;
}

int num_sms() {
    int dev = 0, v = 0;
    CU_CHECK(cudaGetDevice(&dev));
    CU_CHECK(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    return v;
}

// exponents e[R] of the rows of a strided view over the whole K
void row_exponents(Exec &ex, const double *src, int64_t sr, int64_t sk, int64_t R, int64_t K, int64_t Rp, int *e) {
    // start every exponent below any frexp exponent: 0x80 bytes = -2139062144
    CU_CHECK(cudaMemsetAsync(e, 0x80, sizeof(int) * (size_t)Rp, ex.stream));
    if (sk == 1) {
        // K slices so that every row has a few warps when rows are few
        const int kslices = (int)std::max<int64_t>(1, std::min<int64_t>((K + 1023) / 1024, (148 * 64 + R - 1) / R));
        const int64_t warps = R * kslices;
        const int blocks = (int)std::min<int64_t>((warps + 7) / 8, 148 * 16);
        oz_rowexp_kfast_kernel<<<blocks, 256, 0, ex.stream>>>(src, sr, (int)R, (int)K, kslices, e);
        ex.launches++;
        CU_CHECK(cudaGetLastError());
        return;
    }
    const int64_t rb = (R + 31) / 32;
    // enough blocks over K to fill the GPU when there are few row blocks
    const int64_t kb = std::max<int64_t>(1, std::min<int64_t>((K + 31) / 32, (4 * 148 + rb - 1) / rb));
    oz_rowexp_kernel<<<dim3((unsigned)rb, (unsigned)std::min<int64_t>(kb, 65535)), dim3(32, 8), 0, ex.stream>>>(
        src, sr, sk, (int)R, (int)K, e);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

// digits [digits][Rp][Kp] of the K slab of a strided view (the exponents are those of whole rows)
void slab_digits(Exec &ex, const double *src, int64_t sr, int64_t sk, int64_t R, int64_t K, int64_t Rp, int64_t Kp,
                 int digits, const int *e, int8_t *out) {
    if (sk == 1) {
        const int64_t total = Rp * (Kp / 8);
        const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 32);
        oz_digits_kfast_kernel<<<blocks, 256, 0, ex.stream>>>(src, sr, (int)R, (int)K, (int)Rp, (int)Kp, digits, e, out);
        ex.launches++;
        CU_CHECK(cudaGetLastError());
        return;
    }
    oz_digits_kernel<<<dim3((unsigned)(Rp / 32), (unsigned)std::min<int64_t>(Kp / 32, 65535)), dim3(32, 8), 0,
                       ex.stream>>>(src, sr, sk, (int)R, (int)K, (int)Rp, (int)Kp, digits, e, out);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

// N tile of the pair kernel: of the equal cuts of n into multiples of 32 from 64 to 256 columns the one whose
// waves over the pairs cost least.  Per K block an SM's tensor core takes bn / 2 cycles per MMA, and its shared
// memory moves 128 bytes a cycle: per MMA 4 KB of A and 32 bn of B, and once the digit tiles staged.  The
// second is the larger below 224 columns, which is why narrow tiles need the better last wave to win.
int pair_n_tile(int64_t mt, int64_t n, int digits, int64_t pairs) {
    auto cost = [&](int bn) {
        const int per = bn > WBN / 2 ? 2 : 4;
        int tiles = 0;   // digit tiles staged per K block
        for (int nd = per; nd < digits + per; nd += per) tiles += std::min(nd, digits);
        const int64_t units = mt * ((n + bn - 1) / bn);
        const double mmas = digits * (digits + 1) / 2 * (OBK / 32);
        const double smem = (mmas * (OBM * 32 + bn * 32) + tiles * double(A_TILE + bn / 2 * OBK)) / 128.0;
        return double((units + pairs - 1) / pairs) * std::max(mmas * bn / 2.0, smem);
    };
    int best = WBN;
    for (int64_t nt = (n + WBN - 1) / WBN; nt <= (n + 63) / 64; nt++) {
        const int bn = (int)std::min<int64_t>(WBN, round_up((n + nt - 1) / nt, (int64_t)32));
        if (cost(bn) < 0.999 * cost(best)) best = bn;
    }
    return best;
}

}  // namespace

void ozaki_prepare(Exec &ex, bool trans, int64_t rows, int64_t k, const double *X, int64_t ldx, int digits,
                   OzPlanes &out) {
    REQUIRE(rows > 0 && k > 0 && rows < (1ll << 31) && k < (1ll << 31), CCSD_GPU_EINVAL, "ozaki_prepare: bad size");
    REQUIRE(digits >= 4 && digits <= SLOTS, CCSD_GPU_EINVAL, "ozaki_prepare: 4 to 7 digits");
    // rows of op(X): X[r + ldx kk] (N) or X[kk + ldx r] (T), padded to 128 (either operand's tiles)
    const int64_t sr = trans ? ldx : 1, sk = trans ? 1 : ldx;
    const int64_t Rp = round_up(rows, (int64_t)OBM), Kp = round_up(k, (int64_t)OBK);
    const size_t exp_bytes = round_up(sizeof(int) * (size_t)Rp, (size_t)256);
    const size_t need = exp_bytes + (size_t)digits * Rp * Kp;
    if (out.buf.bytes() < need) {
        out.buf.release();
        out.buf.alloc(need, ex.stream);
    }
    out.rows = rows;
    out.k = k;
    out.Rp = Rp;
    out.Kp = Kp;
    out.digits = digits;
    out.exp_bytes = exp_bytes;
    int *e = out.buf.as<int>();
    row_exponents(ex, X, sr, sk, rows, k, Rp, e);
    slab_digits(ex, X, sr, sk, rows, k, Rp, Kp, digits, e, reinterpret_cast<int8_t *>(out.buf.as<uint8_t>() + exp_bytes));
}

void ozaki_gemm(Exec &ex, bool transA, bool transB, int64_t m, int64_t n, int64_t k, double alpha, const double *A,
                int64_t lda, const double *B, int64_t ldb, double beta, double *C, int64_t ldc, int digits,
                const OzPlanes *pa, const OzPlanes *pb) {
    REQUIRE(m > 0 && n > 0 && k > 0, CCSD_GPU_EINVAL, "ozaki_gemm: empty product");
    REQUIRE(!pa || (pa->digits == digits && pa->rows == m && pa->k == k), CCSD_GPU_EINVAL,
            "ozaki_gemm: prepared A does not match");
    REQUIRE(!pb || (pb->digits == digits && pb->rows == n && pb->k == k), CCSD_GPU_EINVAL,
            "ozaki_gemm: prepared B does not match");
    REQUIRE(m < (1ll << 31) && n < (1ll << 31) && k < (1ll << 31), CCSD_GPU_EINVAL, "ozaki_gemm: size too large");
    REQUIRE(digits >= 4 && digits <= SLOTS, CCSD_GPU_EINVAL, "ozaki_gemm: 4 to 7 digits");
    REQUIRE(ex.gemm_err != nullptr, CCSD_GPU_EINVAL, "ozaki_gemm: no error word");
    const int64_t Mp = round_up(m, OBM), Np = round_up(n, OBN);
    // op(A)(r, kk): A[r + lda kk] (N) or A[kk + lda r] (T); op(B)(kk, c) rows c: B[kk + ldb c] (N) or B[c + ldb kk] (T)
    const int64_t a_sr = transA ? lda : 1, a_sk = transA ? 1 : lda;
    const int64_t b_sr = transB ? 1 : ldb, b_sk = transB ? ldb : 1;
    // CTA pairs for every op(A) of more than one 128-row tile: a pair tile stages half the bytes per product that
    // 128 x 128 tiles do, so that even one half empty costs less than they (six digits, single CTAs behind it:
    // 129 x 4000 x 4000 0.14 ms, 0.22; 384 x 4000 x 4000 0.16, 0.23; 4400 x 400 x 40000 1.32, 1.66).
    // CCSD_GPU_PAIR_DIGITS=0 keeps single CTAs
    static const bool pairs_on = [] {
        const char *e = std::getenv("CCSD_GPU_PAIR_DIGITS");
        return !(e && e[0] == '0');
    }();
    const bool pair = pairs_on && m > OBM;
    auto kernel = digits == 7 ? ozaki_gemm_kernel<7> : digits == 6 ? ozaki_gemm_kernel<6>
                : digits == 5 ? ozaki_gemm_kernel<5> : ozaki_gemm_kernel<4>;
    CU_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OSMEM));
    CU_CHECK(cudaFuncSetAttribute(ozaki_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  PairRing<true>::SMEM));
    CU_CHECK(cudaFuncSetAttribute(ozaki_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  PairRing<false>::SMEM));
    const int nsm = num_sms();
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(WTHREADS);
    cfg.dynamicSmemBytes = PairRing<true>::SMEM;
    cfg.stream = ex.stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int max_pairs = 1;
    if (pair) {
        static int cached[128] = {};
        int dev = 0;
        CU_CHECK(cudaGetDevice(&dev));
        int &mp = cached[dev & 127];
        if (mp == 0) {
            cfg.gridDim = dim3((unsigned)(2 * (nsm / 2)));
            int n = 0;
            CU_CHECK(cudaOccupancyMaxActiveClusters(&n, ozaki_pair_kernel<true>, &cfg));
            mp = std::max(1, n);
        }
        max_pairs = mp;
    }
    // scratch: exponents of both operands and the digit planes of one K slab
    const size_t exp_bytes = round_up(sizeof(int) * (size_t)(Mp + Np), 256);
    // the digit planes of K slabs of whole 16384-wide chunks, at most ~4 GB of them at a time (a
    // 21 GB operand would otherwise need 18 GB of planes at once); each slab's launch adds its chunks
    // to C in the order one launch over all K would, so the result does not depend on the slabs
    const int64_t per_chunk = (int64_t)digits * std::max<int64_t>(OBM, (pa ? 0 : Mp) + (pb ? 0 : Np)) * OK_CHUNK;
    int64_t budget = 4ll << 30;
    if (const char *mb = std::getenv("CCSD_GPU_DIGIT_SLAB_MB")) budget = std::max<int64_t>(1, std::atoll(mb)) << 20;
    const int64_t chunks_per_slab = std::max<int64_t>(1, budget / per_chunk);
    const int64_t kslab = std::min<int64_t>(round_up(k, OBK), chunks_per_slab * OK_CHUNK);
    const size_t a_bytes = pa ? 0 : round_up((size_t)digits * Mp * kslab, (size_t)1024);
    const size_t b_bytes = pb ? 0 : (size_t)digits * Np * kslab;
    // the pair kernel's partial sums, a 128 x 256 block per CTA
    const size_t digit_bytes = round_up(a_bytes + b_bytes, (size_t)256);
    const size_t need = exp_bytes + digit_bytes + (pair ? sizeof(double) * OBM * WBN * (size_t)(2 * max_pairs) : 0);
    DBuf local;
    // a buffer grown inside a capture would belong to the graph: there a small arena is left alone
    DBuf *arena = ex.digit_arena && !(ex.capturing && ex.digit_arena->bytes() < need) ? ex.digit_arena : &local;
    if (arena->bytes() < need) {
        arena->release();
        arena->alloc(need, ex.stream);
    }
    uint8_t *base = arena->as<uint8_t>();
    int *ea = reinterpret_cast<int *>(base), *eb = ea + Mp;
    int8_t *da = reinterpret_cast<int8_t *>(base + exp_bytes), *db = da + a_bytes;
    double *scratch = reinterpret_cast<double *>(base + exp_bytes + digit_bytes);
    // a prepared operand brings its exponents and the digit planes of all of K (no conversion here)
    if (pa) ea = pa->buf.as<int>();
    else row_exponents(ex, A, a_sr, a_sk, m, k, Mp, ea);
    if (pb) eb = pb->buf.as<int>();
    else row_exponents(ex, B, b_sr, b_sk, n, k, Np, eb);
    const int64_t num_mt = pair ? round_up(m, (int64_t)(2 * OBM)) / (2 * OBM) : Mp / OBM;
    const int bn = pair ? pair_n_tile(num_mt, n, digits, max_pairs) : OBN;
    const bool wide = bn > WBN / 2;
    auto pkernel = wide ? ozaki_pair_kernel<true> : ozaki_pair_kernel<false>;
    cfg.dynamicSmemBytes = wide ? PairRing<true>::SMEM : PairRing<false>::SMEM;
    for (int64_t k0 = 0; k0 < k; k0 += kslab) {
        const int64_t kk = std::min(kslab, k - k0), Kp = round_up(kk, OBK);
        if (!pa) slab_digits(ex, A + k0 * a_sk, a_sr, a_sk, m, kk, Mp, Kp, digits, ea, da);
        if (!pb) slab_digits(ex, B + k0 * b_sk, b_sr, b_sk, n, kk, Np, Kp, digits, eb, db);
        // prepared planes: the slab starts k0 bytes into each row of the whole-K planes (k0 is a
        // multiple of 16384, so the tensor map base stays 16-byte aligned)
        CUtensorMap ta = pa ? make_i8_map(pa->digits_base() + k0, Mp, Kp, pa->Rp * pa->Kp, digits, OBM, pa->Kp)
                            : make_i8_map(da, Mp, Kp, Mp * Kp, digits);
        CUtensorMap tb = pb ? make_i8_map(pb->digits_base() + k0, Np, Kp, pb->Rp * pb->Kp, digits,
                                          pair ? bn / 2 : OBN, pb->Kp)
                            : make_i8_map(db, Np, Kp, Np * Kp, digits, pair ? bn / 2 : OBN);
        OzMap map{};
        map.bm = pair ? 2 * OBM : OBM;
        map.bn = bn;
        map.num_mt = (int)num_mt;
        map.num_nt = (int)((n + bn - 1) / bn);
        // raster groups of 2048 rows: their A digit panels (2048 x K x digits bytes) stay in L2 while
        // the group's N tiles stream past
        map.group_m = std::min(map.num_mt, pair ? 8 : 16);
        map.nk_all = (int)(Kp / OBK);
        map.kc = OK_CHUNK / OBK;
        map.nchunks = (map.nk_all + map.kc - 1) / map.kc;
        map.digits = digits;
        map.npass = digits > MAX_DIAG_PER_PASS ? 2 : 1;
        map.M = (int)m;
        map.N = (int)n;
        map.ldc = ldc;
        map.alpha = alpha;
        map.beta = k0 == 0 ? beta : 1.0;
        map.C = C;
        map.ea = ea;
        map.eb = eb;
        map.err = ex.gemm_err;
        map.wait_cycles = ex.wait_cycles > 0 ? ex.wait_cycles : OWAIT_CYCLES;
        const int num_tiles = map.num_mt * map.num_nt;
        const int grid = std::min(num_tiles, pair ? max_pairs : nsm);
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (ex.prof && ex.prof->on) {
            CU_CHECK(cudaEventCreate(&e0));
            CU_CHECK(cudaEventCreate(&e1));
            CU_CHECK(cudaEventRecord(e0, ex.stream));
        }
        if (pair) {
            cfg.gridDim = dim3((unsigned)(2 * grid));
            CU_CHECK(cudaLaunchKernelEx(&cfg, pkernel, ta, tb, map, num_tiles, scratch));
        } else {
            kernel<<<grid, OTHREADS, OSMEM, ex.stream>>>(ta, tb, map, num_tiles);
            CU_CHECK(cudaGetLastError());
        }
        ex.launches++;
        if (e0) {
            CU_CHECK(cudaEventRecord(e1, ex.stream));
            ex.prof->oz_events.emplace_back(e0, e1);
            ex.prof->oz_ops.push_back(2.0 * (double)digits * (digits + 1) / 2.0 * (double)m * (double)n * (double)kk);
        }
    }
}

int ozaki_products(int digits) { return digits * (digits + 1) / 2; }

}  // namespace ccsd
