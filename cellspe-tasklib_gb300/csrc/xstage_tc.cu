// K-d2: X stage on the tcgen05 tensor cores (FP16 operands, FP32 accumulate).
//
// Per channel c the visibilities are the Hermitian rank-K product V = X X^H
// of the S x K spectra matrix X = Xr + i Xi (the conjugate MAC of
// genericAddProduct_32fc_conj, architecture.h:427-433, for every product):
//     Re V = Xr Xr^T + Xi Xi^T,      Im V = Xi Xr^T - Xr Xi^T.
// Work is one 128 (i) x 128 (j) tile of one channel that touches the lower
// triangle.  Its two FP32 accumulators live in tensor memory (TMEM): 128 columns
// Re V, 128 columns Im V, lane = row i.  Each k-step issues four kind::f16 MMAs
// (M=128, N=128, K=16); the minus sign of the last product is the instruction
// descriptor's negate-A bit, so no negated copy of the data exists.  Operands are
// K-major (time innermost), loaded by TMA into a shared-memory ring (32 KB
// stages) guarded by mbarriers, one copy per operand bringing its Re and Im
// parts.  A diagonal tile (i0 = j0) loads its rows once and uses them as both
// operands, and needs three MMAs per k-step: its Im columns accumulate
// M = Xi Xr^T and the epilogue forms Im V = M - M^T through shared memory.
//
// k_xmac_tc, one persistent CTA an SM: warp 0 = TMA producer, running ahead into
// the next tile, warps 1 and 2 = MMA issuers of Re V and Im V (a single one's
// instructions took longer than the MMAs), warp 3 = TMEM owner, warps 4..11 =
// epilogue (TMEM -> registers -> global, a quarter of the lanes and every other
// column block each) of one half of TMEM while the MMAs fill the other.  Bound by
// the MMAs' reads of shared memory and, in short integrations, by the stores of
// the visibilities.  200 inputs: 4096 channels of 128, 512 and 960 segments 243,
// 372 and 522 us with a tile a CTA, 172, 270 and 463 so; 16384 channels of 512
// 2.83 -> 2.1 ms.  Up to 128 inputs (one diagonal tile): 100 inputs, 2048 channels
// of 512 150 -> 92 us.
//
// k_xmac_tc_pair: a tile a CTA, two CTAs an SM, for long integrations.
//
// Every mbarrier wait is bounded: on timeout the kernel records an error code,
// drains its own copies (bounded), frees TMEM and returns, and the host reports
// the failure.
//
// Layout in:  __half spectra[C][2][S][K]  (plane 0 = Re, plane 1 = Im), or
//             k-blocked [C][S][K/32][2][32], or channel-grouped k-blocked
//             [C/16][S][K/32][16][2][32]
// Layout out: float2 vis[C][P], p = i(i+1)/2 + j, j <= i
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"
#include "tma.h"

#include <algorithm>
#include <mutex>

namespace {

constexpr int BM = 128, BN = 128, BK = 32;          // tile and k-chunk (64 B of FP16 = one swizzle row)
constexpr int A_BYTES = BM * BK * 2;                // 8 KB
constexpr int B_BYTES = BN * BK * 2;                // 8 KB
constexpr int STAGES = 4;                           // twice as many of half the size when S <= BM
constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;   // Ar, Ai, Br, Bi = 32 KB
constexpr int EPI_WARPS = 8;
constexpr int TC_THREADS = 128 + 32 * EPI_WARPS;
constexpr uint32_t ACC_COLS = 256;                  // TMEM columns of one tile: Re V, then Im V or M
constexpr int MP = BM + 1;                          // pitch of M in shared memory
constexpr size_t TC_SMEM = 1024 + STAGES * STAGE_BYTES + EPI_WARPS * 32 * 16 * 8 + BM * MP * 4 + (4 * STAGES + 6) * 8;
static_assert(TC_SMEM <= 227 * 1024, "shared memory of one SM");
constexpr long long WAIT_CYCLES = 4000000000LL;     // ~2 s at 2 GHz

// error codes
constexpr unsigned ERR_FULL_WAIT = 1, ERR_EMPTY_WAIT = 2, ERR_ACC_WAIT = 3;

using tc::smem_u32;

// K-major operand in shared memory with 64-byte swizzle: 8-row x 64-byte
// atoms stacked along M/N every 512 bytes (stride byte offset).
CS_DEV uint64_t sw64_desc(uint32_t saddr) { return tc::smem_desc(saddr, 16, 512, tc::SW64); }
// the same with 128-byte rows (32 Re and 32 Im halves, or 64 segments of one part)
CS_DEV uint64_t sw128_desc(uint32_t saddr) { return tc::smem_desc(saddr, 16, 1024, tc::SW128); }

// named barrier 1 over the epilogue warps, with an AND vote that every one of
// them reaches
CS_DEV bool group_vote(bool ok, int nthreads)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"(ok ? 1u : 0u), "r"(nthreads)
        : "memory");
    return r != 0;
}

struct TcArgs {
    int S, C, K;
    int64_t P;
    int64_t ntiles;             // tiles of a channel's lower triangle
    int turn;                   // of the CTAs' order, per round
    int stages;                 // of k_xmac_tc_gram's ring
    float2* vis;
    const float* inv_scale;     // [S][scale_stride] or null
    int scale_stride;
    int accumulate;
    int box_rows;               // rows per TMA box: BM, or S rounded up to 8 when S < BM
    int small;                  // S <= BM: one tile per channel whose B operand is its A operand
    int kblock;                 // spectra k-blocked: 1 [C][S][kp/32][2][32],
                                // 2 channel-grouped [C/16][S][kp/32][16][2][32]
    unsigned* err;              // CsErrorWord::code of the job
};

// Tile `round` of this CTA: row and column block and channel, or false.  The CTAs
// take the tiles (a channel's together, so its rows stay in L2) in rounds of one
// each; their order turns by `turn` a round, which gives every CTA diagonal and
// full tiles alike.
struct Tile {
    int i0, j0, c;
};
// columns a tile needs: j < min(j0 + BN, i0 + BM, S), rounded up to 16
CS_DEV uint32_t tile_cols(int S, const Tile& t) { return (uint32_t)((min(min(t.j0 + BN, t.i0 + BM), S) - t.j0 + 15) & ~15); }
CS_DEV Tile tile_at(int n)                                         // n = i(i+1)/2 + j, j <= i
{
    int i = (int)((sqrtf(8.f * (float)n + 1.f) - 1.f) * 0.5f);
    while ((int64_t)i * (i + 1) / 2 > n) i--;
    while ((int64_t)(i + 1) * (i + 2) / 2 <= n) i++;
    return Tile{i * BM, (n - i * (i + 1) / 2) * BN, 0};
}
CS_DEV bool tile_of(const TcArgs& a, int64_t round, Tile& t)
{
    const int64_t w = round * gridDim.x + (int)((blockIdx.x + round * a.turn) % gridDim.x);
    if (w >= (int64_t)a.C * a.ntiles) return false;
    const int c = (int)(w / a.ntiles);
    t = tile_at((int)(w - (int64_t)c * a.ntiles));
    t.c = c;
    return true;
}

__global__ void __launch_bounds__(TC_THREADS, 1) k_xmac_tc(const __grid_constant__ CUtensorMap tmap,
                                                           const __grid_constant__ TcArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // offset from the shared array itself (not an integer round trip), so that
    // the compiler keeps shared-space 32-bit addressing for every access
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    // S <= BM: a stage holds Ar and Ai only (the tile is diagonal, B = A)
    const uint32_t stage_bytes = a.small ? STAGE_BYTES / 2 : STAGE_BYTES;
    const int stages = a.small ? 2 * STAGES : STAGES;
    float2* stg_all = reinterpret_cast<float2*>(smem + STAGES * STAGE_BYTES);        // [EPI_WARPS][32][16]
    float* msh = reinterpret_cast<float*>(stg_all + EPI_WARPS * 32 * 16);            // [BM][MP]
    uint64_t* bars = reinterpret_cast<uint64_t*>(msh + BM * MP);   // full[2 STAGES], empty[2 STAGES], accf[2], acce[2], done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4 * STAGES + 5);
    const uint32_t sbase = smem_u32(smem);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 16 * STAGES, accf = empty0 + 16 * STAGES, acce = accf + 16;
    const uint32_t done = acce + 16;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = a.S;
    const int nk = (a.K + BK - 1) / BK;
    const int64_t rounds = ((int64_t)a.C * a.ntiles + gridDim.x - 1) / gridDim.x;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            tc::mbar_init(full0 + 8 * s, 1);
            tc::mbar_init(empty0 + 8 * s, 2);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(accf + 8 * b, 2);
            tc::mbar_init(acce + 8 * b, EPI_WARPS);
        }
        tc::mbar_init(done, 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
    }
    if (warp == 3) tc::tmem_alloc(smem_u32(tmem_slot), 2 * ACC_COLS);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (tc::elect_one()) {
            // one copy per operand brings both parts of its rows: planes as Re rows
            // then Im rows of 64 bytes, k-blocked as rows of 32 Re and 32 Im halves
            auto load = [&](uint32_t dst, int c, int kc, int row, uint32_t bar) {
                if (a.kblock) tc::tma_load_5d(dst, &tmap, 0, a.kblock == 2 ? c & 15 : 0, kc, row, a.kblock == 2 ? c >> 4 : c, bar);
                else tc::tma_load_4d(dst, &tmap, kc * BK, row, 0, c, bar);
            };
            int s = 0, filled = 0;
            uint32_t ph = 0;                               // of the ring's current turn
            bool ok = true;
            Tile t;
            for (int64_t n = 0; n < rounds && ok && tile_of(a, n, t); n++) {
                const bool diag = t.i0 == t.j0;            // B is A
                // S < 128: the boxes hold the S (rounded up to 8) rows that exist, so a
                // channel's planes are read once; the rows of the operand tiles past them
                // only feed accumulator rows and columns that are never stored
                const uint32_t tx = (diag ? 2u : 4u) * (uint32_t)a.box_rows * BK * 2;
                for (int kc = 0; kc < nk; kc++) {
                    if (!tc::mbar_wait(empty0 + 8 * s, ph ^ 1, a.err, ERR_EMPTY_WAIT, WAIT_CYCLES)) { ok = false; break; }
                    const uint32_t st = sbase + s * stage_bytes, fb = full0 + 8 * s;
                    tc::mbar_expect_tx(fb, tx);
                    load(st, t.c, kc, t.i0, fb);
                    if (!diag) load(st + 2 * A_BYTES, t.c, kc, t.j0, fb);
                    filled = min(filled + 1, stages);
                    if (++s == stages) s = 0, ph ^= 1;
                }
            }
            // drain: every stage this thread filled must have landed before the CTA exits
            for (; filled > 0; filled--) {
                if (--s < 0) s = stages - 1, ph ^= 1;
                tc::mbar_wait(full0 + 8 * s, ph, a.err, ERR_FULL_WAIT, WAIT_CYCLES);
            }
        }
    } else if (warp <= 2) {
        // ---------------- MMA issuers: warp 1 Re V, warp 2 Im V (or M) ----------------
        if (tc::elect_one()) {
            const uint64_t d0 = a.kblock ? sw128_desc(sbase) : sw64_desc(sbase);
            const uint32_t im16 = a.kblock ? 4 : (uint32_t)a.box_rows * BK * 2 / 16;   // Im after Re, in 16 bytes
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            Tile t;
            for (int64_t n = 0; n < rounds && ok && tile_of(a, n, t); n++) {
                const bool diag = t.i0 == t.j0;
                const uint32_t n_eff = tile_cols(S, t);
                const uint32_t id_pos = tc::idesc_f16(BM, n_eff, false, false, false), id_neg = tc::idesc_f16(BM, n_eff, true, false, false);
                const int b = (int)(n & 1);
                if (!tc::mbar_wait(acce + 8 * b, (uint32_t)((n >> 1) & 1) ^ 1, a.err, ERR_ACC_WAIT, WAIT_CYCLES)) break;
                tc::fence_after();
                const uint32_t d = tmem + b * ACC_COLS + (warp == 2 ? ACC_COLS / 2 : 0);
                for (int kc = 0; kc < nk; kc++) {
                    if (!tc::mbar_wait(full0 + 8 * s, ph, a.err, ERR_FULL_WAIT, WAIT_CYCLES)) { ok = false; break; }
                    tc::fence_after();
                    const uint64_t da = d0 + s * (stage_bytes / 16), db = diag ? da : da + 2 * A_BYTES / 16;
#pragma unroll
                    for (int kk = 0; kk < BK / 16; kk++) {
                        // 16 FP16 along K are 32 bytes
                        const uint64_t ar = da + 2 * kk, ai = ar + im16, br = db + 2 * kk, bi = br + im16;
                        const uint32_t acc = (kc | kk) ? 1u : 0u;
                        if (warp == 1) {
                            tc::mma_f16(d, ar, br, id_pos, acc);           // Re += Ar Br^T
                            tc::mma_f16(d, ai, bi, id_pos, 1u);            // Re += Ai Bi^T
                        } else {
                            tc::mma_f16(d, ai, br, id_pos, acc);           // Im += Ai Br^T  (M on a diagonal tile)
                            if (!diag) tc::mma_f16(d, ar, bi, id_neg, 1u); // Im -= Ar Bi^T
                        }
                    }
                    tc::commit(empty0 + 8 * s);                   // stage free once these MMAs finish
                    if (++s == stages) s = 0, ph ^= 1;
                }
                if (ok) tc::commit(accf + 8 * b);
            }
            // `done` completes only after every MMA issued has finished, so TMEM is
            // never freed under one
            tc::commit(done);
        }
        __syncwarp();
    } else if (warp >= 4) {
        // ---------------- epilogue: TMEM -> global ----------------
        const int q = warp & 3, half = (warp - 4) >> 2;            // TMEM lane quarter; even or odd column blocks
        const int r = 32 * q + lane;
        // 32-row x 16-column blocks through shared memory, so that a store
        // instruction writes two 128-byte runs of one output row (columns XORed
        // with the row: conflict-free both ways)
        float2* stg = stg_all + (warp - 4) * 32 * 16;
        Tile t;
        for (int64_t n = 0; n < rounds && tile_of(a, n, t); n++) {
            const int b = (int)(n & 1);
            const bool ok = tc::mbar_wait(accf + 8 * b, (uint32_t)((n >> 1) & 1), a.err, ERR_ACC_WAIT, WAIT_CYCLES);
            // the warps go on together or not at all; the last tile's M is read by now
            if (!group_vote(__all_sync(0xffffffffu, ok), 32 * EPI_WARPS)) break;
            tc::fence_after();
            const bool diag = t.i0 == t.j0;
            const int i = t.i0 + r;
            const uint32_t acc = tmem + b * ACC_COLS + ((uint32_t)(32 * q) << 16);
            const float si = (a.inv_scale && i < S) ? __ldg(a.inv_scale + (int64_t)i * a.scale_stride + t.c) : 1.f;
            const int ncb = (int)(tile_cols(S, t) / 16);
            if (diag) {
                for (int cb = half; cb < ncb; cb += 2) {
                    uint32_t mm[16];
                    tc::tmem_ld_32x32b_x16(acc + ACC_COLS / 2 + cb * 16, mm);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int jj = 0; jj < 16; jj++) msh[r * MP + cb * 16 + jj] = __uint_as_float(mm[jj]);
                }
                group_vote(true, 32 * EPI_WARPS);
            }
            // this warp's rows end before the diagonal's later column blocks
            const int last = diag ? min(ncb, 2 * q + 2) : ncb;
            for (int cb = half; cb < last; cb += 2) {
                uint32_t re[16], im[16];
                tc::tmem_ld_32x32b_x16(acc + cb * 16, re);
                if (!diag) tc::tmem_ld_32x32b_x16(acc + ACC_COLS / 2 + cb * 16, im);
                tc::tmem_ld_wait();
                if (diag) {
#pragma unroll
                    for (int jj = 0; jj < 16; jj++) {
                        const int jl = cb * 16 + jj;                   // column within the tile
                        im[jj] = __float_as_uint(msh[r * MP + jl] - msh[jl * MP + r]);
                    }
                }
#pragma unroll
                for (int jj = 0; jj < 16; jj++) {
                    float f = si;
                    if (a.inv_scale) {
                        const int j = t.j0 + cb * 16 + jj;
                        f *= (j < S) ? __ldg(a.inv_scale + (int64_t)j * a.scale_stride + t.c) : 0.f;
                    }
                    stg[lane * 16 + (jj ^ (lane & 15))] = make_float2(__uint_as_float(re[jj]) * f, __uint_as_float(im[jj]) * f);
                }
                __syncwarp();
                const int col = lane & 15, j = t.j0 + cb * 16 + col;
                int ii = t.i0 + 32 * q + (lane >> 4);
                float2* o = a.vis + (int64_t)t.c * a.P + (int64_t)ii * (ii + 1) / 2 + j;
#pragma unroll 4
                for (int it = 0; it < 16; it++) {
                    const int rr = 2 * it + (lane >> 4);
                    if (ii < S && j <= ii) {
                        float2 v = stg[rr * 16 + (col ^ (rr & 15))];
                        if (a.accumulate) {
                            const float2 old = *o;
                            v.x += old.x;
                            v.y += old.y;
                        }
                        *o = v;
                    }
                    o += 2 * ii + 3;                               // two rows on
                    ii += 2;
                }
                __syncwarp();
            }
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(acce + 8 * b);
        }
        tc::fence_before();
    }
    __syncthreads();
    if (warp == 3) {
        tc::mbar_wait(done, 0, a.err, ERR_ACC_WAIT, WAIT_CYCLES);
        __syncwarp();
        tc::fence_after();
        tc::tmem_dealloc(tmem, 2 * ACC_COLS);
    }
}

// The same with one tile a CTA, two CTAs an SM and one issuer each (6 warps: TMA
// producer, TMEM owner and issuer, epilogue): tiles of long integrations, where a
// ring of three stages each and chunk boundaries that do not meet keep the MMAs
// busier than one CTA does and the epilogue is a small part.  From where it is
// faster, which moves up with the full tiles' share of the work (us, this form
// and the persistent one): 1024 channels, 200 inputs 284 and 263 at 1024 segments,
// 373 and 374 at 1536, 465 and 483 at 2048; 300 inputs 719 and 694 at 1536, 900 and 903
// at 2048; 512 inputs 1709 and 1656 at 2048, of 256 channels 829 and 818 at 4096, 1569
// and 1587 at 8192.
constexpr int pair_min_k(int S) { return S > 192 ? 8 * S : 1536; }
constexpr int P_STAGES = 3, P_THREADS = 192;
constexpr size_t P_SMEM = 1024 + P_STAGES * STAGE_BYTES + 256;
// epilogue shared memory: four warps' 32 x 17 float2 staging blocks, then (on
// a diagonal tile) M as [BM][MP] floats; both inside the operand ring
constexpr int EPI_STG_BYTES = 4 * 32 * 17 * 8;
static_assert(EPI_STG_BYTES + BM * MP * 4 <= P_STAGES * STAGE_BYTES, "epilogue M staging inside the ring");

__global__ void __launch_bounds__(P_THREADS, 1) k_xmac_tc_pair(const __grid_constant__ CUtensorMap tmap,
                                                           const __grid_constant__ TcArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // offset from the shared array itself (not an integer round trip), so that
    // the compiler keeps shared-space 32-bit addressing for every access
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + P_STAGES * STAGE_BYTES);   // full[S], empty[S], acc
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * P_STAGES + 1);
    const uint32_t sbase = smem_u32(smem);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * P_STAGES, accb = full0 + 16 * P_STAGES;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Tile t = tile_at(blockIdx.x);
    const int c = blockIdx.y;
    const int i0 = t.i0, j0 = t.j0;
    const int S = a.S;
    const int nk = (a.K + BK - 1) / BK;
    const uint32_t n_eff = tile_cols(S, t);
    const bool diag = i0 == j0;                        // B is A, Im V = M - M^T
    const uint32_t stage_tx = (diag ? 2u : 4u) * BM * BK * 2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < P_STAGES; s++) {
            tc::mbar_init(full0 + 8 * s, 1);
            tc::mbar_init(empty0 + 8 * s, 1);
        }
        tc::mbar_init(accb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
    }
    if (warp == 1) {
        tc::tmem_alloc(smem_u32(tmem_slot), ACC_COLS);
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (tc::elect_one()) {
            // one copy per operand brings both parts of its rows: planes as Re rows
            // then Im rows of 64 bytes, k-blocked as rows of 32 Re and 32 Im halves
            auto load = [&](uint32_t dst, int kc, int row, uint32_t bar) {
                if (a.kblock) tc::tma_load_5d(dst, &tmap, 0, a.kblock == 2 ? c & 15 : 0, kc, row, a.kblock == 2 ? c >> 4 : c, bar);
                else tc::tma_load_4d(dst, &tmap, kc * BK, row, 0, c, bar);
            };
            int issued = 0;
            bool ok = true;
            for (int kc = 0; kc < nk && ok; kc++) {
                const int s = kc % P_STAGES;
                const uint32_t ph = (kc / P_STAGES) & 1;
                if (!tc::mbar_wait(empty0 + 8 * s, ph ^ 1, a.err, ERR_EMPTY_WAIT, WAIT_CYCLES)) { ok = false; break; }
                const uint32_t st = sbase + s * STAGE_BYTES;
                const uint32_t fb = full0 + 8 * s;
                tc::mbar_expect_tx(fb, stage_tx);
                load(st, kc, i0, fb);
                if (!diag) load(st + 2 * A_BYTES, kc, j0, fb);
                issued = kc + 1;
            }
            // drain: every stage this thread filled must have landed before the CTA exits
            for (int kc = (issued > P_STAGES ? issued - P_STAGES : 0); kc < issued; kc++)
                tc::mbar_wait(full0 + 8 * (kc % P_STAGES), (kc / P_STAGES) & 1, a.err, ERR_FULL_WAIT, WAIT_CYCLES);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (tc::elect_one()) {
            const uint32_t id_pos = tc::idesc_f16(BM, n_eff, false, false, false), id_neg = tc::idesc_f16(BM, n_eff, true, false, false);
            const uint32_t d_re = tmem, d_im = tmem + ACC_COLS / 2;
            const uint64_t d0 = a.kblock ? sw128_desc(sbase) : sw64_desc(sbase);
            const uint32_t im16 = a.kblock ? 4 : BM * BK * 2 / 16;   // Im after Re, in 16 bytes
            bool ok = true;
            for (int kc = 0; kc < nk; kc++) {
                const int s = kc % P_STAGES;
                if (!tc::mbar_wait(full0 + 8 * s, (kc / P_STAGES) & 1, a.err, ERR_FULL_WAIT, WAIT_CYCLES)) { ok = false; break; }
                tc::fence_after();
                const uint64_t da = d0 + s * (STAGE_BYTES / 16), db = diag ? da : da + 2 * A_BYTES / 16;
#pragma unroll
                for (int kk = 0; kk < BK / 16; kk++) {
                    // 16 FP16 along K are 32 bytes
                    const uint64_t ar = da + 2 * kk, ai = ar + im16, br = db + 2 * kk, bi = br + im16;
                    const uint32_t acc = (kc | kk) ? 1u : 0u;
                    tc::mma_f16(d_re, ar, br, id_pos, acc);           // Re += Ar Br^T
                    tc::mma_f16(d_re, ai, bi, id_pos, 1u);            // Re += Ai Bi^T
                    tc::mma_f16(d_im, ai, br, id_pos, acc);           // Im += Ai Br^T  (M on a diagonal tile)
                    if (!diag) tc::mma_f16(d_im, ar, bi, id_neg, 1u);  // Im -= Ar Bi^T
                }
                tc::commit(empty0 + 8 * s);                       // stage free once these MMAs finish
            }
            // Always commit: the barrier then completes only after every MMA
            // issued so far has finished, so TMEM is never freed under one.
            tc::commit(accb);
            if (!ok) tc::record_error(a.err, ERR_FULL_WAIT);
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: TMEM -> global ----------------
        const int q = warp & 3;                                    // TMEM lane quarter
        const int r = 32 * q + lane;
        const int i = i0 + r;
        bool ok = tc::mbar_wait(accb, 0, a.err, ERR_ACC_WAIT, WAIT_CYCLES);
        ok = ok && (*reinterpret_cast<volatile unsigned*>(a.err) == 0u);
        __syncwarp();
        // M - M^T needs the other warps' rows: the four epilogue warps agree
        // (one vote, so all of them or none reach the barrier below)
        bool go = __all_sync(0xffffffffu, ok);
        if (diag) go = group_vote(go, 128);
        if (go) {
            tc::fence_after();
            // Stage each 32-row x 16-column block through shared memory (the
            // operand ring is free once the accumulators are final) so that a
            // store instruction writes two 128-byte runs of one output row.
            float2* stg = reinterpret_cast<float2*>(smem) + (warp - 2) * 32 * 17;
            // diagonal tile: M [BM][MP] after the four warps' staging blocks
            float* msh = reinterpret_cast<float*>(smem + EPI_STG_BYTES);
            const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
            const float si = (a.inv_scale && i < S) ? __ldg(a.inv_scale + (int64_t)i * a.scale_stride + c) : 1.f;
            const int ncb = (int)(n_eff / 16);
            if (diag) {
                for (int cb = 0; cb < ncb; cb++) {
                    uint32_t mm[16];
                    tc::tmem_ld_32x32b_x16(lane_base + ACC_COLS / 2 + cb * 16, mm);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int jj = 0; jj < 16; jj++) msh[r * MP + cb * 16 + jj] = __uint_as_float(mm[jj]);
                }
                group_vote(true, 128);
            }
            for (int cb = 0; cb < ncb; cb++) {
                uint32_t re[16], im[16];
                tc::tmem_ld_32x32b_x16(lane_base + cb * 16, re);
                if (!diag) tc::tmem_ld_32x32b_x16(lane_base + ACC_COLS / 2 + cb * 16, im);
                tc::tmem_ld_wait();
                if (diag) {
#pragma unroll
                    for (int jj = 0; jj < 16; jj++) {
                        const int jl = cb * 16 + jj;                   // column within the tile
                        im[jj] = __float_as_uint(msh[r * MP + jl] - msh[jl * MP + r]);
                    }
                }
#pragma unroll
                for (int jj = 0; jj < 16; jj++) {
                    float f = si;
                    if (a.inv_scale) {
                        const int j = j0 + cb * 16 + jj;
                        f *= (j < S) ? __ldg(a.inv_scale + (int64_t)j * a.scale_stride + c) : 0.f;
                    }
                    stg[lane * 17 + jj] = make_float2(__uint_as_float(re[jj]) * f, __uint_as_float(im[jj]) * f);
                }
                __syncwarp();
#pragma unroll 4
                for (int it = 0; it < 16; it++) {
                    const int rr = 2 * it + (lane >> 4), col = lane & 15;
                    const int ii = i0 + 32 * q + rr, j = j0 + cb * 16 + col;
                    if (ii < S && j <= ii) {
                        float2 v = stg[rr * 17 + col];
                        float2* o = a.vis + (int64_t)c * a.P + (int64_t)ii * (ii + 1) / 2 + j;
                        if (a.accumulate) {
                            const float2 old = *o;
                            v.x += old.x;
                            v.y += old.y;
                        }
                        *o = v;
                    }
                }
                __syncwarp();
            }
        }
        tc::fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, ACC_COLS);
    }
}

// ---------------------------------------------------------------------------
// S <= 64: every product of a channel from a few MMAs per 16 segments.
//   Planes: a stage holds Xr and Xi, RI rows each (S rounded up to 8).
//     [Xr; Xi] Xr^T and, in its upper RI lanes alone, Xi Xi^T go into one accumulator,
//     whose upper rows are then Re V, added in the order of the tiles below (Re, Im,
//     Re, ... : the accumulator truncates, so another order would move every auto by
//     parts in 10^5 at thousands of segments), and whose lower rows are M = Xi Xr^T.
//     (Rows of zeros under Xi in place of the lane mask make NaN of an infinite Xi.)
//   k-blocked (BLK): an operand row holds a block's 32 Re and 32 Im halves; Re V
//     takes two MMAs, M one.
// Im V = M - M^T is put together at the end through shared memory.  One TMA copy
// brings a chunk of 128-byte rows (64 segments of both planes, or 32 of both
// parts): a copy costs the SM's TMA unit about 125 cycles however small it is,
// which bound a form with a copy per plane and 32 segments; four MMAs of S columns per
// 16 segments, at least 32 cycles each, bound the tiles.  32 inputs x 4096
// channels x 4096 segments (2.15 GB, 318 us at the copy rate) take 352 us a call
// where the tiles took 643, 64 x 2048 x 4096 341 where they took 462; for 16 inputs and
// fewer the MMAs' least cost still bounds it (8 x 4096 x 4096: 618 -> 307 us).  The
// accumulators are one TMEM buffer of COLS columns for the whole time axis.  Warps:
// E = COLS / 32 epilogue warps, the TMA producer, the MMA issuer and TMEM owner.
// ---------------------------------------------------------------------------
constexpr int G_ROW = 128;                          // operand row bytes
// Planes take three stages, and two up to 512 segments, where more CTAs on an SM are
// worth more: 64 inputs, 1024 channels of 4088 segments 220 us with two, 204 with three;
// 2048 channels of 200 segments 43 and 49.
template <int COLS, bool BLK> constexpr int gram_stages() { return BLK ? (COLS == 128 ? 6 : 8) : 3; }

template <int COLS, bool BLK>
__global__ void __launch_bounds__(COLS + 64) k_xmac_tc_gram(const __grid_constant__ CUtensorMap tmap,
                                                            const __grid_constant__ TcArgs a)
{
    constexpr int E = COLS / 32, MAX_ST = gram_stages<COLS, BLK>(), SEGS = BLK ? 32 : 64;
    const int ST = a.stages;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x, S = a.S, RI = a.box_rows, nk = (a.K + SEGS - 1) / SEGS;
    const uint32_t plane = (uint32_t)RI * G_ROW, stage_bytes = BLK ? plane : 2 * plane;
    // columns of an accumulator (BLK: Re V and M side by side)
    const uint32_t n = (uint32_t)((S + 15) & ~15);
    // barriers in front, so that the ring and the rows past it end the buffer
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);                   // full[], empty[], acc
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_ST + 1);
    unsigned char* ring = smem + 1024;
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * ST, accb = full0 + 16 * ST;
    const uint32_t sbase = smem_u32(ring);
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) {
            tc::mbar_init(full0 + 8 * s, 1);
            tc::mbar_init(empty0 + 8 * s, 1);
        }
        tc::mbar_init(accb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
    }
    if (warp == E + 1) tc::tmem_alloc(smem_u32(tmem_slot), COLS);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tmem_slot;
    if (warp == E) {
        if (tc::elect_one()) {
            int issued = 0;
            for (int kc = 0; kc < nk; kc++) {
                const int s = kc % ST;
                if (!tc::mbar_wait(empty0 + 8 * s, ((kc / ST) & 1) ^ 1, a.err, ERR_EMPTY_WAIT, WAIT_CYCLES)) break;
                const uint32_t st = sbase + s * stage_bytes, fb = full0 + 8 * s;
                tc::mbar_expect_tx(fb, BLK ? plane : 2 * plane);
                if constexpr (BLK) tc::tma_load_5d(st, &tmap, 0, a.kblock == 2 ? c & 15 : 0, kc, 0, a.kblock == 2 ? c >> 4 : c, fb);
                else tc::tma_load_4d(st, &tmap, kc * SEGS, 0, 0, c, fb);
                issued = kc + 1;
            }
            // drain: every stage this thread filled must have landed before the CTA exits
            for (int kc = (issued > ST ? issued - ST : 0); kc < issued; kc++)
                tc::mbar_wait(full0 + 8 * (kc % ST), (kc / ST) & 1, a.err, ERR_FULL_WAIT, WAIT_CYCLES);
        }
    } else if (warp == E + 1) {
        if (tc::elect_one()) {
            const uint32_t id = tc::idesc_f16(BM, n, false, false, false);
            const uint64_t d0 = sw128_desc(sbase);
            const tc::LaneMask re_lanes = tc::first_lanes(RI);
            for (int kc = 0; kc < nk; kc++) {
                const int s = kc % ST;
                if (!tc::mbar_wait(full0 + 8 * s, (kc / ST) & 1, a.err, ERR_FULL_WAIT, WAIT_CYCLES)) break;
                tc::fence_after();
                const uint64_t d = d0 + s * (stage_bytes / 16);
                const uint32_t acc = kc ? 1u : 0u;
                if constexpr (BLK) {
                    // 16 segments are 32 bytes; the Im halves start at byte 64
#pragma unroll
                    for (int kk = 0; kk < 2; kk++) {
                        const uint64_t re = d + 2 * kk, im = d + 4 + 2 * kk;
                        tc::mma_f16(tmem, re, re, id, kk ? 1u : acc);
                        tc::mma_f16(tmem + n, im, re, id, kk ? 1u : acc);
                        tc::mma_f16(tmem, im, im, id, 1u);
                    }
                } else {
                    const uint64_t di = d + plane / 16;
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        tc::mma_f16(tmem, d + 2 * kk, d + 2 * kk, id, kk ? 1u : acc);
                        tc::mma_f16(tmem, di + 2 * kk, di + 2 * kk, id, 1u, re_lanes);
                    }
                }
                tc::commit(empty0 + 8 * s);
            }
            // always: the barrier then completes only after every MMA issued has finished
            tc::commit(accb);
        }
        __syncwarp();
    } else {
        bool ok = tc::mbar_wait(accb, 0, a.err, ERR_ACC_WAIT, WAIT_CYCLES);
        ok = ok && (*reinterpret_cast<volatile unsigned*>(a.err) == 0u);
        // all or none of the epilogue warps go on (a product needs several rows)
        if (group_vote(__all_sync(0xffffffffu, ok), 32 * E)) {
            tc::fence_after();
            float* g = reinterpret_cast<float*>(ring);           // free: the accumulators are final
            const int rows = BLK ? RI : 2 * RI, cols = BLK ? 2 * (int)n : (int)n, GP = cols + 1;
            if (32 * warp < rows) {
                for (int cb = 0; cb < cols; cb += 16) {
                    uint32_t v[16];
                    tc::tmem_ld_32x32b_x16(tmem + ((uint32_t)(32 * warp) << 16) + cb, v);
                    tc::tmem_ld_wait();
                    if (32 * warp + lane < rows)
#pragma unroll
                        for (int j = 0; j < 16; j++) g[(32 * warp + lane) * GP + cb + j] = __uint_as_float(v[j]);
                }
            }
            group_vote(true, 32 * E);
            float2* out = a.vis + (int64_t)c * a.P;
            for (int p = threadIdx.x; p < (int)a.P; p += 32 * E) {
                int i = (int)((sqrtf(8.f * (float)p + 1.f) - 1.f) * 0.5f);
                if ((i + 1) * (i + 2) / 2 <= p) i++;
                else if (i * (i + 1) / 2 > p) i--;
                const int j = p - i * (i + 1) / 2;
                float2 v;
                if constexpr (BLK) v = make_float2(g[i * GP + j], g[i * GP + n + j] - g[j * GP + n + i]);
                else v = make_float2(g[i * GP + j], g[(RI + i) * GP + j] - g[(RI + j) * GP + i]);
                if (a.inv_scale) {
                    const float f = __ldg(a.inv_scale + (int64_t)i * a.scale_stride + c) *
                                    __ldg(a.inv_scale + (int64_t)j * a.scale_stride + c);
                    v = make_float2(v.x * f, v.y * f);
                }
                if (a.accumulate) {
                    const float2 old = out[p];
                    v.x += old.x;
                    v.y += old.y;
                }
                out[p] = v;
            }
        }
        tc::fence_before();
    }
    __syncthreads();
    if (warp == E + 1) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, COLS);
    }
}

template <int COLS, bool BLK>
int launch_gram(const CUtensorMap& tm, TcArgs a, cudaStream_t st)
{
    const int chunks = (a.K + (BLK ? 32 : 64) - 1) / (BLK ? 32 : 64);
    a.stages = std::min(chunks, !BLK && chunks <= 8 ? 2 : gram_stages<COLS, BLK>());
    // the ring, the rows past it that an MMA of 128 rows reads (lanes never
    // stored), and after the last MMA the accumulators [rows][columns + 1]
    const size_t plane = (size_t)a.box_rows * G_ROW, rows = (BLK ? 1 : 2) * (size_t)a.box_rows;
    const size_t cols = (BLK ? 2 : 1) * (((size_t)a.S + 15) / 16 * 16);
    // an operand of 128 rows from the last stage's Xr (BLK) or Xi on
    const size_t ring = a.stages * (BLK ? plane : 2 * plane) + BM * G_ROW - plane;
    const size_t smem = 2048 + std::max(ring, rows * (cols + 1) * sizeof(float));
    auto kern = k_xmac_tc_gram<COLS, BLK>;
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(kern), (int)smem));
    kern<<<a.C, COLS + 64, smem, st>>>(tm, a), cs_count_launches(1);
    return (int)cudaGetLastError();
}

// Tensor map whose one box is an operand's rows of one chunk, both parts: planes
// [C][2][S][kp] as (segments, inputs, planes, channel) with `segs` segments
// (64-byte rows of 32, 128-byte rows of 64), k-blocked as (64 halves, ...).
// Inputs past S and segments past K read as zeros.
bool encode_map(CsEncodeTiledFn enc, const void* spectra, int kp, int segs, const TcArgs& a, CUtensorMap* tm)
{
    const cuuint64_t S = a.S, C = a.C, K = a.K, pitch = (cuuint64_t)kp * 2, blocks = (cuuint64_t)kp / 32;
    const cuuint32_t rows = a.box_rows, one[5] = {1, 1, 1, 1, 1};
    auto encode = [&](int rank, const cuuint64_t* dim, const cuuint64_t* stride, const cuuint32_t* box) {
        return enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, const_cast<void*>(spectra), dim, stride, box, one,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, box[0] == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!a.kblock) {
        const cuuint64_t dim[4] = {K, S, 2, C}, stride[3] = {pitch, S * pitch, 2 * S * pitch};
        const cuuint32_t box[4] = {(cuuint32_t)segs, rows, 2, 1};
        return encode(4, dim, stride, box);
    }
    const cuuint32_t box[5] = {64, 1, 1, rows, 1};
    if (a.kblock == 2) {
        // [C/16][S][kp/32][16][64]: (64 halves, channel of the group, block, inputs, group)
        const cuuint64_t dim[5] = {64, 16, K / 32, S, C / 16}, stride[4] = {128, 2048, blocks * 2048, S * blocks * 2048};
        return encode(5, dim, stride, box);
    }
    // [C][S][kp/32][64]: (64 halves, -, block, inputs, channel)
    const cuuint64_t dim[5] = {64, 1, K / 32, S, C}, stride[4] = {128, 128, blocks * 128, S * blocks * 128};
    return encode(5, dim, stride, box);
}

int xmac_gram(CsEncodeTiledFn enc, const void* spectra, int kp, const TcArgs& a, cudaStream_t st)
{
    CUtensorMap tm;
    if (!encode_map(enc, spectra, kp, 64, a, &tm)) return CS_ERR_ARG;
    if (a.kblock)
        return a.S <= 16 ? launch_gram<32, true>(tm, a, st)
               : a.S <= 32 ? launch_gram<64, true>(tm, a, st) : launch_gram<128, true>(tm, a, st);
    return a.S <= 16 ? launch_gram<32, false>(tm, a, st)
           : a.S <= 32 ? launch_gram<64, false>(tm, a, st) : launch_gram<128, false>(tm, a, st);
}

// One thread, one barrier that nothing arrives at.
__global__ void k_wait_timeout(unsigned* err)
{
    __shared__ __align__(8) uint64_t bar;
    tc::mbar_init(smem_u32(&bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_wait(smem_u32(&bar), 0, err, ERR_FULL_WAIT, 2000000LL);
}

}  // namespace

CsEncodeTiledFn cs_encode_tiled()
{
    static CsEncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<CsEncodeTiledFn>(p);
    });
    return fn;
}

int cs_xmac_tc_f16(const void* spectra, int S, int C, int K, int kp, float2* vis, const float* inv_scale,
                   int scale_stride, int accumulate, unsigned* err, cudaStream_t st, int kblock)
{
    if (!spectra || !vis || !err || S <= 0 || C <= 0 || K <= 0 || C > 65535 || kp < K) return CS_ERR_ARG;
    if (K % 8 != 0 || kp % 8 != 0 || (uintptr_t)spectra % 16) return CS_ERR_ARG;   // TMA: 16-byte pitch and base
    if (kblock < 0 || kblock > 2 || (kblock && (K % 32 != 0 || kp % 32 != 0)) || (kblock == 2 && C % 16 != 0))
        return CS_ERR_ARG;
    CsEncodeTiledFn enc = cs_encode_tiled();
    if (!enc) return CS_ERR_UNSUPPORTED;
    if (S <= 64) {
        const TcArgs g{S, C, K, (int64_t)S * (S + 1) / 2, 1, 0, 0, vis, inv_scale, scale_stride > 0 ? scale_stride : C,
                       accumulate, (S + 7) / 8 * 8, 1, kblock, err};
        return xmac_gram(enc, spectra, kp, g, st);
    }
    const int64_t nt = (S + BM - 1) / BM, ntiles = nt * (nt + 1) / 2;
    int dev = 0, sms = 0;
    CS_CUDA_TRY(cudaGetDevice(&dev));
    CS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int grid = (int)std::min<int64_t>(sms, ntiles * C);
    // grid + turn = 1 modulo the tiles of a channel: from one round to the next a CTA's tile moves on by one
    const int turn = (int)(((1 - grid) % ntiles + ntiles) % ntiles);
    const TcArgs a{S, C, K, (int64_t)S * (S + 1) / 2, ntiles, turn, 0, vis, inv_scale, scale_stride > 0 ? scale_stride : C,
                   accumulate, S < BM ? (S + 7) / 8 * 8 : BM, S <= BM ? 1 : 0, kblock, err};
    CUtensorMap tm;
    if (!encode_map(enc, spectra, kp, BK, a, &tm)) return CS_ERR_ARG;
    if (S > BM && K >= pair_min_k(S)) {
        CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(k_xmac_tc_pair), (int)P_SMEM));
        k_xmac_tc_pair<<<dim3((unsigned)ntiles, C), P_THREADS, P_SMEM, st>>>(tm, a), cs_count_launches(1);
        return (int)cudaGetLastError();
    }
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(k_xmac_tc), (int)TC_SMEM));
    k_xmac_tc<<<grid, TC_THREADS, TC_SMEM, st>>>(tm, a), cs_count_launches(1);
    return (int)cudaGetLastError();
}

int cs_wait_timeout(unsigned* err, cudaStream_t st)
{
    if (!err) return CS_ERR_ARG;
    k_wait_timeout<<<1, 1, 0, st>>>(err), cs_count_launches(1);
    return (int)cudaGetLastError();
}
