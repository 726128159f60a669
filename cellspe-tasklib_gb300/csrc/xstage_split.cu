// K-d3: X stage of the FP32 path on the tcgen05 tensor cores, from spectra
// held as two FP16 terms.
//
// The F stage writes every FP32 spectrum value x as hi = fp16(s x) and
// lo = fp16(w (s x - hi)), s a power of two for the whole job that keeps |s x|
// below FP16's largest value, w = 1 or 2: 22 significant bits and the sign of
// lo, the same 8 bytes per complex value as FP32.  A product x y is then
// hi hi' + hi lo' + lo hi' (the lo lo' term is below 2^-22 of it), each exact
// in FP32.  X = Xr + i Xi of a channel, V = X X^H.
//
// S <= 64, k_xmac_gram (w = 2): the rows Z = [Xr; Xi] are one operand of 2 R
// rows (R = 16, 32 or 64), and G = Zhi (Zhi + 2 Zlo)^T takes two MMAs per 16
// segments.  V's real and imaginary parts are the symmetric and antisymmetric
// parts of G's blocks (hi hi' counted half in G and half in its transpose), formed
// once at the end through shared memory.  (Nine MMAs of 16 to 64 columns for
// the same products, each paying a minimum of 32 cycles, took 1607 us for 32
// inputs x 4096 channels x 4096 segments, this one 610 to 640: the read of
// 4.3 GB at 7 TB/s, which bounds it; the CUDA cores took 4486.)
//
// S > 64, k_xmac_split (w = 1): 128 x 128 tiles on or below the diagonal,
//     Re V = Xr Xr^T + Xi Xi^T,   Im V = Xi Xr^T - Xr Xi^T,
// twelve MMAs per 16 segments, nine on a diagonal tile (its Im columns
// accumulate M = Xi Xr^T and Im V = M - M^T is formed at the end).
// 200 inputs x 1024 channels x 4096 segments take 2.4 ms (the CUDA cores 26.6 ms), of
// which the MMAs are 1.5 ms at 64 cycles each and most of the rest the waits and
// commits between chunks (tensor pipe 46 %, DRAM 29 %).  Before the issuing lanes were
// elected: 2.59 ms, one issuer 2.67, and with four 64-byte planes per operand
// instead of two of 128 bytes 3.17.
//
// What keeps both at FP32 accuracy is the accumulation: the tensor core adds
// each MMA to its FP32 accumulator without rounding to nearest, a bias that
// grows with the number of MMAs on positive sums.  So an accumulator lives for
// one 32-segment chunk only: the small cross terms go in first, then the hi hi'
// terms, and the epilogue warps add the chunk to FP32 registers in
// round-to-nearest while the other TMEM buffer takes the next chunk.  What the
// cut of one chunk still takes from a sum of positive terms is 1.3e-7 of it
// (S <= 64; two hi hi' MMAs an accumulator) or 2.2e-7 (four).  The autos are
// such sums in every job, so they are added apart, in FP32: the F stage's write-out,
// which holds the FP32 values, sums |X|^2 over its tile of 16 to 64 segments (1/32
// to 1/128 of the spectra's bytes), and k_split_autos adds those, 8 us for 10 inputs
// of 4096 segments and 20 for 200 of 2048.  (Squared here, from the operand rows in
// the ring, by the epilogue's warps or the producer's, 64 inputs took 490 us and not
// 340, 200 inputs of 2048 segments 1508 and not 1258: their work then sets the pace.)
//
// Error against FP64 (inputs that share a tenth of their power; N = 512, 2048,
// 8192 and 32768, S = 9 .. 200) over that of the CUDA cores' serial sum
// (cs_xmac_f32), which grows with K: cross products 0.90 to 0.99 at K = 64, 0.40
// to 0.60 at 512, but 1.00 to 1.09 at 24 and 32, where those are used
// (CS_SPLIT_MIN_K); autos 0.57 to 0.69 at 64, 0.23 to 0.30 at 512.  Cross products of fully
// correlated inputs are positive sums as well: up to 1.2 (S <= 64) and 1.6 at 64
// segments, 1 at 128 and 256, 0.5 and 0.7 at 512.
//
// Warp roles: warps 0 .. E-1 epilogue (warp w reads TMEM lanes 32 (w % 4)
// ..+31), warp E TMA producer, warp E + 1 TMEM owner and MMA issuer.  TMA boxes
// are 128-byte rows (32 hi, 32 lo halves) in 128-byte swizzle.  Every mbarrier
// wait is bounded; on timeout the kernel records an error code, lets the MMAs
// and copies in flight end, frees TMEM and returns.
//
// Layout in:  half [C][S][kp/32][2][64], planes Re and Im of 32 hi and 32 lo
//             halves; segments from K to the next multiple of 32 are zero
// Layout out: float2 vis[C][P], p = i(i+1)/2 + j, j <= i
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"
#include "tma.h"

#include <algorithm>

namespace {

constexpr int BM = 128, BK = 32;                    // tile edge and segments per chunk
constexpr int ROW_BYTES = BK * 4;                   // 32 hi and 32 lo halves
constexpr int MAX_STAGES = 6;
constexpr long long WAIT_CYCLES = 4000000000LL;     // ~2 s at 2 GHz
constexpr unsigned ERR_FULL_WAIT = 1, ERR_EMPTY_WAIT = 2, ERR_ACC_WAIT = 3, ERR_DRAIN_WAIT = 4;

// K-major operand of 128-byte rows; a descriptor's low 14 bits hold the address / 16,
// so an offset within the operand ring is added to them
CS_DEV uint64_t sw128_desc(uint32_t saddr) { return tc::smem_desc(saddr, 16, 8 * ROW_BYTES, tc::SW128); }
// offsets / 16 of a chunk's terms within a row: two k-steps of 16 halves each
CS_DEV constexpr uint32_t hi16(int kk) { return 2 * kk; }
CS_DEV constexpr uint32_t lo16(int kk) { return 4 + 2 * kk; }

// AND vote of the `nthreads` epilogue threads (named barrier 1), which every one of them reaches
CS_DEV bool epi_vote(bool ok, int nthreads)
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

struct SplitArgs {
    int S, K;
    int64_t P;
    float2* vis;
    float inv;                  // 1 / s: every product is scaled by inv twice
    int stages;
    unsigned* err;              // CsErrorWord::code of the job
    uint32_t plane_bytes;       // k_xmac_split: one plane of an operand, box rows x 128 bytes
};

// shared memory after the ring: full[], empty[], accf[2], acce[2], done, the TMEM address
constexpr int BAR_BYTES = (2 * MAX_STAGES + 5) * 8 + 16;

// The barriers and TMEM of a CTA, and the two roles both kernels share.
struct Pipe {
    unsigned* err;                                   // CsErrorWord::code of the job
    uint32_t full0, empty0, accf, acce, done, tmem;
    int stages;
};

// One CTA's set-up: barriers (E epilogue warps release an accumulator), TMEM.
template <int E, int ISSUERS>
CS_DEV Pipe pipe_open(unsigned char* after, int stages, uint32_t tmem_cols, unsigned* err, const CUtensorMap* tmap)
{
    uint64_t* bars = reinterpret_cast<uint64_t*>(after);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 5);
    Pipe p;
    p.err = err;
    p.stages = stages;
    p.full0 = tc::smem_u32(bars);
    p.empty0 = p.full0 + 8 * MAX_STAGES;
    p.accf = p.empty0 + 8 * MAX_STAGES;
    p.acce = p.accf + 16;
    p.done = p.acce + 16;
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            tc::mbar_init(p.full0 + 8 * s, 1);
            tc::mbar_init(p.empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(p.accf + 8 * b, 1);
            tc::mbar_init(p.acce + 8 * b, E);
        }
        tc::mbar_init(p.done, ISSUERS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
    }
    if ((threadIdx.x >> 5) == E + 1) tc::tmem_alloc(tc::smem_u32(slot), tmem_cols);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    p.tmem = *slot;
    return p;
}

// TMA producer (one thread): `load(kc, stage, bar)` issues chunk kc's copies of `bytes` bytes.
template <class Load>
CS_DEV void produce(const Pipe& p, int nk, uint32_t bytes, Load load)
{
    int issued = 0, s = 0;
    uint32_t ph = 1;
    for (int kc = 0; kc < nk; kc++) {
        if (!tc::mbar_wait(p.empty0 + 8 * s, ph, p.err, ERR_EMPTY_WAIT, WAIT_CYCLES)) break;
        tc::mbar_expect_tx(p.full0 + 8 * s, bytes);
        load(kc, s, p.full0 + 8 * s);
        issued = kc + 1;
        if (++s == p.stages) s = 0, ph ^= 1;
    }
    // every stage this thread filled must have landed before the CTA exits
    for (int kc = (issued > p.stages ? issued - p.stages : 0); kc < issued; kc++)
        tc::mbar_wait(p.full0 + 8 * (kc % p.stages), (kc / p.stages) & 1, p.err, ERR_DRAIN_WAIT, WAIT_CYCLES);
}

// MMA issuer (one thread): `mmas(stage, buffer)` issues the MMAs of the chunks
// first, first + step, ...
template <class Mmas>
CS_DEV void issue(const Pipe& p, int nk, int first, int step, Mmas mmas)
{
    for (int kc = first; kc < nk; kc += step) {
        const int b = kc & 1, s = kc % p.stages;
        if (!tc::mbar_wait(p.acce + 8 * b, ((kc >> 1) & 1) ^ 1, p.err, ERR_ACC_WAIT, WAIT_CYCLES)) break;
        if (!tc::mbar_wait(p.full0 + 8 * s, (kc / p.stages) & 1, p.err, ERR_FULL_WAIT, WAIT_CYCLES)) break;
        tc::fence_after();
        mmas(s, b);
        tc::commit(p.empty0 + 8 * s);
        tc::commit(p.accf + 8 * b);
    }
    // TMEM is freed only after every MMA issued has finished
    tc::commit(p.done);
    tc::mbar_wait(p.done, 0, p.err, ERR_DRAIN_WAIT, WAIT_CYCLES);
}

// Epilogue warp: adds each chunk's columns [0, ncol) of `lanes` (TMEM address of
// its lane quarter in buffer 0; buffers `step` columns apart) to acc.
template <int NC>
CS_DEV bool accumulate(const Pipe& p, int nk, uint32_t lanes, uint32_t step, int ncol, float (&acc)[NC])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < NC; j++) acc[j] = 0.f;
    bool ok = true;
    for (int kc = 0; kc < nk; kc++) {
        const int b = kc & 1;
        ok = __all_sync(0xffffffffu, tc::mbar_wait(p.accf + 8 * b, (kc >> 1) & 1, p.err, ERR_ACC_WAIT, WAIT_CYCLES));
        if (!ok) break;
        tc::fence_after();
#pragma unroll
        for (int cb = 0; cb < NC / 32; cb++) {
            if (cb * 32 < ncol) {
                uint32_t u[16], v[16];
                tc::tmem_ld_32x32b_x16(lanes + b * step + cb * 32, u);
                tc::tmem_ld_32x32b_x16(lanes + b * step + cb * 32 + 16, v);
                tc::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    acc[cb * 32 + j] += __uint_as_float(u[j]);
                    acc[cb * 32 + 16 + j] += __uint_as_float(v[j]);
                }
            }
        }
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(p.acce + 8 * b);
    }
    ok = ok && (*reinterpret_cast<volatile unsigned*>(p.err) == 0u);
    return __all_sync(0xffffffffu, ok);
}

CS_DEV unsigned char* align1k(unsigned char* p) { return p + ((1024u - (tc::smem_u32(p) & 1023u)) & 1023u); }

// ---- S <= 64: the Gram matrix of Z = [Xr; Xi], 2 R rows -----------------------
// CTAs per SM by TMEM (two buffers of 2 R columns) and shared memory
template <int R> constexpr int gram_ctas() { return 128 / R; }
template <int R> constexpr uint32_t gram_stage() { return 2 * R * ROW_BYTES; }
// the MMA reads 128 operand rows; those past the stage's 2 R feed lanes never read
template <int R> constexpr uint32_t gram_slack() { return BM * ROW_BYTES - gram_stage<R>(); }

template <int R>
__global__ void __launch_bounds__(2 * R + 64, gram_ctas<R>())
    k_xmac_gram(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ SplitArgs a)
{
    constexpr int E = 2 * R / 32, NC = 2 * R;
    constexpr uint32_t STAGE = gram_stage<R>(), COLS = 2 * NC;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = align1k(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x, nk = (a.K + BK - 1) / BK;
    const Pipe p = pipe_open<E, 1>(smem + a.stages * STAGE + gram_slack<R>(), a.stages, COLS, a.err, &tmap);
    const uint32_t sbase = tc::smem_u32(smem);
    if (warp == E) {
        if (tc::elect_one())
            produce(p, nk, STAGE, [&](int kc, int s, uint32_t bar) {
                tc::tma_load_5d(sbase + s * STAGE, &tmap, 0, 0, 0, kc, c, bar);
            });
    } else if (warp == E + 1) {
        if (tc::elect_one()) {
            const uint32_t id = tc::idesc_f16(BM, NC, false, false, false);
            const uint64_t d0 = sw128_desc(sbase);
            issue(p, nk, 0, 1, [&](int s, int b) {
                const uint64_t d = d0 + s * (STAGE / 16);
                const uint32_t g = p.tmem + b * NC;
                tc::mma_f16(g, d + hi16(0), d + lo16(0), id, 0u);
                tc::mma_f16(g, d + hi16(1), d + lo16(1), id, 1u);
                tc::mma_f16(g, d + hi16(0), d + hi16(0), id, 1u);
                tc::mma_f16(g, d + hi16(1), d + hi16(1), id, 1u);
            });
        }
        __syncwarp();
    } else {
        float acc[NC];
        const bool ok = accumulate<NC>(p, nk, p.tmem + ((uint32_t)(32 * warp) << 16), NC, NC, acc);
        // all or none of the epilogue warps go on; the last chunk's MMAs are
        // done, so the operand ring is free
        constexpr int GP = NC + 1;
        float* g = reinterpret_cast<float*>(smem);
        if (epi_vote(ok, 32 * E)) {
#pragma unroll
            for (int j = 0; j < NC; j++) g[(32 * warp + lane) * GP + j] = acc[j];
            epi_vote(true, 32 * E);
            float2* out = a.vis + (int64_t)c * a.P;
            for (int t = threadIdx.x; t < (int)a.P; t += 32 * E) {
                int i = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
                if ((i + 1) * (i + 2) / 2 <= t) i++;
                else if (i * (i + 1) / 2 > t) i--;
                const int j = t - i * (i + 1) / 2;
                const float re = (g[i * GP + j] + g[j * GP + i]) + (g[(R + i) * GP + R + j] + g[(R + j) * GP + R + i]);
                const float im = (g[(R + i) * GP + j] - g[(R + j) * GP + i]) + (g[j * GP + R + i] - g[i * GP + R + j]);
                out[t] = make_float2(re * a.inv * a.inv * 0.5f, im * a.inv * a.inv * 0.5f);
            }
        }
        tc::fence_before();
    }
    __syncthreads();
    if (warp == E + 1) {
        tc::fence_after();
        tc::tmem_dealloc(p.tmem, COLS);
    }
}

// ---- S > 64: 128 x 128 tiles --------------------------------------------------
constexpr int T_E = 8, T_NC = 64;                   // epilogue warps: 4 row quarters x 2 column halves
constexpr uint32_t T_COLS = 512, T_HALF = 256, T_IM = 128;

__global__ void __launch_bounds__(32 * (T_E + 3), 1)
    k_xmac_split(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ SplitArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = align1k(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.y, S = a.S, nk = (a.K + BK - 1) / BK;
    int bi = 0, bj = blockIdx.x;                     // lower-triangle tile of this CTA, row by row
    while (bj > bi) bj -= ++bi;
    const int i0 = bi * BM, j0 = bj * BM;
    const bool diag = bi == bj;
    const uint32_t n_eff = (uint32_t)((min(j0 + BM, S) - j0 + 15) & ~15);   // columns of this tile
    const uint32_t op_bytes = 2 * a.plane_bytes;
    // S <= 128: the one tile's stages hold one operand; its MMAs may read up to
    // 128 rows of a plane of fewer (lanes never stored)
    const uint32_t stage_bytes = gridDim.x == 1 ? op_bytes : 2 * op_bytes;
    const uint32_t slack = BM * ROW_BYTES - a.plane_bytes;
    const Pipe p = pipe_open<T_E, 2>(smem + a.stages * stage_bytes + slack, a.stages, T_COLS, a.err, &tmap);
    const uint32_t sbase = tc::smem_u32(smem);
    if (warp == T_E) {
        if (tc::elect_one())
            produce(p, nk, diag ? op_bytes : 2 * op_bytes, [&](int kc, int s, uint32_t bar) {
                const uint32_t st = sbase + s * stage_bytes;
                tc::tma_load_5d(st, &tmap, 0, i0, 0, kc, c, bar);
                if (!diag) tc::tma_load_5d(st + op_bytes, &tmap, 0, j0, 0, kc, c, bar);
            });
    } else if (warp > T_E) {
        // two issuers, each with its own TMEM buffer (even and odd chunks): one's
        // waits and commits, about 500 cycles of a chunk, pass behind the other's MMAs
        if (tc::elect_one()) {
            const uint32_t pos = tc::idesc_f16(BM, n_eff, false, false, false);
            const uint32_t neg = tc::idesc_f16(BM, n_eff, true, false, false);
            const uint64_t d0 = sw128_desc(sbase);
            const uint32_t im_plane = a.plane_bytes / 16, st16 = stage_bytes / 16, b_op = diag ? 0 : op_bytes / 16;
            issue(p, nk, warp - (T_E + 1), 2, [&](int s, int b) {
                const uint64_t ar = d0 + s * st16, ai = ar + im_plane, br = ar + b_op, bi_ = br + im_plane;
                const uint32_t re = p.tmem + b * T_HALF, im = re + T_IM;
                // the cross terms of both k-steps first, then hi hi'
#pragma unroll
                for (int kk = 0; kk < 2; kk++) {
                    tc::mma_f16(re, ar + hi16(kk), br + lo16(kk), pos, kk);
                    tc::mma_f16(im, ai + hi16(kk), br + lo16(kk), pos, kk);
                    tc::mma_f16(re, ar + lo16(kk), br + hi16(kk), pos, 1u);
                    tc::mma_f16(im, ai + lo16(kk), br + hi16(kk), pos, 1u);
                    tc::mma_f16(re, ai + hi16(kk), bi_ + lo16(kk), pos, 1u);
                    if (!diag) tc::mma_f16(im, ar + hi16(kk), bi_ + lo16(kk), neg, 1u);
                    tc::mma_f16(re, ai + lo16(kk), bi_ + hi16(kk), pos, 1u);
                    if (!diag) tc::mma_f16(im, ar + lo16(kk), bi_ + hi16(kk), neg, 1u);
                }
#pragma unroll
                for (int kk = 0; kk < 2; kk++) {
                    tc::mma_f16(re, ar + hi16(kk), br + hi16(kk), pos, 1u);
                    tc::mma_f16(im, ai + hi16(kk), br + hi16(kk), pos, 1u);
                    tc::mma_f16(re, ai + hi16(kk), bi_ + hi16(kk), pos, 1u);
                    if (!diag) tc::mma_f16(im, ar + hi16(kk), bi_ + hi16(kk), neg, 1u);
                }
            });
        }
        __syncwarp();
    } else {
        // epilogue: rows 32 q ..+31, columns col0 ..+63, Re then Im
        const int q = warp & 3, col0 = (warp >> 2) * T_NC;
        const int ncol = min(T_NC, (int)n_eff - col0);         // columns of this warp (may be <= 0)
        float accr[T_NC], acci[T_NC];
#pragma unroll
        for (int j = 0; j < T_NC; j++) accr[j] = acci[j] = 0.f;
        const uint32_t lanes = p.tmem + ((uint32_t)(32 * q) << 16) + col0;
        bool ok = true;
        for (int kc = 0; kc < nk; kc++) {
            const int b = kc & 1;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(p.accf + 8 * b, (kc >> 1) & 1, p.err, ERR_ACC_WAIT, WAIT_CYCLES));
            if (!ok) break;
            tc::fence_after();
#pragma unroll
            for (int cb = 0; cb < T_NC / 16; cb++) {
                if (cb * 16 < ncol) {
                    uint32_t re[16], im[16];
                    tc::tmem_ld_32x32b_x16(lanes + b * T_HALF + cb * 16, re);
                    tc::tmem_ld_32x32b_x16(lanes + b * T_HALF + T_IM + cb * 16, im);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        accr[cb * 16 + j] += __uint_as_float(re[j]);
                        acci[cb * 16 + j] += __uint_as_float(im[j]);
                    }
                }
            }
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(p.acce + 8 * b);
        }
        ok = ok && (*reinterpret_cast<volatile unsigned*>(p.err) == 0u);
        // all or none of the epilogue warps go on: M - M^T needs every row.  The last
        // chunk's MMAs are done, so the operand ring is free: a 32 x 17 block
        // per warp, then (diagonal tile) M
        if (epi_vote(__all_sync(0xffffffffu, ok), 32 * T_E)) {
            float2* stg = reinterpret_cast<float2*>(smem) + warp * 32 * 17;
            float* msh = reinterpret_cast<float*>(smem + T_E * 32 * 17 * 8);
            constexpr int MP = BM + 1;
            const int r = 32 * q + lane;
            if (diag) {
#pragma unroll
                for (int j = 0; j < T_NC; j++) msh[r * MP + col0 + j] = acci[j];
                epi_vote(true, 32 * T_E);
            }
            const int row_end = min(S, i0 + 32 * q + 32);      // rows of this warp end here
            float2* out = a.vis + (int64_t)c * a.P;
#pragma unroll
            for (int cb = 0; cb < T_NC / 16; cb++) {
                const int jb = j0 + col0 + cb * 16;            // first column of the block
                if (cb * 16 < ncol && jb < row_end) {
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        float im = acci[cb * 16 + j];
                        if (diag) im -= msh[(col0 + cb * 16 + j) * MP + r];
                        stg[lane * 17 + j] = make_float2(accr[cb * 16 + j] * a.inv * a.inv, im * a.inv * a.inv);
                    }
                    __syncwarp();
#pragma unroll 4
                    for (int it = 0; it < 16; it++) {
                        const int rr = 2 * it + (lane >> 4), i = i0 + 32 * q + rr, j = jb + (lane & 15);
                        if (i < S && j <= i) out[(int64_t)i * (i + 1) / 2 + j] = stg[rr * 17 + (lane & 15)];
                    }
                    __syncwarp();
                }
            }
        }
        tc::fence_before();
    }
    __syncthreads();
    if (warp == T_E + 1) {
        tc::fence_after();
        tc::tmem_dealloc(p.tmem, T_COLS);
    }
}

// ---- the autos -------------------------------------------------------------------
// Input s's auto of 32 channels: eight slices of the F stage's partial sums (32
// channels of one block are 128 bytes), added in order.
constexpr int A_SLICES = 8;
__global__ void __launch_bounds__(32 * A_SLICES)
    k_split_autos(const float* __restrict__ squares, int S, int C, int c_pitch, int nb, int64_t P, float2* __restrict__ vis)
{
    __shared__ float part[A_SLICES][32];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, c = blockIdx.x * 32 + lane, s = blockIdx.y;
    float sum = 0.f;
    if (c < C) {
#pragma unroll 8
        for (int b = slice; b < nb; b += A_SLICES) sum += __ldg(squares + ((int64_t)b * S + s) * c_pitch + c);
    }
    part[slice][lane] = sum;
    __syncthreads();
    if (slice || c >= C) return;
#pragma unroll
    for (int q = 1; q < A_SLICES; q++) sum += part[q][lane];
    vis[(int64_t)c * P + (int64_t)s * (s + 3) / 2] = make_float2(sum, 0.f);
}

// stages of `stage` bytes that fit `ctas` CTAs' rings in an SM's shared memory
int ring_stages(int ctas, uint32_t stage, uint32_t slack)
{
    const uint32_t room = 224u * 1024 / ctas - slack - BAR_BYTES - 2048;
    return (int)std::min<uint32_t>(MAX_STAGES, room / stage);
}

template <int R>
int launch_gram(const CUtensorMap& tm, SplitArgs a, int C, cudaStream_t st)
{
    a.stages = ring_stages(gram_ctas<R>(), gram_stage<R>(), gram_slack<R>());
    const size_t smem = (size_t)a.stages * gram_stage<R>() + gram_slack<R>() + BAR_BYTES + 1024;
    auto kern = k_xmac_gram<R>;
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(kern), (int)smem));
    kern<<<C, 2 * R + 64, smem, st>>>(tm, a), cs_count_launches(1);
    return (int)cudaGetLastError();
}

int launch_autos(const float* squares, int nb, const SplitArgs& a, int C, int c_pitch, cudaStream_t st)
{
    k_split_autos<<<dim3((C + 31) / 32, a.S), 32 * A_SLICES, 0, st>>>(squares, a.S, C, c_pitch, nb, a.P, a.vis), cs_count_launches(1);
    return (int)cudaGetLastError();
}

}  // namespace

float cs_xmac_split_lo(int S) { return S <= 64 ? 2.f : 1.f; }

int cs_xmac_split(const void* spectra, const float* squares, int blocks, int S, int C, int c_pitch, int K, int kp,
                  float2* vis, float inv_scale, unsigned* err, cudaStream_t st)
{
    if (!spectra || !squares || !vis || !err || S > 65535 || S <= 0 || C <= 0 || K <= 0 || C > 65535 || kp % BK || kp < K || (uintptr_t)spectra % 16)
        return CS_ERR_ARG;
    CsEncodeTiledFn enc = cs_encode_tiled();
    if (!enc) return CS_ERR_UNSUPPORTED;
    const int nb = (S + BM - 1) / BM, tiles = nb * (nb + 1) / 2;
    const int rows = S <= 16 ? 16 : S <= 32 ? 32 : S <= 64 ? 64 : S < BM ? (S + 7) / 8 * 8 : BM;
    // (64 halves, inputs, planes, blocks, channels): one box brings both planes
    // of an operand's rows, each plane [rows][64]; inputs past S read as zeros
    CUtensorMap tm;
    const cuuint64_t blk = 2 * ROW_BYTES, row = (cuuint64_t)kp / BK * blk;
    cuuint64_t dim[5] = {2 * BK, (cuuint64_t)S, 2, (cuuint64_t)(K + BK - 1) / BK, (cuuint64_t)C};
    cuuint64_t stride[4] = {row, ROW_BYTES, blk, row * S};
    cuuint32_t box[5] = {2 * BK, (cuuint32_t)rows, 2, 1, 1}, one[5] = {1, 1, 1, 1, 1};
    if (enc(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(spectra), dim, stride, box, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return CS_ERR_ARG;
    SplitArgs a{S, K, (int64_t)S * (S + 1) / 2, vis, inv_scale, 0, err, (uint32_t)rows * ROW_BYTES};
    if (S <= 64) {
        const int rc = S <= 16 ? launch_gram<16>(tm, a, C, st) : S <= 32 ? launch_gram<32>(tm, a, C, st) : launch_gram<64>(tm, a, C, st);
        return rc ? rc : launch_autos(squares, blocks, a, C, c_pitch, st);
    }
    const uint32_t stage = (tiles == 1 ? 2 : 4) * a.plane_bytes, slack = BM * ROW_BYTES - a.plane_bytes;
    a.stages = ring_stages(1, stage, slack);
    const size_t smem = (size_t)a.stages * stage + slack + BAR_BYTES + 1024;
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(k_xmac_split), (int)smem));
    k_xmac_split<<<dim3(tiles, C), 32 * (T_E + 3), smem, st>>>(tm, a), cs_count_launches(1);
    CS_CUDA_TRY(cudaGetLastError());
    return launch_autos(squares, blocks, a, C, c_pitch, st);
}
