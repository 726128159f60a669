// X stage of up to 32 inputs straight from segment-major spectra [S][K][C], FP16 or
// FP32 taken as two FP16 terms.
//
// Transforms of 4096 points and more write each segment's spectrum contiguously,
// and cs_spectra_transpose turns them into time-innermost rows: a read and a
// write of all spectra (32 inputs x 4096 channels x 4096 segments: 730 us in
// FP16, 1690 us in FP32) only so that TMA can bring K-major operands.  Here the
// CTA that multiplies a few channels makes its own operands: one TMA copy brings 32
// bytes of channels (8 in FP16, 4 in FP32: one sector) of every input and
// segment of a chunk (32 KB), and each of eight warps' threads turns eight
// segments of its channels into 16-byte pieces of the swizzled operand rows, up
// to three chunks behind the copies.  The spectra are read once and nothing is
// written.  The arithmetic is k_xmac_tc_gram's (FP16: rows Xr and Xi, Re V and M in
// one accumulator) and k_xmac_gram's (FP32).  Bound by the read of the
// spectra, in FP16 also by the MMAs' least cost: those 32 inputs take 480 us in
// FP16 (2.15 GB, 318 us at the copy rate; 512 CTAs are 3.4 waves) and 870 us in
// FP32, with the transpose 1040 and 2300.  (Register loads instead of TMA: 614 and
// 1285 us, cp.async 1030 and 1700, both with a single MMA per 16 segments; the F
// stage writing blocks of channels for 128-byte TMA rows: 420 and 825, but its
// stores then cost more than that gains.)
//
// Every mbarrier wait is bounded; on timeout the kernel records an error code,
// lets the MMAs and copies in flight end, frees TMEM and returns.
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"
#include "tma.h"

#include <algorithm>

namespace {

constexpr int BM = 128;
constexpr int LOADERS = 256;                         // threads that make operands (8 warps)
constexpr long long WAIT_CYCLES = 4000000000LL;      // ~2 s at 2 GHz
constexpr unsigned ERR_FULL_WAIT = 1, ERR_EMPTY_WAIT = 2, ERR_ACC_WAIT = 3, ERR_DRAIN_WAIT = 4;

struct SegArgs {
    int S, C, K;
    int64_t P;
    float2* vis;                // [C][P]
    const float* inv_scale;     // FP16: [S][scale_stride] or null
    int scale_stride;
    float split, inv;           // FP32: scale of the two terms, 1 / split
    unsigned* err;              // CsErrorWord::code of the job
};

CS_DEV unsigned char* align1k(unsigned char* p) { return p + ((1024u - (tc::smem_u32(p) & 1023u)) & 1023u); }

// A chunk as TMA leaves it, [input][SEGS + 1 segments][32 bytes]: segment 8 kg +
// u of input s, piece h.  The copy brings one segment more than the chunk has, so
// that inputs lie 32 bytes apart in the banks and lanes that differ in h and s
// read without conflicts.  (Segments in another order would do without it, but the
// sums would then differ in the last bit from those of the other X-stage forms.)
template <int RI, int SEGS> struct Raw {
    static constexpr int ROWS = SEGS + 1;
    static constexpr uint32_t BYTES = RI * ROWS * 32;
    static CS_DEV uint32_t at(int s, int kg, int u, int h) { return (s * ROWS + 8 * kg + u) * 32 + h * 16; }
};

// TMA producer (one thread): the channels' chunks in order through DEPTH slots.
template <int DEPTH, int SEGS>
CS_DEV void feed(const CUtensorMap* tmap, uint32_t slots, uint32_t bytes, uint32_t rfull, uint32_t rempty, int nk,
                 unsigned* err)
{
    int issued = 0;
    for (int kc = 0; kc < nk; kc++) {
        const int r = kc % DEPTH;
        if (!tc::mbar_wait(rempty + 8 * r, ((kc / DEPTH) & 1) ^ 1, err, ERR_EMPTY_WAIT, WAIT_CYCLES)) break;
        tc::mbar_expect_tx(rfull + 8 * r, bytes);
        tc::tma_load_3d(slots + r * bytes, tmap, 8 * blockIdx.x, kc * SEGS, 0, rfull + 8 * r);
        issued = kc + 1;
    }
    // every slot this thread filled must have landed before the CTA exits
    for (int kc = (issued > DEPTH ? issued - DEPTH : 0); kc < issued; kc++)
        tc::mbar_wait(rfull + 8 * (kc % DEPTH), (kc / DEPTH) & 1, err, ERR_DRAIN_WAIT, WAIT_CYCLES);
}

// AND vote of `nthreads` threads on named barrier 1, which every one of them reaches
CS_DEV bool vote(bool ok, int nthreads)
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

// product index -> (i, j), j <= i
CS_DEV void product(int p, int& i, int& j)
{
    i = (int)((sqrtf(8.f * (float)p + 1.f) - 1.f) * 0.5f);
    if ((i + 1) * (i + 2) / 2 <= p) i++;
    else if (i * (i + 1) / 2 > p) i--;
    j = p - i * (i + 1) / 2;
}

// ---- FP16 ------------------------------------------------------------------
// RI: inputs rounded up to 16 or 32; eight channels per CTA, with accumulators of
// RI columns.  A chunk of SEGS segments gives each loader one task: 8 segments of 4
// channels of an input.
template <int RI> struct F16Cfg {
    static constexpr int CB = 8, SEGS = RI == 16 ? 64 : 32, ROWB = 2 * SEGS, KG = SEGS / 8;
    using R = Raw<RI, SEGS>;
    static constexpr int COLS = CB * RI;
    static constexpr uint32_t TILE = 2 * RI * ROWB, STAGE = CB * TILE;      // 32 KB
    static constexpr int STAGES = 3, DEPTH = 3;
    static constexpr uint32_t SLACK = (BM - RI) * ROWB;                     // operand rows an MMA reads past the ring
    static_assert(RI * KG * 2 == LOADERS, "one task per loader");
};

template <int RI>
__global__ void __launch_bounds__(LOADERS + 96, 1)
    k_xmac_seg_f16(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ SegArgs a)
{
    using F = F16Cfg<RI>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = align1k(smem_raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);     // full[], empty[], raw full[], raw empty[], acc
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2 * F::STAGES + 2 * F::DEPTH + 1);
    unsigned char* ring = smem + 1024;                       // operands, then (past the rows an MMA may read) raw chunks
    unsigned char* raw = ring + F::STAGES * F::STAGE + F::SLACK;
    const uint32_t full0 = tc::smem_u32(bars), empty0 = full0 + 8 * F::STAGES, rfull = empty0 + 8 * F::STAGES,
                   rempty = rfull + 8 * F::DEPTH, accb = rempty + 8 * F::DEPTH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.x * F::CB, nk = (a.K + F::SEGS - 1) / F::SEGS;
    if (tid == 0) {
        for (int s = 0; s < F::STAGES; s++) {
            tc::mbar_init(full0 + 8 * s, LOADERS / 32);
            tc::mbar_init(empty0 + 8 * s, 2);
        }
        for (int r = 0; r < F::DEPTH; r++) {
            tc::mbar_init(rfull + 8 * r, 1);
            tc::mbar_init(rempty + 8 * r, LOADERS / 32);
        }
        tc::mbar_init(accb, 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == LOADERS / 32) tc::tmem_alloc(tc::smem_u32(slot), F::COLS);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *slot;

    if (warp == LOADERS / 32 + 2) {
        if (tc::elect_one())
            feed<F::DEPTH, F::SEGS>(&tmap, tc::smem_u32(raw), F::R::BYTES, rfull, rempty, nk, a.err);
    } else if (warp >= LOADERS / 32) {
        // two issuers, four channels each: one thread's instructions took as long
        // as the MMAs (611 us with one, 512 unrolled, 487 with two; 474 since one lane is elected, 480 with the lane mask)
        const int ca = (warp - LOADERS / 32) * (F::CB / 2);
        if (tc::elect_one()) {
            const uint32_t id = tc::idesc_f16(BM, RI, false, false, false);
            const uint64_t d0 = tc::smem_desc(tc::smem_u32(ring), 16, 8 * F::ROWB, F::ROWB == 128 ? tc::SW128 : tc::SW64);
            const tc::LaneMask re_lanes = tc::first_lanes(RI);
            for (int kc = 0; kc < nk; kc++) {
                const int s = kc % F::STAGES;
                if (!tc::mbar_wait(full0 + 8 * s, (kc / F::STAGES) & 1, a.err, ERR_FULL_WAIT, WAIT_CYCLES)) break;
                tc::fence_after();
#pragma unroll
                for (int q = 0; q < F::CB / 2; q++) {
                    const int c = ca + q;
                    const uint64_t d = d0 + (s * F::STAGE + c * F::TILE) / 16, di = d + RI * F::ROWB / 16;
#pragma unroll
                    for (int kk = 0; kk < F::SEGS / 16; kk++) {
                        tc::mma_f16(tmem + c * RI, d + 2 * kk, d + 2 * kk, id, (kc | kk) ? 1u : 0u);
                        tc::mma_f16(tmem + c * RI, di + 2 * kk, di + 2 * kk, id, 1u, re_lanes);
                    }
                }
                tc::commit(empty0 + 8 * s);
            }
            // always: completes only after every MMA issued has finished
            tc::commit(accb);
        }
        __syncwarp();
    } else {
        // this thread's task: input si, segments 8 kg ..+7 of a chunk, channels 4 ch ..+3
        const int ch = tid & 1, si = (tid >> 1) % RI, kg = (tid >> 1) / RI;
        const int sw = F::ROWB == 128 ? (si & 7) : ((si >> 1) & 3);       // RI is a multiple of 8: the same for the Im row
        const uint32_t dst = (uint32_t)(4 * ch) * F::TILE + si * F::ROWB + ((kg ^ sw) * 16);
        bool ok = true;
        for (int kc = 0; kc < nk && ok; kc++) {
            const int s = kc % F::STAGES, r = kc % F::DEPTH;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(rfull + 8 * r, (kc / F::DEPTH) & 1, a.err, ERR_FULL_WAIT, WAIT_CYCLES));
            if (!ok) break;
            uint4 v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = *reinterpret_cast<const uint4*>(raw + r * F::R::BYTES + F::R::at(si, kg, u, ch));
            ok = tc::mbar_wait(empty0 + 8 * s, ((kc / F::STAGES) & 1) ^ 1, a.err, ERR_EMPTY_WAIT, WAIT_CYCLES);
            if (__all_sync(0xffffffffu, ok)) {
                unsigned char* st = ring + s * F::STAGE + dst;
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    uint32_t w[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) w[u] = x == 0 ? v[u].x : x == 1 ? v[u].y : x == 2 ? v[u].z : v[u].w;
#pragma unroll
                    for (int im = 0; im < 2; im++) {
                        const uint32_t sel = im ? 0x7632u : 0x5410u;
                        *reinterpret_cast<uint4*>(st + x * F::TILE + im * RI * F::ROWB) =
                            make_uint4(__byte_perm(w[0], w[1], sel), __byte_perm(w[2], w[3], sel),
                                       __byte_perm(w[4], w[5], sel), __byte_perm(w[6], w[7], sel));
                    }
                }
                tc::fence_proxy_async();
            } else {
                ok = false;
            }
            __syncwarp();
            // the raw slot too only after the fence: it orders this thread's reads
            // before the TMA copy that will overwrite them
            if (lane == 0 && ok) {
                tc::mbar_arrive(full0 + 8 * s);
                tc::mbar_arrive(rempty + 8 * r);
            }
        }
        ok = ok && tc::mbar_wait(accb, 0, a.err, ERR_ACC_WAIT, WAIT_CYCLES);
        ok = ok && (*reinterpret_cast<volatile unsigned*>(a.err) == 0u);
        if (vote(__all_sync(0xffffffffu, ok), LOADERS)) {
            tc::fence_after();
            // the ring is free: every channel's Re V rows, then M rows, [2 RI][RI + 1]
            constexpr int GP = RI + 1, Q = 2 * RI / 32;                     // Q: lane quarters in use
            float* g0 = reinterpret_cast<float*>(ring);
            const int q = warp & 3;
            if (q < Q)
                // two warps read each quarter, every other 16 columns
                for (int t = (warp >> 2) * 16; t < F::CB * RI; t += 32) {
                    const int c = t / RI, col = t % RI;
                    uint32_t v[16];
                    tc::tmem_ld_32x32b_x16(tmem + ((uint32_t)(32 * q) << 16) + t, v);
                    tc::tmem_ld_wait();
                    float* g = g0 + (c * 2 * RI + 32 * q + lane) * GP + col;
#pragma unroll
                    for (int j = 0; j < 16; j++) g[j] = __uint_as_float(v[j]);
                }
            vote(true, LOADERS);
            for (int c = 0; c < F::CB; c++) {
                const int cg = c0 + c;
                const float* g = g0 + c * 2 * RI * GP;
                float2* out = a.vis + (int64_t)cg * a.P;
                for (int p = tid; p < (int)a.P; p += LOADERS) {
                    int i, j;
                    product(p, i, j);
                    float2 v = make_float2(g[i * GP + j], g[(RI + i) * GP + j] - g[(RI + j) * GP + i]);
                    if (a.inv_scale) {
                        const float f = __ldg(a.inv_scale + (int64_t)i * a.scale_stride + cg) *
                                        __ldg(a.inv_scale + (int64_t)j * a.scale_stride + cg);
                        v = make_float2(v.x * f, v.y * f);
                    }
                    out[p] = v;
                }
            }
        }
        tc::fence_before();
    }
    __syncthreads();
    if (warp == LOADERS / 32) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, F::COLS);
    }
}

// ---- FP32 as two FP16 terms ------------------------------------------------------
// Four channels per CTA, chunks of 32 segments, operand rows of 32 hi and 32 lo
// halves, accumulators of one chunk added to FP32 registers (k_xmac_gram's
// arithmetic).  Of warps 0 .. 15 those with bit 1 set make operands, the others
// are epilogue warps: channel w / 4, lane quarter w & 1.  Warp 16 issues the MMAs, warp 17 the copies.
template <int RI> struct SplitCfg {
    static constexpr int CB = 4, SEGS = 32, ROWB = 128, N2 = 2 * RI, Q = N2 / 32;
    using R = Raw<RI, SEGS>;
    static constexpr uint32_t TILE = N2 * ROWB, STAGE = CB * TILE;          // 32 or 16 KB
    static constexpr int COLS = 2 * CB * N2, STAGES = RI == 16 ? 4 : 3, DEPTH = RI == 16 ? 6 : 3;
    static constexpr uint32_t SLACK = (BM - N2) * ROWB;
    static constexpr int GROUPS = LOADERS / (RI * 8);                       // loaders work on GROUPS chunks at once
    static constexpr int PARTS = GROUPS * SEGS / 8;                         // loaders that share an input's squares
    static constexpr int E = CB * Q;                                        // epilogue warps
};
constexpr int SPLIT_THREADS = 18 * 32;

template <int RI>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
    k_xmac_seg_split(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ SegArgs a)
{
    using F = SplitCfg<RI>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = align1k(smem_raw);
    // full[], empty[], accf[2], acce[2], done, raw full[], raw empty[]
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2 * F::STAGES + 5 + 2 * F::DEPTH);
    float* sq = reinterpret_cast<float*>(smem + 1024);       // [PARTS][CB][RI], 2 KB
    unsigned char* ring = smem + 3072;                       // operands, then (past the rows an MMA may read) raw chunks
    unsigned char* raw = ring + F::STAGES * F::STAGE + F::SLACK;
    const uint32_t full0 = tc::smem_u32(bars), empty0 = full0 + 8 * F::STAGES, accf = empty0 + 8 * F::STAGES, acce = accf + 16,
                   done = acce + 16, rfull = done + 8, rempty = rfull + 8 * F::DEPTH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.x * F::CB, nk = (a.K + F::SEGS - 1) / F::SEGS;
    if (tid == 0) {
        for (int s = 0; s < F::STAGES; s++) {
            tc::mbar_init(full0 + 8 * s, LOADERS / 32 / F::GROUPS);
            tc::mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(accf + 8 * b, 1);
            tc::mbar_init(acce + 8 * b, F::E);
        }
        for (int r = 0; r < F::DEPTH; r++) {
            tc::mbar_init(rfull + 8 * r, 1);
            tc::mbar_init(rempty + 8 * r, LOADERS / 32 / F::GROUPS);
        }
        tc::mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 16) tc::tmem_alloc(tc::smem_u32(slot), F::COLS);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *slot;

    if (warp == 17) {
        if (tc::elect_one())
            feed<F::DEPTH, F::SEGS>(&tmap, tc::smem_u32(raw), F::R::BYTES, rfull, rempty, nk, a.err);
    } else if (warp == 16) {
        if (tc::elect_one()) {
            const uint32_t id = tc::idesc_f16(BM, F::N2, false, false, false);
            const uint64_t d0 = tc::smem_desc(tc::smem_u32(ring), 16, 8 * F::ROWB, tc::SW128);
            for (int kc = 0; kc < nk; kc++) {
                const int s = kc % F::STAGES, b = kc & 1;
                if (!tc::mbar_wait(acce + 8 * b, ((kc >> 1) & 1) ^ 1, a.err, ERR_ACC_WAIT, WAIT_CYCLES)) break;
                if (!tc::mbar_wait(full0 + 8 * s, (kc / F::STAGES) & 1, a.err, ERR_FULL_WAIT, WAIT_CYCLES)) break;
                tc::fence_after();
#pragma unroll 1
                for (int c = 0; c < F::CB; c++) {
                    // hi halves at byte 0, lo at byte 64, 16 segments are 32 bytes; cross terms first
                    const uint64_t d = d0 + (s * F::STAGE + c * F::TILE) / 16;
                    const uint32_t g = tmem + (b * F::CB + c) * F::N2;
                    tc::mma_f16(g, d, d + 4, id, 0u);
                    tc::mma_f16(g, d + 2, d + 6, id, 1u);
                    tc::mma_f16(g, d, d, id, 1u);
                    tc::mma_f16(g, d + 2, d + 2, id, 1u);
                }
                tc::commit(empty0 + 8 * s);
                tc::commit(accf + 8 * b);
            }
            // TMEM is freed only after every MMA issued has finished
            tc::commit(done);
            tc::mbar_wait(done, 0, a.err, ERR_DRAIN_WAIT, WAIT_CYCLES);
        }
        __syncwarp();
    } else if (warp & 2) {
        // loader: channels 2 ch and 2 ch + 1, segments 8 kg ..+7 of an input, and the
        // sums of their squares: the autos are formed from the FP32 values (see
        // xstage_split.cu), a chunk's eight segments first
        const int t = ((warp >> 2) * 2 + (warp & 1)) * 32 + lane;          // 0 .. 255
        const int grp = t / (RI * 8), u0 = t % (RI * 8);
        const int ch = u0 & 1, si = (u0 >> 1) % RI, kg = (u0 >> 1) / RI;
        const int sw = si & 7;
        const uint32_t row = (uint32_t)(2 * ch) * F::TILE + si * F::ROWB;
        const uint32_t hi_at = row + ((kg ^ sw) * 16), lo_at = row + (((kg + 4) ^ sw) * 16);
        float squares[2] = {0.f, 0.f};
        bool ok = true;
        for (int kc = grp; kc < nk && ok; kc += F::GROUPS) {
            const int s = kc % F::STAGES, r = kc % F::DEPTH;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(rfull + 8 * r, (kc / F::DEPTH) & 1, a.err, ERR_FULL_WAIT, WAIT_CYCLES));
            if (!ok) break;
            uint4 v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = *reinterpret_cast<const uint4*>(raw + r * F::R::BYTES + F::R::at(si, kg, u, ch));
            ok = tc::mbar_wait(empty0 + 8 * s, ((kc / F::STAGES) & 1) ^ 1, a.err, ERR_EMPTY_WAIT, WAIT_CYCLES);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                unsigned char* st = ring + s * F::STAGE;
#pragma unroll
                for (int x = 0; x < 2; x++) {
                    float part = 0.f;
#pragma unroll
                    for (int im = 0; im < 2; im++) {
                        uint32_t h[4], l[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const uint4 e = v[2 * q], o = v[2 * q + 1];
                            const float fa = __uint_as_float(x ? (im ? e.w : e.z) : (im ? e.y : e.x)) * a.split;
                            const float fb = __uint_as_float(x ? (im ? o.w : o.z) : (im ? o.y : o.x)) * a.split;
                            part = fmaf(fa, fa, part);
                            part = fmaf(fb, fb, part);
                            const __half2 hh = __floats2half2_rn(fa, fb);
                            const float2 hf = __half22float2(hh);
                            const __half2 ll = __floats2half2_rn(2.f * (fa - hf.x), 2.f * (fb - hf.y));
                            h[q] = *reinterpret_cast<const uint32_t*>(&hh);
                            l[q] = *reinterpret_cast<const uint32_t*>(&ll);
                        }
                        const uint32_t at = x * F::TILE + im * RI * F::ROWB;
                        *reinterpret_cast<uint4*>(st + hi_at + at) = make_uint4(h[0], h[1], h[2], h[3]);
                        *reinterpret_cast<uint4*>(st + lo_at + at) = make_uint4(l[0], l[1], l[2], l[3]);
                    }
                    squares[x] += part;
                }
                tc::fence_proxy_async();
            }
            __syncwarp();
            // the raw slot too only after the fence: it orders this thread's reads
            // before the TMA copy that will overwrite them
            if (lane == 0 && ok) {
                tc::mbar_arrive(full0 + 8 * s);
                tc::mbar_arrive(rempty + 8 * r);
            }
        }
#pragma unroll
        for (int x = 0; x < 2; x++) sq[((grp * (F::SEGS / 8) + kg) * F::CB + 2 * ch + x) * RI + si] = squares[x];
        asm volatile("bar.arrive 2, %0;" ::"n"(LOADERS + 32 * F::E) : "memory");
    } else if ((warp & 1) < F::Q) {
        // epilogue: channel warp / 4, rows 32 q ..+31 of its G
        const int c = warp >> 2, q = warp & 1;
        float acc[F::N2];
#pragma unroll
        for (int j = 0; j < F::N2; j++) acc[j] = 0.f;
        const uint32_t at = tmem + ((uint32_t)(32 * q) << 16) + c * F::N2;
        bool ok = true;
        for (int kc = 0; kc < nk; kc++) {
            const int b = kc & 1;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(accf + 8 * b, (kc >> 1) & 1, a.err, ERR_ACC_WAIT, WAIT_CYCLES));
            if (!ok) break;
            tc::fence_after();
#pragma unroll
            for (int cb = 0; cb < F::N2; cb += 32) {
                uint32_t u[16], v[16];
                tc::tmem_ld_32x32b_x16(at + b * F::CB * F::N2 + cb, u);
                tc::tmem_ld_32x32b_x16(at + b * F::CB * F::N2 + cb + 16, v);
                tc::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    acc[cb + j] += __uint_as_float(u[j]);
                    acc[cb + 16 + j] += __uint_as_float(v[j]);
                }
            }
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(acce + 8 * b);
        }
        // every loader arrives here, whatever became of its waits
        asm volatile("bar.sync 2, %0;" ::"n"(LOADERS + 32 * F::E) : "memory");
        ok = ok && (*reinterpret_cast<volatile unsigned*>(a.err) == 0u);
        if (vote(__all_sync(0xffffffffu, ok), 32 * F::E)) {
            // the last chunk's MMAs are done, so the ring is free
            constexpr int GP = F::N2 + 1;
            float* g = reinterpret_cast<float*>(ring) + c * F::N2 * GP;
#pragma unroll
            for (int j = 0; j < F::N2; j++) g[(32 * q + lane) * GP + j] = acc[j];
            vote(true, 32 * F::E);
            float2* out = a.vis + (int64_t)(c0 + c) * a.P;
            for (int p = 32 * q + lane; p < (int)a.P; p += 32 * F::Q) {
                int i, j;
                product(p, i, j);
                float re = 0.5f * ((g[i * GP + j] + g[j * GP + i]) + (g[(RI + i) * GP + RI + j] + g[(RI + j) * GP + RI + i]));
                if (i == j) {
                    re = 0.f;
#pragma unroll
                    for (int t = 0; t < F::PARTS; t++) re += sq[(t * F::CB + c) * RI + i];
                }
                const float im = 0.5f * ((g[(RI + i) * GP + j] - g[(RI + j) * GP + i]) + (g[j * GP + RI + i] - g[i * GP + RI + j]));
                out[p] = make_float2(re * a.inv * a.inv, im * a.inv * a.inv);
            }
        }
        tc::fence_before();
    }
    __syncthreads();
    if (warp == 16) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, F::COLS);
    }
}

// (words of a segment, segments, inputs): segments from K and inputs from S on read as zeros
template <class F>
bool encode_map(const void* spectra, const SegArgs& a, int words, int64_t pitch, int ri, CUtensorMap* tm)
{
    CsEncodeTiledFn enc = cs_encode_tiled();
    if (!enc) return false;
    const cuuint64_t dim[3] = {(cuuint64_t)words, (cuuint64_t)a.K, (cuuint64_t)a.S};
    const cuuint64_t stride[2] = {(cuuint64_t)pitch, (cuuint64_t)a.K * pitch};
    const cuuint32_t box[3] = {8, F::R::ROWS, (cuuint32_t)ri}, one[3] = {1, 1, 1};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(spectra), dim, stride, box, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int RI>
int launch_f16(const void* spectra, int64_t pitch, const SegArgs& a, cudaStream_t st)
{
    using F = F16Cfg<RI>;
    CUtensorMap tm;
    if (!encode_map<F>(spectra, a, a.C, pitch, RI, &tm)) return CS_ERR_ARG;
    const size_t ring = F::STAGES * F::STAGE + F::SLACK + F::DEPTH * F::R::BYTES, g = (size_t)F::CB * 2 * RI * (RI + 1) * 4;
    const size_t smem = 2048 + std::max(ring, g);
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(k_xmac_seg_f16<RI>), (int)smem));
    k_xmac_seg_f16<RI><<<a.C / F::CB, LOADERS + 96, smem, st>>>(tm, a), cs_count_launches(1);
    return (int)cudaGetLastError();
}

template <int RI>
int launch_split(const void* spectra, int64_t pitch, const SegArgs& a, cudaStream_t st)
{
    using F = SplitCfg<RI>;
    CUtensorMap tm;
    if (!encode_map<F>(spectra, a, 2 * a.C, pitch, RI, &tm)) return CS_ERR_ARG;
    const size_t ring = F::STAGES * F::STAGE + F::SLACK + F::DEPTH * F::R::BYTES, g = (size_t)F::CB * F::N2 * (F::N2 + 1) * 4;
    static_assert(F::PARTS * F::CB * RI * 4 == 2048, "squares");
    const size_t smem = 4096 + std::max(ring, g);
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(k_xmac_seg_split<RI>), (int)smem));
    k_xmac_seg_split<RI><<<a.C / F::CB, SPLIT_THREADS, smem, st>>>(tm, a), cs_count_launches(1);
    return (int)cudaGetLastError();
}

}  // namespace

bool cs_xmac_seg_supported(int S) { return S <= 32; }

int cs_xmac_seg(const void* spectra, int format, int S, int C, int c_pitch, int K, float2* vis, const float* inv_scale,
                int scale_stride, float split, unsigned* err, cudaStream_t st)
{
    if (!spectra || !vis || !err || S <= 0 || C <= 0 || K <= 0 || !cs_xmac_seg_supported(S)) return CS_ERR_ARG;
    // whole CTAs of channels; TMA: 16-byte pitch and base
    if (C % 8 || c_pitch % 8 || c_pitch < C || (uintptr_t)spectra % 16) return CS_ERR_ARG;
    const bool f16 = format == CS_SPECTRA_F16;
    // FP16 keeps the other tensor-core forms' rule on K
    if (f16 ? K % 8 != 0 : !(split > 0.f)) return CS_ERR_ARG;
    const SegArgs a{S, C, K, (int64_t)S * (S + 1) / 2, vis, inv_scale, scale_stride, split, f16 ? 0.f : 1.f / split, err};
    const int64_t pitch = (int64_t)c_pitch * (f16 ? 4 : 8);
    if (f16) return S <= 16 ? launch_f16<16>(spectra, pitch, a, st) : launch_f16<32>(spectra, pitch, a, st);
    return S <= 16 ? launch_split<16>(spectra, pitch, a, st) : launch_split<32>(spectra, pitch, a, st);
}
