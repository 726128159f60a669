// K-e + K-pcal: spectrometer power accumulation and phase-cal extraction.
//
// Semantics (TaskCoreIPP::doMaths, spectrometer/src/IA-32/TaskCoreIPP.cpp:
// 394-513, one source per subband): spectrum `spec` of subband `sub` is built
// from novl = overlap*K - (overlap-1) FFTs (swspectrometer.cpp:231) that start
// every N/overlap samples from sample spec*K*N; each FFT windows N samples
// (generate_windowfunction :569-605), takes the real FFT, and adds |X_k|^2 for
// k = 1..N/2-1 and X_0^2, X_{N/2}^2 (DC and Nyquist real, :437-447); the sum
// is scaled by 1/novl (:124, :493).
//
// GPU layout: the CTA grid is (chunk of CH FFTs) x (subband, spectrum) x
// (split p).  Inside a CTA, groups of M/16 threads run CtaFft on different
// FFTs of the chunk and accumulate |X|^2 into thread-owned shared-memory bins;
// the CTA writes one partial spectrum per chunk to scratch, and a reduce
// kernel adds the partials in chunk order (deterministic) and applies 1/novl.
// N = 65536 does not fit one SM's shared memory (32768 complex points), so it
// is split across two CTAs by output parity: CTA p computes the M/2-point FFT
// of y_p[n] = (z[n] + (-1)^p z[n + M/2]) W_M^{n p}, which yields
// Z[2m + p]; the real-FFT pairs (k, M-k) keep the parity, so each CTA finishes
// its own bins without exchanging data (input words are read twice, at 0.25 B
// per sample).
//
// Phase-cal (TaskCoreIPP::extract_PCal :633-693, settings
// swspectrometer.cpp:180-184): on the non-overlapped FFTs (every overlap-th),
// i.e. on every sample of the spectrum once, bins[(n mod L) mod T] +=
// x[n] * exp(-2 pi i f_off (n mod L) / fs), L = rotator length, T = tone
// bins.  Tones = DFT(bins)/T, first ntones (PCal.cpp:280-300, getFinalPCal).
#include "common.cuh"
#include "kernels.h"
#include "warpfft.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

namespace {

constexpr int SPEC_CH = CS_SPEC_CHUNK;   // most FFTs per chunk (one partial spectrum each) for N >= 4096

template <int MC> struct SCfg {
    static constexpr int T = MC / 16;
    static constexpr int GROUPS = (T >= 256) ? 1 : 256 / T;
    static constexpr int NT = T * GROUPS;
};

std::mutex g_win_mu;
std::map<std::tuple<int, int, int>, float*> g_win;   // (device, type, n)

const float* window_table(int type, int n)
{
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_win_mu);
    auto key = std::make_tuple(dev, type, n);
    auto it = g_win.find(key);
    if (it != g_win.end()) return it->second;
    std::vector<float> h(n);
    for (int i = 0; i < n; i++) h[i] = (float)cs_window_value(type, i, n);
    float* d = nullptr;
    if (cudaMalloc(&d, sizeof(float) * n) != cudaSuccess) return nullptr;
    cudaMemcpy(d, h.data(), sizeof(float) * n, cudaMemcpyHostToDevice);
    g_win[key] = d;
    return d;
}

// The same window in the order of k_spec_power_m's warps: pairs (2 n, 2 n + 1),
// n = n1 + m1 m, as [m1][1024].
std::map<std::tuple<int, int, int>, float2*> g_winp;
const float2* window_pairs(int type, int n, int m1)
{
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_win_mu);
    auto key = std::make_tuple(dev, type, n);
    auto it = g_winp.find(key);
    if (it != g_winp.end()) return it->second;
    std::vector<float2> h(n / 2);
    for (int i = 0; i < n / 2; i++)
        h[(i % m1) * 1024 + i / m1] = make_float2((float)cs_window_value(type, 2 * i, n), (float)cs_window_value(type, 2 * i + 1, n));
    float2* d = nullptr;
    if (cudaMalloc(&d, sizeof(float2) * (n / 2)) != cudaSuccess) return nullptr;
    cudaMemcpy(d, h.data(), sizeof(float2) * (n / 2), cudaMemcpyHostToDevice);
    g_winp[key] = d;
    return d;
}

std::map<std::tuple<int, int, long long, long long>, float2*> g_rot;

const float2* rotator_table(int L, double off_hz, double fs_hz)
{
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_win_mu);
    auto key = std::make_tuple(dev, L, (long long)llround(off_hz * 1e3), (long long)llround(fs_hz));
    auto it = g_rot.find(key);
    if (it != g_rot.end()) return it->second;
    std::vector<float2> h(L);
    double dphi = 2 * M_PI * (-off_hz / fs_hz);
    for (int i = 0; i < L; i++) h[i] = make_float2((float)std::cos(dphi * i), (float)std::sin(dphi * i));
    float2* d = nullptr;
    if (cudaMalloc(&d, sizeof(float2) * L) != cudaSuccess) return nullptr;
    cudaMemcpy(d, h.data(), sizeof(float2) * L, cudaMemcpyHostToDevice);
    g_rot[key] = d;
    return d;
}

// Samples s and s+1 (s even) of a plane word through a 16-entry table of
// level pairs (one shared-memory read instead of two 4-way selects); blanked
// samples (their bit in the validity mask clear) are 0.0, as mark5access
// decodes them.
CS_DEV float2 sample_pair16(const float2* __restrict__ lut16, uint32_t w, int f, const uint32_t* __restrict__ vmask,
                            int64_t s)
{
    float2 x = lut16[(w >> (2 * f)) & 15u];
    if (vmask) {
        const uint32_t m = __ldg(vmask + (s >> 5)) >> (s & 31);
        x.x = (m & 1u) ? x.x : 0.f;
        x.y = (m & 2u) ? x.y : 0.f;
    }
    return x;
}

template <int MC, int P>
__global__ void __launch_bounds__(SCfg<MC>::NT) k_spec_power(const __grid_constant__ CsSpecArgs a, const float2* __restrict__ tw,
                                                            const float* __restrict__ win, int nchunk, int ch)
{
    using C = SCfg<MC>;
    constexpr int T = C::T, GROUPS = C::GROUPS;
    constexpr int M = MC * P, N = 2 * M;
    constexpr int NACC = M / P + 1;                 // owned bins (local index)
    extern __shared__ __align__(16) unsigned char smem[];
    float2* fb_all = reinterpret_cast<float2*>(smem);
    float* acc_all = reinterpret_cast<float*>(fb_all + GROUPS * fpad_size(MC));

    const int g = threadIdx.x / T, t = threadIdx.x % T;
    float2* fb = fb_all + g * fpad_size(MC);
    float* acc = acc_all + g * NACC;
    const int chunk = blockIdx.x;
    const int row = blockIdx.y;                      // sub * nspec + spec
    const int sub = row / a.nspec, spec = row % a.nspec;
    const int p = (P == 2) ? (int)blockIdx.z : 0;
    const int novl = a.overlap * a.ffts_per_spectrum - (a.overlap - 1);
    const int hop = N / a.overlap;
    const uint32_t* plane = reinterpret_cast<const uint32_t*>(a.planes + (int64_t)sub * a.bytes_per_sub);
    const float lut[4] = {a.lut[0], a.lut[1], a.lut[2], a.lut[3]};
    const uint32_t* vmask = a.valid_mask;

    __shared__ float2 lut16[16];                     // level pairs: entry bits = code0 + 4 code1
    if (threadIdx.x < 16) lut16[threadIdx.x] = make_float2(lut[threadIdx.x & 3], lut[threadIdx.x >> 2]);
    for (int i = threadIdx.x; i < GROUPS * NACC; i += C::NT) acc_all[i] = 0.f;
    __syncthreads();

    const int j_begin = chunk * ch, j_end = min(novl, j_begin + ch);
    auto bar = [] { __syncthreads(); };
    // P = 2, odd outputs: sample pair n = t + r T is rotated by W_N^(2n) =
    // W_N^(2t) W_32^r (2T = N/32), one table load for all windows
    const float2 tw_t = (P == 2) ? twiddle(tw, 2 * t) : make_float2(1.f, 0.f);
    for (int j0 = j_begin; j0 < j_end; j0 += GROUPS) {
        const int j = j0 + g;
        const bool valid = j < j_end;
        const int64_t start = (int64_t)spec * a.ffts_per_spectrum * N + (int64_t)(valid ? j : j_begin) * hop;
        const uint32_t* wsrc = plane + (start >> 4);
        float2 v[16];
#pragma unroll
        for (int r = 0; r < 16; r++) {
            const int n = t + r * T;                 // index into the transformed sequence
            // window values of samples 2n, 2n+1 as one 8-byte load
            const float2* win2 = reinterpret_cast<const float2*>(win);
            if constexpr (P == 1) {
                uint32_t w = __ldg(wsrc + (2 * n >> 4));
                int f = (2 * n) & 15;
                const float2 x = sample_pair16(lut16, w, f, vmask, start + 2 * n);
                const float2 wn = __ldg(win2 + n);
                v[r] = make_float2(x.x * wn.x, x.y * wn.y);
            } else {
                const int n2 = n + MC;
                uint32_t w1 = __ldg(wsrc + (2 * n >> 4)), w2 = __ldg(wsrc + (2 * n2 >> 4));
                int f1 = (2 * n) & 15, f2 = (2 * n2) & 15;
                const float2 x1 = sample_pair16(lut16, w1, f1, vmask, start + 2 * n);
                const float2 x2 = sample_pair16(lut16, w2, f2, vmask, start + 2 * n2);
                // cosine^2: w(i + N/2) = sin^2 = 1 - w(i), so one table read
                // serves both halves (the table pair differs by <= 2^-24)
                const float2 wa = __ldg(win2 + n);
                const float2 wb = (a.window == 2) ? make_float2(1.f - wa.x, 1.f - wa.y) : __ldg(win2 + n2);
                float2 z1 = make_float2(x1.x * wa.x, x1.y * wa.y);
                float2 z2 = make_float2(x2.x * wb.x, x2.y * wb.y);
                v[r] = p ? cmul(csub(z1, z2), rot32(tw_t, r)) : cadd(z1, z2);
            }
        }
        CtaFft<MC, (MC >= 2048)>::run(fb, t, v, tw, N / MC, bar);
        if (valid) {
            const int mmax = (P == 1) ? MC / 2 : (p ? MC / 2 - 1 : MC / 2);
            for (int m = t; m <= mmax; m += T) {
                int k = P * m + p;
                int mb = (P == 1 || p == 0) ? ((MC - m) & (MC - 1)) : (MC - 1 - m);
                float2 Xk, Xm;
                r2c_pair(fb[fpad(m)], fb[fpad(mb)], twiddle(tw, k), Xk, Xm);
                if (k == 0) {
                    acc[0] += Xk.x * Xk.x;
                    acc[M / P] += Xm.x * Xm.x;
                } else {
                    acc[k / P] += Xk.x * Xk.x + Xk.y * Xk.y;
                    if (k != M / 2) acc[(M - k) / P] += Xm.x * Xm.x + Xm.y * Xm.y;
                }
            }
        }
        bar();
    }
    // combine groups, write the chunk partial (owned bins only)
    float* prow = a.partial + ((int64_t)row * nchunk + chunk) * (M + 1);
    for (int l = threadIdx.x; l < NACC; l += C::NT) {
        int k = P * l + p;
        if (k > M) continue;
        float s = 0.f;
#pragma unroll
        for (int gg = 0; gg < GROUPS; gg++) s += acc_all[gg * NACC + l];
        prow[k] = s;
    }
}

// The FFTs of one chunk: the plane words of FFT j as a thread group's cp.async
// copies into its shared buffer, in 16-byte pieces where the FFTs start on
// 16-byte boundaries (hop a multiple of 64 samples), in words otherwise.
CS_DEV void spec_fetch(uint32_t* dst, const uint32_t* __restrict__ plane, int64_t start, int words, int t, int nt, bool vec)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const uint32_t* src = plane + (start >> 4);
    if (vec) {
        for (int i = t; i < words / 4; i += nt)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * i), "l"(src + 4 * i) : "memory");
    } else {
        for (int i = t; i < words; i += nt)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4 * i), "l"(src + i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int PENDING> CS_DEV void spec_fetch_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// Whether any sample of the window [start, start + N) is blanked, as far as
// thread t of nt sees (start a multiple of 16).
CS_DEV bool spec_blanked(const uint32_t* __restrict__ vmask, int64_t start, int N, int t, int nt)
{
    bool any = false;
    if (start & 31) {
        for (int i = t; i < N / 16; i += nt) {
            const int64_t s = start + 16 * i;
            any |= ((__ldg(vmask + (s >> 5)) >> (s & 31)) & 0xffffu) != 0xffffu;
        }
    } else {
        for (int i = t; i < N / 32; i += nt) any |= __ldg(vmask + (start >> 5) + i) != 0xffffffffu;
    }
    return any;
}

// N = 1024 and 2048: a FFT in the registers of L lanes (WarpFft), its powers
// added to registers of the lanes that own the bins, so a group's only shared
// memory traffic is the plane words, the level pairs, the twiddles and one transpose, and
// no group waits on another until the chunk ends.  Bound by instruction issue
// (16 warps per SM; registers).  16 rows x 16383 FFTs of 1024 points: 235 us;
// the radix-16 groups with shared-memory accumulators and CTA barriers took 608.
constexpr int SP_NT = 256;
template <int L, int R, bool MASK>
__global__ void __launch_bounds__(SP_NT, 2) k_spec_power_s(const __grid_constant__ CsSpecArgs a, const float2* __restrict__ tw,
                                                           const float* __restrict__ win, int nchunk, int ch)
{
    using W = WarpFft<L, R>;
    constexpr int M = W::M, N = 2 * M, GROUPS = SP_NT / L, WARPS = SP_NT / 32, WORDS = N / 16;
    extern __shared__ __align__(16) unsigned char smem[];
    float2* tab = reinterpret_cast<float2*>(smem);
    float2* tiles = tab + W::TWIDDLES;
    uint32_t* raw = reinterpret_cast<uint32_t*>(tiles + GROUPS * W::TILE);
    __shared__ float2 lut16[16];
    const int g = threadIdx.x / L, lane = threadIdx.x % L;
    float2* tile = tiles + g * W::TILE;
    uint32_t* rw = raw + g * 2 * WORDS;
    const int chunk = blockIdx.x, row = blockIdx.y;
    const int sub = row / a.nspec, spec = row % a.nspec;
    const int novl = a.overlap * a.ffts_per_spectrum - (a.overlap - 1);
    const int hop = N / a.overlap;
    const bool vec = hop % 64 == 0;
    const uint32_t* plane = reinterpret_cast<const uint32_t*>(a.planes + (int64_t)sub * a.bytes_per_sub);
    const int64_t first = (int64_t)spec * a.ffts_per_spectrum * N;
    const int j_begin = chunk * ch, j_end = min(novl, j_begin + ch);
    // a group past the chunk's end transforms its first FFT again and drops it
    auto start_of = [&](int j) { return first + (int64_t)(j < j_end ? j : j_begin) * hop; };
    spec_fetch(rw, plane, start_of(j_begin + g), WORDS, lane, L, vec);
    if (threadIdx.x < 16) lut16[threadIdx.x] = make_float2(a.lut[threadIdx.x & 3], a.lut[threadIdx.x >> 2]);
    W::fill(tab, tw, 2);
    float2 wh[W::CPL];
#pragma unroll
    for (int c = 0; c < W::CPL; c++) wh[c] = cscale(__ldg(tw + lane + L * c), 0.5f);
    float acc[R], mid = 0.f;
#pragma unroll
    for (int i = 0; i < R; i++) acc[i] = 0.f;
    __syncthreads();
    const float2* win2 = reinterpret_cast<const float2*>(win) + lane;
    const int sh = 4 * (lane & 7);                   // a pair's four bits within its word
    // the mask of the next FFT is looked at while this one is transformed
    bool blank_next = MASK && spec_blanked(a.valid_mask, start_of(j_begin + g), N, lane, L);
    int u = 0;
    for (int j0 = j_begin; j0 < j_end; j0 += GROUPS, u ^= 1) {
        const int j = j0 + g;
        const int64_t start = start_of(j);
        bool blanked = false;
        if constexpr (MASK) blanked = __any_sync(0xffffffffu, blank_next);
        if (j0 + GROUPS < j_end) {
            spec_fetch(rw + (u ^ 1) * WORDS, plane, start_of(j + GROUPS), WORDS, lane, L, vec);
            if constexpr (MASK) blank_next = spec_blanked(a.valid_mask, start_of(j + GROUPS), N, lane, L);
            spec_fetch_wait<1>();
        } else {
            spec_fetch_wait<0>();
        }
        __syncwarp();
        const uint32_t* w = rw + u * WORDS + (lane >> 3);
        float2 v[R];
#pragma unroll
        for (int q = 0; q < R; q++) {
            float2 x = lut16[(w[q * (L / 8)] >> sh) & 15u];
            if (MASK && blanked) {
                const int64_t t = start + 2 * (lane + L * q);
                const uint32_t m = __ldg(a.valid_mask + (t >> 5)) >> (t & 31);
                x = make_float2((m & 1u) ? x.x : 0.f, (m & 2u) ? x.y : 0.f);
            }
            const float2 wn = __ldg(win2 + L * q);
            v[q] = make_float2(x.x * wn.x, x.y * wn.y);
        }
        W::run(v, tile, lane, tab);
        const bool valid = j < j_end;
        W::split(
            v, lane, [&](int c, int k2) { return W::rot_half(wh[c], k2); },
            [&](int i, int, float2 X1, float2 X2) {
                if (!valid) return;
                acc[2 * i] += X1.x * X1.x + X1.y * X1.y;
                acc[2 * i + 1] += X2.x * X2.x + X2.y * X2.y;
            },
            [&](float2 X) {
                if (valid) mid += X.x * X.x + X.y * X.y;
            });
    }
    // the groups' sums: over the warp's groups by shuffles, then over the warps in order
#pragma unroll
    for (int o = L; o < 32; o *= 2) {
#pragma unroll
        for (int i = 0; i < R; i++) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
        mid += __shfl_xor_sync(0xffffffffu, mid, o);
    }
    __syncthreads();
    float* red = reinterpret_cast<float*>(tiles);    // [WARPS][M + 1]
    if ((threadIdx.x & 31) < L) {
        float* r = red + (threadIdx.x >> 5) * (M + 1);
#pragma unroll
        for (int c = 0; c < W::CPL; c++)
#pragma unroll
            for (int k2 = 0; k2 < L / 2; k2++) {
                const int i = c * (L / 2) + k2, k = lane + L * c + R * k2;
                r[k] = acc[2 * i];
                r[M - k] = acc[2 * i + 1];
            }
        if (lane == 0) r[M / 2] = mid;
    }
    __syncthreads();
    float* prow = a.partial + ((int64_t)row * nchunk + chunk) * (M + 1);
    for (int k = threadIdx.x; k <= M; k += SP_NT) {
        float t = red[k];
#pragma unroll
        for (int q = 1; q < WARPS; q++) t += red[q * (M + 1) + k];
        prow[k] = t;
    }
}

// N = 4096, 8192 and 16384: M1 = N / 2048 warps per FFT, decimation in time by
// M1.  Warp n1 transforms z[n1 + M1 m], m < 1024, in registers (WarpFft) and
// parks the result Y_n1 in its tile; after one CTA barrier each thread takes
// mirrored columns kA and 1024 - kA (kA = thread + 32 M1 i; thread 0 also
// columns 0 and 512, each its own mirror):
//     Z[k2 + 1024 k1] = sum_n1 W_M1^(n1 k1) (W_M^(n1 k2) Y_n1[k2]),
// two M1-point DFTs, the second rotated by one as W_M^(n1 (1024 - k2)) =
// W_M1^n1 conj(W_M^(n1 k2)), which holds both ends of every real-FFT pair, and
// adds the powers to its own registers.  The window table is read in the
// warps' order (winp: [M1][1024] pairs).  Bound by instruction issue; 12 rows x
// 1999 FFTs of 8192 points: 285 us (with some blanked windows), the radix-16 groups 430.
template <int M1, bool MASK>
__global__ void __launch_bounds__(32 * M1, 16 / M1) k_spec_power_m(const __grid_constant__ CsSpecArgs a,
                                                                   const float2* __restrict__ tw,
                                                                   const float2* __restrict__ winp, int nchunk, int ch)
{
    using W = WarpFft<32, 32>;
    constexpr int M = 1024 * M1, N = 2 * M, NT = 32 * M1, WORDS = N / 16, TASKS = 512 / NT;
    extern __shared__ __align__(16) unsigned char smem[];
    float2* tab = reinterpret_cast<float2*>(smem);
    float2* tiles = tab + W::TWIDDLES;
    uint32_t* raw = reinterpret_cast<uint32_t*>(tiles + M1 * W::TILE);
    __shared__ float2 lut16[16];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float2* tile = tiles + warp * W::TILE;
    const int chunk = blockIdx.x, row = blockIdx.y;
    const int sub = row / a.nspec, spec = row % a.nspec;
    const int novl = a.overlap * a.ffts_per_spectrum - (a.overlap - 1);
    const int hop = N / a.overlap;
    const bool vec = hop % 64 == 0;
    const uint32_t* plane = reinterpret_cast<const uint32_t*>(a.planes + (int64_t)sub * a.bytes_per_sub);
    const int64_t first = (int64_t)spec * a.ffts_per_spectrum * N;
    const int j_begin = chunk * ch, j_end = min(novl, j_begin + ch);
    spec_fetch(raw, plane, first + (int64_t)j_begin * hop, WORDS, tid, NT, vec);
    if (tid < 16) lut16[tid] = make_float2(a.lut[tid & 3], a.lut[tid >> 2]);
    W::fill(tab, tw, 2 * M1);
    __shared__ float2 w2m[2 * M1];                   // W_(2 M1)^i
    if (tid < 2 * M1) w2m[tid] = __ldg(tw + 1024 * tid);
    const float2 w512 = cscale(__ldg(tw + 512 * (lane & (2 * M1 - 1))), 0.5f);
    float acc[TASKS][2 * M1], extra = 0.f, nyquist = 0.f;
#pragma unroll
    for (int i = 0; i < TASKS; i++)
#pragma unroll
        for (int q = 0; q < 2 * M1; q++) acc[i][q] = 0.f;
    const float2* win2 = winp + 1024 * warp + lane;
    const int n0 = warp + M1 * lane;                 // this lane's first pair; pair q is 32 M1 further on
    const int w0 = n0 >> 3, sh = 4 * (n0 & 7);
    auto power = [](float2 X) { return X.x * X.x + X.y * X.y; };
    // the mask of the next FFT is looked at while this one is transformed
    bool blank_next = MASK && spec_blanked(a.valid_mask, first + (int64_t)j_begin * hop, N, tid, NT);
    int u = 0;
    for (int j = j_begin; j < j_end; j++, u ^= 1) {
        const int64_t start = first + (int64_t)j * hop;
        const bool blank = blank_next;
        if (j + 1 < j_end) {
            spec_fetch(raw + (u ^ 1) * WORDS, plane, start + hop, WORDS, tid, NT, vec);
            if constexpr (MASK) blank_next = spec_blanked(a.valid_mask, start + hop, N, tid, NT);
            spec_fetch_wait<1>();
        } else {
            spec_fetch_wait<0>();
        }
        bool blanked = false;
        // this FFT's words are in, the previous one's columns are read
        if constexpr (MASK) blanked = __syncthreads_or(blank) != 0;
        else __syncthreads();
        {
            const uint32_t* w = raw + u * WORDS + w0;
            float2 v[32];
#pragma unroll
            for (int q = 0; q < 32; q++) {
                float2 x = lut16[(w[4 * M1 * q] >> sh) & 15u];
                if (MASK && blanked) {
                    const int64_t t = start + 2 * (n0 + 32 * M1 * q);
                    const uint32_t m = __ldg(a.valid_mask + (t >> 5)) >> (t & 31);
                    x = make_float2((m & 1u) ? x.x : 0.f, (m & 2u) ? x.y : 0.f);
                }
                const float2 wn = __ldg(win2 + 32 * q);
                v[q] = make_float2(x.x * wn.x, x.y * wn.y);
            }
            W::run(v, tile, lane, tab);
#pragma unroll
            for (int k2 = 0; k2 < 32; k2++) tile[lane + 32 * k2] = v[k2];
        }
        __syncthreads();
        if (warp == M1 - 1) {
            // columns 0 and 512, each paired with itself: bin 512 l is lane l's,
            // Z = sum_n1 Y_n1[512 (l & 1)] W_2M1^(l n1), its pair lane 2 M1 - l's (one
            // thread's pair of columns kept the other warps at the barrier)
            const int l = lane & (2 * M1 - 1);
            float2 z = make_float2(0.f, 0.f);
#pragma unroll
            for (int n1 = 0; n1 < M1; n1++) {
                const float2 y = tiles[n1 * W::TILE + 512 * (l & 1)], w = w2m[(l * n1) & (2 * M1 - 1)];
                z.x = fmaf(y.x, w.x, fmaf(-y.y, w.y, z.x));
                z.y = fmaf(y.x, w.y, fmaf(y.y, w.x, z.y));
            }
            const int lp = (2 * M1 - l) & (2 * M1 - 1);
            const float2 zp = make_float2(__shfl_sync(0xffffffffu, z.x, lp), __shfl_sync(0xffffffffu, z.y, lp));
            float2 Xk, Xm;
            r2c_pair_h(z, zp, w512, Xk, Xm);
            extra += l ? power(Xk) : Xk.x * Xk.x;    // DC and Nyquist are real
            nyquist += Xm.x * Xm.x;
        }
#pragma unroll
        for (int i = 0; i < TASKS; i++) {
            const int kA = tid + NT * i;
            if (kA == 0) continue;                   // columns 0 and 512: above
            float2 ya[M1], yb[M1];
            const float2 u1 = __ldg(tw + 2 * kA);    // W_M^kA
            float2 pw = make_float2(1.f, 0.f);
#pragma unroll
            for (int n1 = 0; n1 < M1; n1++) {
                const float2 za = tiles[n1 * W::TILE + kA], zb = tiles[n1 * W::TILE + 1024 - kA];
                ya[n1] = n1 ? cmul(za, pw) : za;
                yb[n1] = n1 ? cmul_conj(zb, pw) : zb;
                pw = n1 ? cmul(pw, u1) : u1;
            }
            Dft<M1>::run(ya);                        // ya[k1] = Z[kA + 1024 k1]
            Dft<M1>::run(yb);                        // yb[(k1 + 1) % M1] = Z[1024 - kA + 1024 k1]
            const float2 wA = cscale(__ldg(tw + kA), 0.5f);     // W_N^kA / 2
#pragma unroll
            for (int k1 = 0; k1 < M1; k1++) {
                float2 Xk, Xm;
                r2c_pair_h(ya[k1], yb[(M1 - k1) % M1], rot32(wA, (16 / M1) * k1), Xk, Xm);
                acc[i][2 * k1] += power(Xk);
                acc[i][2 * k1 + 1] += power(Xm);
            }
        }
    }
    // every bin has one owner
    float* prow = a.partial + ((int64_t)row * nchunk + chunk) * (M + 1);
#pragma unroll
    for (int i = 0; i < TASKS; i++) {
        const int kA = tid + NT * i;
#pragma unroll
        for (int k1 = 0; k1 < M1; k1++) {
            if (kA) {
                prow[kA + 1024 * k1] = acc[i][2 * k1];
                prow[M - kA - 1024 * k1] = acc[i][2 * k1 + 1];
            }
        }
    }
    if (warp == M1 - 1 && lane < 2 * M1) {
        prow[512 * lane] = extra;
        if (lane == 0) prow[M] = nyquist;
    }
}

// N = 32768 (P = 1) and 65536 (P = 2): the CTA's 16384-point complex FFT as
// a warp four-step with decimation in frequency, so that every input read
// (plane words, window pairs, twiddles) is coalesced across threads:
//   n = 1024 n1 + m (n1 < 16, m < 1024),  k = k1 + 16 k2 (k1 < 16, k2 < 1024)
//   W_MC^(n k) = W_16^(n1 k1) W_MC^(m k1) W_1024^(m k2).
// Column phase: thread t takes columns m = t, t + 512: 16 windowed inputs
// (P = 2: the parity fold of both halves), DFT-16 over n1, twiddle
// W_MC^(m k1), stored to row k1 of a [16][1088] tile.  Row phase: warp k1
// takes row k1: a 1024-point DFT in registers (32 points per lane: DFT-32,
// twiddle, transpose through the row's own padded region, DFT-32) and stores
// Y[k1][k2] back in natural k2 order.  Pair phase: each thread owns fixed
// items (k1, k2) whose real-FFT partner lies in row 16 - k1 (P = 1 and p = 0)
// or 15 - k1 (p = 1), splits them (r2c_pair) and adds |X|^2 into its own
// shared-memory slots [slot][thread] (no two threads share a bin), which the
// CTA writes as the chunk's partial spectrum.  512 threads, one CTA per SM.
constexpr int SW_NT = 512, SW_MC = 16384, SW_ROWP = 1088, SW_SLOTS = 34;

// tile column of index k2 (or m): two float2 of padding after every 32
CS_DEV int sw_pad(int k2) { return k2 + 2 * (k2 >> 5); }

template <int P, bool MASK>
__global__ void __launch_bounds__(SW_NT, 1) k_spec_power_w(const __grid_constant__ CsSpecArgs a, const float2* __restrict__ tw,
                                                           const float* __restrict__ win, int nchunk, int ch)
{
    constexpr int MC = SW_MC, M = MC * P, N = 2 * M;
    extern __shared__ __align__(16) unsigned char smem[];
    float2* tile = reinterpret_cast<float2*>(smem);                       // [16][SW_ROWP]
    float* slots = reinterpret_cast<float*>(tile + 16 * SW_ROWP);         // [SW_SLOTS][SW_NT]
    uint32_t* rawsm = reinterpret_cast<uint32_t*>(slots + SW_SLOTS * SW_NT);   // the FFT's N / 16 plane words
    __shared__ float2 lut16[16];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int chunk = blockIdx.x, row = blockIdx.y;
    const int sub = row / a.nspec, spec = row % a.nspec;
    const int p = (P == 2) ? (int)blockIdx.z : 0;
    const int novl = a.overlap * a.ffts_per_spectrum - (a.overlap - 1);
    const int hop = N / a.overlap;
    const uint32_t* plane = reinterpret_cast<const uint32_t*>(a.planes + (int64_t)sub * a.bytes_per_sub);
    // blanking mask only in the MASK form (framed recordings), so the plain
    // form carries no per-sample mask code
    const uint32_t* vmask = MASK ? a.valid_mask : nullptr;
    const float2* win2 = reinterpret_cast<const float2*>(win);
    if (tid < 16) lut16[tid] = make_float2(a.lut[tid & 3], a.lut[tid >> 2]);
    for (int i = tid; i < SW_SLOTS * SW_NT; i += SW_NT) slots[i] = 0.f;

    // pair items of this thread: (k1, k2) with partner (k1', k2')
    //  P = 1 / p = 0: rows 1..7 (k2 = t, t + 512), row 8 (k2 = t), row 0 (k2 = t; t = 0 also k2 = 512)
    //  p = 1:         rows 0..7 (k2 = t, t + 512)
    const bool odd = P == 2 && p == 1;
    // row-phase twiddles W_1024^(lane e), e < 8 (balanced recurrence), and
    // W_1024^(8 lane), kept in shared memory [e][lane] for every warp
    __shared__ float2 wps[9][32];
    if (warp == 0) {
        float2 wp[8];
        float sn, cs;
        sincospif(-(float)lane / 512.0f, &sn, &cs);
        wp[0] = make_float2(1.f, 0.f);
        wp[1] = make_float2(cs, sn);
#pragma unroll
        for (int e = 2; e < 8; e++) wp[e] = (e & 1) ? cmul(wp[e - 1], wp[1]) : cmul(wp[e / 2], wp[e / 2]);
#pragma unroll
        for (int e = 0; e < 8; e++) wps[e][lane] = wp[e];
        wps[8][lane] = cmul(wp[4], wp[4]);
    }
    // per-thread constants: W_M^m and W_MC^m of the thread's two columns m = t, t + 512;
    // the split twiddle W_N^k of item (k1, k2), k = P (k1 + 16 k2) + p, as
    // ck[k1] = W_N^(P k1 + p) (shared, broadcast) times W_N^(16 P k2) of k2 = t, t + 512
    __shared__ float2 ck[16];
    if (tid < 16) ck[tid] = cscale(__ldg(tw + P * tid + p), 0.5f);
    float2 tmc[2], umc[2], bk[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const int m = tid + SW_NT * c;                   // column-phase columns and pair-phase k2
        tmc[c] = (P == 2) ? __ldg(tw + 2 * m) : make_float2(1.f, 0.f);   // W_M^m
        umc[c] = __ldg(tw + 2 * P * m);                  // W_MC^m
        bk[c] = __ldg(tw + 16 * P * m);                  // W_N^(16 P k2)
    }
    const float2 bk512 = __ldg(tw + 16 * P * 512);       // k2 = 512 (thread 0's extra item)
    __syncthreads();

    const int j_begin = chunk * ch, j_end = min(novl, j_begin + ch);
    // the plane words of FFT j go to shared memory by cp.async (hop is a
    // multiple of 64 samples, so each FFT starts on a 16-byte boundary); the
    // next FFT's are fetched while this one's row and pair phases run
    auto fetch = [&](int jj) {
        const int64_t st = (int64_t)spec * a.ffts_per_spectrum * N + (int64_t)jj * hop;
        const char* src = reinterpret_cast<const char*>(plane + (st >> 4));
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(rawsm);
        for (int i = tid; i < N / 64; i += SW_NT)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(src + 16 * i) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (j_begin < j_end) fetch(j_begin);
    for (int j = j_begin; j < j_end; j++) {
        const int64_t start = (int64_t)spec * a.ffts_per_spectrum * N + (int64_t)j * hop;   // a multiple of 64
        const uint32_t* wsrc = rawsm;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                   // this FFT's words are in
        // ---- column phase: columns m = t, t + 512 ----
        // (the mask is applied only to windows that contain blanked samples)
        auto column_phase = [&](auto masked) {
        const uint32_t* vm = decltype(masked)::value ? vmask : nullptr;
#pragma unroll 1
        for (int c = 0; c < 2; c++) {
            const int m = tid + SW_NT * c;
            float2 v[16];
            const float2 tm = c ? tmc[1] : tmc[0];                                     // W_M^m
#pragma unroll
            for (int n1 = 0; n1 < 16; n1++) {
                const int n = 1024 * n1 + m;
                const float2 x1 = sample_pair16(lut16, wsrc[n >> 3], (2 * n) & 15, vm, start + 2 * n);
                const float2 wa = __ldg(win2 + n);
                const float2 z1 = make_float2(x1.x * wa.x, x1.y * wa.y);
                if constexpr (P == 1) {
                    v[n1] = z1;
                } else {
                    const int n2 = n + MC;
                    const float2 x2 = sample_pair16(lut16, wsrc[n2 >> 3], (2 * n2) & 15, vm, start + 2 * n2);
                    // cosine^2: w(i + N/2) = 1 - w(i) (one table read for both halves)
                    const float2 wb = (a.window == 2) ? make_float2(1.f - wa.x, 1.f - wa.y) : __ldg(win2 + n2);
                    const float2 z2 = make_float2(x2.x * wb.x, x2.y * wb.y);
                    // y_1[n] = (z[n] - z[n + MC]) W_M^n, W_M^(1024 n1 + m) = W_32^n1 W_M^m
                    v[n1] = p ? cmul(csub<false>(z1, z2), rot32(tm, n1)) : cadd<false>(z1, z2);
                }
            }
            Dft<16, false>::run(v);
            // W_MC^(m k1): powers of u = W_MC^m by a balanced recurrence
            const float2 u = c ? umc[1] : umc[0];
            float2 wk[16];
            wk[0] = make_float2(1.f, 0.f);
            wk[1] = u;
#pragma unroll
            for (int e = 2; e < 16; e++) wk[e] = (e & 1) ? cmul(wk[e - 1], u) : cmul(wk[e / 2], wk[e / 2]);
#pragma unroll
            for (int k1 = 0; k1 < 16; k1++) tile[k1 * SW_ROWP + sw_pad(m)] = k1 ? cmul(v[k1], wk[k1]) : v[k1];
        }
        };
        bool blanked = false;
        if constexpr (MASK) {
            // any blanked sample in this window? (N / 32 mask words, a few per thread)
            const uint32_t* mw = vmask + (start >> 5);
            bool mine = false;
            for (int i = tid; i < N / 32; i += SW_NT) mine |= __ldg(mw + i) != 0xffffffffu;
            blanked = __syncthreads_or(mine) != 0;
        }
        if (blanked) column_phase(std::true_type{});
        else column_phase(std::false_type{});
        __syncthreads();                                   // the words are consumed: fetch the next FFT's
        if (j + 1 < j_end) fetch(j + 1);
        // ---- row phase: warp k1 ----
        {
            float2* rowp = tile + warp * SW_ROWP;
            float2 x[32];
#pragma unroll
            for (int e = 0; e < 32; e++) x[e] = rowp[lane + 34 * e];          // m = lane + 32 e
            Dft<32, false>::run(x);
            float2 q = make_float2(1.f, 0.f);
            const float2 w8 = wps[8][lane];
#pragma unroll
            for (int b = 0; b < 4; b++) {
#pragma unroll
                for (int r = 0; r < 8; r++) {
                    if (b == 0 && r == 0) continue;
                    const float2 wr = wps[r][lane];
                    x[8 * b + r] = cmul(x[8 * b + r], b ? cmul(q, wr) : wr);
                }
                q = b ? cmul(q, w8) : w8;
            }
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 32; e++) rowp[e * 33 + lane] = x[e];
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 32; e++) x[e] = rowp[lane * 33 + e];
            Dft<32, false>::run(x);                                                    // x[e] = Y[warp][lane + 32 e]
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 32; e++) rowp[lane + 34 * e] = x[e];          // k2 = lane + 32 e
        }
        __syncthreads();
        // ---- pair phase ----
        int s = 0;
        // SPECIAL: row 0 of the even forms, which holds k = 0 (DC and Nyquist
        // from Z[0]) and k = M/2 (its own partner)
        auto item = [&](int k1, int k2, float2 b, bool special) {
            int k1b, k2b;
            if (odd) k1b = 15 - k1, k2b = 1023 - k2;
            else if (k1 == 0) k1b = 0, k2b = (1024 - k2) & 1023;
            else k1b = 16 - k1, k2b = 1023 - k2;
            const float2 za = tile[k1 * SW_ROWP + sw_pad(k2)], zb = tile[k1b * SW_ROWP + sw_pad(k2b)];
            const int mp = k1 + 16 * k2;                   // index in the CTA's transform
            const int k = P * mp + p;                      // bin of the full real FFT
            float2 Xk, Xm;
            r2c_pair_h(za, zb, cmul(ck[k1], b), Xk, Xm);         // W_N^k / 2
            if (special && k == 0) {
                slots[s * SW_NT + tid] += Xk.x * Xk.x;
                slots[(s + 1) * SW_NT + tid] += Xm.x * Xm.x;
            } else {
                slots[s * SW_NT + tid] += Xk.x * Xk.x + Xk.y * Xk.y;
                if (!special || k != M / 2) slots[(s + 1) * SW_NT + tid] += Xm.x * Xm.x + Xm.y * Xm.y;
            }
            s += 2;
        };
        if (odd) {
#pragma unroll
            for (int k1 = 0; k1 < 8; k1++) item(k1, tid, bk[0], false), item(k1, tid + SW_NT, bk[1], false);
        } else {
#pragma unroll
            for (int k1 = 1; k1 < 8; k1++) item(k1, tid, bk[0], false), item(k1, tid + SW_NT, bk[1], false);
            item(8, tid, bk[0], false);
            item(0, tid, bk[0], true);
            if (tid == 0) item(0, 512, bk512, true);
        }
        __syncthreads();                                   // the tile is rewritten by the next FFT
    }
    // ---- the chunk's partial spectrum: the same items' bins ----
    float* prow = a.partial + ((int64_t)row * nchunk + chunk) * (M + 1);
    int s = 0;
    auto put = [&](int k1, int k2) {
        const int k = P * (k1 + 16 * k2) + p;
        if (k == 0) {
            prow[0] = slots[s * SW_NT + tid];
            prow[M] = slots[(s + 1) * SW_NT + tid];
        } else {
            prow[k] = slots[s * SW_NT + tid];
            if (k != M / 2) prow[M - k] = slots[(s + 1) * SW_NT + tid];
        }
        s += 2;
    };
    if (odd) {
        for (int k1 = 0; k1 < 8; k1++) put(k1, tid), put(k1, tid + SW_NT);
    } else {
        for (int k1 = 1; k1 < 8; k1++) put(k1, tid), put(k1, tid + SW_NT);
        put(8, tid);
        put(0, tid);
        if (tid == 0) put(0, 512);
    }
}

// power[row][k] = scale * sum of the row's chunk partials.  Bound by the read
// of the partials.  A CTA takes 256 / SLICES bins of one row; each slice adds
// every SLICES-th chunk and the slices' sums are added in order, so the sum is
// deterministic.  Eight slices where a thread per bin would leave the chip empty
// (spec_reduce_slices): a row with hundreds of chunks is then not one thread's
// serial chain (16 rows x 512 chunks x 513 bins: 46 us with a thread per bin, 10 us);
// one slice where there are bins enough (16 rows x 32 chunks x 32769 bins: 13 us,
// 20 us with eight).
constexpr int RED_THREADS = 256;
template <int SLICES>
__global__ void __launch_bounds__(RED_THREADS) k_spec_reduce(const float* __restrict__ partial, float* __restrict__ power,
                                                             int nchunk, int nb, float scale)
{
    constexpr int BINS = RED_THREADS / SLICES;
    __shared__ float part[SLICES][BINS];
    const int bin = threadIdx.x % BINS, slice = threadIdx.x / BINS;
    const int r = blockIdx.y, k = blockIdx.x * BINS + bin;
    const float* src = partial + (int64_t)r * nchunk * nb + k;
    float s = 0.f;
    if (k < nb) {
#pragma unroll 8
        for (int c = slice; c < nchunk; c += SLICES) s += __ldg(src + (int64_t)c * nb);
    }
    if constexpr (SLICES > 1) {
        part[slice][bin] = s;
        __syncthreads();
#pragma unroll
        for (int q = 1; q < SLICES; q++) s += part[q][bin];
    }
    if (slice == 0 && k < nb) power[(int64_t)r * nb + k] = s * scale;
}

// one slice from about one full wave of threads (152 SMs x 1024) on
int spec_reduce_slices(int64_t bins, int nchunk) { return bins < 152 * 1024 && nchunk >= 8 ? 8 : 1; }

// PCal fold.  TaskCoreIPP::doMaths folds the overlapped FFT windows whose
// running FFT count is a multiple of the overlap factor (TaskCoreIPP.cpp:
// 414-418).  The count starts at 0 once per call (:358), runs on across the
// spectra of the call and advances after every source's FFT (:434-435), so with
// ns sources source rs folds window j of spectrum s when
// (ns (s novl + j) + rs) % ov == 0: an arithmetic progression j0, j0 + step, ...
// (step = ov / gcd(ns, ov)), possibly empty.  Each window is folded from its
// own start (the rotator index restarts), N samples from j * hop.
//
// Samples whose rotator index l is equal are multiplied by the same value, so
// the fold counts how often each of the four codes occurs per l and applies
// levels and rotator to the counts: exact integers until the last step.  The
// counting is bit-sliced: a plane word holds 16 two-bit codes, and words at
// the same place in the rotator period are added as vertical counters (a
// carry-save adder is two three-input logic operations for 32 positions), the
// AND of a code's two bits in a second set.  About 9 logic operations per word
// instead of 16 level selections and 32 multiply-adds, which bound the fold
// per sample (16 rows x 2^25 samples: 610 us, 61 us now; the read of the planes
// takes 20 us).
// N, L and T are powers of two (L divides N, T divides L), so a thread that
// strides by PCAL_BLOCKS * PCAL_THREADS = 4096 words (65536 samples >= L) keeps
// its place in the rotator period.
CS_DEV int gcd_int(int a, int b) { while (b) { int t = a % b; a = b; b = t; } return a; }

constexpr int PCAL_THREADS = 128;
constexpr int PCAL_BLOCKS = 32;
constexpr int PCAL_POS = 16 * PCAL_THREADS;      // sample positions of a CTA's words
constexpr int PCAL_PLANES = 12;                  // vertical counter planes above 1, 2 and 4

// full adder on 32 positions: s = a ^ b ^ c, carry = majority
CS_DEV void csa(uint32_t& carry, uint32_t& s, uint32_t a, uint32_t b)
{
    const uint32_t u = s;
    s = u ^ a ^ b;
    carry = (u & a) | (u & b) | (a & b);
}

// Vertical counters of 32 positions: weights 1, 2, 4, then 8 2^i in q[i].
struct VCount {
    uint32_t one, two, four, q[PCAL_PLANES];
    CS_DEV void clear()
    {
        one = two = four = 0;
#pragma unroll
        for (int i = 0; i < PCAL_PLANES; i++) q[i] = 0;
    }
    CS_DEV void add8(const uint32_t (&w)[8])
    {
        uint32_t t0, t1, f0, f1, e;
        csa(t0, one, w[0], w[1]);
        csa(t1, one, w[2], w[3]);
        csa(f0, two, t0, t1);
        csa(t0, one, w[4], w[5]);
        csa(t1, one, w[6], w[7]);
        csa(f1, two, t0, t1);
        csa(e, four, f0, f1);
#pragma unroll
        for (int i = 0; i < PCAL_PLANES; i++) {
            const uint32_t t = q[i] & e;
            q[i] ^= e;
            e = t;
        }
    }
    // the count of a position; planes from `np` on are known to be empty
    CS_DEV int count(int pos, int np) const
    {
        int c = (int)((one >> pos) & 1u) + 2 * (int)((two >> pos) & 1u) + 4 * (int)((four >> pos) & 1u);
#pragma unroll
        for (int i = 0; i < PCAL_PLANES; i++)
            if (i < np) c += (int)((q[i] >> pos) & 1u) << (3 + i);
        return c;
    }
};
// words a thread may add before its counters are emptied (a multiple of 8)
constexpr int PCAL_BATCH = (8 << PCAL_PLANES) - 8;

// the 16 validity bits of a plane word, each doubled to its code's two bits
CS_DEV uint32_t double_bits(uint32_t v)
{
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v | (v << 1);
}

template <bool MASK>
__global__ void __launch_bounds__(PCAL_THREADS) k_pcal_fold(
    const uint8_t* __restrict__ planes, int64_t bytes_per_sub, int nspec, int64_t samp_per_spec, int N, int ov, int novl,
    int ns, int rs, int T, int L, const float2* __restrict__ rot, float l0, float l1, float l2, float l3,
    const uint32_t* __restrict__ vmask, float2* __restrict__ partial)
{
    __shared__ int hist[4][PCAL_POS];                // count of each code per position in the period
    __shared__ double2 sums[PCAL_THREADS];
    const int row = blockIdx.y, sub = row / nspec, spec = row % nspec;
    const int tid = threadIdx.x;
    const int LB = min(L, PCAL_POS);                 // rotator positions this CTA touches
    const int LW = max(1, LB / 16);                  // distinct word places among them
    for (int i = tid; i < 4 * PCAL_POS; i += PCAL_THREADS) (&hist[0][0])[i] = 0;
    __syncthreads();
    const uint32_t* plane = reinterpret_cast<const uint32_t*>(planes + (int64_t)sub * bytes_per_sub);
    const int step = ov / gcd_int(ns, ov);
    int j0 = -1;
    for (int j = 0; j < step && j < novl; j++)
        if (((int64_t)ns * ((int64_t)spec * novl + j) + rs) % ov == 0) { j0 = j; break; }
    const int cnt = j0 >= 0 ? (novl - 1 - j0) / step + 1 : 0;
    const int wpw = N / 16, lg = 31 - __clz(wpw);    // 32-bit words per window
    const int64_t nwords = (int64_t)cnt * wpw;
    const int64_t base = ((int64_t)spec * samp_per_spec + (int64_t)max(j0, 0) * (N / ov)) / 16;
    const int64_t win_words = (int64_t)step * (N / ov) / 16;
    constexpr int STRIDE = PCAL_BLOCKS * PCAL_THREADS;
    int64_t w = (int64_t)blockIdx.x * PCAL_THREADS + tid;
    VCount bits, both, val;                          // code bits; their ANDs (two words a set); valid samples
    while (__syncthreads_or(w < nwords)) {
        bits.clear(), both.clear(), val.clear();
        int added = 0, rounds = 0;                   // words and groups of eight counted in this batch
        auto add = [&](uint32_t (&x)[8], uint32_t (&m)[8]) {
            uint32_t av[8];
            if (MASK) {
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const uint32_t d = double_bits(m[u]);
                    x[u] &= d;
                    m[u] = d & 0x55555555u;
                }
#pragma unroll
                for (int u = 0; u < 8; u++) av[u] = u < 4 ? m[2 * u] | (m[2 * u + 1] << 1) : 0u;
                val.add8(av);
            }
            bits.add8(x);
#pragma unroll
            for (int u = 0; u < 8; u++)
                av[u] = u < 4 ? ((x[2 * u] & (x[2 * u] >> 1)) & 0x55555555u) | ((x[2 * u + 1] & (x[2 * u + 1] << 1)) & 0xaaaaaaaau)
                              : 0u;
            both.add8(av);
            rounds++;
            w += 8 * (int64_t)STRIDE;
        };
        // windows back to back (one source): no index arithmetic per word, and
        // the next eight words on their way while eight are added
        if (win_words == wpw && w + 7 * (int64_t)STRIDE < nwords) {
            const uint32_t* p = plane + base;
            const uint32_t* q = vmask + (base >> 1);
            const int half = (int)((base + w) & 1) * 16;
            uint32_t xn[8], mn[8];
            auto load = [&](int64_t at) {
                if (at + 7 * (int64_t)STRIDE >= nwords) return;
#pragma unroll
                for (int u = 0; u < 8; u++) xn[u] = __ldg(p + at + u * STRIDE);
                if (MASK) {
#pragma unroll
                    for (int u = 0; u < 8; u++) mn[u] = __ldg(q + (((base & 1) + at) >> 1) + u * (STRIDE / 2));
                }
            };
            load(w);
            while (rounds < PCAL_BATCH / 8 && w + 7 * (int64_t)STRIDE < nwords) {
                uint32_t x[8], m[8];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    x[u] = xn[u];
                    m[u] = MASK ? mn[u] >> half & 0xffffu : 0u;
                }
                load(w + 8 * (int64_t)STRIDE);
                added += 8;
                add(x, m);
            }
        }
        while (rounds < PCAL_BATCH / 8 && w < nwords) {
            uint32_t x[8], m[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int64_t wu = w + (int64_t)u * STRIDE;
                const bool in = wu < nwords;
                const int64_t wg = base + (wu >> lg) * win_words + (wu & (wpw - 1));
                x[u] = in ? __ldg(plane + wg) : 0u;
                m[u] = MASK && in ? __ldg(vmask + (wg >> 1)) >> ((wg & 1) * 16) & 0xffffu : 0u;
                added += in;
            }
            add(x, m);
        }
        // planes in use: `rounds` groups of eight at most in any lane
        const int np = 32 - __clz(__reduce_max_sync(0xffffffffu, rounds));
        // counts per code, summed over the lanes of the warp at the same place
        // in the period, then over the CTA
#pragma unroll 1
        for (int j = 0; j < 16; j++) {
            const int n01 = both.count(2 * j, np) + both.count(2 * j + 1, np);
            const int n0 = bits.count(2 * j, np), n1 = bits.count(2 * j + 1, np);
            const int nv = MASK ? val.count(2 * j, np) + val.count(2 * j + 1, np) : added;
            int h[4] = {nv - n0 - n1 + n01, n0 - n01, n1 - n01, n01};
            for (int o = 16; o >= LW; o >>= 1) {
#pragma unroll
                for (int c = 0; c < 4; c++) h[c] += __shfl_xor_sync(0xffffffffu, h[c], o);
            }
            if ((tid & 31) < LW) {
#pragma unroll
                for (int c = 0; c < 4; c++) atomicAdd(&hist[c][(16 * tid + j) & (LB - 1)], h[c]);
            }
        }
    }
    __syncthreads();
    // levels and rotator: thread t takes the positions t, t + 128, ... (all of
    // them in bin t % T, as T divides 128), in FP64
    const double lev[4] = {l0, l1, l2, l3};
    double2 s = make_double2(0., 0.);
    for (int i = tid; i < LB; i += PCAL_THREADS) {
        double x = 0.;
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (hist[c][i]) x += (double)hist[c][i] * lev[c];
        const float2 r = __ldg(rot + (((int)blockIdx.x * PCAL_POS + i) & (L - 1)));
        s.x += x * r.x;
        s.y += x * r.y;
    }
    sums[tid] = s;
    __syncthreads();
    if (tid < T) {
        for (int u = tid + T; u < PCAL_THREADS; u += T) {
            s.x += sums[u].x;
            s.y += sums[u].y;
        }
        partial[((int64_t)row * PCAL_BLOCKS + blockIdx.x) * T + tid] = make_float2((float)s.x, (float)s.y);
    }
}

// A CTA per row: bins from the row's partials in CTA order, then the tones
// DFT(bins)/T in FP64, a warp per tone with the T roots of unity in shared
// memory.  (One thread per row for all of it, with a double-precision sine and
// cosine per term, took 868 us at any size; 13 us now.)
constexpr int PCAL_RED = 128;
__global__ void __launch_bounds__(PCAL_RED) k_pcal_reduce(const float2* __restrict__ partial, int nblk, int T, int ntones,
                                                          float2* __restrict__ bins, float2* __restrict__ tones)
{
    __shared__ float2 sb[PCAL_RED];
    __shared__ double2 root[PCAL_RED];
    const int row = blockIdx.x, tid = threadIdx.x;
    if (tid < T) {
        float2 s = make_float2(0.f, 0.f);
        for (int u = 0; u < nblk; u++) {
            const float2 v = partial[((int64_t)row * nblk + u) * T + tid];
            s.x += v.x;
            s.y += v.y;
        }
        bins[(int64_t)row * T + tid] = s;
        sb[tid] = s;
        double sn, cs;
        sincospi(-2.0 * (double)tid / (double)T, &sn, &cs);
        root[tid] = make_double2(cs, sn);
    }
    if (!tones) return;
    __syncthreads();
    const int lane = tid & 31;
    for (int k = tid >> 5; k < ntones; k += PCAL_RED / 32) {
        double re = 0, im = 0;
        for (int n = lane; n < T; n += 32) {
            const double2 w = root[(int)(((int64_t)k * n) % T)];
            re += sb[n].x * w.x - sb[n].y * w.y;
            im += sb[n].x * w.y + sb[n].y * w.x;
        }
        for (int o = 16; o; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (lane == 0) tones[(int64_t)row * ntones + k] = make_float2((float)(re / T), (float)(im / T));
    }
}

// CELLSPE_SPEC_CTA_FFT=1 selects the shared-memory radix-16 kernel for N =
// 32768 and 65536 instead of choosing between it and the warp four-step.
bool spec_cta_fft()
{
    static const bool v = [] {
        const char* e = getenv("CELLSPE_SPEC_CTA_FFT");
        return e && e[0] == '1';
    }();
    return v;
}

// FFTs per chunk (one CTA, one partial spectrum; N = 65536: two CTAs): as many
// as leave about three waves of CTAs on the chip.  Fewer, larger chunks share a
// CTA's start and the writing of its partial spectrum between more FFTs; a small
// job in chunks of 32 would leave most SMs idle (16 rows x 256 FFTs of 4096 points:
// 220 us with 32, 95 with 4).  Not under 16 where a CTA's 16 or 8 groups
// take one FFT each, nor under 4; not above 512, and 32 for N >= 4096, whose
// partial spectra are the larger part of the scratch.
int64_t spec_slots(const CsSpecArgs& a)              // CTAs (pairs for N = 65536) that run at once
{
    const int ctas = a.N <= 2048 ? 2 : a.N == 4096 ? 8 : a.N == 8192 ? 4 : a.N == 16384 ? 2 : 1;   // per SM
    return (int64_t)152 * ctas / (a.N == 65536 ? 2 : 1);
}
int spec_chunk(const CsSpecArgs& a)
{
    if (a.ffts_per_chunk > 0) return a.ffts_per_chunk;
    const int64_t waves = 3 * spec_slots(a);
    const int64_t total = (int64_t)(a.overlap * (int64_t)a.ffts_per_spectrum - (a.overlap - 1)) * a.nsub * a.nspec;
    const int64_t ch = (total + waves - 1) / waves;
    if (a.N <= 2048) return (int)(std::min<int64_t>(512, std::max<int64_t>(16, ch) + 15) / 16 * 16);
    return (int)std::min<int64_t>(SPEC_CH, std::max<int64_t>(4, ch));
}

template <int L, int R>
int launch_power_s(const CsSpecArgs& a, int nchunk, cudaStream_t st)
{
    using W = WarpFft<L, R>;
    constexpr int N = 2 * W::M, GROUPS = SP_NT / L;
    const float2* tw = a.tw_table ? a.tw_table : cs_twiddles(N);
    const float* win = a.win_table ? a.win_table : window_table(a.window, N);
    if (!tw || !win) return CS_ERR_ARG;
    const size_t smem = (size_t)(W::TWIDDLES + GROUPS * W::TILE) * sizeof(float2) + (size_t)GROUPS * 2 * (N / 16) * 4;
    auto kern = a.valid_mask ? k_spec_power_s<L, R, true> : k_spec_power_s<L, R, false>;
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(kern), (int)smem));
    kern<<<dim3(nchunk, a.nsub * a.nspec), SP_NT, smem, st>>>(a, tw, win, nchunk, spec_chunk(a)), cs_count_launches(1);
    return (int)cudaGetLastError();
}

template <int MC, int P> int launch_power(const CsSpecArgs& a, int nchunk, cudaStream_t st);

template <int M1>
int launch_power_m(const CsSpecArgs& a, int nchunk, cudaStream_t st)
{
    using W = WarpFft<32, 32>;
    constexpr int N = 2048 * M1;
    // a caller's own tables come in natural order and without allocation
    if (a.win_table) return launch_power<1024 * M1, 1>(a, nchunk, st);
    const float2* tw = a.tw_table ? a.tw_table : cs_twiddles(N);
    const float2* winp = window_pairs(a.window, N, M1);
    if (!tw || !winp) return CS_ERR_ARG;
    const size_t smem = (size_t)(W::TWIDDLES + M1 * W::TILE) * sizeof(float2) + (size_t)2 * (N / 16) * 4;
    auto kern = a.valid_mask ? k_spec_power_m<M1, true> : k_spec_power_m<M1, false>;
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(kern), (int)smem));
    kern<<<dim3(nchunk, a.nsub * a.nspec), 32 * M1, smem, st>>>(a, tw, winp, nchunk, spec_chunk(a)), cs_count_launches(1);
    return (int)cudaGetLastError();
}

template <int MC, int P>
int launch_power(const CsSpecArgs& a, int nchunk, cudaStream_t st)
{
    using C = SCfg<MC>;
    constexpr int M = MC * P, N = 2 * M;
    const float2* tw = a.tw_table ? a.tw_table : cs_twiddles(N);
    const float* win = a.win_table ? a.win_table : window_table(a.window, N);
    if (!tw || !win) return CS_ERR_ARG;
    size_t smem = (size_t)C::GROUPS * fpad_size(MC) * sizeof(float2) + (size_t)C::GROUPS * (M / P + 1) * sizeof(float);
    auto kern = k_spec_power<MC, P>;
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(kern), (int)smem));
    dim3 grid(nchunk, a.nsub * a.nspec, P);
    kern<<<grid, C::NT, smem, st>>>(a, tw, win, nchunk, spec_chunk(a)), cs_count_launches(1);
    return (int)cudaGetLastError();
}

template <int P>
int launch_power_w(const CsSpecArgs& a, int nchunk, cudaStream_t st)
{
    constexpr int N = 2 * SW_MC * P;
    const float2* tw = a.tw_table ? a.tw_table : cs_twiddles(N);
    const float* win = a.win_table ? a.win_table : window_table(a.window, N);
    if (!tw || !win) return CS_ERR_ARG;
    if ((N / a.overlap) % 64) return launch_power<SW_MC, P>(a, nchunk, st);   // FFT starts not 16-byte aligned
    const size_t smem = (size_t)16 * SW_ROWP * sizeof(float2) + (size_t)SW_SLOTS * SW_NT * sizeof(float) + N / 16 * 4;
    auto kern = a.valid_mask ? k_spec_power_w<P, true> : k_spec_power_w<P, false>;
    CS_CUDA_TRY(cs_smem_at_least(reinterpret_cast<const void*>(kern), (int)smem));
    dim3 grid(nchunk, a.nsub * a.nspec, P);
    kern<<<grid, SW_NT, smem, st>>>(a, tw, win, nchunk, spec_chunk(a)), cs_count_launches(1);
    return (int)cudaGetLastError();
}

// N = 32768 / 65536: the warp four-step or the CTA radix-16 power kernel,
// chosen per (device, N, overlap) by timing both once on the caller's own job
// (both compute the same partial sums, so each runs once warm and once timed
// and the chosen one runs for the result); outside stream capture and where
// the calling thread allows timing (not inside service workers).  Until a
// timed choice exists, and with CELLSPE_SPEC_CTA_FFT=1, fixed choices.
std::mutex g_sp_tune_mu;
std::map<std::tuple<int, int, int>, int> g_sp_choice;   // (device, N, overlap) -> 0 warp, 1 CTA

template <int P>
int launch_power_long(const CsSpecArgs& a, int nchunk, cudaStream_t st)
{
    if (spec_cta_fft()) return launch_power<SW_MC, P>(a, nchunk, st);
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(dev, a.N, a.overlap);
    int choice = -1;
    {
        std::lock_guard<std::mutex> lk(g_sp_tune_mu);
        auto it = g_sp_choice.find(key);
        if (it != g_sp_choice.end()) choice = it->second;
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool can_time = cs_fstage_timing_allowed() && cudaStreamIsCapturing(st, &cap) == cudaSuccess &&
                          cap == cudaStreamCaptureStatusNone;
    if (choice < 0 && can_time) {
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        float t[2] = {1e30f, 1e30f};
        if (cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess) {
            for (int v = 0; v < 2; v++) {
                auto run = [&] { return v ? launch_power<SW_MC, P>(a, nchunk, st) : launch_power_w<P>(a, nchunk, st); };
                if (run() != 0) continue;
                cudaEventRecord(e0, st);
                const int rc = run();
                cudaEventRecord(e1, st);
                if (rc == 0 && cudaEventSynchronize(e1) == cudaSuccess) cudaEventElapsedTime(&t[v], e0, e1);
            }
        }
        cudaGetLastError();
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        choice = t[1] < 0.98f * t[0] ? 1 : 0;
        std::lock_guard<std::mutex> lk(g_sp_tune_mu);
        g_sp_choice[key] = choice;
    }
    return choice == 1 ? launch_power<SW_MC, P>(a, nchunk, st) : launch_power_w<P>(a, nchunk, st);
}

int spec_nchunk(const CsSpecArgs& a)
{
    int novl = a.overlap * a.ffts_per_spectrum - (a.overlap - 1);
    return (novl + spec_chunk(a) - 1) / spec_chunk(a);
}
}  // namespace

const float* cs_window_table(int type, int n) { return window_table(type, n); }

// The no-allocation entry point's choice.  Its transforms of 4096 points and more run in
// k_spec_power and k_spec_power_w, whose CTAs take the same time each: the whole job
// in one wave where chunks of up to 32 allow it, as 3.4 waves of chunks of 9 cost more
// (4 x 2044 FFTs of 16384 points 418 us, 390 in chunks of 32, 339 in one wave of 27).
int cs_spec_noalloc_chunk(const CsSpecArgs& a)
{
    if (a.N < 4096) return 0;
    const int64_t novl = a.overlap * (int64_t)a.ffts_per_spectrum - (a.overlap - 1);
    const int64_t per_row = std::max<int64_t>(1, spec_slots(a) / ((int64_t)a.nsub * a.nspec));
    return (int)std::min<int64_t>(SPEC_CH, std::max<int64_t>(4, (novl + per_row - 1) / per_row));
}

// Scratch layout: chunk partial spectra, then (256-byte aligned: N/2+1 is
// odd, and the phase-cal partials are float2) the phase-cal partials.
int64_t power_partial_floats(const CsSpecArgs& a)
{
    if (a.skip_power) return 0;
    const int64_t power = (int64_t)a.nsub * a.nspec * spec_nchunk(a) * (a.N / 2 + 1);
    return (power + 63) / 64 * 64;
}

int64_t cs_spectrometer_pcal_floats(const CsSpecArgs& a)
{
    return a.tonebins > 0 ? (int64_t)a.nsub * a.nspec * PCAL_BLOCKS * a.tonebins * 2 : 0;
}

int64_t cs_spectrometer_scratch_floats(const CsSpecArgs& a)
{
    return power_partial_floats(a) + cs_spectrometer_pcal_floats(a);
}

int cs_spectrometer(const CsSpecArgs& a, cudaStream_t st)
{
    if (!a.planes || (!a.power && !a.skip_power) || !a.partial || a.nsub <= 0 || a.nspec <= 0 ||
        a.ffts_per_spectrum <= 0)
        return CS_ERR_ARG;
    if (a.overlap < 1 || a.N % (16 * a.overlap) != 0) return CS_ERR_ARG;
    if ((uintptr_t)a.planes % 16 || a.bytes_per_sub % 16) return CS_ERR_ARG;
    // every sample the spectra read must lie inside the subband plane
    if ((int64_t)a.nspec * a.ffts_per_spectrum * a.N > a.bytes_per_sub * 4) return CS_ERR_ARG;
    if (a.nsub * a.nspec > 65535) return CS_ERR_ARG;
    const int nchunk = spec_nchunk(a);
    int rc = 0;
    if (!a.skip_power) switch (a.N) {
        case 1024: rc = launch_power_s<16, 32>(a, nchunk, st); break;
        case 2048: rc = launch_power_s<32, 32>(a, nchunk, st); break;
        case 4096: rc = launch_power_m<2>(a, nchunk, st); break;
        case 8192: rc = launch_power_m<4>(a, nchunk, st); break;
        case 16384: rc = launch_power_m<8>(a, nchunk, st); break;
        case 32768: rc = launch_power_long<1>(a, nchunk, st); break;
        case 65536: rc = launch_power_long<2>(a, nchunk, st); break;
        default: return CS_ERR_UNSUPPORTED;
    }
    if (rc) return rc;
    const int rows = a.nsub * a.nspec, nb = a.N / 2 + 1;
    const int novl = a.overlap * a.ffts_per_spectrum - (a.overlap - 1);
    if (!a.skip_power) {
        const float scale = (float)(1.0 / (double)novl);
        const int slices = spec_reduce_slices((int64_t)rows * nb, nchunk), bins = RED_THREADS / slices;
        (slices == 8 ? k_spec_reduce<8> : k_spec_reduce<1>)<<<dim3((nb + bins - 1) / bins, rows), RED_THREADS, 0, st>>>(
            a.partial, a.power, nchunk, nb, scale),
            cs_count_launches(1);
        CS_CUDA_TRY(cudaGetLastError());
    }

    if (a.tonebins > 0) {
        const int T = a.tonebins, L = a.rotatorlen;
        if (L <= 0 || L % T != 0 || a.N % L != 0 || T > 128 || !a.pcal_bins) return CS_ERR_ARG;
        const float2* rot = a.rot_table ? a.rot_table : rotator_table(L, a.pcal_offset_hz, a.fs_hz);
        if (!rot) return CS_ERR_ARG;
        float2* pp = reinterpret_cast<float2*>(a.partial + power_partial_floats(a));
        int64_t samp_per_spec = (int64_t)a.ffts_per_spectrum * a.N;
        const int ns = a.pcal_sources > 0 ? a.pcal_sources : 1;
        auto fold = a.valid_mask ? k_pcal_fold<true> : k_pcal_fold<false>;
        fold<<<dim3(PCAL_BLOCKS, rows), PCAL_THREADS, 0, st>>>(a.planes, a.bytes_per_sub, a.nspec, samp_per_spec, a.N,
                                                               a.overlap, novl, ns, a.pcal_source, T, L, rot, a.lut[0],
                                                               a.lut[1], a.lut[2], a.lut[3], a.valid_mask, pp),
            cs_count_launches(1);
        CS_CUDA_TRY(cudaGetLastError());
        k_pcal_reduce<<<rows, PCAL_RED, 0, st>>>(pp, PCAL_BLOCKS, T, a.ntones, a.pcal_bins, a.pcal_tones), cs_count_launches(1);
        CS_CUDA_TRY(cudaGetLastError());
    }
    return 0;
}
