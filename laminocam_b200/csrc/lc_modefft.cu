// FFT passes of the NUFFT (fine grid <-> modes) on the register-plan line
// transforms, for even fine-grid lengths L = 2M with a plan for M.
//
//   type 1 (sign +1): L grid values (or a window of them, the others zero) -> n
//     modes k = j - n/2, times a real factor per mode;
//   type 2 (sign -1): n modes, times real factors -> L grid values (or a window).
//
// The fine grid is at least twice as long as the modes, n <= M, so a line runs
// as two transforms of length M in one thread (h(i) = exp(-i pi i / M)):
//   type 1   E, O = DFT+_M of the even and odd grid values;
//            mode m >= 0:  E[m] + conj h(m) O[m],
//            mode m - M < 0 (grid index m + M):  E[m] - conj h(m) O[m]
//   type 2   x[m] = mode m, or mode m - M with the odd half's sign reversed:
//            X[2k] = DFT_M(x)[k],  X[2k+1] = DFT_M(+-h x)[k]
// so no stage works on the zero padding, and one index holds at most one mode.
// The generic kernel (ping-pong shared memory, runtime radices) ran these
// passes: four 1023^2 slices, 4 x 1036 x 2048 cells, x 94 us and y 106 us of a
// backprojection that went from 439 to 380 us; projection of four 511^2 slices
// 101 -> 83 us.
#include <atomic>
#include <cstdint>

#include "lc_fft.hpp"
#include "lc_regfft.cuh"

namespace lc {
namespace {

constexpr int kModeLines = 4;  // rows per CTA, or adjacent columns (32-byte segments)

struct ModeArgs {
    const void *in;
    void *out;
    long n_outer, n_inner, in_ostride, out_ostride, bpo;
    int modes;            // n
    int win, lo;          // grid window: entry j is grid index (j - lo) mod L, j < win
    int real;             // the mode side is real (float)
    const float *fac;     // per mode, or null
    const float *linefac; // per column, or null (type 2)
    float scale;
};

template <int R0, int R1, int R2>
constexpr size_t mode_smem() {
    constexpr int M = RegPlan<R0, R1, R2>::M;
    return (2 * (size_t)M * kModeLines + 2 * (size_t)M) * sizeof(float2);
}

template <int R0, int R1, int R2, bool ROWS, bool TYPE1>
__global__ void __launch_bounds__(RegPlan<R0, R1, R2>::NT *kModeLines) mode_fft_kernel(ModeArgs a) {
    using P = RegPlan<R0, R1, R2>;
    constexpr int M = P::M, RM = P::RM, NT = P::NT, C = kModeLines, L = 2 * M;
    extern __shared__ __align__(16) float2 mode_sm[];
    float2 *tw = mode_sm + 2 * M * C;  // exp(-2 pi i m / M)
    float2 *th = tw + M;               // exp(-pi i m / M)
    load_line_twiddles<M>(tw);
    const int t = ROWS ? (int)threadIdx.x % NT : (int)threadIdx.x / C;
    const int c = ROWS ? (int)threadIdx.x / NT : (int)threadIdx.x % C;
    bool valid;
    long bin, bout, step;
    float lf = a.scale;
    if constexpr (ROWS) {
        const long line = (long)blockIdx.x * C + c;
        valid = line < a.n_outer;
        bin = (valid ? line : 0) * a.in_ostride;
        bout = (valid ? line : 0) * a.out_ostride;
        step = 1;
    } else {
        const long o = (long)blockIdx.x / a.bpo;
        const long col = ((long)blockIdx.x - o * a.bpo) * C + c;
        valid = col < a.n_inner;
        bin = o * a.in_ostride + (valid ? col : 0);
        bout = o * a.out_ostride + (valid ? col : 0);
        step = a.n_inner;
        if (a.linefac && valid) lf *= a.linefac[col];
    }
    const int Q = a.modes / 2, pos = a.modes - Q;  // modes -Q .. pos - 1
    const float2 zero = make_float2(0.f, 0.f);
    const auto at = [&](int q, int i) -> float2 & {
        return ROWS ? mode_sm[q * M * C + c * M + i] : mode_sm[q * M * C + i * C + c];
    };
    float2 v[2][RM];
    constexpr int NA = M / R0, NC = M / R2;
    if constexpr (TYPE1) {
        const float2 *in = static_cast<const float2 *>(a.in) + bin;
        if (t < NA) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const int i = t + r * NA;
                if constexpr (ROWS) {
                    const float4 z = valid ? reinterpret_cast<const float4 *>(in)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[0][r] = make_float2(z.x, z.y);
                    v[1][r] = make_float2(z.z, z.w);
                } else {
                    int j0 = 2 * i + a.lo, j1 = j0 + 1;
                    if (j0 >= L) j0 -= L;
                    if (j1 >= L) j1 -= L;
                    v[0][r] = valid && j0 < a.win ? in[(long)j0 * step] : zero;
                    v[1][r] = valid && j1 < a.win ? in[(long)j1 * step] : zero;
                }
            }
        }
        __syncthreads();  // twiddle tables ready
        xform3<M, R0, R1, R2>(v, at, t, tw, +1);
        if (t < NC && valid) {
#pragma unroll
            for (int r = 0; r < R2; ++r) {
                const int m = t + r * NC;
                int j = -1;
                float sg = 1.f;
                if (m < pos) {
                    j = m + Q;
                } else if (m >= M - Q) {
                    j = m - (M - Q);
                    sg = -1.f;
                }
                if (j < 0) continue;
                const float2 w = cmul(cconj(th[m]), v[1][r]);
                const float s = a.fac ? lf * a.fac[j] : lf;
                const float2 y = make_float2(s * fmaf(sg, w.x, v[0][r].x), s * fmaf(sg, w.y, v[0][r].y));
                if (a.real) static_cast<float *>(a.out)[bout + (long)j * step] = y.x;
                else static_cast<float2 *>(a.out)[bout + (long)j * step] = y;
            }
        }
    } else {
        __syncthreads();  // twiddle tables ready
        if (t < NA) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const int m = t + r * NA;
                int j = -1;
                float sg = 1.f;
                if (m < pos) {
                    j = m + Q;
                } else if (m >= M - Q) {
                    j = m - (M - Q);
                    sg = -1.f;
                }
                float2 x = zero;
                if (valid && j >= 0) {
                    x = a.real ? make_float2(static_cast<const float *>(a.in)[bin + (long)j * step], 0.f)
                               : static_cast<const float2 *>(a.in)[bin + (long)j * step];
                    x = cscale(x, a.fac ? a.fac[j] * lf : lf);
                }
                v[0][r] = x;
                v[1][r] = cscale(cmul(x, th[m]), sg);
            }
        }
        xform3<M, R0, R1, R2>(v, at, t, tw, -1);
        if (t < NC && valid) {
            float2 *out = static_cast<float2 *>(a.out) + bout;
#pragma unroll
            for (int r = 0; r < R2; ++r) {
                const int k = t + r * NC;
                if constexpr (ROWS) {
                    reinterpret_cast<float4 *>(out)[k] = make_float4(v[0][r].x, v[0][r].y, v[1][r].x, v[1][r].y);
                } else {
                    int j0 = 2 * k + a.lo, j1 = j0 + 1;
                    if (j0 >= L) j0 -= L;
                    if (j1 >= L) j1 -= L;
                    if (j0 < a.win) out[(long)j0 * step] = v[0][r];
                    if (j1 < a.win) out[(long)j1 * step] = v[1][r];
                }
            }
        }
    }
}

template <int R0, int R1, int R2, bool ROWS, bool TYPE1>
void launch_mode_t(cudaStream_t st, const ModeArgs &a, long blocks) {
    constexpr size_t smem = mode_smem<R0, R1, R2>();
    auto kern = mode_fft_kernel<R0, R1, R2, ROWS, TYPE1>;
    static std::atomic<unsigned long long> configured{0};
    int dev = 0;
    LC_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load() & bit)) {
        LC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured.fetch_or(bit);
    }
    kern<<<(unsigned)blocks, RegPlan<R0, R1, R2>::NT * kModeLines, smem, st>>>(a);
    LC_CHECK_LAUNCH();
}

template <int R0, int R1, int R2>
void launch_mode_plan(cudaStream_t st, bool rows, bool type1, const ModeArgs &a, long blocks) {
    if (rows && type1) launch_mode_t<R0, R1, R2, true, true>(st, a, blocks);
    else if (rows) launch_mode_t<R0, R1, R2, true, false>(st, a, blocks);
    else if (type1) launch_mode_t<R0, R1, R2, false, true>(st, a, blocks);
    else launch_mode_t<R0, R1, R2, false, false>(st, a, blocks);
}

}  // namespace

bool launch_mode_fft(cudaStream_t st, const AxisFFT &a) {
    if (a.fp64 || a.mid || a.lines_per_cta > 0 || a.L % 2 != 0 || a.cg_parts) return false;
    const int M = a.L / 2;
    if (!line_plan_exists(M)) return false;
    const bool rows = a.n_inner == 1;
    const bool type1 = a.sign > 0;
    // the grid side: every value, or a window with an explicit shift
    const int gmap_in = a.in_map == IN_DIRECT || (a.in_map == IN_MODES && a.in_shift >= 0);
    const int gmap_out = a.out_map == OUT_DIRECT || (a.out_map == OUT_MODES && a.out_shift >= 0);
    ModeArgs m{};
    if (type1) {
        if (!gmap_in || a.out_map != OUT_MODES || a.out_shift >= 0 || a.pre || a.linefac || a.in_t != E_C64) return false;
        m.modes = a.n_out;
        m.win = a.n_in;
        m.lo = a.in_map == IN_MODES ? a.in_shift : 0;
        m.real = a.out_t == E_F32;
        m.fac = static_cast<const float *>(a.post);
    } else {
        if (!gmap_out || a.in_map != IN_MODES || a.in_shift >= 0 || a.post || a.out_t != E_C64) return false;
        m.modes = a.n_in;
        m.win = a.n_out;
        m.lo = a.out_map == OUT_MODES ? a.out_shift : 0;
        m.real = a.in_t == E_F32;
        m.fac = static_cast<const float *>(a.pre);
        m.linefac = static_cast<const float *>(a.linefac);
    }
    if (m.modes > M || m.modes <= 0 || m.lo < 0 || m.lo >= a.L || m.win > a.L) return false;
    if (rows) {
        // whole rows of complex values, two at a time
        const void *grid = type1 ? a.in : a.out;
        const long gs = type1 ? a.in_ostride : a.out_ostride;
        if (m.win != a.L || m.lo != 0 || m.real || m.linefac || gs % 2 != 0 ||
            (reinterpret_cast<uintptr_t>(grid) & 15) != 0)
            return false;
    }
    if (a.n_outer <= 0 || a.n_inner <= 0) return true;
    m.in = a.in;
    m.out = a.out;
    m.n_outer = a.n_outer;
    m.n_inner = a.n_inner;
    m.in_ostride = a.in_ostride;
    m.out_ostride = a.out_ostride;
    m.scale = (float)a.scale;
    m.bpo = (a.n_inner + kModeLines - 1) / kModeLines;
    const long blocks = rows ? (a.n_outer + kModeLines - 1) / kModeLines : a.n_outer * m.bpo;
    LC_REQUIRE(blocks < (1L << 31), "mode FFT: grid too large");
    switch (M) {
#define LC_MODE_CASE(mm, r0, r1, r2) \
    case mm: launch_mode_plan<r0, r1, r2>(st, rows, type1, m, blocks); return true;
        LC_LINE_PLANS(LC_MODE_CASE)
#undef LC_MODE_CASE
        default: return false;
    }
}

}  // namespace lc
