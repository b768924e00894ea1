// Detector-domain DFTs of odd length n by Bluestein's chirp-z convolution on
// the register-plan line kernels.
//
//   X[k] = chirp[k] * sum_j (x[j] chirp[j]) conj(chirp[k - j])
// is a convolution of length L = next 2^p 3^q >= 2n - 1, done as FFT, a
// multiply by the precomputed spectrum V of the chirp kernel, and an inverse
// FFT.  L is even here, and both the padded input and the kept output fit in
// the first M = L/2 points (n <= M), so each of the two transforms runs as
// two transforms of length M in one thread (the even/odd split of the column
// kernels):
//   forward  X[2k] = DFT_M(a)[k],  X[2k+1] = DFT_M(h a)[k],   h(j) = exp(-i pi j / M)
//   inverse  c[j] = DFT+_M(Y_even)[j] + conj h(j) DFT+_M(Y_odd)[j]
// The fftshift/ifftshift rolls are index maps at the load and the store
// (value j of the line is in[(j + d_pre) mod n]; out[k] = X[(k + d_post) mod n]).
// A CTA takes 4 lines: adjacent rows (contiguous lines) or 4 adjacent columns
// (32-byte row segments).  Two real problems go to one line:
//   * real input (rows): rows a and b are transformed as the complex line
//     a + i b, whose DFT Z gives
//       A[k] = (Z[k] + conj Z[n-k]) / 2,   B[k] = (Z[k] - conj Z[n-k]) / (2i)
//     (the DFT of a real sequence is Hermitian), paired through shared memory;
//   * real output: Re DFT(v) = DFT(h) with h[m] = (v[m] + conj v[n-m]) / 2, so
//     lines a and b are transformed as h_a + i h_b and the results are the
//     real and imaginary parts.
// Columns of Hermitian data (AxisDFT::herm) read and transform half of the
// columns, or read half of each column.  (Both passes of a 180 x 361 x 361
// projection: 1.11 ms on the generic kernel with every row, 0.33 ms here with
// half of the rows.  A backprojection of 360 x 511 x 511 values, whose columns
// took 1.19 ms and rows 0.71 ms: 10.4 -> 9.9 ms with half of the columns, the
// spreading then reading half of the lattice.)
#include <atomic>

#include "lc_fft.hpp"
#include "lc_regfft.cuh"

namespace lc {
namespace {

constexpr int kBlueLines = 4;

struct BlueArgs {
    const void *in;
    void *out;
    long n_outer, n_inner, in_ostride, out_ostride, bpo;
    long rows_per, group_stride;
    int odd_rows;       // pairs: whether a group has an odd number of rows, and the
    FastDiv div_lines;  // division of a line's number by the lines of a group
    int n, d_pre, d_post, out_min, out_max, herm;
    float scale;
    const float2 *chirp, *V;
};

template <int R0, int R1, int R2>
constexpr size_t blue_smem() {
    constexpr int M = RegPlan<R0, R1, R2>::M;
    return (2 * (size_t)M * kBlueLines + 2 * (size_t)M) * sizeof(float2);
}

enum BlueKind {
    BK_ROWS_R2C = 0,  // real rows, two to a line
    BK_ROWS_C2C = 1,
    BK_ROWS_C2R = 2,  // real output, two rows to a line
    BK_COLS_C2C = 3,
    BK_COLS_C2R = 4,  // real output, two columns to a line
};

template <int R0, int R1, int R2, int KIND>
__global__ void __launch_bounds__(RegPlan<R0, R1, R2>::NT *kBlueLines) blue_kernel(BlueArgs a) {
    using P = RegPlan<R0, R1, R2>;
    constexpr int M = P::M, RM = P::RM, NT = P::NT, C = kBlueLines;
    constexpr bool ROWS = KIND <= BK_ROWS_C2R;
    constexpr bool C2R = KIND == BK_ROWS_C2R || KIND == BK_COLS_C2R;
    constexpr bool PAIR = C2R || KIND == BK_ROWS_R2C;
    extern __shared__ __align__(16) float2 blue_sm[];
    float2 *tw = blue_sm + 2 * M * C;  // exp(-2 pi i m / M)
    float2 *th = tw + M;               // exp(-pi i m / M)
    load_line_twiddles<M>(tw);
    // ROWS: thread (c, t) with t fastest (contiguous samples); columns: (t, c)
    // with c fastest (adjacent columns)
    const int t = ROWS ? (int)threadIdx.x % NT : (int)threadIdx.x / C;
    const int c = ROWS ? (int)threadIdx.x / NT : (int)threadIdx.x % C;
    const int n = a.n;
    // the line's first element in the input and output, and the second line of
    // a pair at the distances sec_in, sec_out
    long base_in, base_out, step, sec_in = 0, sec_out = 0;
    bool valid, valid_b = false;
    int col = 0;  // column of a C2C column line
    if constexpr (ROWS) {
        if constexpr (PAIR) {
            const unsigned line = blockIdx.x * C + c, g = fast_div(line, a.div_lines);
            const long l0 = 2 * (long)line - (a.odd_rows ? g : 0u);
            valid = l0 < a.n_outer;
            valid_b = l0 + 1 < (long)(g + 1) * a.rows_per && valid;
            base_in = (valid ? l0 : 0) * a.in_ostride;
            base_out = (valid ? l0 : 0) * a.out_ostride;
            sec_in = a.in_ostride;
            sec_out = a.out_ostride;
        } else {
            const long l0 = (long)blockIdx.x * C + c;
            valid = l0 < a.n_outer;
            const long line = valid ? l0 : 0;
            const long g = line / a.rows_per, r = line - g * a.rows_per;
            base_in = g * a.group_stride + r * a.in_ostride;
            base_out = g * a.group_stride + r * a.out_ostride;
        }
        step = 1;
    } else {
        const long o = (long)blockIdx.x / a.bpo;
        const long l0 = (((long)blockIdx.x - o * a.bpo) * C + c) * (PAIR ? 2 : 1) +
                        (KIND == BK_COLS_C2C && a.herm ? a.n_inner / 2 : 0);
        valid = l0 < a.n_inner;
        valid_b = PAIR && l0 + 1 < a.n_inner;
        col = valid ? (int)l0 : 0;
        base_in = o * a.in_ostride + col;
        base_out = o * a.out_ostride + col;
        sec_in = sec_out = 1;
        step = a.n_inner;
    }
    const auto at = [&](int q, int i) -> float2 & {
        return ROWS ? blue_sm[q * M * C + c * M + i] : blue_sm[q * M * C + i * C + c];
    };
    const float2 zero = make_float2(0.f, 0.f);
    float2 v[2][RM];
    constexpr int NA = M / R0;
    if (t < NA) {
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int j = t + r * NA;
            float2 x = zero;
            if (valid && j < n) {
                if constexpr (KIND == BK_ROWS_R2C) {
                    int s = j + a.d_pre;
                    if (s >= n) s -= n;
                    const float *in = static_cast<const float *>(a.in) + base_in + s;
                    x = make_float2(in[0], valid_b ? in[sec_in] : 0.f);
                } else if constexpr (!C2R) {
                    int s = j + a.d_pre;
                    if (s >= n) s -= n;
                    x = static_cast<const float2 *>(a.in)[base_in + (long)s * step];
                } else {
                    const float2 *in = static_cast<const float2 *>(a.in) + base_in;
                    if (KIND == BK_COLS_C2R && a.herm) {
                        // n odd, centre row n / 2: value j of the line is the
                        // conjugate of row n/2 - j, value n - j that row itself
                        const int k = n / 2, m = j <= k ? j : n - j;
                        float2 va = in[(long)(k - m) * step];
                        float2 vb = valid_b ? in[(long)(k - m) * step + sec_in] : zero;
                        if (m == 0) va.y = vb.y = 0.f;
                        x = j <= k ? make_float2(va.x + vb.y, vb.x - va.y) : make_float2(va.x - vb.y, vb.x + va.y);
                    } else {
                        int s = j + a.d_pre, u = (j == 0 ? 0 : n - j) + a.d_pre;
                        if (s >= n) s -= n;
                        if (u >= n) u -= n;
                        const float2 p = in[(long)s * step], q = in[(long)u * step];
                        const float2 pb = valid_b ? in[(long)s * step + sec_in] : zero;
                        const float2 qb = valid_b ? in[(long)u * step + sec_in] : zero;
                        // h_a + i h_b
                        x = make_float2(0.5f * ((p.x + q.x) - (pb.y - qb.y)), 0.5f * ((p.y - q.y) + (pb.x + qb.x)));
                    }
                }
                x = cmul(x, __ldg(a.chirp + j));
            }
            v[0][r] = x;
        }
    }
    __syncthreads();  // twiddle tables ready
    if (t < NA) {
#pragma unroll
        for (int r = 0; r < R0; ++r) v[1][r] = cmul(v[0][r], th[t + r * NA]);
    }
    xform3<M, R0, R1, R2>(v, at, t, tw, -1);
    constexpr int NC = M / R2;
    if (t < NC) {
#pragma unroll
        for (int r = 0; r < R2; ++r) {
            const int k = t + r * NC;
            v[0][r] = cmul(v[0][r], __ldg(a.V + 2 * k));
            v[1][r] = cmul(v[1][r], __ldg(a.V + 2 * k + 1));
        }
    }
    xform3<M, R2, R1, R0>(v, at, t, tw, +1);
    constexpr int NF = M / R0;
    if constexpr (KIND == BK_ROWS_R2C) {
        // Z[q] of the line into its shared-memory row, then the two rows'
        // values from the pairs (q, n - q)
        __syncthreads();  // the transform's last shared-memory reads are done
        if (t < NF) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const int q = t + r * NF;
                if (q < n) {
                    const float2 h = th[q];
                    const float2 y = cadd(v[0][r], cmul(make_float2(h.x, -h.y), v[1][r]));
                    at(0, q) = cscale(cmul(y, __ldg(a.chirp + q)), 0.5f * a.scale);
                }
            }
        }
        __syncthreads();
        if (t < NF && valid) {
            float2 *out = static_cast<float2 *>(a.out) + base_out;
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const int q = t + r * NF;
                if (q < n) {
                    int k = q - a.d_post;
                    if (k < 0) k += n;
                    if (k < a.out_min || k >= a.out_max) continue;
                    const float2 zq = at(0, q), zm = at(0, q == 0 ? 0 : n - q);
                    out[k] = make_float2(zq.x + zm.x, zq.y - zm.y);
                    if (valid_b) out[sec_out + k] = make_float2(zq.y + zm.y, zm.x - zq.x);
                }
            }
        }
        return;
    }
    if (t < NF && valid) {
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int q = t + r * NF;
            if (q < n) {
                const float2 h = th[q];
                float2 y = cadd(v[0][r], cmul(make_float2(h.x, -h.y), v[1][r]));
                y = cscale(cmul(y, __ldg(a.chirp + q)), a.scale);
                int k = q - a.d_post;
                if (k < 0) k += n;
                if constexpr (C2R) {
                    float *out = static_cast<float *>(a.out) + base_out + (long)k * step;
                    out[0] = y.x;
                    if (valid_b) out[sec_out] = y.y;
                } else {
                    float2 *out = static_cast<float2 *>(a.out) + base_out;
                    if (KIND == BK_COLS_C2C && a.herm) {
                        const int mc = (int)a.n_inner - 1 - col;  // the mirrored column, row n - 1 - k
                        if (k <= n / 2) out[(long)k * step] = y;
                        if (mc != col && k >= n / 2)
                            out[(long)(n - 1 - k) * step + (mc - col)] = make_float2(y.x, -y.y);
                    } else {
                        out[(long)k * step] = y;
                    }
                }
            }
        }
    }
}

template <int R0, int R1, int R2, int KIND>
void launch_blue_t(cudaStream_t st, const BlueArgs &a, long blocks) {
    constexpr size_t smem = blue_smem<R0, R1, R2>();
    auto kern = blue_kernel<R0, R1, R2, KIND>;
    static std::atomic<unsigned long long> configured{0};
    int dev = 0;
    LC_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured.load() & bit)) {
        LC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured.fetch_or(bit);
    }
    kern<<<(unsigned)blocks, RegPlan<R0, R1, R2>::NT * kBlueLines, smem, st>>>(a);
    LC_CHECK_LAUNCH();
}

template <int R0, int R1, int R2>
void launch_blue_plan(cudaStream_t st, int kind, const BlueArgs &a, long blocks) {
    switch (kind) {
        case BK_ROWS_R2C: launch_blue_t<R0, R1, R2, BK_ROWS_R2C>(st, a, blocks); break;
        case BK_ROWS_C2C: launch_blue_t<R0, R1, R2, BK_ROWS_C2C>(st, a, blocks); break;
        case BK_ROWS_C2R: launch_blue_t<R0, R1, R2, BK_ROWS_C2R>(st, a, blocks); break;
        case BK_COLS_C2C: launch_blue_t<R0, R1, R2, BK_COLS_C2C>(st, a, blocks); break;
        default: launch_blue_t<R0, R1, R2, BK_COLS_C2R>(st, a, blocks); break;
    }
}

}  // namespace

bool launch_bluestein_lines(cudaStream_t st, const AxisDFT &a, const BluesteinEntry &e) {
    if (e.L % 2 != 0 || a.n > e.L / 2) return false;
    const int M = e.L / 2;
    if (!line_plan_exists(M)) return false;
    const bool rows = a.n_inner == 1, in_real = a.in_t == E_F32, out_real = a.out_t == E_F32;
    // real to real, and columns of real input, take the generic kernel
    if (in_real && (out_real || !rows)) return false;
    if (a.n_outer <= 0 || a.n_inner <= 0) return true;
    const int kind = rows ? (in_real ? BK_ROWS_R2C : (out_real ? BK_ROWS_C2R : BK_ROWS_C2C))
                          : (out_real ? BK_COLS_C2R : BK_COLS_C2C);
    const bool pair = kind == BK_ROWS_R2C || kind == BK_ROWS_C2R || kind == BK_COLS_C2R;
    LC_REQUIRE(a.rows_per == 0 || (rows && a.n_outer % a.rows_per == 0), "DFT: rows come in whole groups");
    LC_REQUIRE(a.group_stride == 0 || (a.rows_per > 0 && !pair), "DFT: real lines follow one another");
    LC_REQUIRE((a.out_min == 0 && a.out_max == 0) || kind == BK_ROWS_R2C, "DFT: only real rows are stored in part");
    LC_REQUIRE(!a.herm || (!rows && a.n % 2 == 1 && (out_real || a.n_inner % 2 == 1)),
               "DFT: Hermitian columns need odd sizes");
    LC_REQUIRE(!a.herm || (a.d_pre == a.n / 2 && a.d_post == (a.n + 1) / 2), "DFT: Hermitian columns are centred");
    BlueArgs b{};
    b.in = a.in;
    b.out = a.out;
    b.n_outer = a.n_outer;
    b.n_inner = a.n_inner;
    b.in_ostride = a.in_ostride;
    b.out_ostride = a.out_ostride;
    b.rows_per = a.rows_per > 0 ? a.rows_per : a.n_outer;
    b.group_stride = a.group_stride;
    b.n = a.n;
    b.d_pre = ((a.d_pre % a.n) + a.n) % a.n;
    b.d_post = ((a.d_post % a.n) + a.n) % a.n;
    b.out_min = a.out_min;
    b.out_max = a.out_max > 0 ? a.out_max : a.n;
    b.herm = a.herm ? 1 : 0;
    b.scale = a.scale;
    b.chirp = e.chirp.get();
    b.V = e.V.get();
    long blocks;
    if (rows) {
        const long lines_per = pair ? (b.rows_per + 1) / 2 : b.rows_per, lines = a.n_outer / b.rows_per * lines_per;
        LC_REQUIRE(lines + kBlueLines < (1L << 31), "DFT: too many lines");
        b.odd_rows = (int)(b.rows_per % 2);
        b.div_lines = make_fastdiv((unsigned)lines_per);
        blocks = (lines + kBlueLines - 1) / kBlueLines;
        b.bpo = 1;
    } else {
        const long cols = pair ? (a.n_inner + 1) / 2 : (a.herm ? a.n_inner - a.n_inner / 2 : a.n_inner);
        b.bpo = (cols + kBlueLines - 1) / kBlueLines;
        blocks = a.n_outer * b.bpo;
    }
    LC_REQUIRE(blocks < (1L << 31), "DFT: grid too large");
    switch (M) {
#define LC_BLUE_CASE(m, r0, r1, r2) \
    case m: launch_blue_plan<r0, r1, r2>(st, kind, b, blocks); return true;
        LC_LINE_PLANS(LC_BLUE_CASE)
#undef LC_BLUE_CASE
        default: return false;
    }
}

}  // namespace lc
