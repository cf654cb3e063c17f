// k_fftg.cu -- the per-frame transforms for frame sizes that are not powers
// of two (or are larger than the radix-2 kernels' 512): any ncols and nrows
// up to kMaxSide.
//
// The reference builds FFTW plans for whatever size its frames have
// (smip-cli/main.cpp:256-259, crosscorrel.h:112-141), so frames such as
// 100 x 100 or a 320 x 240 crop (-s, main.cpp:157-167) are ordinary input.
// These kernels compute the same quantities as k_fft.cu -- the float-float
// forward transform into the spectrum layout S, the power-spectrum partials,
// the FP32 correlation transforms -- and the FP64 lines of the final image,
// with a mixed-radix transform instead of the radix-2 one.
//
// Transform: the Stockham autosort formulation of the mixed-radix FFT
// (Govindaraju, Lloyd, Dotsenko, Smith, Manferdelli, "High performance
// discrete Fourier transforms on graphics processors", SC 2008).  The length
// L is split into factors R_1 R_2 ... (odd primes, then 2, 4 or 8); with Ns
// the product of the earlier factors, the pass of radix R maps x to y by
//     y[(j / Ns) Ns R + q Ns + k] = sum_{r < R} x[j + r L / R] w^(r (k + q Ns) L / (Ns R)),
//     j in [0, L / R), k = j mod Ns, q in [0, R),  w = exp(-2 pi i / L).
// Radices up to 8 are butterflies: a thread takes the R inputs of one j into
// registers, multiplies them by the twiddles w^(r k L / (Ns R)) (one table
// lookup each, exponents below L) and forms their R-point transform, for an
// odd R from the sums and differences of the inputs r and R - r.  A larger
// prime is summed per output, its twiddle and its DFT folded into one lookup
// per term.  Results come out in natural order.  Odd factors go first: their
// first pass's strided stores then fall into different banks.
// Arithmetic per the caller's type: float-float (dfc, the same error-free
// two_prod / two_sum steps as the radix-2 forward transform), FP32, or FP64.
//
// Bound by FP32 issue and shared-memory latency.  A sum per output for every
// radix cost R - 1 complex products an element and pass; with butterflies and
// two real rows per transform, 200 frames of 640 x 480 take 627 us in the row
// kernel, 1111 in the column kernel and 294 in the correlation rows (2662,
// 2306 and 1506 before).  Four CTAs of 256 threads an SM are worth the registers
// that they cost (three: 731 us, row kernel; unbounded: 909 and 1319).
#include "smip_dev.cuh"

namespace smip_gpu {

// ---------------------------------------------------------------- arithmetic
__device__ __forceinline__ float2 gmac(float2 acc, float2 x, float2 w)
{
    acc.x = fmaf(x.x, w.x, fmaf(-x.y, w.y, acc.x));
    acc.y = fmaf(x.x, w.y, fmaf(x.y, w.x, acc.y));
    return acc;
}
__device__ __forceinline__ double2 gmac(double2 acc, double2 x, double2 w)
{
    acc.x = fma(x.x, w.x, fma(-x.y, w.y, acc.x));
    acc.y = fma(x.x, w.y, fma(x.y, w.x, acc.y));
    return acc;
}
__device__ __forceinline__ dfc gmac(const dfc& acc, const dfc& x, const dfc& w) { return df_cadd(acc, df_cmul(x, w)); }
__device__ __forceinline__ float2 gconj(float2 w) { return make_float2(w.x, -w.y); }
__device__ __forceinline__ double2 gconj(double2 w) { return make_double2(w.x, -w.y); }
__device__ __forceinline__ dfc gconj(dfc w) { return tw_conj(w); }
__device__ __forceinline__ float2 gnorm(float2 v) { return v; }
__device__ __forceinline__ double2 gnorm(double2 v) { return v; }
__device__ __forceinline__ dfc gnorm(dfc v)
{
    df_norm(v.h.x, v.l.x);
    df_norm(v.h.y, v.l.y);
    return v;
}

// --------------------------------------------------------- butterflies
__device__ __forceinline__ float2 gadd(float2 a, float2 b) { return cadd(a, b); }
__device__ __forceinline__ float2 gsub(float2 a, float2 b) { return csub(a, b); }
__device__ __forceinline__ float2 gmul(float2 a, float2 w) { return cmul(a, w); }
__device__ __forceinline__ double2 gadd(double2 a, double2 b) { return cadd(a, b); }
__device__ __forceinline__ double2 gsub(double2 a, double2 b) { return csub(a, b); }
__device__ __forceinline__ double2 gmul(double2 a, double2 w) { return cmul(a, w); }
__device__ __forceinline__ dfc gadd(const dfc& a, const dfc& b) { return df_cadd(a, b); }
__device__ __forceinline__ dfc gsub(const dfc& a, const dfc& b) { return df_csub(a, b); }
__device__ __forceinline__ dfc gmul(const dfc& a, const dfc& w) { return df_cmul(a, w); }
__device__ __forceinline__ double2 mul_mi(double2 b, int sign) { return sign > 0 ? make_double2(-b.y, b.x) : make_double2(b.y, -b.x); }

// acc + a * (real part of w), acc + a * (minus the imaginary part of w)
__device__ __forceinline__ float2 gmacr(float2 acc, float2 a, float2 w) { return make_float2(fmaf(a.x, w.x, acc.x), fmaf(a.y, w.x, acc.y)); }
__device__ __forceinline__ float2 gmaci(float2 acc, float2 a, float2 w) { return make_float2(fmaf(-a.x, w.y, acc.x), fmaf(-a.y, w.y, acc.y)); }
__device__ __forceinline__ double2 gmacr(double2 acc, double2 a, double2 w) { return make_double2(fma(a.x, w.x, acc.x), fma(a.y, w.x, acc.y)); }
__device__ __forceinline__ double2 gmaci(double2 acc, double2 a, double2 w) { return make_double2(fma(-a.x, w.y, acc.x), fma(-a.y, w.y, acc.y)); }
__device__ __forceinline__ void df_mac(float& h, float& l, float ah, float al, float sh, float sl)
{
    const float p = __fmul_rn(ah, sh);
    const float e = fmaf(al, sh, fmaf(ah, sl, fmaf(ah, sh, -p)));
    df_add_lazy(h, l, p, e, h, l);
}
__device__ __forceinline__ dfc gmacr(dfc acc, const dfc& a, const dfc& w)
{
    df_mac(acc.h.x, acc.l.x, a.h.x, a.l.x, w.h.x, w.l.x);
    df_mac(acc.h.y, acc.l.y, a.h.y, a.l.y, w.h.x, w.l.x);
    return acc;
}
__device__ __forceinline__ dfc gmaci(dfc acc, const dfc& a, const dfc& w)
{
    df_mac(acc.h.x, acc.l.x, a.h.x, a.l.x, -w.h.y, -w.l.y);
    df_mac(acc.h.y, acc.l.y, a.h.y, a.l.y, -w.h.y, -w.l.y);
    return acc;
}

template <typename C> __device__ __forceinline__ void dft4(C& a, C& b, C& c, C& d, int sign)
{
    const C s0 = gadd(a, c), d0 = gsub(a, c), s1 = gadd(b, d), d1 = mul_mi(gsub(b, d), sign);
    a = gadd(s0, s1);
    c = gsub(s0, s1);
    b = gadd(d0, d1);
    d = gsub(d0, d1);
}

// The R-point transform of v in place; tw: the length-L table, lr = L / R.
template <int R, typename C> __device__ __forceinline__ void dft_small(C* v, const C* tw, int lr, int sign)
{
    if constexpr (R == 2) {
        const C a = v[0];
        v[0] = gadd(a, v[1]);
        v[1] = gsub(a, v[1]);
    } else if constexpr (R == 4) {
        dft4(v[0], v[1], v[2], v[3], sign);
    } else if constexpr (R == 8) {
        const C w = sign > 0 ? gconj(tw[lr]) : tw[lr]; // exp(-+ i pi / 4)
        dft4(v[0], v[2], v[4], v[6], sign);
        dft4(v[1], v[3], v[5], v[7], sign);
        const C t1 = gmul(v[3], w), t2 = mul_mi(v[5], sign), t3 = mul_mi(gmul(v[7], w), sign);
        const C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = gadd(e0, o0);
        v[4] = gsub(e0, o0);
        v[1] = gadd(e1, t1);
        v[5] = gsub(e1, t1);
        v[2] = gadd(e2, t2);
        v[6] = gsub(e2, t2);
        v[3] = gadd(e3, t3);
        v[7] = gsub(e3, t3);
    } else { // odd: V[q], V[R - q] = (v0 + sum s_r cos) -+ i (sum d_r sin)
        constexpr int h = (R - 1) / 2;
        C s[h], d[h];
#pragma unroll
        for (int r = 1; r <= h; ++r) {
            s[r - 1] = gadd(v[r], v[R - r]);
            d[r - 1] = gsub(v[r], v[R - r]);
        }
        const C v0 = v[0];
#pragma unroll
        for (int r = 0; r < h; ++r)
            v[0] = gadd(v[0], s[r]);
#pragma unroll
        for (int q = 1; q <= h; ++q) {
            C A = v0, B {};
#pragma unroll
            for (int r = 1; r <= h; ++r) {
                const C w = tw[(r * q % R) * lr];
                A = gmacr(A, s[r - 1], w);
                B = gmaci(B, d[r - 1], w);
            }
            B = mul_mi(B, sign);
            v[q] = gadd(A, B);
            v[R - q] = gsub(A, B);
        }
    }
}

// One pass of radix R over nl lines (line stride ls) from x to y.
template <int R, typename C>
__device__ __forceinline__ void stockham_pass(const C* x, C* y, int L, int Ns, const unsigned* mp, int nl, int ls,
                                              const C* tw, int sign)
{
    const int LR = L / R;
    for (int idx = threadIdx.x; idx < nl * LR; idx += blockDim.x) {
        const int line = idx / LR, j = idx - line * LR;
        const unsigned m = __ldg(mp + j); // first output, twiddle exponent of r = 1: no divisions
        const int o0 = (int)(m & 0xffffu), k1 = (int)(m >> 16);
        const C* X = x + line * ls + j;
        C v[R];
        v[0] = X[0];
#pragma unroll
        for (int r = 1; r < R; ++r)
            v[r] = X[r * LR];
        if (Ns > 1) {
#pragma unroll
            for (int r = 1; r < R; ++r) {
                const C w = tw[r * k1];
                v[r] = gmul(v[r], sign > 0 ? gconj(w) : w);
            }
        }
        dft_small<R>(v, tw, LR, sign);
        C* Y = y + line * ls + o0;
#pragma unroll
        for (int q = 0; q < R; ++q)
            Y[q * Ns] = v[q];
    }
}

// Stockham passes over nl lines of length p.L (line stride ls) in shared
// memory, ping-ponging between x and y; returns the buffer with the result.
// tw: p.L entries exp(-2 pi i k / L); sign -1 forward, +1 inverse
// (unnormalised).  Called by all threads of the block.
template <typename C>
__device__ C* stockham(C* x, C* y, const GenPlan& p, int nl, int ls, const C* tw, int sign)
{
    const int L = p.L;
    int Ns = 1;
    for (int f = 0; f < p.nf; ++f) {
        const int R = p.fac[f];
        const unsigned* mp = p.map + f * L;
        switch (R) {
        case 2: stockham_pass<2>(x, y, L, Ns, mp, nl, ls, tw, sign); break;
        case 3: stockham_pass<3>(x, y, L, Ns, mp, nl, ls, tw, sign); break;
        case 4: stockham_pass<4>(x, y, L, Ns, mp, nl, ls, tw, sign); break;
        case 5: stockham_pass<5>(x, y, L, Ns, mp, nl, ls, tw, sign); break;
        case 7: stockham_pass<7>(x, y, L, Ns, mp, nl, ls, tw, sign); break;
        case 8: stockham_pass<8>(x, y, L, Ns, mp, nl, ls, tw, sign); break;
        default: { // a larger prime: one output per thread
            const int LR = L / R;
            for (int idx = threadIdx.x; idx < nl * L; idx += blockDim.x) {
                const int line = idx / L, o = idx - line * L;
                const unsigned m = __ldg(mp + o); // first input, exponent step
                const int j = (int)(m & 0xffffu), e0 = (int)(m >> 16);
                const C* X = x + line * ls + j;
                C acc = X[0];
                int e = 0;
                for (int r = 1; r < R; ++r) {
                    e += e0;
                    if (e >= L)
                        e -= L;
                    const C w = sign > 0 ? gconj(tw[e]) : tw[e];
                    acc = gmac(acc, X[r * LR], w);
                }
                y[line * ls + o] = gnorm(acc);
            }
        }
        }
        __syncthreads();
        C* tmp = x;
        x = y;
        y = tmp;
        Ns *= R;
    }
    return x;
}

template <typename C> __device__ void load_table(C* dst, const C* src, int n)
{
    for (int k = threadIdx.x; k < n; k += blockDim.x)
        dst[k] = src[k];
}

// a pixel as a float pair (hi, lo)
template <typename T> __device__ __forceinline__ float2 pix_pair(const T* p, long long i)
{
    return make_float2((float)p[i], 0.f); // u8/u16/f32 are exact in FP32
}
template <> __device__ __forceinline__ float2 pix_pair<double>(const double* p, long long i)
{
    const double v = p[i];
    const float h = (float)v;
    return make_float2(h, (float)(v - (double)h));
}

__device__ __forceinline__ float2 dfc_round(const dfc& v) { return make_float2(v.h.x + v.l.x, v.h.y + v.l.y); }

// ---------------------------------------------------------------- row pass
// rb rows (an even number) of one frame per CTA, two real rows per float-float
// transform (x0 + i x1), separated afterwards: writes G'(a, y) = sum_x f(x, y)
// exp(+2 pi i a x / W) = conj X(a), a < hw, stored [f][a][y] (the layout of
// k_fft.cu's row pass).  copy_out: the frames as read, written to device memory
// (mapped host input).
template <typename T>
__global__ void __launch_bounds__(256, 4) gen_row_kernel(const T* __restrict__ frames, long long fstride, int H, int hw,
                                                      int rb, const GenPlan pw, const dfc* __restrict__ tw_g,
                                                      dfc* __restrict__ Gt, T* __restrict__ copy_out,
                                                      SqSum<T>* __restrict__ rowsq)
{
    extern __shared__ dfc smg[];
    __shared__ SqSum<T> sqpart[8];
    SqLane<T> sq {}; // of this thread's pixels, for the correlation's error bound (k_xcorr.cu)
    const int W = pw.L;
    dfc* tw = smg;
    dfc* X = tw + W;
    dfc* Y = X + rb / 2 * W;
    const int f = blockIdx.y;
    const int y0 = blockIdx.x * rb;
    const int nr = min(rb, H - y0), nl = (nr + 1) / 2;
    const T* fr = frames + (long long)f * fstride + (long long)y0 * W;
    T* co = copy_out ? copy_out + (long long)f * fstride + (long long)y0 * W : nullptr;
    load_table(tw, tw_g, W);
    for (int i = threadIdx.x; i < nl * W; i += blockDim.x) {
        const int l = i / W, x = i - l * W, at = 2 * l * W + x;
        const bool two = 2 * l + 1 < nr; // the last row of an odd block goes alone
        const T v0 = fr[at], v1 = two ? fr[at + W] : T(0);
        const float2 p0 = pix_pair(&v0, 0), p1 = pix_pair(&v1, 0);
        dfc d;
        d.h = make_float2(p0.x, p1.x);
        d.l = make_float2(p0.y, p1.y);
        sq_add(sq, v0);
        sq_add(sq, v1);
        X[i] = d;
        if (co) {
            co[at] = v0;
            if (two)
                co[at + W] = v1;
        }
    }
    sq_store_warp(sq, sqpart);
    __syncthreads();
    const dfc* Z = stockham(X, Y, pw, nl, W, tw, -1);
    dfc* out = Gt + (long long)f * hw * H;
    for (int i = threadIdx.x; i < hw * nr; i += blockDim.x) {
        const int a = i / nr, r = i - a * nr;
        const dfc* z = Z + (r >> 1) * W;
        const dfc za = z[a], zb = z[a == 0 ? 0 : W - a];
        dfc g;
        if ((r & 1) == 0) { // conj of X0 = (Z(a) + conj Z(-a)) / 2
            df_add_lazy(za.h.x, za.l.x, zb.h.x, zb.l.x, g.h.x, g.l.x);
            df_add_lazy(zb.h.y, zb.l.y, -za.h.y, -za.l.y, g.h.y, g.l.y);
        } else { // conj of X1 = (Z(a) - conj Z(-a)) / 2i
            df_add_lazy(za.h.y, za.l.y, zb.h.y, zb.l.y, g.h.x, g.l.x);
            df_add_lazy(za.h.x, za.l.x, -zb.h.x, -zb.l.x, g.h.y, g.l.y);
        }
        g.h.x *= 0.5f; g.l.x *= 0.5f; g.h.y *= 0.5f; g.l.y *= 0.5f;
        out[(long long)a * H + y0 + r] = g;
    }
    // (here: before the transform it costs spills, 110 us at 200 frames of 640 x 480)
    sq_store_block(sqpart, rowsq + (long long)f * gridDim.x + blockIdx.x);
}

// ------------------------------------------------------------- column pass
// One CTA per (a, chunk of frames), cl columns at a time: float-float forward
// transform along y gives F(-a, y); writes S[f][a][c] = F(-a, c - H/2) (row
// pitch Hs, rounded to FP32), the power partials |F|^2 summed in float-float
// in frame order, and the FP32 inverse y-transform of conj(R) * F into T.
// first: frame 0 is the reference, whose column every CTA transforms first
// (k_fft.cu).
__global__ void __launch_bounds__(256, 4) gen_col_kernel(const dfc* __restrict__ Gt, float2* __restrict__ S,
                                                      int Hs, float2* __restrict__ Rbuf,
                                                      float2* __restrict__ T, double* __restrict__ Ppart, int nframes,
                                                      int fpc, int first, int hw, int cl, const GenPlan ph,
                                                      const dfc* __restrict__ twd_g, const float2* __restrict__ tw_g)
{
    extern __shared__ dfc smg[];
    const int H = ph.L;
    dfc* twd = smg;                                                // [H]
    dfc* X = twd + H;                                              // [cl][H]
    dfc* Y = X + cl * H;                                           // [cl][H]
    float2* tw = reinterpret_cast<float2*>(Y + cl * H);            // [H]
    float2* R = tw + H;                                            // [H]
    float2* pacc = R + H;                                          // [H] float-float (hi, lo)
    const int a = blockIdx.x;
    const int chunk = blockIdx.y;
    const int fbeg = chunk * fpc;
    const int fend = min(nframes, fbeg + fpc);
    const long long gstride = (long long)hw * H;
    const long long sstride = (long long)hw * Hs;
    const int hh = H / 2;
    load_table(twd, twd_g, H);
    load_table(tw, tw_g, H);
    for (int y = threadIdx.x; y < H; y += blockDim.x) {
        if (first != 1)
            R[y] = Rbuf[(long long)a * H + y];
        pacc[y] = make_float2(0.f, 0.f);
    }
    if (first == 1) {
        for (int y = threadIdx.x; y < H; y += blockDim.x)
            X[y] = Gt[(long long)a * H + y];
        __syncthreads();
        const dfc* Fr = stockham(X, Y, ph, 1, H, twd, -1);
        for (int y = threadIdx.x; y < H; y += blockDim.x) {
            R[y] = dfc_round(Fr[y]);
            if (chunk == 0)
                Rbuf[(long long)a * H + y] = R[y];
        }
    }
    for (int f0 = fbeg; f0 < fend; f0 += cl) {
        const int nl = min(cl, fend - f0);
        __syncthreads();
        for (int i = threadIdx.x; i < nl * H; i += blockDim.x) {
            const int l = i / H, y = i - l * H;
            X[i] = Gt[(f0 + l) * gstride + (long long)a * H + y];
        }
        __syncthreads();
        dfc* Fm = stockham(X, Y, ph, nl, H, twd, -1); // Fm[l][y] = F(-a, y)
        // the FP32 transform's buffers: the other one, then Fm's own
        float2* X2 = reinterpret_cast<float2*>(Fm == X ? Y : X);
        float2* Y2 = reinterpret_cast<float2*>(Fm);
        for (int i = threadIdx.x; i < nl * H; i += blockDim.x) {
            const int l = i / H, c = i - l * H;
            int y = c - hh;
            y += y < 0 ? H : 0;
            S[(f0 + l) * sstride + (long long)a * Hs + c] = dfc_round(Fm[l * H + y]);
        }
        // power spectrum, frames in order per element, float-float sums
        for (int c = threadIdx.x; c < H; c += blockDim.x) {
            int y = c - hh;
            y += y < 0 ? H : 0;
            float ah = pacc[c].x, al = pacc[c].y;
            for (int l = 0; l < nl; ++l) {
                dfc v = Fm[l * H + y];
                df_norm(v.h.x, v.l.x); // the butterflies leave lazy pairs
                df_norm(v.h.y, v.l.y);
                float rh, rl, ih, il, sh, sl;
                df_mul(v.h.x, v.l.x, v.h.x, v.l.x, rh, rl);
                df_mul(v.h.y, v.l.y, v.h.y, v.l.y, ih, il);
                df_add(rh, rl, ih, il, sh, sl);
                df_add(ah, al, sh, sl, ah, al);
            }
            pacc[c] = make_float2(ah, al);
        }
        // correlation product conj(R) * F in FP32, inverse y-transform
        for (int i = threadIdx.x; i < nl * H; i += blockDim.x) {
            const int y = i % H;
            const float2 r = R[y], v = dfc_round(Fm[i]);
            X2[i] = make_float2(r.x * v.x + r.y * v.y, r.x * v.y - r.y * v.x);
        }
        __syncthreads();
        const float2* Tz = stockham(X2, Y2, ph, nl, H, tw, +1);
        for (int i = threadIdx.x; i < nl * H; i += blockDim.x) {
            const int l = i / H, y = i - l * H;
            if (first && f0 + l == 0)
                continue;
            T[(f0 + l) * gstride + (long long)a * H + y] = Tz[i];
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < H; c += blockDim.x)
        Ppart[(long long)chunk * gstride + (long long)a * H + c] = (double)pacc[c].x + (double)pacc[c].y;
}

// ------------------------------------------------------- correlation rows
// c2r along x of T(-a, y), two rows per complex transform (z0 + i z1): Z(0) =
// Re T(0); Z(k) = conj T(a = k) for 0 < k < W/2; Re T(W/2) at the Nyquist
// column of an even W (FFTW's c2r ignores those imaginary parts); Z(k) =
// T(a = W - k) above.  Output: the correlation c[y][x] and each row's maximum.
// rb rows (an even number) per CTA; T is read with the rows fastest.
__global__ void __launch_bounds__(256) gen_xrows_kernel(const float2* __restrict__ Tg, float* __restrict__ corr,
                                                        float* __restrict__ rowmax, int H, int hw, int rb,
                                                        const GenPlan pw, const float2* __restrict__ tw_g)
{
    extern __shared__ float2 smx[];
    const int W = pw.L;
    float2* tw = smx;
    float2* X = tw + W;
    float2* Y = X + rb / 2 * W;
    const int f = blockIdx.y;
    const int y0 = blockIdx.x * rb;
    const int nr = min(rb, H - y0), nl = (nr + 1) / 2;
    const float2* T = Tg + (long long)f * hw * H;
    load_table(tw, tw_g, W);
    for (int i = threadIdx.x; i < nl * hw; i += blockDim.x) { // one a of two rows: the elements k = a and W - a
        const int a = i / nl, l = i - a * nl;
        const float2 z0 = T[(long long)a * H + y0 + 2 * l];
        const float2 z1 = 2 * l + 1 < nr ? T[(long long)a * H + y0 + 2 * l + 1] : make_float2(0.f, 0.f);
        float2* x = X + l * W;
        if (a == 0 || 2 * a == W) {
            x[a] = make_float2(z0.x, z1.x);
        } else {
            x[a] = make_float2(z0.x + z1.y, z1.x - z0.y);     // conj z0 + i conj z1
            x[W - a] = make_float2(z0.x - z1.y, z1.x + z0.y); // z0 + i z1
        }
    }
    __syncthreads();
    const float2* Z = stockham(X, Y, pw, nl, W, tw, +1);
    float* out = corr + (long long)f * W * H + (long long)y0 * W;
    // each row, and its maximum: one warp per two rows
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int l = warp; l < nl; l += blockDim.x >> 5) {
        float m0 = -INFINITY, m1 = -INFINITY;
        const bool two = 2 * l + 1 < nr;
        for (int x = lane; x < W; x += 32) {
            const float2 v = Z[l * W + x];
            out[2 * l * W + x] = v.x;
            m0 = fmaxf(m0, v.x);
            if (two) {
                out[(2 * l + 1) * W + x] = v.y;
                m1 = fmaxf(m1, v.y);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
            m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
        }
        if (lane == 0) {
            rowmax[(long long)f * H + y0 + 2 * l] = m0;
            if (two)
                rowmax[(long long)f * H + y0 + 2 * l + 1] = m1;
        }
    }
}

// -------------------------------------------------------------- FP64 lines
// nlb lines per CTA of length p.L (element stride es, line stride ls), in place.
__global__ void __launch_bounds__(256) gen_lines_d_kernel(double2* __restrict__ data, int nlines, long long ls,
                                                          long long es, int sign, int nlb, const GenPlan p,
                                                          const double2* __restrict__ tw_g)
{
    extern __shared__ double2 smd2[];
    const int L = p.L;
    double2* tw = smd2;
    double2* X = tw + L;
    double2* Y = X + nlb * L;
    const int l0 = blockIdx.x * nlb;
    const int nl = min(nlb, nlines - l0);
    load_table(tw, tw_g, L);
    for (int i = threadIdx.x; i < nl * L; i += blockDim.x) {
        const int l = i / L, k = i - l * L;
        X[i] = data[(l0 + l) * ls + k * es];
    }
    __syncthreads();
    const double2* Z = stockham(X, Y, p, nl, L, tw, sign);
    for (int i = threadIdx.x; i < nl * L; i += blockDim.x) {
        const int l = i / L, k = i - l * L;
        data[(l0 + l) * ls + k * es] = Z[i];
    }
}

// ------------------------------------------------------------- launchers
// Blocking per launch, chosen so that a CTA's shared memory stays below
// kGenSmem for every length up to kMaxSide.
constexpr size_t kGenSmem = 200 * 1024;
// Lines per CTA: as many as fit in about 64 KB of shared memory, so that
// several CTAs share an SM and hide each other's shared-memory latency
// (48 KB: rows 1272 us, columns 1879; 96 KB: 800 and 1234, correlation rows 396
// instead of 294; all without the bound on registers).
constexpr long kGenTarget = 64 * 1024;

static int row_block(int W) { return 2 * (int)std::max(1L, std::min(8L, (kGenTarget / (16L * W) - 1) / 2)); }
static size_t row_smem(int W, int rb) { return sizeof(dfc) * (size_t)W * (1 + rb); }
static int col_lines(int H)
{
    const long per = (long)H * 2 * sizeof(dfc); // one more column
    const long fixed = (long)H * (sizeof(dfc) + 3 * sizeof(float2));
    return (int)std::max(1L, std::min(8L, (kGenTarget - fixed) / per));
}
static size_t col_smem(int H, int cl)
{
    return (size_t)H * (sizeof(dfc) * (1 + 2 * cl) + sizeof(float2) * 3);
}
static int xrow_block(int W) { return 2 * (int)std::max(1L, std::min(8L, (kGenTarget / (8L * W) - 1) / 2)); }
static size_t xrow_smem(int W, int rb) { return sizeof(float2) * (size_t)W * (1 + rb); }
static int lines_block(int L) { return (int)std::max(1L, std::min(8L, (kGenTarget / (16L * L) - 1) / 2)); }
static size_t lines_smem(int L, int nlb) { return sizeof(double2) * (size_t)L * (1 + 2 * nlb); }

template <typename K> static cudaError_t allow(K kern, size_t bytes)
{
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

size_t gen_max_smem() { return kGenSmem; }
int gen_row_blocks(const Geometry& g) { return (g.H + row_block(g.W) - 1) / row_block(g.W); }

cudaError_t launch_gen_row_pass(int dtype, const void* frames, long long fstride, int nframes, const Geometry& g,
                                dfc* Gt, void* rowsq, const dfc* twW, cudaStream_t st, void* copy_out)
{
    const int rb = row_block(g.W);
    const dim3 grid((g.H + rb - 1) / rb, nframes);
    const size_t smem = row_smem(g.W, rb);
    cudaError_t e = cudaSuccess;
#define SMIP_GEN_ROW(TY)                                                                                          \
    if ((e = allow(gen_row_kernel<TY>, kGenSmem)) != cudaSuccess)                                                 \
        return e;                                                                                                  \
    gen_row_kernel<TY><<<grid, 256, smem, st>>>((const TY*)frames, fstride, g.H, g.hw, rb, g.pW, twW, Gt,         \
                                                (TY*)copy_out, (SqSum<TY>*)rowsq);
    switch (dtype) {
    case 0: SMIP_GEN_ROW(uint8_t) break;
    case 1: SMIP_GEN_ROW(uint16_t) break;
    case 2: SMIP_GEN_ROW(float) break;
    default: SMIP_GEN_ROW(double) break;
    }
#undef SMIP_GEN_ROW
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_gen_col_pass(const dfc* Gt, float2* S, float2* Rbuf, float2* T, double* Ppart, int nframes, int fpc,
                                int first, const Geometry& g, const dfc* twH, const float2* twH32, cudaStream_t st)
{
    const int cl = col_lines(g.H);
    const dim3 grid(g.hw, (nframes + fpc - 1) / fpc);
    cudaError_t e = allow(gen_col_kernel, kGenSmem);
    if (e != cudaSuccess)
        return e;
    gen_col_kernel<<<grid, 256, col_smem(g.H, cl), st>>>(Gt, S, g.Hs, Rbuf, T, Ppart, nframes, fpc, first, g.hw, cl,
                                                         g.pH, twH, twH32);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_gen_xcorr_rows(const float2* T, float* corr, float* rowmax, int nframes, const Geometry& g,
                                  const float2* twW32, cudaStream_t st)
{
    const int rb = xrow_block(g.W);
    const dim3 grid((g.H + rb - 1) / rb, nframes);
    cudaError_t e = allow(gen_xrows_kernel, kGenSmem);
    if (e != cudaSuccess)
        return e;
    gen_xrows_kernel<<<grid, 256, xrow_smem(g.W, rb), st>>>(T, corr, rowmax, g.H, g.hw, rb, g.pW, twW32);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_gen_lines_d(double2* data, const GenPlan& p, int nlines, long long ls, long long es, int sign,
                               const double2* tw, cudaStream_t st)
{
    const int nlb = lines_block(p.L);
    cudaError_t e = allow(gen_lines_d_kernel, kGenSmem);
    if (e != cudaSuccess)
        return e;
    gen_lines_d_kernel<<<(nlines + nlb - 1) / nlb, 256, lines_smem(p.L, nlb), st>>>(data, nlines, ls, es, sign, nlb,
                                                                                    p, tw);
    note_launches(1);
    return cudaGetLastError();
}

// Factors of L for the Stockham passes: the odd primes in increasing order,
// then the twos as 4s (so that none is left alone, unless there is only one)
// and 8s.
GenPlan make_gen_plan(int L)
{
    GenPlan p {};
    p.L = L;
    int n = L, twos = 0;
    while (n % 2 == 0) {
        n /= 2;
        ++twos;
    }
    for (int q = 3; q <= n; q += 2)
        while (n % q == 0) {
            p.fac[p.nf++] = q;
            n /= q;
        }
    if (twos == 1) {
        p.fac[p.nf++] = 2;
        twos = 0;
    }
    for (; twos % 3 != 0; twos -= 2)
        p.fac[p.nf++] = 4;
    for (; twos > 0; twos -= 3)
        p.fac[p.nf++] = 8;
    return p;
}

} // namespace smip_gpu
