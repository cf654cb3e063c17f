// k_reco.cu -- closure-phase recovery.
//
// Replaces reconstruct_phases / calc_phase (include/phasereco.h:33-123).  The
// reference walks the spiral of NextRecoIndex (src/phasereco.cpp:17-36) and,
// for every unflagged point w, averages the unit phasors
//     phi(u) phi(v) conj(B(u,v) / |B(u,v)|)    over u + v = w,
// u and v flagged, |B| > DBL_EPSILON, v inside the bispectrum's v range.
// Each point may use phases set earlier in the same ring, so the walk is a
// serial chain.  Most of a point's pairs, though, read phases that were final
// long before: a pair is "recent" only when u or v was visited within the
// kRecoLag visits before w (the arc of the ring just behind w; at most 64
// pairs, a fact of the lag).  Which pairs are recent depends only on the visit
// list, so spiral_plan_kernel lists them ahead of the walk with everything
// else that does not depend on the chain; phase_walk_kernel is the walk.
//
// Precision: per-pair products in FP32 from an FP32 mirror of the phase map
// (~1e-7 rad per pair); the non-recent share is summed in FP32 per lane and in
// float-float over the lanes, and the recent pairs are added to it in
// float-float, because at low-consistency points the mean phasor is a large
// cancellation; the mean, |mean| (consistency) and the stored phase are FP64.
// B is read through a device replica of Bispectrum::get_element's index
// arithmetic, aliasing included.
#include <type_traits>

#include "smip_dev.cuh"

namespace smip_gpu {

constexpr int kRecoThreads = 512;
constexpr int kMaxWords = (65 * 65 + 31) / 32; // words of a pair-slot mask at the largest depth

__device__ __forceinline__ int wrap_idx(int x, int y, int W, int H)
{
    return (x < 0 ? x + W : x) + (y < 0 ? y + H : y) * W;
}

// Unit phasor of B in FP32 without overflow (scale by a power of two), and
// the reference's test |B| > DBL_EPSILON = 2^-52 (phasereco.h:100) decided
// from the binary exponent, without FP64 arithmetic.
__device__ __forceinline__ bool unit_phasor(float2 b, float2* out)
{
    const float m = fmaxf(fabsf(b.x), fabsf(b.y));
    if (!(m > 0.f))
        return false;
    int e;
    frexpf(m, &e); // m = f * 2^e, f in [0.5, 1)
    const float sx = ldexpf(b.x, -e), sy = ldexpf(b.y, -e);
    const float n2 = sx * sx + sy * sy; // |B|^2 / 4^e, in [0.25, 2)
    // |B| = 2^e sqrt(n2) with sqrt(n2) in [0.5, sqrt 2)
    if (e <= -53)
        return false;
    if (e == -52 && !(n2 > 1.f))
        return false;
    const float r = rsqrtf(n2);
    *out = make_float2(sx * r, sy * r);
    return true;
}

// float-float accumulation (Knuth two-sum).  The _rn intrinsics are never
// contracted with a product the caller passes in.
__device__ __forceinline__ void ff_add(float& hi, float& lo, float bh, float bl)
{
    const float s = __fadd_rn(hi, bh);
    const float bb = __fsub_rn(s, hi);
    float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(bh, bb));
    e = __fadd_rn(e, __fadd_rn(lo, bl));
    hi = __fadd_rn(s, e);
    lo = __fsub_rn(e, __fsub_rn(hi, s));
}

// phi(u) phi(v) conj(b), every rounding spelt out: a visit's terms are formed in
// several places, and the compiler may contract the same expression differently
// in each.
__device__ __forceinline__ float2 pair_product(float2 u, float2 v, float bx, float by)
{
    const float2 m = make_float2(__fmaf_rn(u.x, v.x, -__fmul_rn(u.y, v.y)), __fmaf_rn(u.y, v.x, __fmul_rn(u.x, v.y)));
    return make_float2(__fmaf_rn(m.x, bx, __fmul_rn(m.y, by)), __fmaf_rn(m.y, bx, -__fmul_rn(m.x, by)));
}
// For normal arguments, 0 and NaN: rsqrtf without its scaling of subnormals.
__device__ __forceinline__ float rsqrt_ftz(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float norm2(float2 p) { return __fmaf_rn(p.x, p.x, __fmul_rn(p.y, p.y)); }

// ----------------------------------------------------------------- plan
// The bispectrum side of every pair the walk can use depends only on (w, v),
// not on the chain: plan[q][t] = unit phasor of B(w_q - v_t, v_t), or
// (0, 0) when the pair never contributes (u outside the map, |B| <= eps,
// w skipped by calc_phase), or NaN where Bispectrum::get_element would throw.
// Fully parallel over (visit, v).  (The ring-parallel estimator's; the spiral
// walk's plan, with its recent pairs taken out, is spiral_plan_kernel's.)
__global__ void __launch_bounds__(256) reco_plan_kernel(const RecoJob* __restrict__ jobs)
{
    const RecoJob J = jobs[blockIdx.y];
    const int W = J.W, H = J.H, De = J.De;
    const int nside = De + 1, nv = nside * nside;
    BispecDims d;
    const int szW = (W / 2) * 2 + 1, szH = (H / 2) * 2 + 1, szD = De + 1;
    d.sizes[0] = szW; d.sizes[1] = szH; d.sizes[2] = szD; d.sizes[3] = szD;
    d.base[0] = szW - szW / 2; d.base[1] = szH; d.base[2] = szD - szD / 2; d.base[3] = szD;
    for (int n = 0; n < 4; ++n) {
        d.mn[n] = -(d.sizes[n] / 2);
        d.mx[n] = d.sizes[n] + d.mn[n] - 1;
    }
    d.base_size = (long long)d.base[0] * d.base[1] * d.base[2] * d.base[3];
    const int pmin0 = -(W >> 1), pmin1 = -(H >> 1);
    const int pmax0 = -W / 2 + W - 1, pmax1 = -H / 2 + H - 1;
    const long long total = (long long)J.nvisits * nv;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int q = (int)(e / nv), t = (int)(e - (long long)q * nv);
        const int2 w = J.visits[q];
        float2 out = make_float2(0.f, 0.f);
        const bool wok = !(w.x < pmin0 || w.x > pmax0 || w.y < pmin1 || w.y > pmax1) && (abs(w.x) + abs(w.y) > 1)
                         && !(w.x < d.mn[0] || w.x > d.mx[0] || w.y < d.mn[1] || w.y > d.mx[1]);
        if (wok) {
            const int vx = -De / 2 + t % nside, vy = -De / 2 + t / nside;
            const int ux = w.x - vx, uy = w.y - vy;
            if (!(ux < pmin0 || ux > pmax0 || uy < pmin1 || uy > pmax1)) {
                int cj = 0;
                const long long off = bispec_get_offset(d, ux, uy, vx, vy, &cj);
                if (off < 0) {
                    out = make_float2(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
                } else {
                    float2 b = __ldg(&J.B[off]);
                    if (cj)
                        b.y = -b.y;
                    float2 bh;
                    if (unit_phasor(b, &bh))
                        out = bh;
                }
            }
        }
        J.plan[e] = out;
    }
}

// ----------------------------------------------------------- the spiral
// The walk's inputs that do not depend on the chain, one warp per visit q:
//   plan[q][t]: the unit phasor of B(w - v_t, v_t) of every non-recent pair,
//     or NaN for a pair that the sum leaves out (u outside the map, |B| <= eps,
//     a recent pair), so that one test of the product tells a usable pair;
//   rec[q][64]: the recent pairs in increasing slot order (at most 32 by u and
//     32 by v): phasor, slot and the ages ku, kv (q - the last visit of u, v
//     within the lag; 0: none);
//   meta[q]: the point's place in the padded map (-1: outside), its FFT-order
//     index, the number of recent pairs, the age of the point's own last visit
//     within the lag, and its slot when it lies in the v box.
// A visit with at most 32 recent pairs of which at most one has age 1 is
// "fast": its list is stored permuted by XOR with that pair's position, which
// puts the pair into lane 0 and leaves the order of a butterfly sum as it is.
// A phasor whose real part is NaN (Bispectrum::get_element would throw, or B is
// not a number) has the payload kOorBits; one whose imaginary part alone is NaN
// (that of B is infinite) has kNanBits: its pair counts and makes the point's sum
// NaN.  Both raise J.oor, which has the walk look for them.
// Bound by the scattered reads of B (one 32-byte sector per pair): 64 M pairs
// at 256 x 256, d = 32.
constexpr unsigned kUnusable = 0x7fc00000u;
constexpr unsigned kOorBits = 0x7fc00001u;
constexpr unsigned kNanBits = 0x7fc00002u;
constexpr int kPlanWarps = 8;

// rec code: slot t (13 bits) | ku << 13 | kv << 19
// meta.z: recent pairs | kc << 8 | fast << 16 | runnable << 17
__global__ void __launch_bounds__(32 * kPlanWarps) spiral_plan_kernel(const RecoJob* __restrict__ jobs)
{
    extern __shared__ int slot_xy[]; // [nwords * 32] vx | vy << 16
    __shared__ unsigned mask_s[kPlanWarps][kMaxWords];
    __shared__ unsigned short list_s[kPlanWarps][kRecentMax];
    __shared__ unsigned code_s[kPlanWarps][kRecentMax];
    const RecoJob J = jobs[blockIdx.y];
    const int W = J.W, H = J.H, De = J.De, e = De / 2;
    const int nside = De + 1, nv = nside * nside, nwords = (nv + 31) / 32, row = nwords * 32;
    for (int t = threadIdx.x; t < row; t += blockDim.x) {
        const int vx = -e + t % nside, vy = -e + t / nside;
        slot_xy[t] = (int)(((unsigned)vx & 0xffffu) | ((unsigned)vy << 16));
    }
    __syncthreads();
    BispecDims d;
    const int szW = (W / 2) * 2 + 1, szH = (H / 2) * 2 + 1, szD = De + 1;
    d.sizes[0] = szW; d.sizes[1] = szH; d.sizes[2] = szD; d.sizes[3] = szD;
    d.base[0] = szW - szW / 2; d.base[1] = szH; d.base[2] = szD - szD / 2; d.base[3] = szD;
    for (int n = 0; n < 4; ++n) {
        d.mn[n] = -(d.sizes[n] / 2);
        d.mx[n] = d.sizes[n] + d.mn[n] - 1;
    }
    d.base_size = (long long)d.base[0] * d.base[1] * d.base[2] * d.base[3];
    const int pmin0 = -(W >> 1), pmin1 = -(H >> 1);
    const int pmax0 = -W / 2 + W - 1, pmax1 = -H / 2 + H - 1;
    auto in_map = [&](int x, int y) { return x >= pmin0 && x <= pmax0 && y >= pmin1 && y <= pmax1; };
    auto pack = [](int x, int y) { return (int)(((unsigned)x & 0xffffu) | ((unsigned)y << 16)); };
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned* mask = mask_s[warp];
    unsigned short* list = list_s[warp];
    unsigned* code = code_s[warp];
    const float2 nan2 = make_float2(__uint_as_float(kUnusable), __uint_as_float(kUnusable));
    for (int q = blockIdx.x * kPlanWarps + warp; q < J.nvisits; q += gridDim.x * kPlanWarps) {
        const int2 w = J.visits[q];
        if (!in_map(w.x, w.y)) {
            if (lane == 0)
                J.meta[q] = make_int4(-1, 0, 0, -1);
            continue;
        }
        // lane j: the visit of age j + 1
        const int pq = q - 1 - lane;
        int2 pj = make_int2(0, 0);
        if (pq >= 0)
            pj = J.visits[pq];
        const bool inj = pq >= 0 && in_map(pj.x, pj.y);
        const int pkj = inj ? pack(pj.x, pj.y) : (int)0x80008000; // not a point of any map
        for (int i = lane; i < nwords; i += 32)
            mask[i] = 0u;
        __syncwarp();
        if (inj) {
            const int ux = w.x - pj.x, uy = w.y - pj.y; // the pair's other member
            if (abs(pj.x) <= e && abs(pj.y) <= e && in_map(ux, uy)) { // v = pj
                const int t = (pj.y + e) * nside + pj.x + e;
                atomicOr(&mask[t >> 5], 1u << (t & 31));
            }
            if (abs(ux) <= e && abs(uy) <= e) { // u = pj
                const int t = (uy + e) * nside + ux + e;
                atomicOr(&mask[t >> 5], 1u << (t & 31));
            }
        }
        __syncwarp();
        int rc = 0;
        for (int w0 = 0; w0 < nwords; w0 += 32) {
            const unsigned bits = w0 + lane < nwords ? mask[w0 + lane] : 0u;
            if (!__any_sync(0xffffffffu, bits != 0u))
                continue;
            const int c = __popc(bits);
            int incl = c; // inclusive prefix over the lanes
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o)
                    incl += y;
            }
            int pos = rc + incl - c;
            for (unsigned b = bits; b; b &= b - 1)
                list[pos++] = (unsigned short)((w0 + lane) * 32 + __ffs(b) - 1);
            rc += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
        const int ta = lane < rc ? list[lane] : 0, tb = lane + 32 < rc ? list[lane + 32] : 0;
        const int va = slot_xy[ta], vb = slot_xy[tb];
        const int ua = pack(w.x - (short)va, w.y - (va >> 16)), ub = pack(w.x - (short)vb, w.y - (vb >> 16));
        int kua = 0, kva = 0, kub = 0, kvb = 0;
        for (int k = 32; k >= 1; --k) { // the smallest age is kept
            const int p = __shfl_sync(0xffffffffu, pkj, k - 1);
            kua = p == ua ? k : kua;
            kva = p == va ? k : kva;
            kub = p == ub ? k : kub;
            kvb = p == vb ? k : kvb;
        }
        const unsigned late_a = __ballot_sync(0xffffffffu, lane < rc && (kua == 1 || kva == 1));
        const unsigned late_b = __ballot_sync(0xffffffffu, lane + 32 < rc && (kub == 1 || kvb == 1));
        const unsigned own = __ballot_sync(0xffffffffu, pkj == pack(w.x, w.y));
        const int kc = own ? __ffs(own) : 0;
        const bool fast = rc <= 32 && __popc(late_a) + __popc(late_b) <= 1 && kc == 0;
        const int perm = fast && late_a ? __ffs(late_a) - 1 : 0;
        const bool run = abs(w.x) + abs(w.y) > 1; // phasereco.h:84
        if (lane < rc)
            code[lane] = (unsigned)(ta | kua << 13 | kva << 19);
        if (lane + 32 < rc)
            code[lane + 32] = (unsigned)(tb | kub << 13 | kvb << 19);
        if (lane == 0) {
            const int bx = w.x - pmin0 + e, by = w.y - pmin1 + e;
            const int vs = abs(w.x) <= e && abs(w.y) <= e ? (w.y + e) * nside + w.x + e : -1;
            J.meta[q] = make_int4(by * (W + De) + bx, wrap_idx(w.x, w.y, W, H),
                                  rc | kc << 8 | (fast ? 1 << 16 : 0) | (run ? 1 << 17 : 0), vs);
        }
        __syncwarp();
        if (!run)
            continue;
        uint4* rec = J.rec + (long long)q * kRecentMax;
        const uint4 none = make_uint4(kUnusable, kUnusable, 0u, 0u);
        if (lane >= rc)
            rec[lane ^ perm] = none;
        if (rc > 32 && lane + 32 >= rc)
            rec[lane + 32] = none;
        float2* prow = J.plan + (long long)q * row;
        int before = 0; // recent pairs in the words before word i
        bool oor = false;
        for (int i = 0; i < nwords; ++i) {
            const int t = lane + 32 * i;
            float2 out = nan2;
            if (t < nv) {
                const int xy = slot_xy[t];
                const int vx = (short)xy, vy = xy >> 16;
                const int ux = w.x - vx, uy = w.y - vy;
                if (in_map(ux, uy)) {
                    int cj = 0;
                    const long long off = bispec_get_offset(d, ux, uy, vx, vy, &cj);
                    unsigned bad = off < 0 ? kOorBits : 0u;
                    if (!bad) {
                        float2 b = __ldg(&J.B[off]);
                        if (cj)
                            b.y = -b.y;
                        float2 bh;
                        if (unit_phasor(b, &bh)) {
                            bad = isnan(bh.x) ? kOorBits : isnan(bh.y) ? kNanBits : 0u;
                            out = bh;
                        }
                    }
                    if (bad) {
                        out = make_float2(__uint_as_float(bad), __uint_as_float(bad));
                        oor = true;
                    }
                }
            }
            const unsigned bits = mask[i];
            if ((bits >> lane) & 1u) {
                const int pos = before + __popc(bits & ((1u << lane) - 1u));
                rec[pos ^ perm] = make_uint4(__float_as_uint(out.x), __float_as_uint(out.y), code[pos], 0u);
                out = nan2;
            }
            before += __popc(bits);
            prow[t] = out;
        }
        if (oor)
            atomicOr(J.oor, 1);
        __syncwarp();
    }
}

// The walk: one cluster of CTAs per job (or one CTA, where the caller asks for it
// or the GPU places no cluster).
//   warp 0 of rank 0 (the serial warp) runs the visits in order;
//   the writer, on another sub-partition, copies what the serial warp found
//     into the phase map in global memory and publishes the progress, first to
//     its own CTA, whose warps need no release at cluster scope;
//   loading warps bring visit q's recent pairs into slot q mod kRing of rank 0
//     once the progress has reached q - kRecoLag, with the members that lie
//     outside the lag;
//   summing warps form the share of the non-recent pairs, at the same progress,
//     and post it to that slot (st.async, whose completion the slot's mbarrier
//     counts: a plain store and a release at cluster scope held the summing warp
//     for 2,200 cycles a visit);
//   gathering warps wait for both, add a visit's parts and set the tag that the
//     serial warp looks at.
// In a cluster rank 0 sums nothing; in a lone CTA the summing warps are those
// of the other three SM sub-partitions, so that the serial warp keeps the
// issue slots of its own.
//
// What a visit must wait for is the phase of the visit just before it.  The
// serial warp therefore does everything else of visit q + 1 while the chain of
// visit q runs: the terms of the pairs of age >= 2, and their butterfly sum
// over the lanes (real parts in the lower half warp, imaginary parts in the
// upper, after its first level), of which lanes 0 and 16 keep the sibling sums
// that they receive.  Every lane forms the first pair's term, the only one of
// age 1: that, five additions of the sibling sums (bit for bit the butterfly's
// result), the float-float addition to the share, one exchange between lanes 0
// and 16 and the phase are the chain.  Visits that are "wide" (two pairs of age
// 1, more than 32 recent pairs, or a point visited within the lag: near the
// origin, 2 % of the visits at 256 x 256) form their sum at once, as 32 or 64
// terms.
//
// A share waits for its u's, which come from L2 (the other SMs write them).  The
// plan row of a visit does not depend on the chain: a bulk copy brings it into
// the summing CTA's shared memory before the visit may be summed, so that up to
// 20 gathers a lane are in flight with 2 registers each (10 with the row's
// elements in registers beside them: 1,800 cycles a batch; now 3,300 for 19 or 20
// words).
//
// The phase map is kept centred with De / 2 points of padding and holds NaN
// where there is no phase, so that a pair's u is one address and needs no
// bounds or flag test: a product with an unflagged or outside point is NaN.
// Every wait is bounded; on a timeout the walk stops and the error is recorded.
//
// Bound by the serial warp, which waits for instructions as much as for the
// chain (200 cycles): a visit takes 458 / 442 / 428 cycles at depths 24 / 32 / 48
// (495 / 472 / 465 with the recent pairs loaded by the summing warps, the whole
// butterfly in one step and addresses formed in the loop; 2,000 with everything
// in the serial warp).  128 x 128, d = 24, R = 48 in 2.04 ms (2.34, 7.8), 256 x
// 256, d = 32, R = 128 in 13.7 (15.3, 58.2), 512 x 512, d = 48, R = 200 in 34.9
// (41.5, 163), normalisation and plan included.  A sum of the recent pairs by age instead
// of by slot needs no butterfly at all and takes 330 cycles, but rounds
// otherwise: the phases then differ by up to 5e-7.
constexpr int kRing = 64;
constexpr int kMaxParts = 6;
constexpr int kStep = 4;                 // visits between two looks of the serial warp at the other warps
constexpr int kGroups = kRing / kStep;
// Words of a plan row that a summing warp of a cluster keeps in shared memory.  The
// function's limit is one number: the box of the largest depth, 16 warps' rows of
// 40 words and the static arrays take 225,168 of 232,448 bytes; 43 words would not
// fit.  Only depths 36 and 38 have longer parts (43, 48 words in one part; 39 at
// depth 34, 18 in three at 40) and read their rows from global memory: 411 and 420
// ns a visit at 144 x 144, R = 64 (254 at depths 34 and 40).  With rows of 48 words
// and a limit of these depths' own they took 270 and 275 at 128 x 128 (373 and 378
// without).
constexpr int kRowWords = 40;
constexpr unsigned long long kRecoWaitNs = 2000000000ull;
static_assert(kRing > kRecoLag + 8, "ring slots outlive the lag and the serial warp's look-ahead");

// parts per visit share from depth kPartsDepth on: about 16 words of pair
// slots (512 slots) each, so that a visit's sum is short enough for the lag
constexpr int kPartsDepth = 40;
__host__ __device__ __forceinline__ int share_parts(int De, int nwords)
{
    const int p = De < kPartsDepth ? 1 : nwords / 16;
    return p < 1 ? 1 : (p > kMaxParts ? kMaxParts : p);
}

// CTA-scope acquire load / release store on shared memory: they order the
// accesses after (before) them without waiting for this thread's other
// outstanding loads, as a full fence would.
__device__ __forceinline__ void st_release_cta(int* p, int v)
{
    asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_cta(const int* p)
{
    int v;
    asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}
// a plan row is read once: not kept in L1, which holds the phase map
__device__ __forceinline__ float2 ld_stream(const float2* p)
{
    float2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

// Dynamic shared memory, offsets in bytes.  What the serial warp reads and writes
// lies at constant offsets, so that a slot's number is its only address
// arithmetic.  Ranks above 0 keep their plan rows there instead.  v's phase and
// map offset are at the end.
constexpr int kShareAt = 0;                      // float4 [kRing]: sum of the non-recent pairs (re hi, lo, im hi, lo)
constexpr int kCtlAt = kShareAt + 16 * kRing;    // float4 [kRing]: phase the point already has (or NaN), kCtl bits, number of those pairs (far below 0: the point has its phase, or can have none)
constexpr int kSumAt = kCtlAt + 16 * kRing;      // float4 [kRing]: sums of the last visits, for the writer
constexpr int kPhaseAt = kSumAt + 16 * kRing;    // float4 [kRing]: phases of the last visits, pairs of a point that got its phase
constexpr int kHeadAt = kPhaseAt + 16 * kRing;   // float4 [kRing]: the first recent pair: phasor, offsets of u's and v's phase
constexpr int kPairAt = kHeadAt + 16 * kRing;    // float4 [kRing][kRecentMax]: phasor, the member outside the lag
constexpr int kPlaceAt = kPairAt + 16 * kRing * kRecentMax; // uint2 [kRing][kRecentMax]: offsets of u's and v's phase
constexpr int kRingBytes = kPlaceAt + 8 * kRing * kRecentMax;
// kCtl: age of the point's own last visit | two sets of pairs << 8 | the first pair's u, v is the last phase << 9, << 10
__host__ __device__ constexpr size_t box_bytes(int nslots) { return (size_t)nslots * (sizeof(float2) + sizeof(int)); }
// words of a visit's longest part, and whether they fit
__host__ __device__ __forceinline__ int part_words(int De, int nwords) { return (nwords + share_parts(De, nwords) - 1) / share_parts(De, nwords); }
static size_t walk_smem(int De, int nslots, bool multi)
{
    size_t most = (size_t)kRingBytes; // of any depth up to De: the jobs of a launch may differ
    for (int d = 0; multi && d <= De; d += 2) {
        const int pw = part_words(d, ((d + 1) * (d + 1) + 31) / 32);
        const size_t rows = pw <= kRowWords ? (size_t)pw * 256 * (kRecoThreads / 32) : 0;
        most = rows > most ? rows : most;
    }
    return box_bytes(nslots) + most;
}

// CTAs per job: as few as keep the serial warp busy, because jobs that share
// the GPU need the other SMs.  Cycles a visit with 2 / 4 / 8 CTAs: 459 / 456 /
// 455 at depth 24, 528 / 440 / 435 at depth 32; with 4 / 8: 479 / 428 at depth 48.
// (A lone CTA, asked for or where no cluster can be placed: 1,108 and 1,240 at
// depths 24 and 32, the whole call.)
static int walk_ctas(int De) { return De < 28 ? 2 : (De < kPartsDepth ? 4 : 8); }

template <bool MULTI> // a cluster of CTAs per job, or one CTA
__global__ void __launch_bounds__(kRecoThreads, 1) phase_walk_kernel(const RecoJob* __restrict__ jobs)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ float4 shr[kMaxParts][kRing];     // a part's sum over the non-recent pairs: re hi, lo, im hi, lo
    __shared__ int shn[kMaxParts][kRing];        // its number of pairs
    __shared__ float4 shc[kRing];                // number of pairs of part 0, the phase that the point already has
    __shared__ int tag_s[kMaxParts][kRing];      // visit + 1 whose part has landed (lone CTA)
    __shared__ int gtag[kRing];                  // 2 (visit + 1) + wide: the visit is ready for the serial warp
    __shared__ int lhead[kRing];                 // kCtl bits of the visit's first pair
    __shared__ int ltag[kRing];                  // visit + 1 whose recent pairs have been loaded
    __shared__ __align__(8) uint64_t row_bar[kRecoThreads / 32]; // a summing warp's plan row has arrived
    __shared__ __align__(8) uint64_t ring_bar[kRing];   // cluster: visit q's parts have landed in slot q mod kRing
    __shared__ __align__(8) uint64_t done_bar[kGroups]; // the serial warp has finished kStep more visits
    __shared__ int progress;   // visits whose phases are published (a copy in every CTA)
    __shared__ int abort_walk;
    const uint32_t rank = MULTI ? cluster_rank() : 0u, ncta = MULTI ? cluster_size() : 1u;
    const RecoJob J = jobs[blockIdx.x / ncta];
    const int W = J.W, H = J.H, De = J.De, e = De / 2;
    const int nside = De + 1, nv = nside * nside, nwords = (nv + 31) / 32, nslots = nwords * 32;
    const int nparts = share_parts(De, nwords);
    const int PW = W + De;
    unsigned box_at; // the same in every CTA of the cluster
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(box_at));
    box_at -= (unsigned)box_bytes(nslots);
    float2* vt = reinterpret_cast<float2*>(smraw + box_at); // [nslots] phase of v
    int* voff = reinterpret_cast<int*>(vt + nslots);        // [nslots] map offset of v
    float2* rows = reinterpret_cast<float2*>(smraw);        // ranks above 0: a plan row per warp
    float4* share = reinterpret_cast<float4*>(smraw + kShareAt);
    float4* ctl = reinterpret_cast<float4*>(smraw + kCtlAt);
    float4* res_s = reinterpret_cast<float4*>(smraw + kSumAt);
    float4* res_p = reinterpret_cast<float4*>(smraw + kPhaseAt);
    float4* head = reinterpret_cast<float4*>(smraw + kHeadAt);
    float4* ent = reinterpret_cast<float4*>(smraw + kPairAt);
    uint2* place = reinterpret_cast<uint2*>(smraw + kPlaceAt);
    auto phase_at = [&](unsigned off) { return *reinterpret_cast<const float2*>(smraw + off); };
    const float nanf_ = __uint_as_float(kUnusable);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = threadIdx.x; t < nslots; t += blockDim.x) {
        const int vx = -e + t % nside, vy = -e + t / nside;
        float2 v = make_float2(nanf_, nanf_);
        if (t < nv && abs(vx) + abs(vy) <= 1) { // seeds (phasereco.h:42-54)
            v.x = 1.f;
            v.y = vx < 0 || vy < 0 ? -0.f : 0.f;
            if (rank == 0) {
                const int p = wrap_idx(vx, vy, W, H);
                J.pmap[(vy + (H >> 1) + e) * PW + vx + (W >> 1) + e] = make_float2(v.x, v.y);
                J.sums[p] = make_float4(0.f, 0.f, 0.f, 0.f);
                J.cnt[p] = -1;
            }
        }
        vt[t] = v;
        voff[t] = t < nv ? vy * PW + vx : 0;
    }
    for (int i = threadIdx.x; i < kMaxParts * kRing; i += blockDim.x)
        (&tag_s[0][0])[i] = 0;
    for (int i = threadIdx.x; i < kRing; i += blockDim.x)
        ltag[i] = gtag[i] = 0;
    // a slot may be read before anything is posted to it: its offsets are
    // places of phases at all times
    if (rank == 0) {
        for (int i = threadIdx.x; i < kRing * kRecentMax; i += blockDim.x) {
            place[i] = make_uint2(kPhaseAt, kPhaseAt);
            ent[i] = make_float4(nanf_, nanf_, nanf_, nanf_);
        }
        for (int i = threadIdx.x; i < kRing; i += blockDim.x) {
            share[i] = res_s[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            ctl[i] = res_p[i] = make_float4(nanf_, nanf_, 0.f, 0.f);
            head[i] = make_float4(nanf_, nanf_, __uint_as_float(kPhaseAt), __uint_as_float(kPhaseAt));
        }
    }
    if (threadIdx.x == 0) {
        progress = 0;
        abort_walk = 0;
        for (int i = 0; i < kRing; ++i)
            mbar_init(&ring_bar[i], nparts); // an arrival per part
        for (int i = 0; i < kGroups; ++i)
            mbar_init(&done_bar[i], 1);
        for (int i = 0; i < kRecoThreads / 32; ++i)
            mbar_init(&row_bar[i], 1);
        fence_mbar_init();
    }
    __threadfence(); // the seeds in the map
    if constexpr (MULTI)
        cluster_sync_all();
    else
        __syncthreads();

    auto aborted = [&]() {
        if constexpr (MULTI)
            return dsmem_ld_relaxed(dsmem_addr(&abort_walk, 0)) != 0;
        else
            return *reinterpret_cast<volatile int*>(&abort_walk) != 0;
    };
    auto give_up = [&]() {
        if constexpr (MULTI)
            dsmem_st_relaxed(dsmem_addr(&abort_walk, 0), 1);
        else
            *reinterpret_cast<volatile int*>(&abort_walk) = 1;
    };
    // bounded wait on a condition; false on a timeout or when another warp
    // gave up (then the walk stops)
    auto wait_until = [&](auto cond, unsigned sleep) {
        if (cond())
            return true;
        const unsigned long long t0 = globaltimer_ns();
        for (;;) {
            for (int i = 0; i < 64; ++i) {
                if (cond())
                    return true;
                if (sleep)
                    __nanosleep(sleep);
            }
            if (aborted())
                return false;
            if (globaltimer_ns() - t0 > kRecoWaitNs) {
                record_error(J.err, SMIP_DEV_ERR_TIMEOUT);
                give_up();
                return false;
            }
        }
    };
    const bool oor_any = *J.oor != 0; // some phasor is marked
    // a pair of a marked phasor b, used: true where it makes the sum NaN
    auto marked = [&](float bx, float2 U, float2 V) {
        const unsigned b = __float_as_uint(bx);
        const bool used = (b == kOorBits || b == kNanBits) && !isnan(U.x) && !isnan(V.x);
        if (used && b == kOorBits) // get_element would throw
            record_error(J.err, SMIP_DEV_ERR_OUT_OF_RANGE);
        return used && b == kNanBits;
    };

    // which warp does what (a nibble each): 0 the serial warp, 1 the writer,
    // 2.. loading, 6.. gathering, 14 summing, 15 nothing.  In a cluster rank 0
    // sums nothing; the serial warp's sub-partition (warp % 4) is its own in a
    // cluster, and free of summing warps in a lone CTA.
    constexpr unsigned long long kRoles = MULTI ? 0xFB5F432FA91F8760ull : 0xEEE2EEE6EEE1EEE0ull;
    constexpr int kLoaders = MULTI ? 4 : 1, kGatherers = MULTI ? 6 : 1;
    const int role = MULTI && rank != 0 ? 14 : (int)(kRoles >> (4 * warp)) & 15;
    // the map: other SMs write it in a cluster (read from L2), this SM in a lone CTA
    auto map_at = [&](long long i) { return MULTI ? __ldcg(J.pmap + i) : *(J.pmap + i); };
    // this CTA's copy of the progress has reached v
    auto reached = [&](int v) { return __all_sync(0xffffffffu, wait_until([&] { return ld_acquire_cta(&progress) >= v; }, 20u) ? 1 : 0); };
    if (role == 0) {
        // ------------------------------------------------ serial warp
        auto term = [&](float2 U, float2 V, float2 bh, float2& p, float& r) {
            p = pair_product(U, V, bh.x, bh.y);
            const float n2 = norm2(p);
            r = rsqrt_ftz(n2);
            return !isnan(n2);
        };
        // visits [q, q + kStep) (or up to the last) are ready, and which of them
        // are wide: relaxed polls and one fence of this CTA's scope, which costs
        // nothing (a fence of the cluster's takes 300 cycles)
        auto ready = [&](int q, unsigned& wide) {
            const int at = q + (lane & (kStep - 1)), v = at < J.nvisits ? at : J.nvisits - 1;
            const volatile int* tag = &gtag[v & (kRing - 1)];
            unsigned long long t0 = 0;
            for (int n = 1;; ++n) {
                const int t = *tag;
                if (__all_sync(0xffffffffu, t >> 1 == v + 1)) {
                    __threadfence_block();
                    wide = __ballot_sync(0xffffffffu, lane < kStep && (t & 1) && at < J.nvisits);
                    return true;
                }
                if (n & 63)
                    continue;
                const unsigned long long now = globaltimer_ns();
                t0 = t0 ? t0 : now;
                const bool late = now - t0 > kRecoWaitNs;
                if (late && lane == 0) {
                    record_error(J.err, SMIP_DEV_ERR_TIMEOUT);
                    give_up();
                }
                if (__any_sync(0xffffffffu, late || aborted()))
                    return false;
            }
        };
        const int nqs = (J.nvisits + kStep - 1) / kStep * kStep; // the writer leaves out what lies past the last visit
        const bool imag = lane >= 16; // lanes 0 and 16 form the real and the imaginary part
        float2 last = make_float2(nanf_, nanf_);
        uint2 lc = {}, hc = {};            // places of visit q + 1's members: the lane's pair, the first pair
        float2 hU = {}, hV = {}, hb = {};  // visit q's first pair
        float sib0 = 0.f, level = 0.f;     // visit q's recent pairs in the butterfly: the first pair's sibling, and its first level
        float en = 0.f;                    // its recent pairs but the first
        // what can be known of visit q before the phase of visit q - 1: the terms
        // of the lanes' pairs (the first's is left out) and the first level of
        // their butterfly sum, from which on the lower lanes hold real parts and the
        // upper ones imaginary parts.  The other levels run beside the next step's
        // chain: all of them in one step would make it as long as they are.
        auto early = [&](float2 U, float2 V, float2 b) {
            float2 p;
            float r;
            const bool ok = term(U, V, b, p, r);
            const float x = ok ? fmaf(p.x, r, 0.f) : 0.f, y = ok ? fmaf(p.y, r, 0.f) : 0.f;
            en = (float)__popc(__ballot_sync(0xffffffffu, ok) & ~1u);
            float a = imag ? y : x;
            const float o = __shfl_xor_sync(0xffffffffu, imag ? x : y, 16);
            sib0 = imag ? a : o;
            level = __fadd_rn(a, o);
        };
        // The sum of a visit from its recent pairs' (lanes 0 and 16) and its
        // share, its phase and what is kept of it.  FP64 values are formed after
        // the walk; a sum above the limit has a normal square; a point without
        // any pair has no phase.
        auto finish = [&](float part, float2 sh, float4 ct, float cnt, float2& kept) {
            const float s = __fadd_rn(sh.x, part), bb = __fsub_rn(s, sh.x);
            const float e = __fadd_rn(__fadd_rn(__fsub_rn(sh.x, __fsub_rn(s, bb)), __fsub_rn(part, bb)), sh.y);
            kept = make_float2(s, e);
            const float h = __fadd_rn(s, e);
            const float2 f = make_float2(__shfl_sync(0xffffffffu, h, 0), __shfl_sync(0xffffffffu, h, 16));
            const float s2 = norm2(f), r = rsqrt_ftz(s2), lim = 2.220446049250313e-16f * cnt;
            const bool has = cnt > 0.f, normal = has && s2 > lim * lim;
            float2 now = make_float2(has ? 0.f : ct.x, has ? 0.f : ct.y);
            now.x = normal ? f.x * r : now.x;
            now.y = normal ? f.y * r : now.y;
            return now;
        };
        auto share_of = [&](int s) { return *reinterpret_cast<const float2*>(smraw + kShareAt + 16 * s + (imag ? 8 : 0)); };
        auto keep = [&](int s, float cnt, float2 kept) {
            res_p[s] = make_float4(last.x, last.y, cnt, 0.f); // the same in every lane
            if ((lane & 15) == 0)
                *reinterpret_cast<float2*>(smraw + kSumAt + 16 * s + (imag ? 8 : 0)) = kept;
            __syncwarp();
        };
        // visit q; the chain (the first pair's term, five additions, the share,
        // the phase) and the early part of visit q + 1 overlap
        auto step = [&](int q) {
            const int s = q & (kRing - 1), s1 = (q + 1) & (kRing - 1), s2 = (q + 2) & (kRing - 1);
            const float2 sh = share_of(s);
            const float4 ct = ctl[s];
            const float2 nU = phase_at(lc.x), nV = phase_at(lc.y), nhU = phase_at(hc.x), nhV = phase_at(hc.y);
            const float4* ne = &ent[s1 * kRecentMax + lane];
            const float2 nb = make_float2(ne->x, ne->y), nhb = make_float2(head[s1].x, head[s1].y);
            lc = place[s2 * kRecentMax + lane];
            hc = make_uint2(__float_as_uint(head[s2].z), __float_as_uint(head[s2].w));
            const int bits = __float_as_int(ct.z);
            const bool lu = bits & (1 << 9), lv = bits & (1 << 10);
            // sibling sums on the first pair's way down the butterfly (lanes 0, 16)
            float sib[5] = { sib0 };
#pragma unroll
            for (int l = 1; l < 5; ++l) {
                sib[l] = __shfl_xor_sync(0xffffffffu, level, 16 >> l);
                level = __fadd_rn(level, sib[l]);
            }
            float2 p, kept;
            float r;
            const bool ok = term(make_float2(lu ? last.x : hU.x, lu ? last.y : hU.y),
                                 make_float2(lv ? last.x : hV.x, lv ? last.y : hV.y), hb, p, r);
            float a = ok ? fmaf(imag ? p.y : p.x, r, 0.f) : 0.f;
#pragma unroll
            for (int l = 0; l < 5; ++l)
                a = __fadd_rn(a, sib[l]);
            const float cnt = ct.w + en + (ok ? 1.f : 0.f);
            early(nU, nV, nb);
            last = finish(a, sh, ct, cnt, kept);
            keep(s, cnt, kept);
            hU = nhU;
            hV = nhV;
            hb = nhb;
        };
        // a visit with up to 64 recent pairs, several of age 1, or whose point may
        // have got its phase within the lag: all terms now, the phases up to the
        // last lie in their slots
        auto wide_step = [&](int q) {
            const int s = q & (kRing - 1), s1 = (q + 1) & (kRing - 1), s2 = (q + 2) & (kRing - 1);
            const float2 sh = share_of(s);
            const float4 ct = ctl[s];
            const int bits = __float_as_int(ct.z), kc = bits & 63;
            const bool two = bits & (1 << 8);
            const uint2 ca = place[s * kRecentMax + lane], cb = place[s * kRecentMax + 32 + lane];
            const float4 ba = ent[s * kRecentMax + lane], bb = ent[s * kRecentMax + 32 + lane];
            const float2 Ua = phase_at(ca.x), Va = phase_at(ca.y), Ub = phase_at(cb.x), Vb = phase_at(cb.y);
            const float4 own = res_p[(q - kc) & (kRing - 1)];
            float2 pa, pb, kept;
            float ra, rb;
            bool oka = term(Ua, Va, make_float2(ba.x, ba.y), pa, ra);
            bool okb = term(Ub, Vb, make_float2(bb.x, bb.y), pb, rb) && two;
            if (oor_any && q < J.nvisits && !(kc && !isnan(own.x))) { // (a NaN term is then a pair like any other)
                oka = marked(ba.x, Ua, Va) || oka;
                okb = (two && marked(bb.x, Ub, Vb)) || okb;
            }
            float sr = oka ? fmaf(pa.x, ra, 0.f) : 0.f, si = oka ? fmaf(pa.y, ra, 0.f) : 0.f;
            sr = okb ? fmaf(pb.x, rb, sr) : sr;
            si = okb ? fmaf(pb.y, rb, si) : si;
            float cnt = ct.w + (float)(__popc(__ballot_sync(0xffffffffu, oka)) + __popc(__ballot_sync(0xffffffffu, okb)));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sr = __fadd_rn(sr, __shfl_xor_sync(0xffffffffu, sr, o));
                si = __fadd_rn(si, __shfl_xor_sync(0xffffffffu, si, o));
            }
            float2 now = finish(imag ? si : sr, sh, ct, cnt, kept);
            if (kc && !isnan(own.x)) { // its point, visited within the lag, has its phase
                now = make_float2(own.x, own.y);
                cnt = 0.f;
            }
            const float4* ne = &ent[s1 * kRecentMax + lane];
            early(phase_at(lc.x), phase_at(lc.y), make_float2(ne->x, ne->y));
            hU = phase_at(hc.x);
            hV = phase_at(hc.y);
            hb = make_float2(head[s1].x, head[s1].y);
            lc = place[s2 * kRecentMax + lane];
            hc = make_uint2(__float_as_uint(head[s2].z), __float_as_uint(head[s2].w));
            last = now;
            keep(s, cnt, kept);
        };
        unsigned wide = 0u, more = 0u; // wide visits from q on
        bool go = ready(0, wide) && ready(2, more);
        wide = (wide & 3u) | more << 2;
        if (go) {
            const float4* e0 = &ent[lane];
            const uint2 c0 = place[lane];
            early(phase_at(c0.x), phase_at(c0.y), make_float2(e0->x, e0->y));
            hb = make_float2(head[0].x, head[0].y);
            hU = phase_at(__float_as_uint(head[0].z));
            hV = phase_at(__float_as_uint(head[0].w));
            lc = place[kRecentMax + lane];
            hc = make_uint2(__float_as_uint(head[1].z), __float_as_uint(head[1].w));
        }
        for (int q = 0; go && q < nqs;) {
            // a loop of one block without branches; unrolled it was slower (493
            // cycles a visit instead of 428 at depth 48), as with both forms in
            // one loop (568): the warp waits for instructions
            if ((wide & ((1u << kStep) - 1u)) == 0u) {
#pragma unroll 1
                for (int k = 0; k < kStep; ++k)
                    step(q + k);
            } else {
#pragma unroll 1
                for (int k = 0; k < kStep; ++k) {
                    if ((wide >> k) & 1u)
                        wide_step(q + k);
                    else
                        step(q + k);
                }
            }
            q += kStep;
            wide >>= kStep;
            // tell the writer, look ahead
            if (lane == 0)
                mbar_arrive(&done_bar[(q / kStep - 1) & (kGroups - 1)]);
            go = ready(q + 2, more);
            wide |= more << 2;
        }
    } else if (role == 1) {
        // ------------------------------------------------------ writer
        const int ngroups = (J.nvisits + kStep - 1) / kStep;
        for (int g = 0; g < ngroups;) {
            // groups of kStep visits, as many as are done (up to 32 visits)
            const int q = kStep * g + lane, s = q & (kRing - 1);
            int4 m = make_int4(-1, 0, 0, -1);
            if (q < J.nvisits)
                m = J.meta[q];
            auto is_done = [&](int h) { return mbar_test_wait(&done_bar[h & (kGroups - 1)], (uint32_t)(h / kGroups) & 1u); };
            if (!__all_sync(0xffffffffu, wait_until([&] { return is_done(g); }, 20u) ? 1 : 0))
                break;
            const unsigned m8 = __ballot_sync(0xffffffffu, lane < 32 / kStep && g + lane < ngroups && is_done(g + lane)) | 1u;
            const int n = __ffs(~m8) - 1;
            float4 rp = make_float4(0.f, 0.f, 0.f, 0.f), rs = rp;
            if (lane < kStep * n && q < J.nvisits) {
                rp = res_p[s];
                rs = res_s[s];
            }
            const int cnt = (int)rp.z;
            const float2 pf = make_float2(rp.x, rp.y);
            if (cnt > 0) { // a point got its phase
                J.pmap[m.x] = pf;
                if (m.w >= 0)
                    vt[m.w] = pf;
            }
            g += n;
            __syncwarp();
            // release: the stores above come before it for whoever acquires it,
            // first in this CTA, whose warps wait for nothing else
            if (lane == 0)
                st_release_cta(&progress, kStep * g);
            if constexpr (MULTI) {
                if (cnt > 0 && m.w >= 0)
                    for (uint32_t c = 1; c < ncta; ++c)
                        dsmem_st_f2(dsmem_addr(&vt[m.w], c), pf);
                __syncwarp();
                if (lane > 0 && lane < (int)ncta)
                    dsmem_st_release(dsmem_addr(&progress, lane), kStep * g);
            }
            if (cnt > 0) { // read after the walk only
                J.sums[m.y] = rs;
                J.cnt[m.y] = cnt;
            }
            __syncwarp();
        }
    } else if (role < 6) {
        // ------- loading warps: a visit's recent pairs, with their members
        // outside the lag, whose phases are final
        int4 nm = make_int4(-1, 0, 0, -1);
        uint4 na = make_uint4(kUnusable, kUnusable, 0u, 0u), nb = na;
        auto fetch = [&](int q) { // the list of a point that is not runnable was never written
            if (q < J.nvisits) {
                nm = J.meta[q];
                na = J.rec[(long long)q * kRecentMax + lane];
                nb = J.rec[(long long)q * kRecentMax + 32 + lane];
            }
        };
        fetch(role - 2);
        for (int q = role - 2; q < J.nvisits; q += kLoaders) {
            const int4 m = nm;
            const uint4 ra = na, rb = nb;
            const int s = q & (kRing - 1);
            fetch(q + kLoaders);
            if (!reached(q - kRecoLag))
                break;
            auto post = [&](int at, uint4 r) {
                const int t = r.z & 0x1fff, ku = (r.z >> 13) & 63, kv = (r.z >> 19) & 63;
                float2 x = vt[t]; // v, unless u is the one outside the lag
                if (!ku && kv)
                    x = map_at((long long)m.x - voff[t]);
                ent[s * kRecentMax + at] = make_float4(__uint_as_float(r.x), __uint_as_float(r.y), x.x, x.y);
                const unsigned own = kPairAt + 16u * (s * kRecentMax + at) + 8u;
                const uint2 c = make_uint2(ku ? kPhaseAt + 16u * ((q - ku) & (kRing - 1)) : own,
                                           kv ? kPhaseAt + 16u * ((q - kv) & (kRing - 1)) : own);
                place[s * kRecentMax + at] = c;
                if (at == 0) {
                    head[s] = make_float4(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(c.x), __uint_as_float(c.y));
                    lhead[s] = (ku == 1 ? 1 << 9 : 0) | (kv == 1 ? 1 << 10 : 0);
                }
            };
            if ((m.z >> 17) & 1) {
                post(lane, ra);
                if ((m.z & 255) > 32)
                    post(lane + 32, rb);
            }
            __syncwarp();
            if (lane == 0)
                st_release_cta(&ltag[s], q + 1);
        }
    } else if (role < 14) {
        // gathering warps: a visit's parts, in part order, and what its point has
        int4 nm = make_int4(-1, 0, 0, -1);
        if (role - 6 < J.nvisits)
            nm = J.meta[role - 6];
        for (int q = role - 6; q < J.nvisits; q += kGatherers) {
            const int s = q & (kRing - 1);
            const int4 m = nm;
            if (q + kGatherers < J.nvisits)
                nm = J.meta[q + kGatherers];
            const volatile int* tag = &tag_s[lane < nparts ? lane : 0][s];
            const volatile int* lt = &ltag[s];
            if (!__all_sync(0xffffffffu, wait_until([&] {
                                return MULTI ? mbar_try_wait_cluster(&ring_bar[s], (uint32_t)(q / kRing) & 1u) : *tag == q + 1;
                            }, MULTI ? 0u : 20u) && wait_until([&] { return *lt == q + 1; }, 20u) ? 1 : 0))
                break;
            __threadfence_block();
            float4 sum = shr[0][s];
            const float4 c = shc[s];
            int n = __float_as_int(c.x);
            for (int pp = 1; pp < nparts; ++pp) {
                const float4 op = shr[pp][s];
                ff_add(sum.x, sum.y, op.x, op.y);
                ff_add(sum.z, sum.w, op.z, op.w);
                n += shn[pp][s];
            }
            if (lane == 0) {
                // a point outside the map, a seed, or one that has its phase: nothing to sum
                const int rc = m.z & 255, kc = (m.z >> 8) & 63;
                const bool skip = !((m.z >> 17) & 1) || (kc == 0 && !isnan(c.y));
                const bool wide = !skip && (!((m.z >> 16) & 1) || oor_any);
                share[s] = sum;
                ctl[s] = make_float4(c.y, c.z, __int_as_float(kc | (rc > 32 ? 1 << 8 : 0) | (skip ? 0 : lhead[s])), skip ? -1e6f : (float)n);
                st_release_cta(&gtag[s], 2 * (q + 1) + (wide ? 1 : 0));
            }
            __syncwarp();
        }
    } else if (role == 14) {
        // ------------------------------------------- non-recent shares
        // Warp g takes part g % nparts of the visits g / nparts, + at_once, ..
        const int nsum = MULTI ? (int)(ncta - 1) * (kRecoThreads / 32) : kRecoThreads / 32 * 3 / 4;
        const int g = MULTI ? warp * (int)(ncta - 1) + (int)(rank - 1) : (warp >> 2) * 3 + (warp & 3) - 1;
        const int at_once = nsum / nparts, part = g % nparts, q0 = g < at_once * nparts ? g / nparts : J.nvisits;
        const int wb = part * nwords / nparts, we = (part + 1) * nwords / nparts;
        // In a cluster a visit's plan row comes into shared memory before the
        // visit may be summed, and only the gathers of u stand between the
        // progress and the sum: kB of them a lane in flight (2 registers each), in
        // batches of equal length (10, 18 or 20 words compiled; 7, 9 or 12 at a time
        // were slower at depths 24, 32 and 48).
        constexpr int kB = 20, kBDirect = 10;
        const int nbat = (we - wb + kB - 1) / kB, nbw = (we - wb + nbat - 1) / nbat; // batches, words of one
        const bool staged = MULTI && part_words(De, nwords) <= kRowWords;
        float2* row = rows + warp * part_words(De, nwords) * 32;
        auto is_run = [&](const int4& m) { return ((m.z >> 17) & 1) != 0; };
        bool flying = false; // a copy of a row is on its way, or has not been waited for
        uint32_t phase = 0u;
        auto stage = [&](int q, const int4& m) {
            flying = staged && is_run(m);
            if (flying && lane == 0) {
                const uint32_t bytes = (uint32_t)(we - wb) * 256u;
                mbar_arrive_expect_tx(&row_bar[warp], bytes);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(row)),
                             "l"(J.plan + (long long)q * nslots + 32 * wb), "r"(bytes), "r"(smem_u32(&row_bar[warp]))
                             : "memory");
            }
        };
        int4 nm = make_int4(-1, 0, 0, -1); // the next visit's meta, and the phase that its point has so far
        float nx = nanf_;
        if (q0 < J.nvisits) {
            nm = J.meta[q0];
            stage(q0, nm);
        }
        for (int q = q0; q < J.nvisits; q += at_once) {
            const int4 m = nm;
            const int kc = (m.z >> 8) & 63;
            // a point outside the map, a seed, or one that has its phase: nothing
            // to sum (a phase once set stays; a point that has none yet is looked
            // at again below)
            bool skip = !is_run(m) || (kc == 0 && !isnan(nx));
            if (q + at_once < J.nvisits) {
                nm = J.meta[q + at_once];
                if (lane == 0) // the next visit's plan row on its way into L2
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(J.plan + (long long)(q + at_once) * nslots + 32 * wb),
                                 "r"((we - wb) * 32 * (int)sizeof(float2))
                                 : "memory");
            }
            if (!__all_sync(0xffffffffu, wait_until([&] {
                                const int pr = MULTI ? dsmem_ld_acquire(dsmem_addr(&progress, rank)) : ld_acquire_cta(&progress);
                                return pr >= q - kRecoLag;
                            }, 20u) ? 1 : 0))
                break;
            // The errors of a point that has its phase do not count, however long
            // ago it was visited.  One that gets its phase within the lag was
            // formed then from every pair that is summed here, errors included.
            if (oor_any && !skip)
                skip = !isnan(map_at(m.x).x);
            float2 cur = make_float2(nanf_, nanf_); // waited for at the end
            if (m.x >= 0)
                cur = map_at(m.x);
            skip = __all_sync(0xffffffffu, skip);
            float sr = 0.f, si = 0.f;
            int cnt = 0;
            const float2* mb = J.pmap + m.x;
            const float2* prow = J.plan + (long long)q * nslots + lane;
            // the part's words in order, NB gathers at a time
            auto sum_pairs = [&](auto nb, auto rowed) {
                constexpr int NB = decltype(nb)::value;
                constexpr bool ROW = decltype(rowed)::value;
                for (int i0 = wb; i0 < we; i0 += NB) {
                    float2 u[NB], bh[ROW ? 1 : NB];
#pragma unroll
                    for (int k = 0; k < NB; ++k) {
                        const int i = i0 + k < we ? 32 * (i0 + k) : 32 * i0;
                        const float2* up = mb - voff[i + lane];
                        u[k] = MULTI ? __ldcg(up) : *up;
                        if constexpr (!ROW)
                            bh[k] = ld_stream(prow + i);
                    }
#pragma unroll
                    for (int k = 0; k < NB; ++k) { // no branch: the words' latencies overlap
                        const bool in = i0 + k < we;
                        const int i = in ? i0 + k : i0;
                        const float2 v = vt[32 * i + lane];
                        float2 b;
                        if constexpr (ROW)
                            b = row[32 * (i - wb) + lane];
                        else
                            b = bh[k];
                        const float2 p = pair_product(u[k], v, b.x, b.y);
                        const float n2 = norm2(p);
                        const float r = rsqrt_ftz(n2);
                        const bool use = in && !isnan(n2);
                        sr = use ? fmaf(p.x, r, sr) : sr;
                        si = use ? fmaf(p.y, r, si) : si;
                        cnt += use ? 1 : 0;
                    }
                }
            };
            if (flying) { // also of a visit that is skipped: the buffer must be free for the next
                if (!__all_sync(0xffffffffu, wait_until([&] { return mbar_try_wait(&row_bar[warp], phase); }, 0u) ? 1 : 0))
                    break;
                phase ^= 1u;
                flying = false;
            }
            if (!skip) {
                using Yes = std::true_type;
                using No = std::false_type;
                if (!staged)
                    sum_pairs(std::integral_constant<int, kBDirect> {}, No {});
                else if (nbw <= 10)
                    sum_pairs(std::integral_constant<int, 10> {}, Yes {});
                else if (nbw <= 18)
                    sum_pairs(std::integral_constant<int, 18> {}, Yes {});
                else
                    sum_pairs(std::integral_constant<int, kB> {}, Yes {});
                if (oor_any)
                    for (int i = wb; i < we; ++i) {
                        const float2 v = vt[32 * i + lane], *up = mb - voff[32 * i + lane];
                        if (marked(ld_stream(prow + 32 * i).x, MULTI ? __ldcg(up) : *up, v)) {
                            sr = si = nanf_;
                            ++cnt;
                        }
                    }
                if (kc == 0 && !isnan(cur.x)) { // it had its phase
                    sr = si = 0.f;
                    cnt = 0;
                }
            }
            __syncwarp();
            nx = nanf_;
            if (q + at_once < J.nvisits) {
                stage(q + at_once, nm);
                if (nm.x >= 0)
                    nx = map_at(nm.x).x; // on its way during what follows
            }
            // float-float over the lanes, lane 0's order
            float rh = sr, rl = 0.f, ih = si, il = 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float a = __shfl_xor_sync(0xffffffffu, rh, o), b = __shfl_xor_sync(0xffffffffu, rl, o);
                const float c = __shfl_xor_sync(0xffffffffu, ih, o), f = __shfl_xor_sync(0xffffffffu, il, o);
                ff_add(rh, rl, a, b);
                ff_add(ih, il, c, f);
            }
            cnt = __reduce_add_sync(0xffffffffu, cnt);
            const int s = q & (kRing - 1);
            if (lane == 0) {
                const float4 sum = make_float4(rh, rl, ih, il), c = make_float4(__int_as_float(cnt), cur.x, cur.y, 0.f);
                if constexpr (MULTI) {
                    const uint32_t bar = dsmem_addr(&ring_bar[s], 0);
                    dsmem_mbar_arrive_expect_tx(bar, part == 0 ? 32u : 20u);
                    dsmem_st_async_f4(dsmem_addr(&shr[part][s], 0), sum, bar);
                    if (part == 0)
                        dsmem_st_async_f4(dsmem_addr(&shc[s], 0), c, bar);
                    else
                        dsmem_st_async_i(dsmem_addr(&shn[part][s], 0), cnt, bar);
                } else {
                    shr[part][s] = sum;
                    if (part == 0)
                        shc[s] = c;
                    else
                        shn[part][s] = cnt;
                    st_release_cta(&tag_s[part][s], q + 1);
                }
            }
            __syncwarp();
        }
        if (flying) // the walk was given up: no copy outlives its CTA
            mbar_wait_bounded(&row_bar[warp], phase, kRecoWaitNs);
    }
    if constexpr (MULTI)
        cluster_sync_all(); // no CTA touches another's shared memory after this
}

// FP64 mean, consistency and phase of every point (phasereco.h:110-122) and
// the flag map, once the walk is done.
__global__ void __launch_bounds__(256) phase_final_kernel(const RecoJob* __restrict__ jobs)
{
    const RecoJob J = jobs[blockIdx.y];
    const int W = J.W, H = J.H, e = J.De / 2;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < W * H; p += gridDim.x * blockDim.x) {
        int x = p % W, y = p / W; // FFT order -> the centred map
        x -= x > -W / 2 + W - 1 ? W : 0;
        y -= y > -H / 2 + H - 1 ? H : 0;
        const float2 pf = J.pmap[(long long)(y + (H >> 1) + e) * (W + J.De) + x + (W >> 1) + e];
        const bool f = !isnan(pf.x);
        J.flags[p] = f;
        if (!f)
            continue;
        const int n = J.cnt[p];
        if (n < 0) { // seed
            J.phases[p] = make_double2(1.0, pf.y);
            J.cons[p] = 1.0;
            continue;
        }
        const float4 s = J.sums[p];
        const double mr = ((double)s.x + (double)s.y) / (double)n;
        const double mi = ((double)s.z + (double)s.w) / (double)n;
        const double ab = sqrt(mr * mr + mi * mi);
        J.cons[p] = ab;
        J.phases[p] = ab > 2.220446049250313080847263336181640625e-16 ? make_double2(mr / ab, mi / ab)
                                                                      : make_double2(0.0, 0.0);
    }
}

// ------------------------------------------ ring-parallel estimator (opt-in)
// A different estimator from the reference's spiral, offered as an option:
// the spiral's visits are grouped by the radius r at which NextRecoIndex makes
// them (one ring per r, each point once per ring), and every point of ring k
// is formed in parallel from the pairs whose u and v got their phases in
// rings before k.  The spiral also uses phases set earlier in the same ring,
// so the two differ; the phase difference is measured, not bounded by the
// reference.  fring[p]: the ring in which point p got its phase (seeds 0),
// -1 while it has none; only rings < k are read while ring k is written, so
// the result does not depend on the order in which the ring's warps run.
__global__ void ring_seed_kernel(const RecoJob* __restrict__ jobs, int* __restrict__ fring)
{
    const RecoJob J = jobs[0];
    if (threadIdx.x < 5) { // seeds (phasereco.h:42-54), as in the spiral walk
        const int sx[5] = { 0, 1, 0, -1, 0 }, sy[5] = { 0, 0, 1, 0, -1 };
        const int p = wrap_idx(sx[threadIdx.x], sy[threadIdx.x], J.W, J.H);
        const float im = threadIdx.x < 3 ? 0.f : -0.f;
        J.phf[p] = make_float2(1.f, im);
        J.sums[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        J.cnt[p] = -1;
        fring[p] = 0;
    }
}

// One warp per visit of ring `ring`: rq[0..n) are the ring's visit indices.
__global__ void __launch_bounds__(256) ring_pass_kernel(const RecoJob* __restrict__ jobs, const int* __restrict__ rq,
                                                        int n, int ring, int* __restrict__ fring)
{
    const RecoJob J = jobs[0];
    const int gw = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (gw >= n) // whole warps leave together
        return;
    const int W = J.W, H = J.H, De = J.De, nside = De + 1, nv = nside * nside;
    const int q = rq[gw];
    const int2 w = J.visits[q];
    const int pmin0 = -(W >> 1), pmin1 = -(H >> 1);
    const int pmax0 = -W / 2 + W - 1, pmax1 = -H / 2 + H - 1;
    const int szW = (W / 2) * 2 + 1, szH = (H / 2) * 2 + 1;
    const int umn0 = -(szW / 2), umx0 = szW - szW / 2 - 1, umn1 = -(szH / 2), umx1 = szH - szH / 2 - 1;
    if (w.x < pmin0 || w.x > pmax0 || w.y < pmin1 || w.y > pmax1)
        return;
    const int pw = wrap_idx(w.x, w.y, W, H);
    if (fring[pw] >= 0 || abs(w.x) + abs(w.y) <= 1                          // phasereco.h:84
        || w.x < umn0 || w.x > umx0 || w.y < umn1 || w.y > umx1)
        return;
    const float2* prow = J.plan + (long long)q * nv;
    float sr = 0.f, si = 0.f;
    int cnt = 0;
    // kB slots per lane at a time: every gather of the group is issued before
    // any is used, so their latencies overlap; the sums take the slots in
    // increasing order as a one-slot loop would
    constexpr int kB = 8;
    for (int t0 = lane; t0 < nv; t0 += 32 * kB) {
        float2 bh[kB], pa[kB], pb[kB];
        int fu[kB], fv[kB];
        bool use[kB];
#pragma unroll
        for (int k = 0; k < kB; ++k) {
            const int t = t0 + 32 * k;
            use[k] = t < nv;
            bh[k] = use[k] ? prow[t] : make_float2(0.f, 0.f);
            const int vx = -De / 2 + t % nside, vy = -De / 2 + t / nside;
            const int ux = w.x - vx, uy = w.y - vy;
            use[k] = use[k] && !(ux < pmin0 || ux > pmax0 || uy < pmin1 || uy > pmax1);
            const int pu = use[k] ? wrap_idx(ux, uy, W, H) : 0, pv = use[k] ? wrap_idx(vx, vy, W, H) : 0;
            fu[k] = use[k] ? fring[pu] : -1;
            fv[k] = use[k] ? fring[pv] : -1;
            pa[k] = use[k] ? J.phf[pu] : make_float2(0.f, 0.f);
            pb[k] = use[k] ? J.phf[pv] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < kB; ++k) {
            if (!use[k] || (bh[k].x == 0.f && bh[k].y == 0.f)) // the plan's zero: never contributes
                continue;
            if (fu[k] < 0 || fu[k] >= ring || fv[k] < 0 || fv[k] >= ring)
                continue;
            if (isnan(bh[k].x)) {
                record_error(J.err, SMIP_DEV_ERR_OUT_OF_RANGE);
                continue;
            }
            const float2 ph = cmul(cmul(pa[k], pb[k]), make_float2(bh[k].x, -bh[k].y));
            const float r = rsqrtf(ph.x * ph.x + ph.y * ph.y);
            sr += ph.x * r;
            si += ph.y * r;
            ++cnt;
        }
    }
    float rh = sr, rl = 0.f, ih = si, il = 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float a = __shfl_xor_sync(0xffffffffu, rh, o), b = __shfl_xor_sync(0xffffffffu, rl, o);
        const float c = __shfl_xor_sync(0xffffffffu, ih, o), e = __shfl_xor_sync(0xffffffffu, il, o);
        ff_add(rh, rl, a, b);
        ff_add(ih, il, c, e);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    if (lane == 0 && cnt > 0) {
        const float s2 = rh * rh + ih * ih;
        const float lim = 2.220446049250313e-16f * (float)cnt;
        float2 pf = make_float2(0.f, 0.f);
        if (s2 > lim * lim) {
            const float r = rsqrtf(s2);
            pf = make_float2(rh * r, ih * r);
        }
        J.phf[pw] = pf;
        J.sums[pw] = make_float4(rh, rl, ih, il);
        J.cnt[pw] = cnt;
        fring[pw] = ring;
    }
}

// FP64 mean, consistency and phase of every point and the flag map, as the
// spiral walk's final pass forms them.
__global__ void ring_final_kernel(const RecoJob* __restrict__ jobs, const int* __restrict__ fring)
{
    const RecoJob J = jobs[0];
    const int np = J.W * J.H;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
        const unsigned char f = fring[p] >= 0 ? 1 : 0;
        J.flags[p] = f;
        if (!f)
            continue;
        const int n = J.cnt[p];
        if (n < 0) {
            J.phases[p] = make_double2(1.0, J.phf[p].y);
            J.cons[p] = 1.0;
            continue;
        }
        const float4 s = J.sums[p];
        const double mr = ((double)s.x + (double)s.y) / (double)n;
        const double mi = ((double)s.z + (double)s.w) / (double)n;
        const double ab = sqrt(mr * mr + mi * mi);
        J.cons[p] = ab;
        J.phases[p] = ab > 2.220446049250313080847263336181640625e-16 ? make_double2(mr / ab, mi / ab)
                                                                      : make_double2(0.0, 0.0);
    }
}

cudaError_t launch_ring_reco(const RecoJob* job_dev, int* fring, const int* rq, const std::vector<int>& roff, int W,
                             int H, cudaStream_t st)
{
    reco_plan_kernel<<<dim3(1024, 1), 256, 0, st>>>(job_dev);
    note_launches(1);
    cudaError_t e = cudaMemsetAsync(fring, 0xff, sizeof(int) * (size_t)W * H, st); // -1: no phase yet
    if (e != cudaSuccess)
        return e;
    ring_seed_kernel<<<1, 32, 0, st>>>(job_dev, fring);
    note_launches(1);
    for (size_t k = 1; k + 1 < roff.size(); ++k) {
        const int n = roff[k + 1] - roff[k];
        if (n <= 0)
            continue;
        ring_pass_kernel<<<(n * 32 + 255) / 256, 256, 0, st>>>(job_dev, rq + roff[k], n, (int)k, fring);
        note_launches(1);
    }
    const int np = W * H;
    ring_final_kernel<<<(np + 255) / 256 < 2048 ? (np + 255) / 256 : 2048, 256, 0, st>>>(job_dev, fring);
    note_launches(1);
    return cudaGetLastError();
}

// Runs the device get_element index replica on a list of 4-index tuples.
__global__ void bispec_offset_probe_kernel(BispecDims d, const int4* __restrict__ idx, long long n,
                                           long long* __restrict__ off, int* __restrict__ conj)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int4 i = idx[q];
        int cj = 0;
        off[q] = bispec_get_offset(d, i.x, i.y, i.z, i.w, &cj);
        conj[q] = off[q] < 0 ? 0 : cj;
    }
}

cudaError_t launch_offset_probe(const Geometry& g, const int* idx, long long n, long long* off, int* conj,
                                cudaStream_t st)
{
    BispecDims d;
    const int szW = (g.W / 2) * 2 + 1, szH = (g.H / 2) * 2 + 1, szD = g.De + 1;
    d.sizes[0] = szW; d.sizes[1] = szH; d.sizes[2] = szD; d.sizes[3] = szD;
    d.base[0] = szW - szW / 2; d.base[1] = szH; d.base[2] = szD - szD / 2; d.base[3] = szD;
    for (int k = 0; k < 4; ++k) {
        d.mn[k] = -(d.sizes[k] / 2);
        d.mx[k] = d.sizes[k] + d.mn[k] - 1;
    }
    d.base_size = (long long)d.base[0] * d.base[1] * d.base[2] * d.base[3];
    bispec_offset_probe_kernel<<<256, 256, 0, st>>>(d, reinterpret_cast<const int4*>(idx), n, off, conj); note_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_phase_reco(const RecoJob* jobs_dev, int njobs, int max_W, int max_H, int max_De, int ctas,
                              cudaStream_t st)
{
    const int nv = (max_De + 1) * (max_De + 1), nslots = (nv + 31) / 32 * 32;
    spiral_plan_kernel<<<dim3(1216, njobs), 32 * kPlanWarps, sizeof(int) * nslots, st>>>(jobs_dev);
    note_launches(1);
    // the limit is that of any depth (the attribute is per function; a launch of
    // another shape must never lower it under this one)
    const int smem_max = (int)(box_bytes(kMaxWords * 32) + (size_t)kRowWords * 256 * (kRecoThreads / 32));
    size_t smem = walk_smem(max_De, nslots, true);
    int ncta = ctas ? ctas : walk_ctas(max_De);
    cudaError_t e = cudaSuccess;
    if (ncta > 1) {
        // a cluster per job, or the largest that the GPU can place
        e = cudaFuncSetAttribute(phase_walk_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
        if (e != cudaSuccess)
            return e;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.blockDim = dim3(kRecoThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        for (; ncta > 1; ncta /= 2) {
            attr[0].val.clusterDim.x = ncta;
            cfg.gridDim = dim3(ncta);
            int nclusters = 0;
            if (cudaOccupancyMaxActiveClusters(&nclusters, phase_walk_kernel<true>, &cfg) == cudaSuccess && nclusters >= 1)
                break;
            cudaGetLastError();
        }
        if (ncta > 1) {
            cfg.gridDim = dim3(njobs * ncta);
            e = cudaLaunchKernelEx(&cfg, phase_walk_kernel<true>, jobs_dev);
            note_launches(1);
        }
    }
    if (ncta <= 1) {
        e = cudaFuncSetAttribute(phase_walk_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
        if (e != cudaSuccess)
            return e;
        smem = walk_smem(max_De, nslots, false);
        phase_walk_kernel<false><<<njobs, kRecoThreads, smem, st>>>(jobs_dev);
        note_launches(1);
    }
    if (e != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess)
        return e;
    const int np = max_W * max_H;
    phase_final_kernel<<<dim3((np + 255) / 256, njobs), 256, 0, st>>>(jobs_dev);
    note_launches(1);
    return cudaGetLastError();
}

} // namespace smip_gpu
