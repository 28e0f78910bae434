// serial_grid.cuh -- the reference's serial fp32 delta formed by a whole
// resident grid.  Included by loopy.cu (it uses the binade arithmetic of
// block_serial_sum and the grid barrier there).
//
// Inside one binade of the running sum each add moves m (s = m U) by an
// increment that depends on m only through its parity, so a run of terms is
// a pair of increments (SumStep) and runs compose.  Every block takes one
// slice of the terms and every warp a part of it; from the slice's f64 prefix
// it guesses the binade(s) the running sum has there -- one, or the two on
// either side of a crossing -- and composes its terms' steps for each guess.
// One warp then walks the slices in order: the walk knows the exact running
// sum, so a slice's pair counts only when it was made for the binade the sum
// is in and the sum stays below the binade's top; otherwise that slice is
// walked warp part by warp part, a part that crosses lane run by lane run, and
// the run that crosses (or a part guessed wrong) is added term by term.  The
// guesses decide the speed, never the value: the result is the one-by-one sum
// bit for bit.
//
// Before, one block of the grid formed the sum while the others waited (600k
// terms 1.1 ms, 80k terms after an interval narrowed from the terms' errors
// had not decided).  Now 80k terms (79 blocks) take 50 us and 600k terms (782
// blocks) 70 us, two sums at once the same: half of it the walk, a few
// thousand cycles for each of the half dozen slices that cross, the rest four
// grid barriers.  10M terms: 0.5 ms.
#pragma once

// doubles of scratch per block behind the grid's 2 x G delta partials: two
// sums' slice sum, record, warps' pairs and lanes' pairs
constexpr uint32_t kSumScratch = 2 * (1 + 4 + 16 + 512);
constexpr int32_t kAnyUnit = 0x7fffffff;   // an empty slice: nothing to add in any binade

constexpr uint32_t kSumBlocks = 1184;   // eight per SM: bounds the scratch

struct SumRec {
    int32_t ua, ub;   // unit exponents the two pairs were made for
    SumStep a, b;
    uint32_t pad[2];
};
static_assert(sizeof(SumRec) == 32, "two 16-byte loads");

// the scratch arrays of sum j (0: the check's terms, 1: the previous check's)
struct SumScr {
    double *slice;   // [G]
    SumRec *rec;     // [G]
    uint4 *part;     // [G][8] the warps' pairs: a.e, a.o, b.e, b.o
    uint4 *lane;     // [G][8][32] the lanes' pairs
    __device__ SumScr(double *partials, uint32_t G, int j) {
        double *base = partials + 2 * (size_t)gridDim.x;
        slice = base + (size_t)j * G;
        rec = reinterpret_cast<SumRec *>(base + 2 * (size_t)G) + (size_t)j * G;
        part = reinterpret_cast<uint4 *>(base + 10 * (size_t)G) + (size_t)j * G * 8;
        lane = reinterpret_cast<uint4 *>(base + 42 * (size_t)G) + (size_t)j * G * 256;
    }
};

// unit exponent of the binade of a positive double, within fp32's range
__device__ __forceinline__ int32_t sum_unit(double s) {
    if (!(s >= 0x1p-126)) return -149;
    return min(ilogb(s), 127) - 23;
}

// The units guessed for a slice with f64 prefix P and sum `own` among n terms:
// the fp32 sum lies within n 2^-24 of the prefix (a half at most).  From 5.6M
// terms on that can span three binades; a slice inside one then takes its own
// and the nearer neighbour's, which leaves a drift of 29 % or more to either
// side unguessed.  The lowest and the highest of the three, without the
// prefix's own, made 10M terms take 46 ms; a third pair made every sum's code,
// and the loop around it, spill (40,000 edges of 2 states 2.4 % slower).
__device__ __forceinline__ void sum_guess(double P, double own, uint64_t n, int32_t &ua, int32_t &ub) {
    const double wide = fmin(0.5, (double)n * 0x1p-24);
    ua = sum_unit(P * (1.0 - wide));
    ub = sum_unit((P + own) * (1.0 + wide));
    if (wide > 1.0 / 3.0 && ub - ua >= 2) {
        ua = sum_unit(P);
        ub = sum_unit(P + own);
        if (ua == ub) {
            if (sum_unit(P * 0x1.6a09e667f3bcdp+0) == ua) ua -= 1;   // P below sqrt(2) of its binade
            else ub += 1;
        }
    }
}

// sum_term's pair without its branches: term t added in the binade with unit
// 2^eu; an inf saturates
__device__ __forceinline__ SumStep sum_step(float t, int32_t eu) {
    const uint32_t tb = __float_as_uint(t), Et = (tb >> 23) & 0xffu;
    const uint32_t Mt = Et ? ((tb & 0x7fffffu) | 0x800000u) : (tb & 0x7fffffu);
    const int32_t shift = (Et ? (int32_t)Et - 150 : -149) - eu;
    const uint32_t sh = (uint32_t)min(max(-shift, 0), 31);
    const uint32_t one = 1u << sh, half = one >> 1, rem = Mt & (one - 1u);
    uint32_t fl = shift > 0 ? (shift >= 7 ? kSumSat : min(Mt << shift, kSumSat)) : Mt >> sh;
    if (Mt == 0u) fl = 0u;
    if (Et == 0xffu) fl = kSumSat;
    const uint32_t tie = half != 0u && rem == half ? 1u : 0u, up = rem > half ? 1u : 0u;
    SumStep st;
    st.e = fl + (up | (tie & fl & 1u));
    st.o = fl + (up | (tie & ~fl & 1u));
    return st;
}

// terms x[lo, hi) in order, composed for unit exponents ua and ub; lane 0 of
// the warp gets the pairs.  Each lane takes a run of them, four loads ahead,
// and leaves its run's pairs in `lanes`.
__device__ __forceinline__ void warp_sum_steps(const float *__restrict__ x, uint64_t lo, uint64_t hi, int32_t ua,
                                               int32_t ub, SumStep &A, SumStep &B, uint4 *lanes) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t k = (hi - lo + 31u) / 32u;
    const uint64_t p0 = min(lo + lane * k, hi), p1 = min(p0 + k, hi);
    A = B = SumStep{0u, 0u};
    float t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = p0 + i < p1 ? __ldcg(x + p0 + i) : 0.0f;
#pragma unroll 1
    for (uint64_t p = p0; p < p1; p += 4) {
        float n[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) n[i] = p + 4 + i < p1 ? __ldcg(x + p + 4 + i) : 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            A = sum_compose(A, sum_step(t[i], ua));   // a 0 past the end adds nothing
            if (ub != ua) B = sum_compose(B, sum_step(t[i], ub));
            t[i] = n[i];
        }
    }
    if (ub == ua) B = A;
    lanes[lane] = make_uint4(A.e, A.o, B.e, B.o);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        SumStep oa, ob;
        oa.e = __shfl_down_sync(0xffffffffu, A.e, d);
        oa.o = __shfl_down_sync(0xffffffffu, A.o, d);
        ob.e = __shfl_down_sync(0xffffffffu, B.e, d);
        ob.o = __shfl_down_sync(0xffffffffu, B.o, d);
        if ((lane & (2u * d - 1u)) == 0u) {
            A = sum_compose(A, oa);
            B = sum_compose(B, ob);
        }
    }
}

// a float's binade: unit exponent, m, and the m the binade ends at
__device__ __forceinline__ void sum_split(float s, int32_t &eu, uint32_t &m, uint32_t &top, uint32_t &Es) {
    const uint32_t sb = __float_as_uint(s);
    Es = sb >> 23;
    eu = Es ? (int32_t)Es - 150 : -149;
    m = Es ? ((sb & 0x7fffffu) | 0x800000u) : sb;
    top = Es ? 0x1000000u : 0x800000u;
}

__device__ __forceinline__ float sum_join(uint32_t Es, uint32_t m) {
    return __uint_as_float((Es << 23) + m - (Es ? 0x800000u : 0u));
}

// s plus the terms x[lo, hi), one add after another; a whole warp, the same s
// in every lane.  The terms go through 128 floats of shared memory, so that
// the chain is the adds alone (out of shuffles it took 32 cycles a term).
__device__ __forceinline__ float warp_serial_add(float s, const float *__restrict__ x, uint64_t lo, uint64_t hi,
                                                 float *buf) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 1
    for (uint64_t p = lo; p < hi; p += 128) {
        float t[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint64_t k = p + 32u * i + lane;
            t[i] = k < hi ? __ldcg(x + k) : 0.0f;   // adding 0 past the end leaves s as it is
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) buf[32u * i + lane] = t[i];
        __syncwarp();
        const uint32_t n = (uint32_t)min(hi - p, (uint64_t)128);
#pragma unroll 1
        for (uint32_t k = 0; k < n; k += 32) {
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const float4 *>(buf + k + 4 * i);
#pragma unroll
            for (int i = 0; i < 8; ++i) s = FADD(FADD(FADD(FADD(s, v[i].x), v[i].y), v[i].z), v[i].w);
        }
    }
    return s;
}

// the pairs of 32 consecutive runs (lane l: its run's, for the binade the sum
// s is in) from run `pos` on, applied up to the first that leaves the binade
// or has no pair for it; returns that run (32: none)
__device__ __forceinline__ uint32_t warp_sum_apply(float &s, uint32_t pos, bool any, int32_t ua, int32_t ub, SumStep a,
                                                   SumStep b) {
    const uint32_t lane = threadIdx.x & 31u;
    int32_t eu;
    uint32_t m, top, Es;
    sum_split(s, eu, m, top, Es);
    SumStep inc{0u, 0u};
    if (lane >= pos && !any) inc = ua == eu ? a : (ub == eu ? b : SumStep{kSumSat, kSumSat});
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        SumStep o;
        o.e = __shfl_up_sync(0xffffffffu, inc.e, d);
        o.o = __shfl_up_sync(0xffffffffu, inc.o, d);
        if ((int)lane >= d) inc = sum_compose(o, inc);
    }
    const uint32_t ma = sum_apply(m, inc);
    const uint32_t fails = __ballot_sync(0xffffffffu, ma >= top);
    const uint32_t f = fails ? (uint32_t)__ffs(fails) - 1u : 32u;
    if (f > pos) s = sum_join(Es, __shfl_sync(0xffffffffu, ma, f - 1));
    return f;
}

__device__ __forceinline__ bool sum_is_inf(float s) { return __float_as_uint(s) >> 23 >= 0xffu; }

// the walk over the slices (one warp; see the file header)
__device__ float warp_sum_walk(const float *__restrict__ x, uint64_t n, uint64_t L, uint64_t LW, uint32_t nw,
                               const SumScr &scr, uint32_t G, float *buf) {
    const uint32_t lane = threadIdx.x & 31u;
    float s = 0.0f;
    const uint4 none = make_uint4((uint32_t)kAnyUnit, 0, 0, 0);
    auto record = [&](uint32_t k, int half) {
        return k < G ? __ldcg(reinterpret_cast<const uint4 *>(scr.rec + k) + half) : none;
    };
    uint4 n0 = record(lane, 0), n1 = record(lane, 1);
    for (uint32_t base = 0; base < G; base += 32) {
        const uint32_t cnt = min(32u, G - base);
        SumRec r;
        r.ua = (int32_t)n0.x;
        r.ub = (int32_t)n0.y;
        r.a = SumStep{n0.z, n0.w};
        r.b = SumStep{n1.x, n1.y};
        n0 = record(base + 32 + lane, 0);   // the next 32 records, while these are walked
        n1 = record(base + 32 + lane, 1);
        for (uint32_t pos = 0; pos < cnt;) {
            if (sum_is_inf(s)) return s;   // inf stays
            const uint32_t f = warp_sum_apply(s, pos, r.ua == kAnyUnit, r.ua, r.ub, r.a, r.b);
            if (f >= cnt) break;
            pos = f + 1;
            // slice base + f, one warp's part after another
            const uint32_t b = base + f;
            const uint64_t lo = min(n, (uint64_t)b * L), hi = min(n, lo + L);
            const int32_t ua = __shfl_sync(0xffffffffu, r.ua, f), ub = __shfl_sync(0xffffffffu, r.ub, f);
            const uint4 part = lane < nw ? __ldcg(scr.part + (size_t)b * 8 + lane) : make_uint4(0, 0, 0, 0);
            for (uint32_t w = 0; w < nw; ++w) {
                const uint64_t p0 = min(hi, lo + w * LW), p1 = min(hi, p0 + LW);
                if (p0 >= p1) break;
                int32_t eu;
                uint32_t m, top, Es;
                sum_split(s, eu, m, top, Es);
                if (Es >= 0xffu) return s;
                if (ua != eu && ub != eu) {
                    s = warp_serial_add(s, x, p0, p1, buf);
                    continue;
                }
                SumStep st;
                st.e = __shfl_sync(0xffffffffu, ua == eu ? part.x : part.z, w);
                st.o = __shfl_sync(0xffffffffu, ua == eu ? part.y : part.w, w);
                const uint32_t mw = sum_apply(m, st);
                if (mw < top) {
                    s = sum_join(Es, mw);
                    continue;
                }
                // the part crosses: its lanes' runs, the crossing one term by term
                const uint4 lp = __ldcg(scr.lane + ((size_t)b * 8 + w) * 32 + lane);
                const uint64_t k = (p1 - p0 + 31u) / 32u;
                for (uint32_t q = 0; q < 32u;) {
                    if (sum_is_inf(s)) return s;
                    const uint32_t g = warp_sum_apply(s, q, false, ua, ub, SumStep{lp.x, lp.y}, SumStep{lp.z, lp.w});
                    if (g >= 32u) break;
                    const uint64_t q0 = min(p0 + g * k, p1), q1 = min(q0 + k, p1);
                    s = warp_serial_add(s, x, q0, q1, buf);
                    q = g + 1;
                    sum_split(s, eu, m, top, Es);
                    if (q < 32u && ua != eu && ub != eu) {   // a binade nobody guessed: the rest one by one
                        s = warp_serial_add(s, x, q1, p1, buf);
                        break;
                    }
                }
            }
        }
    }
    return s;
}

// the serial sums of x0[0, n) and, when x1 is not null, of x1[0, n), by the
// whole grid (at most 8 warps per block); every thread gets them.  false when
// a barrier gave up.
template <int NT>
__device__ __noinline__ bool grid_serial_sums(double *partials, const float *x0, const float *x1, uint64_t n,
                                              LoopyCtl *ctl, GridBar &gb, uint32_t *s_fail, double *red, float &sum0,
                                              float &sum1) {
    static_assert(NT <= 256, "eight warps' pairs per block");
    constexpr uint32_t NW = NT / 32;
    __shared__ uint4 s_part[2][NW];
    __shared__ __align__(16) float s_add[2][128];
    // the first kSumBlocks blocks take a slice each
    const uint32_t G = min(gridDim.x, kSumBlocks), b = blockIdx.x, tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    const bool grid = gridDim.x > 1;
    const uint64_t L = ((n + G - 1) / G + 3) & ~3ull, LW = (L + NW - 1) / NW;
    const uint64_t lo = min(n, (uint64_t)b * L), hi = min(n, lo + L);
    const int nsum = x1 ? 2 : 1;
    double own[2] = {0.0, 0.0};
    for (int j = 0; b < G && j < nsum; ++j) {
        const float *x = j ? x1 : x0;
        double v = 0.0;
#pragma unroll 4
        for (uint64_t k = lo + tid; k < hi; k += NT) v += (double)__ldcg(x + k);
        own[j] = broadcast_sum(block_sum<NT>(v, red));
        if (tid == 0) SumScr(partials, G, j).slice[b] = own[j];
    }
    if (grid && !grid_barrier(gb, s_fail)) return false;
    for (int j = 0; b < G && j < nsum; ++j) {
        const SumScr scr(partials, G, j);
        double v = 0.0;
        for (uint32_t k = tid; k < b; k += NT) v += __ldcg(scr.slice + k);
        const double P = broadcast_sum(block_sum<NT>(v, red));
        int32_t ua, ub;
        sum_guess(P, own[j], n, ua, ub);
        const uint64_t p0 = min(hi, lo + w * LW), p1 = min(hi, p0 + LW);
        SumStep A, B;
        warp_sum_steps(j ? x1 : x0, p0, p1, ua, ub, A, B, scr.lane + ((size_t)b * 8 + w) * 32);
        if (lane == 0) {
            const uint4 r = make_uint4(A.e, A.o, B.e, B.o);
            s_part[j][w] = r;
            scr.part[(size_t)b * 8 + w] = r;
        }
        __syncthreads();
        if (tid == 0) {
            SumRec r;
            r.a = r.b = SumStep{0u, 0u};
            for (uint32_t k = 0; k < NW; ++k) {
                r.a = sum_compose(r.a, SumStep{s_part[j][k].x, s_part[j][k].y});
                r.b = sum_compose(r.b, SumStep{s_part[j][k].z, s_part[j][k].w});
            }
            r.ua = lo < hi ? ua : kAnyUnit;
            r.ub = ub;
            r.pad[0] = r.pad[1] = 0;
            scr.rec[b] = r;
        }
    }
    if (grid) {
        if (!grid_barrier(gb, s_fail)) return false;
    } else {
        __syncthreads();
    }
    if (b == 0 && w < (uint32_t)nsum) {
        const float s = warp_sum_walk(w ? x1 : x0, n, L, LW, NW, SumScr(partials, G, (int)w), G, s_add[w]);
        if (lane == 0) {
            if (w) ctl->fb_p = s;
            else ctl->fb_s = s;
        }
    }
    if (grid) {
        if (!grid_barrier(gb, s_fail)) return false;
    } else {
        __syncthreads();
    }
    sum0 = *(volatile float *)&ctl->fb_s;
    sum1 = x1 ? *(volatile float *)&ctl->fb_p : 0.0f;
    return true;
}

// the narrowed intervals of an undecided check in the one-launch loop,
// grid-wide: each block takes one slice of the terms (of s, and of the
// previous delta when that is neither exact nor narrowed yet); slice sums,
// a barrier, each slice's errors from its exact prefix, a barrier, and
// every block sums the same slices in the same order, so all blocks end with
// the same intervals.  xs: the check's terms, xp: the previous check's.
// Scratch: 8 doubles per block after the partials (the sums' own scratch,
// not in use yet).  false when a barrier gave up.
template <int NT>
__device__ __noinline__ bool grid_refine(double *partials, const float *xs, const float *xp, uint64_t n, float tol,
                                         GridBar &gb, uint32_t *s_fail, SerialCheck &x, double *red) {
    constexpr uint32_t cap = 8 * NT;
    __shared__ __align__(16) float buf[cap];
    __shared__ double s_b[4];
    __shared__ double s_v[NT / 32][6];
    __shared__ double s_t[6];
    const double c0 = refine_c0(n);
    if (c0 == 0.0) return true;
    const bool do_p = !x.p_exact && !x.p_ref;
    ++x.refines;
    const uint32_t G = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
    double *scr = partials + 2 * (size_t)G;
    const uint64_t L = ((n + G - 1) / G + 3) & ~3ull;
    const uint64_t lo = min(n, (uint64_t)b * L), hi = min(n, lo + L);
    double ls = 0.0, lp = 0.0;
    for (uint64_t k = lo + tid; k < hi; k += NT) {
        ls += (double)__ldcg(xs + k);
        if (do_p) lp += (double)__ldcg(xp + k);
    }
    ls = block_sum<NT>(ls, red);
    lp = block_sum<NT>(lp, red);
    if (tid == 0) {
        scr[b] = ls;
        scr[G + b] = lp;
    }
    if (gridDim.x > 1) {
        if (!grid_barrier(gb, s_fail)) return false;
    } else {
        __syncthreads();
    }
    // prefixes before this slice, and the totals (the same in every block)
    double ps = 0.0, ts = 0.0, pp = 0.0, tp = 0.0;
    for (uint32_t k = tid; k < G; k += NT) {
        const double vs = __ldcg(scr + k), vp = __ldcg(scr + G + k);
        ts += vs;
        tp += vp;
        if (k < b) {
            ps += vs;
            pp += vp;
        }
    }
    ps = block_sum<NT>(ps, red);
    ts = block_sum<NT>(ts, red);
    pp = block_sum<NT>(pp, red);
    tp = block_sum<NT>(tp, red);
    if (tid == 0) {
        s_b[0] = ps;
        s_b[1] = ts;
        s_b[2] = pp;
        s_b[3] = tp;
    }
    __syncthreads();
    ps = s_b[0];
    ts = s_b[1];
    pp = s_b[2];
    tp = s_b[3];
    double pe;
    const Refine rs = refine_segment<NT>(xs, lo, hi, ps, c0, buf, cap, pe);
    Refine rp{0.0, 0.0, 0.0, false};
    if (do_p) rp = refine_segment<NT>(xp, lo, hi, pp, c0, buf, cap, pe);
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    if (tid == 0) {
        scr[2 * (size_t)G + b] = rs.E;
        scr[3 * (size_t)G + b] = rs.A;
        scr[4 * (size_t)G + b] = rs.bad ? inf : rs.B;
        scr[5 * (size_t)G + b] = rp.E;
        scr[6 * (size_t)G + b] = rp.A;
        scr[7 * (size_t)G + b] = rp.bad ? inf : rp.B;
    }
    if (gridDim.x > 1) {
        if (!grid_barrier(gb, s_fail)) return false;
    } else {
        __syncthreads();
    }
    // the same totals in every block: fixed per-thread slices, then a fixed
    // reduction order; the bounds (j = 2, 5) rounded up
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (uint32_t k = tid; k < G; k += NT) {
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            const double y = __ldcg(scr + (size_t)(2 + j) * G + k);
            v[j] = (j == 2 || j == 5) ? __dadd_ru(v[j], y) : v[j] + y;
        }
    }
#pragma unroll
    for (int j = 0; j < 6; ++j)
        for (int d = 16; d > 0; d >>= 1) {
            const double y = __shfl_xor_sync(0xffffffffu, v[j], d);
            v[j] = (j == 2 || j == 5) ? __dadd_ru(v[j], y) : v[j] + y;
        }
    if ((tid & 31u) == 0u)
        for (int j = 0; j < 6; ++j) s_v[tid >> 5][j] = v[j];
    __syncthreads();
    if (tid == 0)
        for (int j = 0; j < 6; ++j) {
            double t = 0.0;
            for (int w = 0; w < NT / 32; ++w) t = (j == 2 || j == 5) ? __dadd_ru(t, s_v[w][j]) : t + s_v[w][j];
            s_t[j] = t;
        }
    __syncthreads();
    double lo2, hi2;
    const Refine Rs{s_t[0], s_t[1], s_t[2], !(s_t[2] < inf)};
    if (!Rs.bad) {
        refine_interval(ts, Rs, n, lo2, hi2);
        serial_narrow(x, 0, lo2, hi2);
    }
    if (do_p) {
        const Refine Rp{s_t[3], s_t[4], s_t[5], !(s_t[5] < inf)};
        if (!Rp.bad) {
            refine_interval(tp, Rp, n, lo2, hi2);
            serial_narrow(x, 1, lo2, hi2);
        }
    }
    x.d = serial_decide(x.lo, x.hi, x.s_exact, x.plo, x.phi, x.p_exact, tol);
    __syncthreads();   // s_t and s_b are free
    return true;
}

// one serial-mode check of a one-launch loop, undecided by the bounds: the
// interval narrowed from the terms' own errors, then the serial sum of the
// check's terms and, where the previous delta is not exact yet, of the previous
// check's decide.  Narrowing costs two barriers and decides where deltas
// differ (80k terms: 29 us against 50 for the sums; 900k: 45 against 85); where
// they creep it decides nothing, so after one such check (`narrow` false) the
// run goes straight to the sums.  Every block of the grid calls it with the
// same x and narrow.
template <int NT>
__device__ __noinline__ bool grid_serial_form(SerialCheck &x, const float *terms, const float *prev_terms,
                                                 uint64_t n, float tol, LoopyCtl *ctl, double *partials, GridBar &gb,
                                                 uint32_t *s_fail, double *red, bool &narrow) {
    if (narrow) {
        if (!grid_refine<NT>(partials, terms, prev_terms, n, tol, gb, s_fail, x, red)) return false;
        if (x.d >= 0) return true;
        narrow = false;
        if (gridDim.x > 1) {   // the scratch is the sums' now
            if (!grid_barrier(gb, s_fail)) return false;
        } else {
            __syncthreads();
        }
    }
    const float *xp = x.p_exact ? nullptr : prev_terms;
    float s, p;
    if (!grid_serial_sums<NT>(partials, terms, xp, n, ctl, gb, s_fail, red, s, p)) return false;
    x.s = s;
    x.lo = x.hi = (double)s;
    x.s_exact = true;
    x.s_ref = false;
    ++x.sums;
    if (xp) {
        x.plo = x.phi = (double)p;
        x.p_exact = x.p_new = true;
        ++x.sums;
    }
    x.d = serial_decide(x.lo, x.hi, true, x.plo, x.phi, true, tol);
    return true;
}

// the returned delta and previous delta of a finished one-launch run, where
// the loop decided without forming them
template <int NT>
__device__ __noinline__ bool grid_serial_final(LoopyCtl &sc, LoopyCtl *ctl, double *partials, const float *absdiff,
                                                  GridBar &gb, uint32_t *s_fail, double *red) {
    const bool cur = !sc.delta_exact, prev = !sc.prev_exact;
    if (!cur && !prev) return true;
    const float *xc = absdiff + (size_t)sc.cur_buf * sc.ad_stride, *xp = absdiff + (size_t)sc.prev_buf * sc.ad_stride;
    float s, p;
    if (!grid_serial_sums<NT>(partials, cur ? xc : xp, cur && prev ? xp : nullptr, sc.n_terms, ctl, gb, s_fail, red,
                              s, p))
        return false;
    __syncthreads();   // every thread has read sc
    if (threadIdx.x == 0) {
        if (cur) sc.delta_f = s;
        if (prev) sc.prev_f = cur ? p : s;
        sc.delta_exact = sc.prev_exact = 1;
    }
    __syncthreads();
    return true;
}
