// flood_loop.cuh -- small graphs: every iteration of the flooding schedule in
// one cooperative launch, a block per node tile, the tile's data on chip.
// Included by loopy.cu (it uses the tile, control-block, barrier and delta
// machinery there).
//
// When each tile has a block of its own on the GPU at once (a cooperative
// launch guarantees co-residency), an iteration is a chain of latencies: the
// gather of the sources' send buffers, the messages, the products, and a grid
// barrier.  So what does not have to cross blocks never leaves the SM:
//  * the tile's messages live in shared memory for the whole run (the last
//    two, or three with the serial delta), and go to HBM once at the end;
//    source ids too, and tables while few tiles share an SM; beliefs and row
//    ranges live in registers;
//  * the |diff| terms of a serial check are formed from those messages only
//    when a check is undecided, instead of scattered to HBM every iteration;
//  * the barrier is one flag per block: a block stores its own after its send
//    buffers and delta partial, and every block polls all of them, with no
//    atomic and no second hop (kFlagBlocks blocks at most; more meet at the
//    counter barrier);
//  * the next iteration's gathers are issued before the stopping decision of
//    the last one, which then costs no time of its own;
//  * a graph of one tile keeps its send buffers in shared memory and meets
//    nobody.
// A tile whose messages do not fit its block's shared memory runs flood_tile
// on global memory beside the others (its send buffers cross blocks the same
// way).
//
// Each edge belongs to the thread k_flood gives it, and the partials are
// summed in k_flood's order, so results and the f64 delta equal the
// one-launch-per-iteration loop's bit for bit.
//
// What bounds it: the instruction stream of the few warps of a tile more than the
// memory, and with the serial delta its spills (20-110 bytes in the wide form of
// 1-4 states at 128 registers, 330-690 in the narrow one):
// 10,000 nodes, 40,000 edges, 2 states take 6.0 us an iteration with the f64
// delta (8.2 before) and 7.5 with the serial one (11.7), 61 nodes of 2-4
// states (one tile) 2.3 and 3.3 (5.7 and 6.8).
#pragma once

// blocks that meet by polling each other's flags: every block reads every
// flag, so the polling traffic grows with the square
constexpr uint32_t kFlagBlocks = 512;

// resident blocks per SM the registers are capped for, and in-edges per
// thread whose gathers are in flight at once: few tiles per SM get the
// registers for more gathers, many get the residency
template <int MS, bool WIDE> constexpr int loop_unroll() { return WIDE ? (MS <= 2 ? 4 : (MS <= 4 ? 2 : 1)) : 1; }
template <int MS, bool WIDE> constexpr int loop_min_blocks() {
    return WIDE ? (MS > 2 && MS <= 4 ? 2 : 4) : (MS <= 2 ? 12 : (MS <= 4 ? 4 : 6));
}
// floats between tables in shared memory: 16-byte rows whose starts fall in
// different banks for eight consecutive edges
template <int MS> constexpr uint32_t loop_table_stride() {
    return (MS * MS) % 4 ? MS * MS : ((MS * MS) % 8 ? MS * MS : (MS == 2 ? 4 : MS * MS + 4));
}

struct LoopArgs {
    FloodArgs f;
    uint32_t *bar;       // the graph's grid barrier
    uint64_t *flags;     // [G] one per block, rising over the runs of a graph
    uint64_t run_tag;    // above every tag of earlier runs; + iteration + 1
    uint32_t smem;       // dynamic shared memory per block, bytes
};

// every block's flag at `tag` or above (this block's is set here); the wait is
// bounded as grid_barrier's, and the same test hook holds a block back: it
// never sets its flag and does not wait at its first barrier
__device__ __forceinline__ bool flag_barrier(LoopyCtl *c, uint64_t *flags, uint64_t tag, bool skip, bool first,
                                             uint32_t wait_ms, uint32_t *s_fail) {
    __syncthreads();
    if (threadIdx.x == 0 && !skip) {
        fence_acq_rel();
        st_relaxed(flags + blockIdx.x, tag);
    }
    if (!(skip && first)) {
#pragma unroll 1
        for (uint32_t k = threadIdx.x; k < gridDim.x; k += blockDim.x) {
            uint64_t t0 = 0;
#pragma unroll 1
            for (uint32_t spin = 0; ld_relaxed(flags + k) < tag; ++spin) {
                if ((spin & 255u) != 255u) continue;
                if (*(volatile uint32_t *)s_fail) break;
                const uint64_t t = global_ns();
                if (t0 == 0) t0 = t;
                if (t - t0 > (wait_ms ? (uint64_t)wait_ms * 1000000ull : kBarrierWaitNs)) {
                    *(volatile uint32_t *)s_fail = 1;
                    atomicExch(&c->bar_fail, 1u);
                    break;
                }
            }
        }
        fence_acq_rel();
    }
    __syncthreads();
    return *(volatile uint32_t *)s_fail == 0;
}

// The steady loop is kept small -- runtime loops not unrolled, everything rare
// out of line -- since a handful of warps per SM run straight through it every
// iteration and wait for instructions otherwise.

// |diff| terms of the tile's message buffers `from` and `to`, at their edge ids
template <int MS, bool UNI>
__device__ __noinline__ void loop_write_terms(float *dst, const float *from, const float *to, const uint32_t *srcs,
                                              const uint32_t *pos_edge, uint32_t ne) {
#pragma unroll 1
    for (uint32_t i = threadIdx.x; i < ne; i += flood_nt<MS>()) {
        const int x = UNI ? MS : (int)(srcs[i] >> 24 & 15u);
        float ad[MS];
#pragma unroll
        for (int k = 0; k < MS; ++k) {
            float d = 0.0f;
            if (UNI || k < x) {
                d = FSUB(from[(size_t)i * MS + k], to[(size_t)i * MS + k]);
                if (d != d) d = 0.0f;
                d = fabsf(d);
            }
            ad[k] = d;
        }
        stv<MS>(dst + (size_t)pos_edge[i] * MS, ad);
    }
}

// flood_tile on global memory, for a tile too large for its block
template <int MS, bool UNI>
__device__ __noinline__ double loop_flood_tile(const FloodArgs &a, bool want, float *absd, uint32_t t, uint32_t mp0,
                                               uint32_t qp0, float *sm) {
    const int mp = (int)((mp0 + t) & 1u), qp = (int)((qp0 + t) & 1u);
    double dsum = 0.0;
    flood_tile<MS, UNI, 1>(a, blockIdx.x, want, absd, mp ? a.msg1 : a.msg0, mp ? a.msg0 : a.msg1, qp ? a.q1 : a.q0,
                           qp ? a.q0 : a.q1, 0, sm, dsum);
    return dsum;
}

// acc *= the messages of positions [r0, r1) in order (combine)
template <int MS, bool UNI>
__device__ __forceinline__ void node_product(const float *m, uint32_t r0, uint32_t r1, int S, float *acc) {
#pragma unroll 1
    for (uint32_t p = r0; p < r1; ++p) {
        float mm[MS];
        ldv<MS>(m + (size_t)p * MS, mm);
        combine<MS, UNI>(acc, mm, S);
    }
}

template <int MS, bool UNI, bool SER, bool WIDE>
__global__ void __launch_bounds__(flood_nt<MS>(), loop_min_blocks<MS, WIDE>()) k_flood_loop(const LoopArgs la) {
    constexpr int NT = flood_nt<MS>();
    constexpr int FU = loop_unroll<MS, WIDE>();
    constexpr uint32_t EMAX = flood_smem_floats<MS>() / MS;
    constexpr uint32_t NB = SER ? 3 : 2;   // message buffers
    constexpr uint32_t TS = loop_table_stride<MS>();
    extern __shared__ __align__(16) unsigned char dyn[];
    constexpr int NW = NT / 32;
    __shared__ double red[NW], red_t[NW], red_b[NW];
    __shared__ LoopyCtl s_ctl;
    __shared__ uint32_t s_fail;

    const FloodArgs &a = la.f;
    LoopyCtl *ctl = a.ctl;
    const uint32_t tid = threadIdx.x, G = gridDim.x;
    GridBar gb(ctl, la.bar);
    if (tid == 0) {
        s_ctl = *ctl;
        s_fail = 0;
    }
    // the tile: nodes [v0, vend), positions [e0, e1)
    const uint32_t v0 = blockIdx.x * NT, vend = min(v0 + NT, a.V), v = v0 + tid;
    const bool has = v < a.V, solo = G == 1;
    const uint32_t e0 = a.in_ptr[v0], e1 = a.in_ptr[vend], ne = e1 - e0;
    // dynamic shared memory: [send buffers of a lone tile][messages][source
    // ids][tables], as far as they fit.  A tile of more than EMAX in-edges
    // keeps k_flood's chunks, whose edge-to-thread assignment starts over at
    // each chunk, unless a chunk is a whole number of rounds.
    float *const qs = reinterpret_cast<float *>(dyn);
    const uint32_t q_fl = solo ? 2u * NT * MS : 0u;
    float *const ms = qs + q_fl;
    const uint32_t m_fl = (NB * ne * MS + 3u) & ~3u;
    uint32_t *const srcs = reinterpret_cast<uint32_t *>(ms + m_fl);
    const uint32_t s_fl = (ne + 3u) & ~3u;
    float *const js = reinterpret_cast<float *>(srcs + s_fl);
    const bool resident = (EMAX % NT == 0 || ne <= EMAX) &&
                          4ull * (q_fl + (uint64_t)NB * ne * MS + 4u + s_fl) <= la.smem;
    const bool tables = resident && 4ull * (q_fl + (uint64_t)m_fl + s_fl + (uint64_t)TS * ne) <= la.smem;

    uint32_t r0 = 0, r1 = 0;
    int S = MS;
    float b[MS];
#pragma unroll
    for (int i = 0; i < MS; ++i) b[i] = 0.0f;
    if (has) {
        r0 = a.in_ptr[v] - e0;
        r1 = a.in_ptr[v + 1] - e0;
        if (!UNI) S = a.node_s[v];
    }
    __syncthreads();
    const uint32_t mp0 = s_ctl.msg_parity0 & 1u, qp0 = s_ctl.q_parity0 & 1u, ce = s_ctl.check_every;
    // the terms of a check are formed from the messages on chip when every
    // iteration is checked; else each check writes them
    const bool lazy = resident && ce <= 1;
    if (resident) {
        if (has) ldv<MS>(a.belief + (size_t)v * MS, b);
        const float *m0 = mp0 ? a.msg1 : a.msg0;
#pragma unroll 1
        for (uint32_t i = tid; i < ne; i += NT) {
            // the state counts beside the source (node ids of a graph this
            // small are below 2^24)
            uint32_t sv = a.in_src[e0 + i];
            if (!UNI) sv |= (uint32_t)a.pos_dims[e0 + i] << 24;
            srcs[i] = sv;
            float m[MS];
            ldv<MS>(m0 + (size_t)(e0 + i) * MS, m);
            stv<MS>(ms + (size_t)i * MS, m);
            if (tables) {
                if constexpr (MS * MS <= 16) {
                    float j[MS * MS];
                    ldv<MS * MS, kStream>(a.joint + (size_t)(e0 + i) * (MS * MS), j);
                    stv<MS * MS>(js + (size_t)i * TS, j);
                } else {
#pragma unroll
                    for (int k = 0; k < MS; ++k) {
                        float j[MS];
                        ldv<MS, kStream>(a.joint + (size_t)(e0 + i) * (MS * MS) + k * MS, j);
                        stv<MS>(js + (size_t)i * TS + k * MS, j);
                    }
                }
            }
        }
        if (solo && has) {
            float q[MS];
            ldv<MS>((qp0 ? a.q1 : a.q0) + (size_t)v * MS, q);
            stv<MS>(qs + (size_t)(qp0 * NT + tid) * MS, q);
        }
    }
    __syncthreads();

    auto write_terms = [&](float *dst, const float *from, const float *to) {
        loop_write_terms<MS, UNI>(dst, from, to, srcs, a.pos_edge + e0, ne);
    };

    // the decision's running state, the same in every thread of every block:
    // each thread takes each decision itself, and the control block is
    // written once at the end
    const uint32_t max_it = s_ctl.max_it, wait_ms = s_ctl.wait_ms;
    const float tol = s_ctl.tol;
    const bool skip = s_ctl.bar_skip == blockIdx.x + 1u;
    // f64 sum, interval of the serial sum, whether it is the sum itself and
    // its check: of the last check (d) and of the one before (p), which stays
    // where it is at the last allowed iteration, as the reference's does
    double d_d = 0.0, dlo = 0.0, dhi = 0.0, p_d = s_ctl.prev_d, plo = s_ctl.plo, phi = s_ctl.phi;
    float d_f = 0.0f, p_f = s_ctl.prev_f;
    bool d_exact = true, p_exact = true, stop = false;
    uint32_t d_buf = 0, p_buf = 0, sums = 0, refines = 0, it = 0;
    bool narrow = true, d_ref = false, p_ref = false;   // intervals narrowed
    double tot = 0.0;   // a lone tile's sum needs no exchange
    uint32_t cur = 0;   // buffer of the latest messages
    bool ok = true;
    for (uint32_t t = 0;; ++t) {
        const uint32_t qp = (qp0 + t) & 1u;
        const float *q_in = qp ? a.q1 : a.q0;
        float *q_out = qp ? a.q0 : a.q1;
        // the first round's gathers, before the last iteration's decision
        float q[FU][MS];
        auto gather = [&](uint32_t i, float *o) {
            const uint32_t s = UNI ? srcs[i] : srcs[i] & 0xffffffu;
            if (solo) {
                ldv<MS>(qs + (size_t)(qp * NT + s) * MS, o);
            } else {
                const float *p = q_in + (size_t)s * MS;
                if constexpr (MS % 4 == 0) {
#pragma unroll
                    for (int k = 0; k < MS / 4; ++k) {
                        const float4 w = __ldcg(reinterpret_cast<const float4 *>(p) + k);
                        o[4 * k] = w.x; o[4 * k + 1] = w.y; o[4 * k + 2] = w.z; o[4 * k + 3] = w.w;
                    }
                } else if constexpr (MS % 2 == 0) {
#pragma unroll
                    for (int k = 0; k < MS / 2; ++k) {
                        const float2 w = __ldcg(reinterpret_cast<const float2 *>(p) + k);
                        o[2 * k] = w.x; o[2 * k + 1] = w.y;
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < MS; ++k) o[k] = __ldcg(p + k);
                }
            }
        };
        if (resident) {
#pragma unroll
            for (int u = 0; u < FU; ++u)
                if (tid + u * NT < ne) gather(tid + u * NT, q[u]);
        }
        if (t) {
            // the decision of iteration t - 1 (the reference's stopping rule)
            const bool want = (ce <= 1) || (t % ce == 0);
            if (!solo && want) {
                const double *part = a.partials + (size_t)((t - 1) & 1u) * G;
                double acc = 0.0;
#pragma unroll 1
                for (uint32_t k = tid; k < G; k += NT) acc += __ldcg(part + k);
                acc = warp_sum(acc);
                if ((tid & 31u) == 0) red_t[tid >> 5] = acc;
                __syncthreads();
                tot = warps_total<NW>(red_t);
            }
            it = t;
            if (want) {
                if (t > ce) {
                    p_d = d_d;
                    p_f = d_f;
                    plo = dlo;
                    phi = dhi;
                    p_exact = d_exact;
                    p_ref = d_ref;
                    p_buf = d_buf;
                }
                d_d = tot;
                d_f = (float)tot;
                if constexpr (SER) {
                    SerialCheck x;
                    x.T = tot;
                    x.plo = plo;
                    x.phi = phi;
                    x.p_exact = p_exact;
                    x.p_ref = p_ref;
                    x.s_exact = x.s_ref = x.p_new = false;
                    x.sums = x.refines = 0;
                    x.cb = d_buf = check_index(t - 1, ce) % 3u;
                    x.s = d_f;
                    serial_interval(tot, s_ctl.n_terms, x.lo, x.hi);
                    x.d = serial_decide(x.lo, x.hi, false, plo, phi, p_exact, tol);
                    if (x.d < 0) {
                        float *const tc = a.absdiff + (size_t)d_buf * s_ctl.ad_stride;
                        float *const tp = a.absdiff + (size_t)p_buf * s_ctl.ad_stride;
                        if (lazy) {
                            const uint32_t p1 = (cur + 2u) % 3u, p2 = (cur + 1u) % 3u;
                            write_terms(tc, ms + (size_t)p1 * ne * MS, ms + (size_t)cur * ne * MS);
                            if (!p_exact) write_terms(tp, ms + (size_t)p2 * ne * MS, ms + (size_t)p1 * ne * MS);
                        }
                        if (solo) __syncthreads();
                        else if (ce <= 1) ok = grid_barrier(gb, &s_fail);
                        ok = ok && grid_serial_form<NT>(x, tc, tp, s_ctl.n_terms, tol, ctl, a.partials, gb, &s_fail,
                                                         red_b, narrow);
                        refines += x.refines;
                        if (!ok) break;
                        if (x.p_exact) p_f = (float)x.plo;
                        plo = x.plo;
                        phi = x.phi;
                        p_exact = x.p_exact;
                        p_ref = x.p_ref;
                        sums += x.sums;
                    }
                    d_f = x.s;
                    dlo = x.lo;
                    dhi = x.hi;
                    d_exact = x.s_exact;
                    d_ref = x.s_ref;
                    stop = x.d == 1;
                } else {
                    stop = tot < (double)tol || fabs(tot - p_d) < (double)tol;
                }
                if (stop) break;
            }
            if ((ce <= 1 || want) && t >= max_it) break;
        }
        const bool want = (ce <= 1) || ((t + 1) % ce == 0);
        float *absd = SER && !lazy && want ? a.absdiff + (size_t)(check_index(t, ce) % 3u) * s_ctl.ad_stride : nullptr;
        double dsum = 0.0;
        if (!resident) {
            dsum = loop_flood_tile<MS, UNI>(a, want, absd, t, mp0, qp0, reinterpret_cast<float *>(dyn));
        } else {
            const float *mo = ms + (size_t)cur * ne * MS;
            cur = cur + 1u == NB ? 0u : cur + 1u;
            float *mn = ms + (size_t)cur * ne * MS;
#pragma unroll 1
            for (uint32_t base = tid; base < ne; base += NT * FU) {
                if (base != tid) {
#pragma unroll
                    for (int u = 0; u < FU; ++u)
                        if (base + u * NT < ne) gather(base + u * NT, q[u]);
                }
#pragma unroll
                for (int u = 0; u < FU; ++u) {
                    const uint32_t i = base + u * NT;
                    if (i >= ne) break;
                    const uint32_t sv = UNI ? 0u : srcs[i];
                    const int x = UNI ? MS : (int)(sv >> 24 & 15u), y = UNI ? MS : (int)(sv >> 28);
                    float m[MS], o[MS];
                    ldv<MS>(mo + (size_t)i * MS, o);
                    if (tables) {
                        if constexpr (MS * MS <= 16) {
                            float j[MS * MS];
                            ldv<MS * MS>(js + (size_t)i * TS, j);
                            send_msg_regs<MS, UNI>(j, q[u], x, y, m);
                        } else {
                            send_msg_rows<MS, UNI>(js + (size_t)i * TS, q[u], x, y, m);
                        }
                    } else {
                        send_msg<MS, UNI>(a.joint + (size_t)(e0 + i) * (MS * MS), q[u], x, y, m);
                    }
                    stv<MS>(mn + (size_t)i * MS, m);
                    if (want) {
                        float ad[MS];
#pragma unroll
                        for (int k = 0; k < MS; ++k) {
                            float d = 0.0f;
                            if (UNI || k < x) {
                                d = FSUB(o[k], m[k]);
                                if (d != d) d = 0.0f;
                                d = fabsf(d);
                            }
                            ad[k] = d;
                            dsum += (double)d;
                        }
                        if (SER && absd) stv<MS>(absd + (size_t)a.pos_edge[e0 + i] * MS, ad);
                    }
                }
            }
        }
        dsum = warp_sum(dsum);
        if ((tid & 31u) == 0) red[tid >> 5] = dsum;
        __syncthreads();
        if (resident) {
            // the node: marginalise, then the next send buffer (flood_tile's
            // phase 2)
            const float *mn = ms + (size_t)cur * ne * MS;
            if (has) {
                float prod[MS];
#pragma unroll
                for (int i = 0; i < MS; ++i) prod[i] = 1.0f;
                node_product<MS, UNI>(mn, r0, r1, S, prod);
                if (r1 > r0) {
#pragma unroll
                    for (int i = 0; i < MS; ++i)
                        if (UNI || i < S) b[i] = FMUL(b[i], prod[i]);
                }
                normalise<MS, UNI>(b, S);
                float qo[MS];
#pragma unroll
                for (int i = 0; i < MS; ++i) qo[i] = b[i];
                node_product<MS, UNI>(mn, r0, r1, S, qo);
                if (solo) stv<MS>(qs + (size_t)((qp ^ 1u) * NT + tid) * MS, qo);
                else stv<MS>(q_out + (size_t)v * MS, qo);
            }
        }
        if (solo) tot = warps_total<NW>(red);
        else if (tid == 0) a.partials[(size_t)(t & 1u) * G + blockIdx.x] = warps_total<NW>(red);
        if (solo) __syncthreads();
        else if (G <= kFlagBlocks) ok = flag_barrier(ctl, la.flags, la.run_tag + t + 1u, skip, t == 0, wait_ms, &s_fail);
        else ok = grid_barrier(gb, &s_fail);
        if (!ok) break;
    }

    // the reference's loop variables at exit (graph.c:1313-1318; _acc:
    // :1410-1414), which finalize_with keeps iteration by iteration
    if (tid == 0 && ok) {
        s_ctl.it = it;
        s_ctl.done = stop ? 1u : 2u;
        if (ce <= 1) {
            s_ctl.ret = s_ctl.final_i = stop ? it - 1u : max_it;
        } else {
            s_ctl.num_iter = stop ? it - ce : it;
            s_ctl.ret = s_ctl.num_iter;
            s_ctl.final_i = stop ? it - ce : it;
            if (!stop) {   // the _acc loop keeps the last check as the previous one too
                p_d = d_d;
                p_f = d_f;
                plo = dlo;
                phi = dhi;
                p_buf = d_buf;
            }
        }
        s_ctl.delta_f = d_f;
        s_ctl.delta_d = d_d;
        s_ctl.prev_f = p_f;
        s_ctl.prev_d = p_d;
        if (SER) {
            s_ctl.delta_exact = d_exact;
            s_ctl.prev_exact = ce > 1 && !stop ? d_exact : p_exact;
            s_ctl.cur_buf = d_buf;
            s_ctl.prev_buf = p_buf;
            s_ctl.serial_sums = sums;
            s_ctl.serial_refines = refines;
        }
    }
    __syncthreads();
    if (ok && SER) {
        // the returned deltas where the loop decided without them
        if (lazy) {
            const uint32_t p1 = (cur + 2u) % 3u, p2 = (cur + 1u) % 3u;
            if (!s_ctl.delta_exact)
                write_terms(a.absdiff + (size_t)s_ctl.cur_buf * s_ctl.ad_stride, ms + (size_t)p1 * ne * MS,
                            ms + (size_t)cur * ne * MS);
            if (!s_ctl.prev_exact)
                write_terms(a.absdiff + (size_t)s_ctl.prev_buf * s_ctl.ad_stride, ms + (size_t)p2 * ne * MS,
                            ms + (size_t)p1 * ne * MS);
        }
        if (!s_ctl.delta_exact || !s_ctl.prev_exact) {
            if (solo) __syncthreads();
            else ok = grid_barrier(gb, &s_fail);
            ok = ok && grid_serial_final<NT>(s_ctl, ctl, a.partials, a.absdiff, gb, &s_fail, red_b);
        }
    }
    if (ok && resident) {
        float *ml = ((mp0 + it) & 1u) ? a.msg1 : a.msg0, *mo = ((mp0 + it) & 1u) ? a.msg0 : a.msg1;
        const uint32_t old = cur ? cur - 1u : NB - 1u;
#pragma unroll 1
        for (uint32_t i = tid; i < ne; i += NT) {
            float m[MS];
            ldv<MS>(ms + ((size_t)cur * ne + i) * MS, m);
            stv<MS>(ml + (size_t)(e0 + i) * MS, m);
            ldv<MS>(ms + ((size_t)old * ne + i) * MS, m);
            stv<MS>(mo + (size_t)(e0 + i) * MS, m);
        }
        if (has) stv<MS>(a.belief + (size_t)v * MS, b);
    }
    if (blockIdx.x == 0 && tid == 0 && !s_fail) publish_ctl(ctl, s_ctl);
}
