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
// 10,000 nodes, 40,000 edges, 2 states, per iteration: 8.2 -> 7.0 us with the
// f64 delta, 11.7 -> 8.2 us with the serial one; 61 nodes of 2-4 states (one
// tile): 5.7 -> 4.3 us.
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
    uint64_t *flags;     // [G] one per block, rising over the runs of a graph
    uint64_t run_tag;    // above every tag of earlier runs; + iteration + 1
    uint32_t smem;       // dynamic shared memory per block, bytes
};

// every block's flag at `tag` or above (this block's is set here); the wait is
// bounded as grid_barrier's, and the same test hook holds a block back: it
// never sets its flag and does not wait at its first barrier
__device__ __forceinline__ bool flag_barrier(LoopyCtl *c, uint64_t *flags, uint64_t tag, bool first, uint32_t *s_fail) {
    __syncthreads();
    const bool skip = c->bar_skip == blockIdx.x + 1u;
    if (threadIdx.x == 0 && !skip) {
        __threadfence();
        *(volatile uint64_t *)(flags + blockIdx.x) = tag;
    }
    if (!(skip && first)) {
        const uint64_t limit = c->wait_ms ? (uint64_t)c->wait_ms * 1000000ull : kBarrierWaitNs;
        for (uint32_t k = threadIdx.x; k < gridDim.x; k += blockDim.x) {
            uint64_t t0 = 0;
            for (uint32_t spin = 0; *(volatile uint64_t *)(flags + k) < tag; ++spin) {
                if ((spin & 255u) != 255u) continue;
                if (*(volatile uint32_t *)s_fail) break;
                const uint64_t t = global_ns();
                if (t0 == 0) t0 = t;
                if (t - t0 > limit) {
                    *(volatile uint32_t *)s_fail = 1;
                    atomicExch(&c->bar_fail, 1u);
                    break;
                }
            }
        }
    }
    __threadfence();
    __syncthreads();
    return *(volatile uint32_t *)s_fail == 0;
}

template <int MS, bool UNI, bool SER, bool WIDE>
__global__ void __launch_bounds__(flood_nt<MS>(), loop_min_blocks<MS, WIDE>()) k_flood_loop(const LoopArgs la) {
    constexpr int NT = flood_nt<MS>();
    constexpr int FU = loop_unroll<MS, WIDE>();
    constexpr uint32_t EMAX = flood_smem_floats<MS>() / MS;
    constexpr uint32_t NB = SER ? 3 : 2;   // message buffers
    constexpr uint32_t TS = loop_table_stride<MS>();
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ double red[NT / 32];
    __shared__ LoopyCtl s_ctl;
    __shared__ uint32_t s_fail;

    const FloodArgs &a = la.f;
    LoopyCtl *ctl = a.ctl;
    const uint32_t tid = threadIdx.x, G = gridDim.x;
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
        for (uint32_t i = tid; i < ne; i += NT) {
            srcs[i] = a.in_src[e0 + i];
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

    // |diff| terms of messages buffers `from` and `to` at their edge ids
    auto write_terms = [&](float *dst, const float *from, const float *to) {
        for (uint32_t i = tid; i < ne; i += NT) {
            int x = MS;
            if (!UNI) x = a.pos_dims[e0 + i] & 15;
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
            stv<MS>(dst + (size_t)a.pos_edge[e0 + i] * MS, ad);
        }
    };

    uint32_t gen = 0;
    uint32_t cur = 0;   // buffer of the latest messages
    bool ok = true;
    for (uint32_t t = 0;; ++t) {
        const uint32_t qp = (qp0 + t) & 1u;
        const float *q_in = qp ? a.q1 : a.q0;
        float *q_out = qp ? a.q0 : a.q1;
        // the first round's gathers, before the last iteration's decision
        float q[FU][MS];
        auto gather = [&](uint32_t i, float *o) {
            const uint32_t s = srcs[i];
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
            const double *part = a.partials + (size_t)((t - 1) & 1u) * G;
            double acc = 0.0;
            for (uint32_t k = tid; k < G; k += NT) acc += __ldcg(part + k);
            const double tot = block_sum<NT>(acc, red);
            if (SER && want) {
                SerialCheck x = serial_check(&s_ctl, broadcast_sum(tot));
                if (x.d < 0) {
                    if (lazy) {
                        const uint32_t p1 = (cur + 2u) % 3u, p2 = (cur + 1u) % 3u;
                        write_terms(a.absdiff + (size_t)x.cb * s_ctl.ad_stride, ms + (size_t)p1 * ne * MS,
                                    ms + (size_t)cur * ne * MS);
                        if (!x.p_exact)
                            write_terms(a.absdiff + (size_t)s_ctl.prev_buf * s_ctl.ad_stride,
                                        ms + (size_t)p2 * ne * MS, ms + (size_t)p1 * ne * MS);
                    }
                    if (solo) __syncthreads();
                    else if (lazy || ce <= 1) ok = grid_barrier(ctl, gen, &s_fail);
                    ok = ok && grid_serial_form<NT>(x, s_ctl, ctl, a.partials, a.absdiff, gen, &s_fail, red);
                    if (!ok) break;
                }
                __syncthreads();   // every thread has read s_ctl
                if (tid == 0) serial_commit(&s_ctl, x);
            } else if (tid == 0) {
                finalize(&s_ctl, want, (float)tot, tot);
            }
            __syncthreads();
            if (s_ctl.done) break;
        }
        const bool want = (ce <= 1) || ((t + 1) % ce == 0);
        float *absd = SER && !lazy ? check_buffer(&s_ctl, a.absdiff, t, want) : nullptr;
        double dsum = 0.0;
        if (!resident) {
            const int mp = (int)((mp0 + t) & 1u);
            flood_tile<MS, UNI, FU>(a, blockIdx.x, want, absd, mp ? a.msg1 : a.msg0, mp ? a.msg0 : a.msg1, q_in, q_out,
                                    0, reinterpret_cast<float *>(dyn), dsum);
        } else {
            const float *mo = ms + (size_t)cur * ne * MS;
            cur = cur + 1u == NB ? 0u : cur + 1u;
            float *mn = ms + (size_t)cur * ne * MS;
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
                    int x = MS, y = MS;
                    if (!UNI) {
                        const uint8_t d = a.pos_dims[e0 + i];
                        x = d & 15;
                        y = d >> 4;
                    }
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
            __syncthreads();
            // the node: marginalise, then the next send buffer (flood_tile's
            // phase 2)
            if (has) {
                float prod[MS];
#pragma unroll
                for (int i = 0; i < MS; ++i) prod[i] = 1.0f;
                for (uint32_t p = r0; p < r1; ++p) {
                    float mm[MS];
                    ldv<MS>(mn + (size_t)p * MS, mm);
                    combine<MS, UNI>(prod, mm, S);
                }
                if (r1 > r0) {
#pragma unroll
                    for (int i = 0; i < MS; ++i)
                        if (UNI || i < S) b[i] = FMUL(b[i], prod[i]);
                }
                normalise<MS, UNI>(b, S);
                float qo[MS];
#pragma unroll
                for (int i = 0; i < MS; ++i) qo[i] = b[i];
                for (uint32_t p = r0; p < r1; ++p) {
                    float mm[MS];
                    ldv<MS>(mn + (size_t)p * MS, mm);
                    combine<MS, UNI>(qo, mm, S);
                }
                if (solo) stv<MS>(qs + (size_t)((qp ^ 1u) * NT + tid) * MS, qo);
                else stv<MS>(q_out + (size_t)v * MS, qo);
            }
        }
        const double part = block_sum<NT>(dsum, red);
        if (tid == 0) a.partials[(size_t)(t & 1u) * G + blockIdx.x] = part;
        if (solo) __syncthreads();
        else if (G <= kFlagBlocks) ok = flag_barrier(ctl, la.flags, la.run_tag + t + 1u, t == 0, &s_fail);
        else ok = grid_barrier(ctl, gen, &s_fail);
        if (!ok) break;
    }

    if (ok && SER) {
        // the returned deltas where the loop decided without them
        if (lazy && s_ctl.done) {
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
            else ok = grid_barrier(ctl, gen, &s_fail);
            ok = ok && grid_serial_final<NT>(s_ctl, ctl, a.partials, a.absdiff, gen, &s_fail, red);
        }
    }
    if (ok && resident) {
        const uint32_t it = s_ctl.it;
        float *ml = ((mp0 + it) & 1u) ? a.msg1 : a.msg0, *mo = ((mp0 + it) & 1u) ? a.msg0 : a.msg1;
        const uint32_t old = cur ? cur - 1u : NB - 1u;
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
