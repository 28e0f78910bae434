// edge_loop.cuh -- the edge-centric schedule's whole run in one cooperative
// launch.  Included by loopy.cu (it uses the control-block, barrier and delta
// machinery there).
//
// loopy_propagate_until_edge (graph.c:1186-1276) and its _acc form
// (graph.c:1444-1547), reproduced with their quirks:
//  * copy: num_edges * MAX_STATES BYTES of current into previous
//    (graph.c:1211), i.e. the first 2.5E floats of the reference's padded
//    array; the _acc form copies every float and swaps the two roles after
//    each iteration;
//  * send from the beliefs themselves (no incoming product);
//  * combine: belief(dest) *= message for each edge in edge order, no NaN
//    check; the _acc form multiplies by the message of edge i, the batch's
//    first iteration index (graph.c:1485);
//  * normalise: node 0's belief, once per node with that node's state count
//    (the base pointer is passed, graph.c:1225, :1505).
//
// Per iteration a resident grid runs two phases with a grid barrier after
// each: the edges (copy, send and |diff| in one pass: each message array is
// read and written once), then the nodes (combine; node 0 also normalised)
// beside the stopping decision, which every block takes from the same
// partials.  Five launches per iteration, one of them a pass over the copied
// floats and one a re-read of both arrays for the delta, did this before.
//
// What bounded it: node 0's normalisation is a map of a few floats applied V
// times, one thread's chain of dependent adds and divides.  It was applied
// until it stopped changing the belief, but rounding often leaves it in a
// short cycle, and then all V applications ran: 2.1 ms of every iteration on
// 50,001 nodes x 3 states.  The orbit is now followed only until its period
// is known (Brent's method), and the rest taken modulo the period.
// 50,001 nodes, 200,003 edges, 3 states, serial delta, 50 iterations:
// 105.4 -> 3.6 ms per solve (the rest of it forms the serial sum in the 38 checks
// that need it, serial_grid.cuh); f64 delta 0.75 ms.  Mixed state counts: the
// map changes with every run of equal counts, and in no order there are about
// as many runs as nodes, each applied by that one thread: 3000 nodes of 2 and 8
// states 337 us an iteration (540 before), of 8 alone 11.5.
#pragma once

struct EdgeArgs {
    uint32_t V, E;
    const uint32_t *in_ptr, *in_src, *pos_edge, *edge_pos;
    const uint8_t *node_s, *pos_dims;
    const float *joint;
    float *belief;
    float *msg0, *msg1;
    double *partials;
    float *absdiff;
    LoopyCtl *ctl;
    const uint32_t *run_len;
    const uint8_t *run_s;
    uint32_t nruns;
    uint32_t *bar;       // the graph's grid barrier
};

constexpr int kEdgeThreads = 256;

// b = normalised once with its first s slots (a sum that is not positive
// leaves it, graph.c:1046-1061); whether any bit changed
template <int MS>
__device__ __forceinline__ bool edge_normalise_once(float *b, int s) {
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < MS; ++i)
        if (i < s) sum = FADD(sum, b[i]);
    if (!(sum > 0.0f)) return false;
    float nb[MS];
#pragma unroll
    for (int i = 0; i < MS; ++i) nb[i] = b[i];
    divide_by_sum<MS, true>(nb, sum, s);
    bool changed = false;
#pragma unroll
    for (int i = 0; i < MS; ++i)
        if (i < s) {
            changed |= __float_as_uint(nb[i]) != __float_as_uint(b[i]);
            b[i] = nb[i];
        }
    return changed;
}

// b = normalised `len` times with s slots.  The map is deterministic on a
// finite set, so its orbit ends in a cycle: Brent's method keeps one earlier
// point, moved at powers of two; when the orbit returns to it the period is
// known and the remaining applications are taken modulo the period (a fixed
// point is a period of one).
template <int MS>
__device__ __forceinline__ void edge_normalise_run(float *b, int s, uint32_t len) {
    float seen[MS];
#pragma unroll
    for (int i = 0; i < MS; ++i) seen[i] = b[i];
    uint32_t power = 1, lam = 0;
    bool cycle = false;
    for (uint32_t left = len; left; --left) {
        if (!edge_normalise_once<MS>(b, s)) return;
        if (cycle) continue;
        ++lam;
        bool same = true;
#pragma unroll
        for (int i = 0; i < MS; ++i) same = same && (i >= s || __float_as_uint(b[i]) == __float_as_uint(seen[i]));
        if (same) {
            cycle = true;
            left = (left - 1) % lam + 1;   // the loop takes one off
        } else if (lam == power) {
#pragma unroll
            for (int i = 0; i < MS; ++i) seen[i] = b[i];
            power *= 2;
            lam = 0;
        }
    }
}

template <int MS, bool UNI, bool SER>
__global__ void __launch_bounds__(kEdgeThreads) k_edge_loop(const EdgeArgs a) {
    constexpr int NT = kEdgeThreads;
    __shared__ double red[NT / 32];
    __shared__ LoopyCtl s_ctl;
    __shared__ uint32_t s_fail;

    LoopyCtl *ctl = a.ctl;
    GridBar gb(ctl, a.bar);
    if (threadIdx.x == 0) {
        s_ctl = *ctl;
        s_fail = 0;
    }
    __syncthreads();
    const uint64_t first = (uint64_t)blockIdx.x * NT + threadIdx.x, step = (uint64_t)gridDim.x * NT;
    // the copied part of the padded array, in floats and odd bytes
    const uint64_t nbytes = (uint64_t)a.E * 10u, nfull = nbytes / 4u;
    const uint32_t keep = 0xffffffffu << (8u * (uint32_t)(nbytes & 3u));
    bool narrow = true;   // narrowing has decided every check that needed it so far
    while (!s_ctl.done) {
        const uint32_t it = s_ctl.it, ce = s_ctl.check_every;
        const bool acc = s_ctl.acc_edge != 0;
        const bool want = (ce <= 1) || ((it + 1) % ce == 0);
        // previous/current roles: the _acc form swaps them every iteration
        const int pr = (int)((s_ctl.msg_parity0 + (acc ? it : 0u)) & 1u);
        float *prev = pr ? a.msg1 : a.msg0, *curr = pr ? a.msg0 : a.msg1;
        float *absd = SER ? check_buffer(&s_ctl, a.absdiff, it, want) : nullptr;

        // the edges: copy, send, and the |diff| of the copied and the new
        // message (the _acc form's delta reads the swapped roles: the same
        // two, the other way round)
        double dsum = 0.0;
        for (uint64_t p = first; p < a.E; p += step) {
            const uint32_t s = a.in_src[p];
            const uint32_t e = a.pos_edge[p];
            int x = MS, y = MS;
            if (!UNI) {
                const uint8_t d = a.pos_dims[p];
                x = d & 15;
                y = d >> 4;
            }
            float o[MS], m[MS], q[MS];
            ldv<MS>(prev + p * MS, o);
            ldv<MS>(a.belief + (size_t)s * MS, q);
            const uint64_t f0 = (uint64_t)e * 10u;   // float index of slot 0 in the padded layout
            if (acc || f0 <= nfull) {
                float c[MS];
                ldv<MS>(curr + p * MS, c);
#pragma unroll
                for (int k = 0; k < MS; ++k) {
                    if (acc || f0 + k < nfull) o[k] = c[k];
                    else if (f0 + k == nfull && (nbytes & 3u))
                        o[k] = __uint_as_float((__float_as_uint(o[k]) & keep) | (__float_as_uint(c[k]) & ~keep));
                }
                stv<MS>(prev + p * MS, o);
            }
            send_msg<MS, UNI>(a.joint + p * (MS * MS), q, x, y, m);
            stv<MS>(curr + p * MS, m);
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
                if (SER && absd) stv<MS>(absd + (size_t)e * MS, ad);
            }
        }
        const double t = block_sum<NT>(dsum, red);
        double *part = a.partials + (size_t)(it & 1u) * gridDim.x;
        if (threadIdx.x == 0) part[blockIdx.x] = t;
        if (!grid_barrier(gb, &s_fail)) break;

        // the nodes: combine, in edge order
        const uint32_t i_batch = (it / 10u) * 10u;
        if (!acc || i_batch < a.E) {
            float mb[MS];
            if (acc) ldv<MS>(curr + (size_t)a.edge_pos[i_batch] * MS, mb);
            for (uint64_t v = first; v < a.V; v += step) {
                const int S = UNI ? MS : a.node_s[v];
                const uint32_t r0 = a.in_ptr[v], r1 = a.in_ptr[v + 1];
                if (r0 == r1) continue;
                float b[MS];
                ldv<MS>(a.belief + v * MS, b);
                for (uint32_t p = r0; p < r1; ++p) {
                    float mm[MS];
                    if (acc) {
#pragma unroll
                        for (int i = 0; i < MS; ++i) mm[i] = mb[i];
                    } else {
                        ldv<MS>(curr + (size_t)p * MS, mm);
                    }
#pragma unroll
                    for (int i = 0; i < MS; ++i)
                        if (UNI || i < S) b[i] = FMUL(b[i], mm[i]);
                }
                stv<MS>(a.belief + v * MS, b);
            }
        }
        // node 0 (this grid's first thread combined it): normalised once per
        // node, runs of equal state counts in node order
        if (first == 0 && a.V) {
            float b[MS];
            ldv<MS>(a.belief, b);
            for (uint32_t r = 0; r < a.nruns; ++r) edge_normalise_run<MS>(b, a.run_s[r], a.run_len[r]);
            stv<MS>(a.belief, b);
        }

        // the decision, the same in every block
        double sum = 0.0;
        for (uint32_t k = threadIdx.x; k < gridDim.x; k += NT) sum += __ldcg(part + k);
        const double tot = block_sum<NT>(sum, red);
        if (SER && want) {
            SerialCheck x = serial_check(&s_ctl, broadcast_sum(tot));
            if (x.d < 0 && !grid_serial_form<NT>(x, a.absdiff + (size_t)x.cb * s_ctl.ad_stride,
                                                 a.absdiff + (size_t)s_ctl.prev_buf * s_ctl.ad_stride, s_ctl.n_terms,
                                                 s_ctl.tol, ctl, a.partials, gb, &s_fail, red, narrow))
                break;
            __syncthreads();   // every thread has read s_ctl
            if (threadIdx.x == 0) serial_commit(&s_ctl, x);
        } else if (threadIdx.x == 0) {
            finalize(&s_ctl, want, (float)tot, tot);
        }
        __syncthreads();
        // the next iteration's sends read the beliefs combined here
        if (!s_ctl.done && !grid_barrier(gb, &s_fail)) break;
    }
    if (SER && !s_fail && s_ctl.done) grid_serial_final<NT>(s_ctl, ctl, a.partials, a.absdiff, gb, &s_fail, red);
    if (first == 0 && !s_fail) publish_ctl(ctl, s_ctl);
}
