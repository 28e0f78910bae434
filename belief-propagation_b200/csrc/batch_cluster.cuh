// batch_cluster.cuh -- the large networks of a batch, a thread-block cluster
// each.  Included by batch.cu.
//
// A network solved by one block runs at one SM's rate: the largest of a batch
// (4096 nodes, 24,000 edges of 8 states) takes 60 ms for its 200 iterations
// while the GPU's other SMs have run out of networks.  Here kBatchCluster
// blocks share a network.  Each owns a run of nodes with about the same
// number of in-edges and all of those edges, so messages never leave the
// block: they live in its shared memory (with the source ids, and the tables
// where they fit) for the whole solve.  What crosses blocks is the send
// buffers, through L2, and one f64 partial of the delta per block and
// iteration, written into every block's shared memory; a cluster barrier per
// iteration orders both, and every block takes the same stopping decision
// from the same partials in rank order.
//
// Which batches take clusters: clusters_pay (batch.cu).
//
// 1024 networks of 32-4096 nodes, 2-8 states, 200 iterations at most: 103 ms
// with a block per network, 26.7 ms with clusters from 1024 edges on (28.4 from
// 512, 30.2 from 2048, 51 from 4096).  Blocks per SM, their threads and shared
// memory (2 x 256 x 108 KB, 3 x 256 x 70 KB, 4 x 128 x 54 KB) and clusters of
// 4 lie within 5 % of each other.  The networks of 8 states take 17 ms of it
// and read their tables from L2 (every iteration all of them: most do not fit
// these 70 KB); the others are bound by the instruction streams of 24 warps per
// SM and a cluster barrier per iteration.
#pragma once

constexpr int kBatchCluster = 8;           // the largest portable cluster
constexpr int kClusterThreads = 256;
constexpr int kClusterPerSm = 3;           // resident blocks per SM
constexpr uint32_t kClusterSmem = 70u << 10;

// floats between tables in shared memory: 16-byte rows whose starts fall in
// different banks for eight consecutive edges
constexpr uint32_t cluster_table_stride(uint32_t S) {
    return (S * S) % 4 ? S * S : ((S * S) % 8 ? S * S : (S == 2 ? 4 : S * S + 4));
}

// whether the tables of a network's block fit its shared memory beside the
// messages and source ids (a block of ne edges, an eighth of the network's)
inline bool cluster_tables_fit(uint32_t S, uint32_t E) {
    const uint64_t ne = E / kBatchCluster + 1;
    return 4 * ne * (2 * S + 1 + cluster_table_stride(S)) + 64 <= kClusterSmem;
}

template <int S>
__device__ __forceinline__ void ldcg_state(const float *p, float *o) {
    if constexpr (S % 4 == 0) {
#pragma unroll
        for (int k = 0; k < S / 4; ++k) {
            const float4 w = __ldcg(reinterpret_cast<const float4 *>(p) + k);
            o[4 * k] = w.x; o[4 * k + 1] = w.y; o[4 * k + 2] = w.z; o[4 * k + 3] = w.w;
        }
    } else if constexpr (S % 2 == 0) {
#pragma unroll
        for (int k = 0; k < S / 2; ++k) {
            const float2 w = __ldcg(reinterpret_cast<const float2 *>(p) + k);
            o[2 * k] = w.x; o[2 * k + 1] = w.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < S; ++k) o[k] = __ldcg(p + k);
    }
}

// eight floats from a 32-byte aligned address, one whole sector a lane
__device__ __forceinline__ void ld_sector(const float *p, float *o) {
    asm("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]), "=f"(o[6]), "=f"(o[7])
        : "l"(p));
}

// send_msg on a table in global memory.  Eight states: a row is a 32-byte
// sector, loaded whole, every row before the first is used -- as pairs of
// 16-byte loads, each sector crossed from L2 twice (1024 networks: 38 ms against
// 27.5).
template <int S>
__device__ __forceinline__ void cluster_send(const float *__restrict__ J, const float *x, float *m) {
    if constexpr (S == 8) {
        float j[S][S];
#pragma unroll
        for (int i = 0; i < S; ++i) ld_sector(J + i * S, j[i]);
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < S; ++i) {
            float partial = 0.0f;
#pragma unroll
            for (int c = 0; c < S; ++c) partial = FADD(partial, FMUL(j[i][c], x[c]));
            sum = FADD(sum, partial);
            m[i] = partial;
        }
        divide_message<S, true>(m, sum, S);
    } else {
        send_msg<S, true>(J, x, S, S, m);
    }
}

// network n by the calling cluster (f64 delta); dyn: kClusterSmem bytes,
// part[2][kBatchCluster]: the blocks' delta partials by iteration parity
template <int S>
__device__ void cluster_solve(const BatchArgs &a, uint32_t n, cooperative_groups::cluster_group &cluster, float *dyn,
                              double (*part)[kBatchCluster], double *red, uint32_t *bound) {
    constexpr uint32_t T = kClusterThreads, C = kBatchCluster, TS = cluster_table_stride(S);
    const NetInfo ni = a.info[n];
    const uint32_t V = ni.V, E = ni.E, tid = threadIdx.x, rank = cluster.block_rank();
    const uint32_t *ptr = a.in_ptr + ni.ptr_off;
    // this block's nodes: from the first whose row starts at or after its
    // share of the edges
    if (tid < 2) {
        const uint32_t r = rank + tid;
        uint32_t lo = 0, hi = V;
        const uint32_t want = (uint32_t)((uint64_t)E * r / C);
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if (ptr[mid] < want) lo = mid + 1;
            else hi = mid;
        }
        bound[tid] = r == 0 ? 0u : (r == C ? V : lo);
    }
    __syncthreads();
    const uint32_t v0 = bound[0], v1 = bound[1], e0 = ptr[v0], ne = ptr[v1] - e0;
    const uint32_t *src = a.in_src + ni.edge_off + e0;
    const float *J = a.joint + ni.joint_off + (size_t)e0 * S * S;
    float *b = a.belief + ni.node_off;
    const size_t m_off = ni.msg_off + (size_t)e0 * S;
    float *q[2] = {a.q0 + ni.node_off, a.q1 + ni.node_off};
    const int latest = a.latest[n];
    // [messages x 2][source ids][tables] in shared memory, as far as they fit
    const uint32_t m_fl = (2u * ne * S + 3u) & ~3u, s_fl = (ne + 3u) & ~3u;
    const bool chip = 4ull * ((uint64_t)m_fl + s_fl) <= kClusterSmem;
    const bool tables = chip && 4ull * ((uint64_t)m_fl + s_fl + (uint64_t)TS * ne) <= kClusterSmem;
    uint32_t *const ss = reinterpret_cast<uint32_t *>(dyn + m_fl);
    float *const js = dyn + m_fl + s_fl;
    float *m[2];   // m[0]: the latest messages
    if (chip) {
        m[0] = dyn;
        m[1] = dyn + (size_t)ne * S;
    } else {
        m[0] = (latest ? a.msg1 : a.msg0) + m_off;
        m[1] = (latest ? a.msg0 : a.msg1) + m_off;
    }
    if (chip) {
        for (uint32_t i = tid; i < ne; i += T) ss[i] = src[i];
        src = ss;
        if (tables) {
            for (uint32_t i = tid; i < ne * S; i += T) {   // a row per thread
                float r[S];
                ldv<S, kStream>(J + (size_t)i * S, r);
                stv<S>(js + (size_t)(i / S) * TS + (i % S) * S, r);
            }
        }
    }
    __syncthreads();
    auto send = [&](uint32_t i, const float *x, float *o) {
        if (tables) send_msg_rows<S, true>(js + (size_t)i * TS, x, S, S, o);
        else cluster_send<S>(J + (size_t)i * S * S, x, o);
    };
    if (a.init) {   // init_previous_edge (graph.c:725-751)
        for (uint32_t i = tid; i < ne; i += T) {
            float x[S], o[S];
            ldcg_state<S>(b + (size_t)src[i] * S, x);
            send(i, x, o);
            stv<S>(m[0] + (size_t)i * S, o);
        }
    } else if (chip) {
        const float *g = (latest ? a.msg1 : a.msg0) + m_off;
        for (uint32_t i = tid; i < ne * S; i += T) m[0][i] = g[i];
    }
    // the beliefs every block sent from are rewritten in the first iteration
    cluster.sync();
    // Q_1 = b * prod of the latest messages (graph.c:860-882)
    for (uint32_t v = v0 + tid; v < v1; v += T) {
        float bb[S];
        ldv<S>(b + (size_t)v * S, bb);
        for (uint32_t p = ptr[v] - e0; p < ptr[v + 1] - e0; ++p) {
            float mm[S];
            ldv<S>(m[0] + (size_t)p * S, mm);
            combine<S, true>(bb, mm, S);
        }
        stv<S>(q[0] + (size_t)v * S, bb);
    }
    cluster.sync();

    double prev = -1.0, tot = 0.0, last_prev = -1.0;
    uint32_t it = 0, converged = 0;
    for (; it < a.max_it; ++it) {
        const float *q_in = q[it & 1];
        float *q_out = q[(it + 1) & 1];
        double dsum = 0.0;
#pragma unroll 1
        for (uint32_t i = tid; i < ne; i += T) {
            float x[S], o[S], c[S];
            ldcg_state<S>(q_in + (size_t)src[i] * S, x);
            ldv<S>(m[0] + (size_t)i * S, o);
            send(i, x, c);
#pragma unroll
            for (int k = 0; k < S; ++k) {
                float d = FSUB(o[k], c[k]);
                if (d != d) d = 0.0f;
                dsum += (double)fabsf(d);
            }
            stv<S>(m[1] + (size_t)i * S, c);
        }
        dsum = warp_sum(dsum);
        if ((tid & 31u) == 0) red[tid >> 5] = dsum;
        __syncthreads();
        if (tid < C) *cluster.map_shared_rank(&part[it & 1][rank], tid) = warps_total<T / 32>(red);
#pragma unroll 1
        for (uint32_t v = v0 + tid; v < v1; v += T) {
            const uint32_t r0 = ptr[v] - e0, r1 = ptr[v + 1] - e0;
            float prod[S], bb[S];
#pragma unroll
            for (int i = 0; i < S; ++i) prod[i] = 1.0f;
            for (uint32_t p = r0; p < r1; ++p) {
                float mm[S];
                ldv<S>(m[1] + (size_t)p * S, mm);
                combine<S, true>(prod, mm, S);
            }
            ldv<S>(b + (size_t)v * S, bb);
            if (r1 > r0) {
#pragma unroll
                for (int i = 0; i < S; ++i) bb[i] = FMUL(bb[i], prod[i]);
            }
            normalise<S, true>(bb, S);
            stv<S>(b + (size_t)v * S, bb);
            for (uint32_t p = r0; p < r1; ++p) {
                float mm[S];
                ldv<S>(m[1] + (size_t)p * S, mm);
                combine<S, true>(bb, mm, S);
            }
            stv<S>(q_out + (size_t)v * S, bb);
        }
        float *t = m[0];
        m[0] = m[1];
        m[1] = t;
        cluster.sync();
        // the stopping rule (graph.c:1300-1318), the same in every thread
        tot = 0.0;
#pragma unroll
        for (uint32_t r = 0; r < C; ++r) tot += part[it & 1][r];
        last_prev = prev;
        if (tot < (double)a.tol || fabs(tot - prev) < (double)a.tol) {
            converged = 1;
            break;
        }
        prev = tot;
    }
    const uint32_t executed = converged ? it + 1 : a.max_it;
    const int now = latest ^ (int)(executed & 1u);
    if (chip) {
        float *g0 = (now ? a.msg1 : a.msg0) + m_off, *g1 = (now ? a.msg0 : a.msg1) + m_off;
        for (uint32_t i = tid; i < ne * S; i += T) {
            g0[i] = m[0][i];
            g1[i] = m[1][i];
        }
    }
    if (rank == 0 && tid == 0) {
        NetResult r;
        r.iterations = converged ? it : a.max_it;
        r.executed = executed;
        r.converged = converged;
        r.latest = (uint32_t)now;
        r.delta = (float)tot;
        r.prev_delta = (float)last_prev;
        r.delta_d = tot;
        a.res[n] = r;
        a.latest[n] = (uint8_t)now;
    }
    __syncthreads();   // shared memory is free for the next network
}

template <int S>
__global__ void __cluster_dims__(kBatchCluster, 1, 1) __launch_bounds__(kClusterThreads, kClusterPerSm)
    k_batch_cluster(const BatchArgs a, const uint32_t *__restrict__ order, uint32_t count, uint32_t *queue) {
    extern __shared__ __align__(16) float dyn[];
    __shared__ double part[2][kBatchCluster];
    __shared__ double red[kClusterThreads / 32];
    __shared__ uint32_t s_next, s_bound[2];
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    // a block's shared memory may be written by its peers only once it runs:
    // every block of the cluster has started behind this barrier
    cluster.sync();
    for (;;) {
        if (cluster.block_rank() == 0 && threadIdx.x == 0) {
            const uint32_t k = atomicAdd(queue, 1u);
            for (uint32_t r = 0; r < kBatchCluster; ++r) *cluster.map_shared_rank(&s_next, r) = k;
        }
        cluster.sync();
        const uint32_t k = s_next;
        if (k >= count) break;
        cluster_solve<S>(a, order[k], cluster, dyn, part, red, s_bound);
        cluster.sync();   // every block has read s_next and the partials
    }
}
