// Block triangular solve as one launch: the whole forward (L y = B) or
// backward (L^T x = B) sweep of pobtas (src/serinv/algs/pobtas.py:65-161).
//
// What bounds it.  A sweep is a chain over the blocks, and inside a block over
// its rows; with one right-hand side the arithmetic of a block (about 1.6 b^2
// FMAs) is small next to what a launch, or a barrier over the whole GPU,
// costs.  Launched product by product (two or three launches per block, and
// the full inverse of every diagonal block first) the sweep ran at 86 us per
// block for b = 512 and one right-hand side and 420 us with sixteen; as it is 22
// and 54 us.
//
// Here a cluster of G CTAs walks the whole chain and exchanges values through
// distributed shared memory: asynchronous stores that count their bytes on the
// receiver's mbarrier, so no fence and no barrier over the cluster sits on the
// chain (a release fence also waits for the stores of B: with cluster barriers
// the sweep took 3.4 us per sub-block at b = 64).  A diagonal block is cut into
// sub-blocks of at most kSub rows whose inverses the caller supplies: the
// longer the sub-block the fewer exchanges, but the inverses cost b s^2 / 6
// FMAs per block on the FP64 pipe, which at s = b = 512 is more than the rest
// of the sweep.  128 is where the two meet for b >= 128.  Right-hand sides are
// independent, so they go to different clusters (NR per cluster): that is what
// fills the GPU when there are many.
//
// Per sub-block q of block j, with every row owned by one CTA (the rows of
// each sub-block are spread evenly over the cluster):
//   chain (warps 0-3)  y_q = Linv_qq x_q for its own rows, to every CTA;
//                      x_{q+1} = acc - L_{q+1,q} y_q for its own rows of the
//                      next sub-block (the first of the next block after the
//                      last q), to every CTA;
//   bulk (warps 4-11)  acc -= L_{r,q} y_q for its own rows of everything else
//                      below, beside the chain's next step.
// The backward sweep is the same with the transposed entries and the order
// reversed.  The last "block" is the arrow tip.  Running rows stay in shared
// memory until they are solved, so B is read and written once.
//
// Why no buffer is overwritten early.  x and y have two buffers each.  Every
// CTA contributes to every exchange (a credit if it owns no row there), so a
// complete y_q means that all CTAs have read x_q, and a complete x_{q+2},
// which a CTA sends only after its bulk(q) (named barriers 1, 2), means that all
// have read y_q.
//
// A warp issues one FP64 instruction per 64 cycles, one lane or all, and the
// SM one per 16 to 19: four warps on two rows each (16 lanes per row) give a chain
// step the fewest cycles (12 instructions a warp at k = 128, of which four
// reduce).  In the bulk update one warp forms RW outputs at once and the
// reduction halves the outputs a lane carries at every shuffle step (V - 1 +
// log2(32 / V) additions for V values instead of 5 V).
#include <math.h>
#include <string.h>

#include <mutex>
#include <type_traits>

#include "sgb_internal.cuh"

namespace sgb {

namespace {

constexpr int NC = 4;                // chain warps
constexpr int NB = 8;                // bulk warps
constexpr int NT = 32 * (NC + NB);
constexpr int kSub = 128;            // rows of a sub-block at most
constexpr int KU = kSub / 32;        // k values per lane, 32 lanes to an output
constexpr int KH = kSub / 16;        // k values per lane, 16 lanes to an output
constexpr int kMaxCluster = 16;
constexpr size_t kMaxSmem = 200 * 1024;
constexpr int kCtl = 64;             // bytes in front of the buffers: four mbarriers, the failure flag

template <typename T>
struct SolveArgs {
    const T* D;
    const T* Lo;
    const T* Ar;
    const T* Tp;
    const T* Li;   // (n, b, b): inverses of the diagonal sub-blocks (transposed when li_trans)
    const T* Lti;  // (a, a): the same for the tip, never transposed
    T* B;
    int64_t n, ldb, nrhs;
    int32_t* status;  // SGB_ERR_TIMEOUT if a wait gives up
    long long spin;   // poll limit of every wait
    int32_t b, a;
    int32_t trans, li_trans;
    int32_t s, st;      // sub-block rows of a block and of the tip
    int32_t warm;       // the matrix does not fit L2: fetch ahead of the chain
    int32_t rpc, rpct;  // most rows of a sub-block owned by one CTA
};

__device__ __forceinline__ unsigned sm_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// v to address p of another CTA of the cluster; its bytes count on mbarrier `bar` there.
__device__ __forceinline__ void send(unsigned p, unsigned bar, double v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(p),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send(unsigned p, unsigned bar, float v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(p),
                 "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sm_u32(bar)), "r"(bytes) : "memory");
}
// Bounded wait for the phase of that parity; after a failure anywhere in the
// CTA every wait returns at once (the sweep runs out, its result is marked).
__device__ __forceinline__ void bar_wait(uint64_t* bar, unsigned parity, volatile int* fail, long long spin) {
    for (long long i = 0;; ++i) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n"
            " mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(sm_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return;
        if (*fail) return;
        if (i >= spin) {
            *fail = 1;
            return;
        }
    }
}

// Sums of V values over W lanes: on return lane l holds in v[0] the total of
// value (l % W) / (W / V).
template <typename T, int V, int W>
__device__ __forceinline__ void lane_sums(T (&v)[V]) {
    const int lane = threadIdx.x & 31;
    int off = W / 2;
#pragma unroll
    for (int m = V / 2; m >= 1; m /= 2, off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < m; ++i) {
            const T give = up ? v[i] : v[i + m];
            const T keep = up ? v[i + m] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
    }
#pragma unroll
    for (; off >= 1; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
}

// Volatile, so that the loads stay where they are written: ahead of the wait
// for the values they multiply (the compiler otherwise moves read-only loads
// down to their use, which put an L2 latency on every step of the chain).
__device__ __forceinline__ double ld_now(const double* p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_now(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// Entries of R outputs along this lane's k (32 lanes to an output).
template <typename T, int R>
__device__ __forceinline__ void fetch(T (&l)[R][KU], const T* M, int64_t so, int64_t sk, int nout, int K) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int u = 0; u < KU; ++u) {
            const int k = lane + 32 * u;
            l[r][u] = (r < nout && k < K) ? ld_now(M + r * so + k * sk) : T(0);
        }
}

template <typename T, int R, int NR>
__device__ __forceinline__ void mults(T (&v)[R * NR], const T (&l)[R][KU], const T* y, int K) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < R * NR; ++i) v[i] = T(0);
#pragma unroll
    for (int u = 0; u < KU; ++u) {
        const int k = lane + 32 * u;
        if (32 * u >= K) break;
        if (k < K) {
            T yv[NR];
#pragma unroll
            for (int c = 0; c < NR; ++c) yv[c] = y[k * NR + c];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < NR; ++c) v[r * NR + c] = fma(l[r][u], yv[c], v[r * NR + c]);
        }
    }
}

// The chain's form: one output per half warp.
template <typename T>
__device__ __forceinline__ void fetch_half(T (&l)[KH], const T* M, int64_t sk, bool on, int K) {
    const int h = threadIdx.x & 15;
#pragma unroll
    for (int u = 0; u < KH; ++u) {
        const int k = h + 16 * u;
        l[u] = (on && k < K) ? ld_now(M + k * sk) : T(0);
    }
}
// Multiplies only k in [k_lo, k_hi): what B holds in rows outside the triangle
// does not reach rows that do not depend on it.
template <typename T, int NR>
__device__ __forceinline__ void mults_half(T (&v)[NR], const T (&l)[KH], const T* y, int K, int k_lo, int k_hi) {
    const int h = threadIdx.x & 15;
#pragma unroll
    for (int i = 0; i < NR; ++i) v[i] = T(0);
#pragma unroll
    for (int u = 0; u < KH; ++u) {
        const int k = h + 16 * u;
        if (16 * u >= K) break;
        if (k >= k_lo && k < k_hi) {
#pragma unroll
            for (int c = 0; c < NR; ++c) v[c] = fma(l[u], y[k * NR + c], v[c]);
        }
    }
}

// One block of the chain: a diagonal block, or (j == n) the tip.
template <typename T>
struct Block {
    const T* D;
    const T* Li;
    int64_t row0;  // first row in B
    int m, s, rpc, nsub;
    int li_trans;
    __device__ int rows(int sb) const { return min(s, m - sb * s); }
};

template <typename T>
__device__ __forceinline__ Block<T> block_of(const SolveArgs<T>& a, int64_t j) {
    Block<T> r;
    const bool tip = j == a.n;
    const int64_t bb = (int64_t)a.b * a.b;
    r.D = tip ? a.Tp : a.D + j * bb;
    r.Li = tip ? a.Lti : a.Li + j * bb;
    r.row0 = j * a.b;
    r.m = tip ? a.a : a.b;
    r.s = tip ? a.st : a.s;
    r.rpc = tip ? a.rpct : a.rpc;
    r.nsub = (r.m + r.s - 1) / r.s;
    r.li_trans = tip ? 0 : a.li_trans;
    return r;
}

// Share `part` of `parts` of the cnt elements at p towards L2.  (One bulk
// request: `prefetch.global.L2` line by line held up the loads that followed
// by 2500 cycles a step.)
template <typename T>
__device__ __forceinline__ void warm_l2(const T* p, int64_t cnt, int part, int parts) {
    const uintptr_t lo = ((uintptr_t)(p + cnt * part / parts) + 15) & ~(uintptr_t)15;
    const uintptr_t hi = (uintptr_t)(p + cnt * (part + 1) / parts) & ~(uintptr_t)15;
    if (hi > lo) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((unsigned)(hi - lo)) : "memory");
}

// The rows of a sub-block of `rows` rows owned by a CTA: first and count.
// (G = 1 << lg CTAs)
__device__ __forceinline__ void own_of(int rows, int lg, unsigned rank, int& first, int& cnt) {
    const int per = (rows + (1 << lg) - 1) >> lg;
    first = min(rows, (int)rank * per);
    cnt = min(rows, first + per) - first;
}

template <typename T, int NR>
__global__ void __launch_bounds__(NT, 1) k_solve(const __grid_constant__ SolveArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned G, rank;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(G));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int lg = 31 - __clz((int)G);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int64_t cl = blockIdx.x >> lg;      // this cluster's right-hand sides
    const int64_t c0 = cl * NR;
    const int nr = (int)(a.nrhs - c0 < NR ? a.nrhs - c0 : NR);
    const bool tr = a.trans != 0;
    const int64_t bb = (int64_t)a.b * a.b, ab = (int64_t)a.a * a.b;
    const int nsb = (a.b + a.s - 1) / a.s, nst = a.a ? (a.a + a.st - 1) / a.st : 0;
    const int ownb = nsb * a.rpc, ownt = nst * a.rpct;
    uint64_t* bx = (uint64_t*)smem_raw;   // [2] x complete, [2] y complete
    uint64_t* by = bx + 2;
    volatile int* fail = (volatile int*)(by + 2);
    T* xbuf = (T*)(smem_raw + kCtl);         // [2][kSub + kMaxCluster][NR]: rows, then the credits
    constexpr int kBuf = (kSub + kMaxCluster) * NR;
    T* ybuf = xbuf + 2 * kBuf;               // the same
    T* ytip = ybuf + 2 * kBuf;               // [a + kMaxCluster][NR] (backward: the solved tip)
    T* acc0 = ytip + ((size_t)a.a + kMaxCluster) * NR;  // [3][ownb][NR] running rows of the current block and two more
    T* acct = acc0 + 3 * (size_t)ownb * NR;  // [ownt][NR] running rows of the tip

    const int64_t jfirst = tr ? (a.a ? a.n : a.n - 1) : 0, jlast = tr ? 0 : (a.a ? a.n : a.n - 1);
    const int64_t dj = tr ? -1 : 1;
    // running rows of the block `ahead` places after the one in buffer ring
    auto acc_of = [&](int64_t j, int ring, int ahead) {
        const int r = ring + ahead;
        return j == a.n ? acct : acc0 + (size_t)(r < 3 ? r : r - 3) * ownb * NR;
    };
    int ring = 0;
    // own rows of block j from B, by threads t0, t0 + nt, ...
    auto load_acc = [&](const Block<T>& K, T* acc, int t0, int nt) {
        for (int e = t0; e < K.nsub * K.rpc * NR; e += nt) {
            const int c = e % NR, lr = e / NR, sb = lr / K.rpc, o = lr % K.rpc;
            int f, cnt;
            own_of(K.rows(sb), lg, rank, f, cnt);
            acc[e] = (o < cnt && c < nr) ? a.B[(K.row0 + sb * K.s + f + o) * a.ldb + c0 + c] : T(0);
        }
    };

    Block<T> cur = block_of(a, jfirst);
    load_acc(cur, acc_of(jfirst, 0, 0), tid, NT);
    if (jfirst != jlast && jfirst + dj != a.n) load_acc(block_of(a, jfirst + dj), acc_of(jfirst + dj, 0, 1), tid, NT);
    if (!tr && a.a && jfirst != a.n) load_acc(block_of(a, a.n), acct, tid, NT);
    {
        const int q0 = tr ? cur.nsub - 1 : 0;
        for (int e = tid; e < cur.rows(q0) * NR; e += NT) {
            const int c = e % NR, row = q0 * cur.s + e / NR;
            xbuf[e] = c < nr ? a.B[(cur.row0 + row) * a.ldb + c0 + c] : T(0);
        }
    }
    if (tid == 0) {
        for (int i = 0; i < 4; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm_u32(bx + i)) : "memory");
        *fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");

    // bytes of an exchange of `rows` rows: every row, and a credit from every CTA without one
    auto count = [&](int rows) {
        const int per = (rows + (int)G - 1) >> lg, with = (rows + per - 1) / per;
        return (unsigned)((rows * NR + (int)G - with) * (int)sizeof(T));
    };
    const int rest_b = a.b - (nsb - 1) * a.s, rest_t = a.a ? a.a - (nst - 1) * a.st : 1;
    const unsigned full_b = count(a.s), last_b = count(rest_b), full_t = count(a.st), last_t = count(rest_t);
    auto xbytes = [&](const Block<T>& K, int sb) {
        const bool tip = K.row0 == a.n * a.b, lst = sb == K.nsub - 1;
        return tip ? (lst ? last_t : full_t) : (lst ? last_b : full_b);
    };
    // matrix that couples block j to the next one: the stride of its output
    // (row of the next block) index is so, of its k (row of block j) index sk
    auto coupling = [&](int64_t j) -> const T* {
        if (!tr) return j < a.n - 1 ? a.Lo + j * bb : a.Ar + j * ab;
        return j == a.n ? a.Ar + (j - 1) * ab : a.Lo + (j - 1) * bb;
    };
    unsigned step = 0;  // exchanges so far: buffer step & 1, phase parity (step >> 1) & 1

    if (w < NC) {
        // ---------------- chain
        const int half = lane >> 4, h = lane & 15;
        const int o0 = 2 * w + half;  // this half warp's first own row
        constexpr int LC = 16 / NR;   // lanes that hold the same sum
        const int c = h / LC;
        T la[KH], l1[KH], ld;
        int f, cnt;
        // the CTAs this lane sends a sum to: base of their shared memory
        constexpr int NG = kMaxCluster / LC;
        const unsigned base = sm_u32(smem_raw);
        unsigned to[NG];
#pragma unroll
        for (int i = 0; i < NG; ++i) to[i] = map_rank(base, min((unsigned)(h % LC + i * LC), G - 1));
        auto send_all = [&](const T* p, const uint64_t* bar, T v) {
            const unsigned po = sm_u32(p) - base, bo = sm_u32(bar) - base;
#pragma unroll
            for (int i = 0; i < NG; ++i)
                if (h % LC + i * LC < (int)G) send(to[i] + po, to[i] + bo, v);
        };
        auto send_credit = [&](const T* p, const uint64_t* bar) {
            if (w == 0 && lane < (int)G) {
                const unsigned r = map_rank(base, lane);
                send(r + (sm_u32(p) - base), r + (sm_u32(bar) - base), T(0));
            }
        };
        auto fetch_inv = [&](const Block<T>& K, int sb, int o) {
            const int K0 = sb * K.s;
            const bool row_major = (K.li_trans != 0) == tr;  // the output index walks rows of the stored matrix
            const T* M = K.Li + (int64_t)K0 * K.m + K0;
            int ff, cc;
            own_of(K.rows(sb), lg, rank, ff, cc);
            fetch_half<T>(la, M + (row_major ? (int64_t)(ff + o) * K.m : (int64_t)(ff + o)), row_major ? 1 : K.m, o < cc,
                          K.rows(sb));
            ld = o < cc ? ld_now(M + (int64_t)(ff + o) * (K.m + 1)) : T(0);
        };
        fetch_inv(cur, tr ? cur.nsub - 1 : 0, o0);
        for (int64_t j = jfirst;; j += dj) {
            const bool last_block = j == jlast;
            const Block<T> nxt = last_block ? cur : block_of(a, j + dj);
            const T* Cn = last_block ? nullptr : coupling(j);
            for (int qi = 0; qi < cur.nsub; ++qi, ++step) {
                const int q = tr ? cur.nsub - 1 - qi : qi;
                const bool last_q = qi == cur.nsub - 1, end = last_block && last_q;
                const int K0 = q * cur.s, K = cur.rows(q);
                const unsigned p = step & 1, ph = (step >> 1) & 1;
                T* y = (tr && j == a.n) ? ytip + (size_t)K0 * NR : ybuf + p * kBuf;
                // credits land behind the rows (behind all of the tip's)
                T* ycr = (tr && j == a.n) ? ytip + (size_t)a.a * NR : y + kSub * NR;
                // nobody reads the last y: it is not exchanged (see the end of the kernel)
                if (tid == 0 && !end && !*fail) bar_expect(by + p, xbytes(cur, q));
                // y_q = Linv_qq x_q, own rows
                if (step > 0) bar_wait(bx + (p ^ 1), ((step - 1) >> 1) & 1, fail, a.spin);
                own_of(K, lg, rank, f, cnt);
                const bool mute = end || *fail;
                if (cnt == 0 && !mute) send_credit(ycr + rank, by + p);
                for (int o = o0; o - half < cnt; o += 2 * NC) {
                    if (o != o0) fetch_inv(cur, q, o);
                    T v[NR];
                    const T* xs = step > 0 ? xbuf + (p ^ 1) * kBuf : xbuf;
                    // the diagonal's term by itself and last: in the lanes' sums four more of
                    // them would round at its size (FP64 b=70 a=40, N and C: relative errors
                    // 1.23e-16 and 1.44e-16 so, 0.79e-16 and 0.87e-16 here, for 1 % of the
                    // time at b=64..512)
                    const T xd = o < cnt ? xs[(f + o) * NR + c] : T(0);
                    mults_half<T, NR>(v, la, xs, K, tr ? f + o + 1 : 0, tr ? K : f + o);
                    lane_sums<T, NR, 16>(v);
                    v[0] = fma(ld, xd, v[0]);
                    if (o < cnt) {
                        if (!mute) send_all(y + (f + o) * NR + c, by + p, v[0]);
                        if (h % LC == 0 && c < nr) a.B[(cur.row0 + K0 + f + o) * a.ldb + c0 + c] = v[0];
                    }
                }
                if (end) break;
                // the next sub-block (of this block, or the first of the next one)
                const Block<T>& nb = last_q ? nxt : cur;
                const int nq = last_q ? (tr ? nxt.nsub - 1 : 0) : (tr ? q - 1 : q + 1);
                const int64_t ld = last_q ? a.b : cur.m, so = tr ? 1 : ld, sk = tr ? ld : 1;
                int fn, on;
                own_of(nb.rows(nq), lg, rank, fn, on);
                // entry (output o of sub-block nq, k of sub-block q)
                const T* Mn = (last_q ? Cn : cur.D) + (int64_t)(nq * nb.s + fn) * so + (int64_t)K0 * sk;
                const T* an = last_q ? acc_of(j + dj, ring, 1) : acc_of(j, ring, 0);
                fetch_half<T>(l1, Mn + o0 * so, sk, o0 < on, K);
                T* xn = xbuf + p * kBuf;
                if (tid == 0 && !*fail) bar_expect(bx + p, xbytes(nb, nq));
                bar_wait(by + p, ph, fail, a.spin);
                asm volatile("bar.sync %0, 384;" ::"r"(1 + (int)p) : "memory");  // the bulk update of the step before is done
                // x of the next sub-block, own rows
                const bool dead2 = *fail;
                if (on == 0 && !dead2) send_credit(xn + kSub * NR + rank, bx + p);
                for (int o = o0; o - half < on; o += 2 * NC) {
                    if (o != o0) fetch_half<T>(l1, Mn + o * so, sk, o < on, K);
                    T v[NR];
                    mults_half<T, NR>(v, l1, y, K, 0, K);
                    lane_sums<T, NR, 16>(v);
                    if (o < on) {
                        const T xv = an[(nq * nb.rpc + o) * NR + c] - v[0];
                        if (!dead2) send_all(xn + (fn + o) * NR + c, bx + p, xv);
                    }
                }
                fetch_inv(nb, nq, o0);
            }
            if (last_block) break;
            cur = nxt;
            ring = ring == 2 ? 0 : ring + 1;
        }
    } else {
        // ---------------- bulk
        const int bw = w - NC, bt = tid - 32 * NC;
        constexpr int RW = NR == 4 ? 4 : 8;  // outputs per warp
        T l[RW][KU];
        // outputs [0, no) of the rows at M against y, into A
        const T* M = nullptr;
        T* A = nullptr;
        int64_t ms = 0, mk = 0;
        int no = 0;
        auto apply = [&](auto rows, const T* y, int K) {
            constexpr int R = decltype(rows)::value, V = R * NR;
            T v[V];
            mults<T, R, NR>(v, reinterpret_cast<const T(&)[R][KU]>(l), y, K);
            lane_sums<T, V, 32>(v);
            const int i = lane / (32 / V);
            if (lane % (32 / V) == 0 && i / NR < no) A[i] -= v[0];
        };
        using RowsAll = std::integral_constant<int, RW>;
        using RowsFew = std::integral_constant<int, 2>;
        // B_j -= Ar_j^T y_tip for the own rows of block j
        auto tip_part = [&](const Block<T>& K, int64_t j, T* acc) {
            const int per = (K.rpc + RW - 1) / RW;
            for (int t = bw; t < K.nsub * per; t += NB) {
                const int sb = t / per, o0 = (t % per) * RW;
                int f, cnt;
                own_of(K.rows(sb), lg, rank, f, cnt);
                no = min(cnt - o0, RW);
                if (no <= 0) continue;
                A = acc + (sb * K.rpc + o0) * NR;
                M = a.Ar + j * ab + (sb * K.s + f + o0);
                for (int k0 = 0; k0 < a.a; k0 += kSub) {
                    fetch<T, RW>(l, M + (int64_t)k0 * a.b, 1, a.b, no, a.a - k0);
                    apply(RowsAll{}, ytip + (size_t)k0 * NR, min(kSub, a.a - k0));
                    __syncwarp();
                }
            }
        };
        // Chain step s waits on barrier 1 + (s & 1) for the bulk update of step
        // s - 1; two barriers, because a bulk update may finish before every
        // chain warp has come to wait for the one before it.  None is due at
        // the first step.
        if (jfirst != jlast || cur.nsub > 1) asm volatile("bar.arrive 1, 384;" ::: "memory");
        for (int64_t j = jfirst;; j += dj) {
            const bool last_block = j == jlast;
            const Block<T> nxt = last_block ? cur : block_of(a, j + dj);
            const T* Cn = last_block ? nullptr : coupling(j);
            T* acc = acc_of(j, ring, 0);
            T* accn = acc_of(j + dj, ring, 1);
            // the next block's matrices towards L2, a share per CTA and step, one cluster per block
            const bool warm_next = a.warm && !last_block && j + dj < a.n && (j % (int64_t)(gridDim.x >> lg)) == cl;
            for (int qi = 0; qi < cur.nsub; ++qi, ++step) {
                const int q = tr ? cur.nsub - 1 - qi : qi;
                const bool last_q = qi == cur.nsub - 1;
                if (last_block && last_q) break;
                const int K0 = q * cur.s, K = cur.rows(q);
                const unsigned p = step & 1, ph = (step >> 1) & 1;
                const T* y = (tr && j == a.n) ? ytip + (size_t)K0 * NR : ybuf + p * kBuf;
                if (last_q && !last_block && j + dj != jlast && !(tr && j == a.n)) {
                    // rows of the block after the next; backward, less the solved tip's part
                    const int64_t j2 = j + 2 * dj;
                    const Block<T> far = block_of(a, j2);
                    T* accf = acc_of(j2, ring, 2);
                    if (j2 != a.n) load_acc(far, accf, bt, 32 * NB);
                    if (tr && a.a) {
                        asm volatile("bar.sync 3, 256;" ::: "memory");
                        tip_part(far, j2, accf);
                    }
                }
                // the rest of this block, the next block, (forward) the tip
                const int nD = cur.nsub - 2 - qi > 0 ? cur.nsub - 2 - qi : 0;
                const int nN = last_block ? 0 : nxt.nsub - (last_q ? 1 : 0);
                const int nT = (!tr && a.a && j < a.n - 1) ? nst : 0;
                // few rows: two to a warp, so that no warp's turn is long
                const int R = nD * cur.rpc + nN * nxt.rpc + nT * a.rpct <= 2 * NB ? 2 : RW;
                const int perc = (cur.rpc + R - 1) / R, pern = (nxt.rpc + R - 1) / R, pert = (a.rpct + R - 1) / R;
                const int tD = nD * perc, tN = nN * pern, total = tD + tN + nT * pert;
                auto unit = [&](int t) {
                    int f, cnt, sb, o0;
                    if (t < tD) {
                        sb = tr ? q - 2 - t / perc : q + 2 + t / perc;
                        o0 = (t % perc) * R;
                        own_of(cur.rows(sb), lg, rank, f, cnt);
                        ms = tr ? 1 : cur.m;
                        mk = tr ? cur.m : 1;
                        M = cur.D + (int64_t)(sb * cur.s + f + o0) * ms + (int64_t)K0 * mk;
                        A = acc + (sb * cur.rpc + o0) * NR;
                    } else if (t < tD + tN) {
                        const int tt = t - tD, i = tt / pern + (last_q ? 1 : 0);
                        sb = tr ? nxt.nsub - 1 - i : i;
                        o0 = (tt % pern) * R;
                        own_of(nxt.rows(sb), lg, rank, f, cnt);
                        ms = tr ? 1 : a.b;
                        mk = tr ? a.b : 1;
                        M = Cn + (int64_t)(sb * nxt.s + f + o0) * ms + (int64_t)K0 * mk;
                        A = accn + (sb * nxt.rpc + o0) * NR;
                    } else {
                        const int tt = t - tD - tN;
                        sb = tt / pert;
                        o0 = (tt % pert) * R;
                        own_of(min(a.st, a.a - sb * a.st), lg, rank, f, cnt);
                        ms = a.b;
                        mk = 1;
                        M = a.Ar + j * ab + (int64_t)(sb * a.st + f + o0) * ms + K0;
                        A = acct + (sb * a.rpct + o0) * NR;
                    }
                    no = min(cnt - o0, R);
                };
                if (bw < total) {  // the first unit's entries are on their way before y is
                    unit(bw);
                    fetch<T, RW>(l, M, ms, mk, no, K);
                }
                bar_wait(by + p, ph, fail, a.spin);
                for (int t = bw; t < total; t += NB) {
                    if (t != bw) {
                        unit(t);
                        if (no > 0) fetch<T, RW>(l, M, ms, mk, no, K);
                    }
                    if (no <= 0) continue;
                    if (R == 2) apply(RowsFew{}, y, K);
                    else apply(RowsAll{}, y, K);
                }
                if (tr && j == a.n && last_q && j + dj != jlast) {  // the tip is solved: the second block's part
                    const int64_t j2 = j + 2 * dj;
                    const Block<T> far = block_of(a, j2);
                    T* accf = acc_of(j2, ring, 2);
                    load_acc(far, accf, bt, 32 * NB);
                    asm volatile("bar.sync 3, 256;" ::: "memory");
                    tip_part(far, j2, accf);
                }
                if (warm_next && bw == NB - 1) {
                    const int64_t jn = j + dj;
                    const int part = (int)rank * cur.nsub + qi, parts = (int)G * cur.nsub;
                    if (lane == 0) {
                        warm_l2(a.D + jn * bb, bb, part, parts);
                        if (tr ? jn > 0 : jn < a.n - 1) warm_l2(a.Lo + (tr ? jn - 1 : jn) * bb, bb, part, parts);
                        if (a.a) warm_l2(a.Ar + (tr && jn > 0 ? jn - 1 : jn) * ab, ab, part, parts);
                    }
                    for (int r = part + parts * lane; r < a.b; r += parts * 32) {  // diagonal sub-blocks of the inverse
                        const int x = r / a.s * a.s;
                        warm_l2(a.Li + jn * bb + (int64_t)r * a.b + x, min(a.s, a.b - x), 0, 1);
                    }
                }
                // updates of one row come from different warps in different steps
                asm volatile("bar.sync 3, 256;" ::: "memory");
                const bool next_is_last = last_block ? qi == cur.nsub - 2 : (last_q && j + dj == jlast && nxt.nsub == 1);
                if (!next_is_last) asm volatile("bar.arrive %0, 384;" ::"r"(1 + (int)((step + 1) & 1)) : "memory");
            }
            if (last_block) break;
            cur = nxt;
            ring = ring == 2 ? 0 : ring + 1;
        }
    }
    // No CTA leaves while a peer may still store into it.  A cluster barrier does
    // not cover st.async, whose completion shows on the receiver's mbarrier only;
    // so every exchange that is sent is waited for by its receivers: each y by the
    // chain's wait for it, each x by the next step's, and the last y is not sent.
    // A CTA whose wait gave up has neither armed nor sent anything since.  What its
    // peers sent it before they stopped (all have when the barrier below lets it
    // pass) may be on its way to phases that never complete: it stays for 2^14
    // polls of each barrier, some thousand times as long as a store takes.
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (*fail) {  // the result is not one
        if (tid < 4) {
            volatile int never = 0;
            for (unsigned parity = 0; parity < 2; ++parity) bar_wait(bx + tid, parity, &never, 1 << 14);
        }
        if (tid == 0) atomicExch(a.status, SGB_ERR_TIMEOUT);
        __syncthreads();
        const int64_t N = a.n * a.b + a.a;
        for (int64_t e = tid; e < N * nr; e += NT) a.B[(e / nr) * a.ldb + c0 + e % nr] = T(NAN);
    }
}

template <typename T>
size_t solve_smem(const SolveArgs<T>& a, int NR) {
    const size_t nsb = (a.b + a.s - 1) / a.s, nst = a.a ? (a.a + a.st - 1) / a.st : 0;
    return kCtl + sizeof(T) * NR * (4 * (size_t)(kSub + kMaxCluster) + a.a + kMaxCluster + 3 * nsb * a.rpc + nst * a.rpct);
}

std::mutex g_mu;
int g_max_cluster[64] = {};  // largest cluster the device runs (16, or 8); 0: not asked yet
int g_room[64][5] = {};      // clusters of 1, 2, 4, 8, 16 CTAs that run side by side

template <typename T, int NR>
cudaError_t prepare_kernel() {
    cudaError_t e = cudaFuncSetAttribute(k_solve<T, NR>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_solve<T, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
    return e;
}

void solve_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int G, int clusters, size_t smem, cudaStream_t s) {
    memset(&cfg, 0, sizeof(cfg));
    memset(at, 0, sizeof(*at));
    cfg.gridDim = dim3((unsigned)(G * clusters));
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)G;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

cudaError_t max_cluster(int* out, const int** room) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_max_cluster[dev] == 0) {
        for (cudaError_t x : {prepare_kernel<double, 1>(), prepare_kernel<double, 2>(), prepare_kernel<double, 4>(),
                              prepare_kernel<float, 1>(), prepare_kernel<float, 2>(), prepare_kernel<float, 4>()})
            if (x != cudaSuccess) return x;
        for (int k = 0; k < 5; ++k) {
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute at;
            solve_config(cfg, &at, 1 << k, 1, kMaxSmem, nullptr);
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, k_solve<double, 4>, &cfg) != cudaSuccess) {
                cudaGetLastError();
                n = 0;
            }
            g_room[dev][k] = n;
        }
        g_max_cluster[dev] = g_room[dev][4] >= 1 ? kMaxCluster : 8;
    }
    *out = g_max_cluster[dev];
    *room = g_room[dev];
    return cudaSuccess;
}

}  // namespace

int solve_sub() { return kSub; }

namespace {

struct Shape {
    int G, NR;
    size_t smem;
};

// Cluster size: about eight rows of a sub-block per CTA, two per chain warp.
// Half of it made b = 512 1.5 times and b = 200 1.4 times slower (a CTA's rows
// keep its FP64 pipe busy longer), and at b = 64 neither side gained (505 and
// 492 us at n = 128 with 8 and 16 CTAs, 626 with 4).
// Right-hand sides per cluster: one while the GPU has room for that many
// clusters (7 of 16 CTAs, 15 of 8), more beyond that; a second wave of
// clusters costs more than wider ones (b = 512, 16 columns: 6.6 ms with four
// clusters of four against 8.4 ms with sixteen of one in two waves).  In a
// batch plan's graph the other matrices fill the GPU: one cluster takes up to
// four right-hand sides and reads L once.
// Very many columns: the products' launches fill the GPU by themselves once
// there are waves of clusters to wait for.  b = 512, n = 64, FP64: 15.0 ms
// here against 27.0 ms at 128 columns, 29.6 against 32.6 at 256, 55.8 against
// 44.5 at 512; FP32 (whose products are not held up by the FP64 pipe): 2.4
// against 5.4 ms at 64, 7.6 against 5.4 at 256.
template <typename T>
cudaError_t shape_of(const sgb_bta* m, int64_t nrhs, cudaStream_t s, SolveArgs<T>& a, Shape& h) {
    if (nrhs < 1) return cudaErrorNotSupported;
    int gmax = 8;
    const int* rooms = nullptr;
    cudaError_t e = max_cluster(&gmax, &rooms);
    if (e != cudaSuccess) return e;
    const bool shared_gpu = capture_panel_grid() > 0 && capturing(s);
    if (shared_gpu && gmax > 8) gmax = 8;
    a.n = m->n;
    a.nrhs = nrhs;
    a.b = (int32_t)m->b;
    a.a = (int32_t)m->a;
    a.s = a.b < kSub ? a.b : kSub;
    a.st = a.a < 1 ? 1 : (a.a < kSub ? a.a : kSub);
    int lg = 0;
    while ((1 << lg) < gmax && a.s > (8 << lg)) ++lg;
    h.G = 1 << lg;
    const int room = rooms[lg] > 1 ? rooms[lg] : 1;
    h.NR = 1;
    while (h.NR < 4 && (shared_gpu ? h.NR < nrhs : h.NR * room < nrhs)) h.NR *= 2;
    if (ceil_div(nrhs, 4) > (sizeof(T) == 8 ? 8 : 3) * room) return cudaErrorNotSupported;
    a.rpc = (a.s + h.G - 1) / h.G;
    a.rpct = (a.st + h.G - 1) / h.G;
    h.smem = solve_smem(a, h.NR);
    return h.smem > kMaxSmem ? cudaErrorNotSupported : cudaSuccess;  // very wide blocks or tips
}

}  // namespace

template <typename T>
bool solve_chain_ok(const sgb_bta* m, int64_t nrhs, cudaStream_t s) {
    SolveArgs<T> a;
    Shape h;
    return shape_of<T>(m, nrhs, s, a, h) == cudaSuccess;
}

template <typename T>
cudaError_t solve_chain(const sgb_bta* m, T* B, int64_t nrhs, int64_t ldb, bool trans, const T* Li, bool li_trans,
                        const T* Lti, int32_t* status, cudaStream_t s) {
    SolveArgs<T> a;
    Shape h;
    cudaError_t e = shape_of<T>(m, nrhs, s, a, h);
    if (e != cudaSuccess) return e;
    a.D = (const T*)m->diag;
    a.Lo = (const T*)m->lower;
    a.Ar = (const T*)m->arrow;
    a.Tp = (const T*)m->tip;
    a.Li = Li;
    a.Lti = Lti;
    a.B = B;
    a.ldb = ldb;
    a.trans = trans;
    a.li_trans = li_trans;
    a.status = status;
    a.spin = spin_limit();
    a.warm = (double)a.n * a.b * (2.0 * a.b + a.a) * sizeof(T) > 48e6;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    solve_config(cfg, &at, h.G, (int)ceil_div(nrhs, h.NR), h.smem, s);
    const double bd = a.b, ad = a.a;
    prof_before(s, SGB_KCLASS_GEMM);
    switch (h.NR) {
        case 1: e = cudaLaunchKernelEx(&cfg, k_solve<T, 1>, a); break;
        case 2: e = cudaLaunchKernelEx(&cfg, k_solve<T, 2>, a); break;
        default: e = cudaLaunchKernelEx(&cfg, k_solve<T, 4>, a); break;
    }
    prof_after(SGB_KCLASS_GEMM, s, (double)nrhs * ((double)a.n * (3.0 * bd * bd + 2.0 * ad * bd) + ad * ad));
    return e;
}

#define SGB_INST(T)                                                                                       \
    template bool solve_chain_ok<T>(const sgb_bta*, int64_t, cudaStream_t);                               \
    template cudaError_t solve_chain<T>(const sgb_bta*, T*, int64_t, int64_t, bool, const T*, bool, const T*, \
                                        int32_t*, cudaStream_t);
SGB_INST(double)
SGB_INST(float)

}  // namespace sgb
