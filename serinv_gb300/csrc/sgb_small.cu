// Small blocks: pobtaf, pobtasi and pobtas (src/serinv/algs/pobtaf.py:97-183,
// pobtasi.py:92-172, pobtas.py:65-161), each in one launch of one CTA (the solve:
// one per four right-hand sides).
//
// What bounds it.  A block step of these sizes is a few microseconds of
// arithmetic on one SM, but it took two or three launches whatever its size:
// 14 to 25 us a block for the factorization, 7 to 22 for the selected inverse,
// 3 for either sweep of the solve.  Here everything a step needs stays in shared
// memory, the next block's values are on their way to registers meanwhile, and
// a block costs its chain: per column the reciprocal of the pivot (or a
// multiplication by it), one update of the columns behind, one CTA barrier.
// n = 128, us a call, start of this file's calls -> now: factorization FP64 b=3
// 3587 -> 567, b=8 3783 -> 877, b=16 4114 -> 1650, FP32 b=16 2535 -> 651, b=32
// 3849 -> 1996; selected inverse FP64 b=3 2255 -> 508, b=8 2778 -> 751, FP32 b=16
// 1682 -> 581; both sweeps of the solve FP64 b=3 3869 -> 324, b=8 3992 -> 590,
// FP32 b=32 2955 -> 671.
// The lines: an SM issues one FP64 warp instruction per 19 cycles, so with
// larger blocks the launches over many SMs win (FP64 factorization b=24 3807
// here against 2843 with the column-block kernel, b=16 1650 / 2464; selected
// inverse b=12 1313 / 985, b=8 751 / 925; solve b=12 845 / 775, b=8 590 / 781; FP32
// selected inverse b=20 1194 / 665, b=16 581 / 790).  With few blocks the other
// paths' launches ahead of the chain weigh more (FP64 selected inverse n=4
// b=16 131 against 210 at the start), so the lines lie higher there.
#include <math.h>

#include "sgb_internal.cuh"
#include "sgb_tile.cuh"

namespace sgb {

namespace {

constexpr int NT = 256;
constexpr int kMaxTip = 32;

template <typename T, int MB>
struct SmallSmem {
    T P[2 * MB + kMaxTip][MB + 1];  // rows of D_i, Lo_i, Ar_i
    T tip[kMaxTip][kMaxTip + 1];
    T col[2][2 * MB + kMaxTip];  // the column being eliminated
    T rs[MB > kMaxTip ? MB : kMaxTip];
    int fail;
};

// Right-looking elimination of the columns of a stack of `rows` rows whose
// first nc <= NC rows are the diagonal block: on return the unscaled columns a'
// are in X and d^{-1/2} in rs, so that L = X diag(rs) below the diagonal.  row0:
// pivot number reported for the first column.  Warp w keeps columns w, w + 8,
// ... in registers, a row to a lane, so a column costs one pass: with column j
// in shared memory every warp takes the reciprocal of the pivot itself, updates
// its later columns, and the owner of column j + 1 publishes it.  An element's
// updates are summed apart and taken from it at once, when its column's turn
// comes: in sequence each would round at the element's size (FP32 rows at b =
// 32 1.1e-7 off so, 6.5e-8 as sums).
template <typename T, int NC, int NR, int LD>
__device__ void eliminate(T (*X)[LD], T (*col)[NR], T* rs, int* fail, int nc, int rows, int row0) {
    constexpr int CP = (NC + 7) / 8, RG = (NR + 31) / 32;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    T v[CP][RG], s[CP][RG];
#pragma unroll
    for (int p = 0; p < CP; ++p)
#pragma unroll
        for (int g = 0; g < RG; ++g) {
            const int r = lane + 32 * g, c = w + 8 * p;
            v[p][g] = r < rows && c < nc ? X[r][c] : T(0);
            s[p][g] = T(0);
        }
    if (w == 0)
#pragma unroll
        for (int g = 0; g < RG; ++g)
            if (lane + 32 * g < rows) col[0][lane + 32 * g] = v[0][g];
    __syncthreads();
    for (int j = 0; j < nc; ++j) {
        const T* x = col[j & 1];
        const T d = x[j];
        Rcp<T> rc;
        rc.first(d);
        T xr[RG], ac[CP];
#pragma unroll
        for (int g = 0; g < RG; ++g) xr[g] = lane + 32 * g < rows ? x[lane + 32 * g] : T(0);
#pragma unroll
        for (int p = 0; p < CP; ++p) ac[p] = w + 8 * p < nc ? x[w + 8 * p] : T(0);
        T inv = rc.second();
        if (!Rcp<T>::plain(d)) {
            const bool ok = pivot_ok(d);
            inv = ok ? T(1) / d : T(NAN);
            if (!ok && tid == 0 && *fail == 0) *fail = row0 + j + 1;
        }
#pragma unroll
        for (int p = 0; p < CP; ++p) {
            const int c = w + 8 * p;
            if (c <= j || c >= nc) continue;
            const T m = ac[p] * inv;
#pragma unroll
            for (int g = 0; g < RG; ++g) s[p][g] = fma(xr[g], m, s[p][g]);
            if (c == j + 1)
#pragma unroll
                for (int g = 0; g < RG; ++g) {
                    v[p][g] -= s[p][g];
                    if (lane + 32 * g < rows) col[c & 1][lane + 32 * g] = v[p][g];
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < CP; ++p)
#pragma unroll
        for (int g = 0; g < RG; ++g) {
            const int r = lane + 32 * g, c = w + 8 * p;
            if (r < rows && c < nc) X[r][c] = v[p][g];
        }
    __syncthreads();
    if (tid < nc) {
        const T d = X[tid][tid];
        rs[tid] = pivot_ok(d) ? rsq<T>(d) : T(NAN);
    }
    __syncthreads();
}

template <typename T>
struct SmallArgs {
    T* D;
    T* Lo;
    T* Ar;
    T* Tp;
    int64_t n;
    int32_t b, a, last;  // last: factor the last block and the tip too
    int32_t* info;
    int32_t* status;
};

template <typename T, int MB>
__global__ void __launch_bounds__(NT) k_small_factor(const __grid_constant__ SmallArgs<T> A) {
    __shared__ SmallSmem<T, MB> S;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int b = A.b, a = A.a, bb = b * b, ab = a * b;
    constexpr int U = (MB * MB + NT - 1) / NT, UA = (kMaxTip * MB + NT - 1) / NT;
    auto rows_at = [&](int e, int base) -> T& { return S.P[base + e / b][e % b]; };
    for (int e = tid; e < bb; e += NT) {
        rows_at(e, 0) = A.D[e];
        if (A.n > 1) rows_at(e, b) = A.Lo[e];
    }
    for (int e = tid; e < ab; e += NT) rows_at(e, 2 * b) = A.Ar[e];
    for (int e = tid; e < a * a; e += NT) S.tip[e / a][e % a] = A.Tp[e];
    if (tid == 0) S.fail = 0;
    __syncthreads();
    for (int64_t i = 0; i < A.n; ++i) {
        const bool end = i == A.n - 1;
        if (end && !A.last) break;
        // the next block on its way
        T nd[U], nl[U], na[UA];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = tid + u * NT;
            nd[u] = (!end && e < bb) ? A.D[(i + 1) * bb + e] : T(0);
            nl[u] = (i + 2 < A.n && e < bb) ? A.Lo[(i + 1) * bb + e] : T(0);
        }
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            const int e = tid + u * NT;
            na[u] = (!end && e < ab) ? A.Ar[(i + 1) * ab + e] : T(0);
        }
        // (after the last block's D the rows of the block before stand in the
        // place of Lo: they are eliminated along and not used)
        eliminate<T, MB, 2 * MB + kMaxTip, MB + 1>(S.P, S.col, S.rs, &S.fail, b, 2 * b + a, (int)(i * b));
        for (int e = tid; e < bb; e += NT) {
            const int r = e / b, c = e % b;
            const T x = S.P[r][c];
            A.D[i * bb + e] = c < r ? x * S.rs[c] : c == r ? x * S.rs[c] : T(0);
            if (!end) {
                const T y = S.P[b + r][c] * S.rs[c];
                A.Lo[i * bb + e] = y;
                S.P[b + r][c] = y;
            }
        }
        for (int e = tid; e < ab; e += NT) {
            const T y = rows_at(e, 2 * b) * S.rs[e % b];
            A.Ar[i * ab + e] = y;
            rows_at(e, 2 * b) = y;
        }
        __syncthreads();
        // Schur products: the next block's D goes over this one's, which is done
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = tid + u * NT;
            if (!end && e < bb) {
                const int r = e / b, c = e % b;
                T s = T(0);
                if (c <= r || !A.last)
                    for (int k = 0; k < b; ++k) s = fma(S.P[b + r][k], S.P[b + c][k], s);
                S.P[r][c] = nd[u] - s;
            }
        }
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            const int e = tid + u * NT;
            if (!end && e < ab) {
                const int r = e / b, c = e % b;
                T s = T(0);
                for (int k = 0; k < b; ++k) s = fma(S.P[2 * b + r][k], S.P[b + c][k], s);
                na[u] -= s;
            }
        }
        for (int r = ty; r < a; r += 16)
            for (int c = tx; c < a; c += 16) {
                if (c > r && A.last) continue;
                T s = T(0);
                for (int k = 0; k < b; ++k) s = fma(S.P[2 * b + r][k], S.P[2 * b + c][k], s);
                S.tip[r][c] -= s;
            }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = tid + u * NT;
            if (e < bb) rows_at(e, b) = nl[u];
        }
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            const int e = tid + u * NT;
            if (!end && e < ab) rows_at(e, 2 * b) = na[u];
        }
        __syncthreads();
    }
    if (A.last) {
        eliminate<T, kMaxTip, 2 * MB + kMaxTip, kMaxTip + 1>(S.tip, S.col, S.rs, &S.fail, a, a, (int)(A.n * b));
        for (int e = tid; e < a * a; e += NT) {
            const int r = e / a, c = e % a;
            A.Tp[e] = c <= r ? S.tip[r][c] * S.rs[c] : T(0);
        }
    } else {  // the last block and the tip as the elimination leaves them
        for (int e = tid; e < bb; e += NT) A.D[(A.n - 1) * bb + e] = rows_at(e, 0);
        for (int e = tid; e < ab; e += NT) A.Ar[(A.n - 1) * ab + e] = rows_at(e, 2 * b);
        for (int e = tid; e < a * a; e += NT) A.Tp[e] = S.tip[e / a][e % a];
    }
    if (tid == 0) {
        if (A.info != nullptr) *A.info = S.fail;
        if (A.status != nullptr) *A.status = 0;
    }
}

// ---- selected inverse ------------------------------------------------------
// pobtasi (src/serinv/algs/pobtasi.py:92-172) in one launch, block by block from
// the bottom with everything the next step needs in shared memory.  As in the
// launched sweep, with G = Lo_i L_ii^{-1}, H = Ar_i L_ii^{-1}:
//   [X_{i+1,i}; X_{A,i}] = -[X_{i+1,i+1} X_{A,i+1}^T; X_{A,i+1} X_T] [G; H]
//   X_ii = L_ii^{-T} L_ii^{-1} - X_{i+1,i}^T G - X_{A,i}^T H
// L_ii^{-1}, G and H come from one substitution with the rows of [I; Lo_i; Ar_i].
template <typename T, int MB>
struct InvSmem {
    T Q[2 * MB + kMaxTip][MB + 1];  // rows of L_ii^{-1}, G, H
    T L[kMaxTip > MB ? kMaxTip : MB][(kMaxTip > MB ? kMaxTip : MB) + 1];
    T XD[MB][MB + 1], XL[MB][MB + 1], XA[2][kMaxTip][MB + 1];
    T XT[kMaxTip][kMaxTip + 1];
    T col[2][2 * MB + kMaxTip];
    T rd[kMaxTip > MB ? kMaxTip : MB];
};

// rows of X <- rows L^{-1} (back substitution over the columns, last first;
// rd: reciprocals of L's diagonal), in the layout of eliminate().
template <typename T, int NC, int NR, int LDX, int LDL>
__device__ void right_solve(T (*X)[LDX], const T (*L)[LDL], const T* rd, T (*col)[NR], int nc, int rows) {
    constexpr int CP = (NC + 7) / 8, RG = (NR + 31) / 32;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    T v[CP][RG], s[CP][RG];
#pragma unroll
    for (int p = 0; p < CP; ++p) {
        const int c = w + 8 * p;
#pragma unroll
        for (int g = 0; g < RG; ++g) {
            const int r = lane + 32 * g;
            v[p][g] = r < rows && c < nc ? X[r][c] : T(0);
            s[p][g] = T(0);
        }
        if (c == nc - 1)
#pragma unroll
            for (int g = 0; g < RG; ++g) {
                v[p][g] *= rd[c];
                if (lane + 32 * g < rows) col[c & 1][lane + 32 * g] = v[p][g];
            }
    }
    __syncthreads();
    for (int j = nc - 1; j > 0; --j) {
        const T* x = col[j & 1];
        T xr[RG];
#pragma unroll
        for (int g = 0; g < RG; ++g) xr[g] = lane + 32 * g < rows ? x[lane + 32 * g] : T(0);
#pragma unroll
        for (int p = 0; p < CP; ++p) {
            const int c = w + 8 * p;
            if (c >= j) continue;
            const T l = L[j][c];
#pragma unroll
            for (int g = 0; g < RG; ++g) s[p][g] = fma(xr[g], l, s[p][g]);
            if (c == j - 1)
#pragma unroll
                for (int g = 0; g < RG; ++g) {
                    v[p][g] = (v[p][g] - s[p][g]) * rd[c];
                    if (lane + 32 * g < rows) col[c & 1][lane + 32 * g] = v[p][g];
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < CP; ++p)
#pragma unroll
        for (int g = 0; g < RG; ++g) {
            const int r = lane + 32 * g, c = w + 8 * p;
            if (r < rows && c < nc) X[r][c] = v[p][g];
        }
    __syncthreads();
}

template <typename T, int MB>
__global__ void __launch_bounds__(NT) k_small_inverse(const __grid_constant__ SmallArgs<T> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    InvSmem<T, MB>& S = *(InvSmem<T, MB>*)smem_raw;
    const int tid = threadIdx.x;
    const int b = A.b, a = A.a, bb = b * b, ab = a * b;
    constexpr int U = (MB * MB + NT - 1) / NT, UA = (kMaxTip * MB + NT - 1) / NT;
    if (A.last && a) {  // X_T = L_T^{-T} L_T^{-1}; Q's rows are too short for the tip, L_T's place is XT's
        for (int e = tid; e < a * a; e += NT) {
            S.L[e / a][e % a] = A.Tp[e];
            S.XT[e / a][e % a] = T(e / a == e % a ? 1 : 0);
        }
        if (tid < a) S.rd[tid] = T(1) / A.Tp[tid * a + tid];
        __syncthreads();
        right_solve<T, kMaxTip, 2 * MB + kMaxTip>(S.XT, S.L, S.rd, S.col, a, a);
        T t[(kMaxTip * kMaxTip + NT - 1) / NT];
#pragma unroll
        for (int u = 0; u < (kMaxTip * kMaxTip + NT - 1) / NT; ++u) {
            const int e = tid + u * NT;
            T s = T(0);
            if (e < a * a)
                for (int k = a - 1; k >= max(e / a, e % a); --k) s = fma(S.XT[k][e / a], S.XT[k][e % a], s);
            t[u] = s;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < (kMaxTip * kMaxTip + NT - 1) / NT; ++u) {
            const int e = tid + u * NT;
            if (e < a * a) A.Tp[e] = S.XT[e / a][e % a] = t[u];
        }
    } else {
        for (int e = tid; e < a * a; e += NT) S.XT[e / a][e % a] = A.Tp[e];
    }
    int64_t i = A.n - 1;
    int cur = 0;
    if (!A.last) {  // the last block is given inverted
        for (int e = tid; e < bb; e += NT) S.XD[e / b][e % b] = A.D[i * bb + e];
        for (int e = tid; e < ab; e += NT) S.XA[0][e / b][e % b] = A.Ar[i * ab + e];
        --i;
    }
    T nd[U], nl[U], na[UA];
    auto fetch = [&](int64_t j) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = tid + u * NT;
            nd[u] = (j >= 0 && e < bb) ? A.D[j * bb + e] : T(0);
            nl[u] = (j >= 0 && j < A.n - 1 && e < bb) ? A.Lo[j * bb + e] : T(0);
        }
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            const int e = tid + u * NT;
            na[u] = (j >= 0 && e < ab) ? A.Ar[j * ab + e] : T(0);
        }
    };
    fetch(i);
    for (; i >= 0; --i) {
        const bool next = i < A.n - 1;
        __syncthreads();  // the previous step's reads are done
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = tid + u * NT, r = e / b, c = e % b;
            if (e < bb) {
                S.L[r][c] = nd[u];
                S.Q[r][c] = T(r == c ? 1 : 0);
                S.Q[b + r][c] = nl[u];
                if (r == c) S.rd[r] = T(1) / nd[u];
            }
        }
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            const int e = tid + u * NT;
            if (e < ab) S.Q[2 * b + e / b][e % b] = na[u];
        }
        fetch(i - 1);
        __syncthreads();
        right_solve<T, MB, 2 * MB + kMaxTip>(S.Q, S.L, S.rd, S.col, b, 2 * b + a);
        T(*XA)[MB + 1] = S.XA[cur ^ 1];
        T(*XP)[MB + 1] = S.XA[cur];  // X_{A,i+1}
        for (int e = tid; e < (next ? bb : 0) + ab; e += NT) {
            const bool low = next && e < bb;
            const int f = next && !low ? e - bb : e, r = f / b, c = f % b;
            T s0 = T(0), s1 = T(0);
            if (low) {
                for (int k = 0; k < b; ++k) s0 = fma(S.XD[r][k], S.Q[b + k][c], s0);
                for (int k = 0; k < a; ++k) s1 = fma(XP[k][r], S.Q[2 * b + k][c], s1);
                A.Lo[i * bb + f] = S.XL[r][c] = -(s0 + s1);
            } else {
                if (next)
                    for (int k = 0; k < b; ++k) s0 = fma(XP[r][k], S.Q[b + k][c], s0);
                for (int k = 0; k < a; ++k) s1 = fma(S.XT[r][k], S.Q[2 * b + k][c], s1);
                A.Ar[i * ab + f] = XA[r][c] = -(s0 + s1);
            }
        }
        __syncthreads();
        for (int e = tid; e < bb; e += NT) {
            const int r = e / b, c = e % b;
            // the dominant term last: each smaller one added to it would round at its size
            // (relative error of the inverse, FP64 b=8 a=21: 1.33e-16 so, 0.91e-16 here)
            T s0 = T(0), s1 = T(0), s2 = T(0);
            const int m = max(r, c);
            for (int k = b - 1; k > m; --k) s0 = fma(S.Q[k][r], S.Q[k][c], s0);
            if (next)
                for (int k = 0; k < b; ++k) s1 = fma(S.XL[k][r], S.Q[b + k][c], s1);
            for (int k = 0; k < a; ++k) s2 = fma(XA[k][r], S.Q[2 * b + k][c], s2);
            A.D[i * bb + e] = S.XD[r][c] = fma(S.Q[m][r], S.Q[m][c], s0 - (s1 + s2));
        }
        cur ^= 1;
    }
    if (tid == 0 && A.status != nullptr) *A.status = 0;
}

// ---- solve --------------------------------------------------------------------
// pobtas (src/serinv/algs/pobtas.py:65-161) by substitution, one right-hand side
// per warp (lane = row of the block), four to a CTA; the other four warps stage
// the blocks: M = L diag(L)^{-1} (so that a row costs the chain one shuffle and
// one FMA), the reciprocal diagonal, Lo and Ar, two blocks ahead.
constexpr int kSolveCols = 4;

// x / d from d's reciprocal: the product with it would round twice (relative error
// of an FP64 solve with L, b=8 a=21, in the mean: so 8.6e-17, with the product 9.4e-17;
// 5 % of the time at b=8, 10 at b=3).  Where the remainder is not finite (x or d
// infinite or NaN, a product past the range) the product stays.
template <typename T>
__device__ __forceinline__ T quotient(T x, T d, T rd) {
    const T q = x * rd, c = fma(fma(-d, q, x), rd, q);
    bool ok;  // by the exponent: comparisons take the FP64 pipe as long as an FMA does
    if constexpr (sizeof(T) == 8) ok = (__double2hiint(c) & 0x7ff00000) != 0x7ff00000;
    else ok = (__float_as_int(c) & 0x7f800000) != 0x7f800000;
    return ok ? c : q;
}

template <typename T, int MB>
struct SolveSmem {
    T M[2][MB][MB + 1], Lo[2][MB][MB + 1], Ar[2][kMaxTip][MB + 1], d[2][MB], rd[2][MB];
    T tm[kMaxTip][kMaxTip + 1], td[kMaxTip], trd[kMaxTip];
};

template <typename T>
struct SmallSolve {
    const T* D;
    const T* Lo;
    const T* Ar;
    const T* Tp;
    T* B;
    int64_t n, ldb, nrhs;
    int32_t b, a, trans;
    int32_t* status;
};

template <typename T, int MB>
__global__ void __launch_bounds__(256) k_small_solve(const __grid_constant__ SmallSolve<T> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SolveSmem<T, MB>& S = *(SolveSmem<T, MB>*)smem_raw;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int b = A.b, a = A.a, bb = b * b, ab = a * b;
    const int64_t n = A.n;
    const bool tr = A.trans != 0;
    // block of step s; backward: Lo of the block before it
    auto blk = [&](int64_t s) { return tr ? n - 1 - s : s; };
    const int lt = tid - 128;
    constexpr int U = (MB * MB + 127) / 128, UA = (kMaxTip * MB + 127) / 128;
    T nd[U], ndk[U], nl[U], na[UA];
    auto fetch = [&](int64_t s) {
        const int64_t i = s < n ? blk(s) : 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = lt + u * 128;
            const bool on = s < n && e < bb;
            nd[u] = on ? __ldg(A.D + i * bb + e) : T(1);
            ndk[u] = on ? __ldg(A.D + i * bb + (e % b) * (b + 1)) : T(1);  // the diagonal entry of this column
            nl[u] = on && i < n - 1 ? __ldg(A.Lo + i * bb + e) : T(0);
        }
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            const int e = lt + u * 128;
            na[u] = s < n && e < ab ? __ldg(A.Ar + i * ab + e) : T(0);
        }
    };
    auto park = [&](int p) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = lt + u * 128, r = e / b, c = e % b;
            if (e < bb) {
                const T rd = ndk[u] > T(0) ? rcp_pivot(ndk[u]) : T(1) / ndk[u];
                S.M[p][r][c] = nd[u] * rd;
                if (r == c) {
                    S.d[p][c] = ndk[u];
                    S.rd[p][c] = rd;
                }
                S.Lo[p][r][c] = nl[u];
            }
        }
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            const int e = lt + u * 128;
            if (e < ab) S.Ar[p][e / b][e % b] = na[u];
        }
    };
    for (int e = tid; e < a * a; e += 256) {
        const T d = A.Tp[(e % a) * (a + 1)];
        const T rd = d > T(0) ? rcp_pivot(d) : T(1) / d;
        S.tm[e / a][e % a] = A.Tp[e] * rd;
        if (e / a == e % a) {
            S.td[e % a] = d;
            S.trd[e % a] = rd;
        }
    }
    if (tid == 0 && blockIdx.x == 0) *A.status = 0;
    if (w >= 4) {
        fetch(0);
        park(0);
        fetch(1);
    }
    const int64_t col = (int64_t)blockIdx.x * kSolveCols + w;
    const bool on = w < kSolveCols && col < A.nrhs;
    T* Bc = A.B + (on ? col : 0);
    T x = T(0), xn = T(0), t = T(0);
    if (on) {
        if (lane < b) x = Bc[(blk(0) * b + lane) * A.ldb];
        if (lane < a) t = Bc[(n * b + lane) * A.ldb];
    }
    __syncthreads();
    // v <- unit triangular solve with M (forward: below the diagonal; backward:
    // its transpose).  Products are summed by themselves and taken from v at
    // once: small terms do not round at the size of v one by one (that doubled
    // the error at b = 16).
    auto substitute = [&](T v, auto M, int m) {
        const T v0 = v;
        T s = T(0);
        if (!tr) {
            for (int k = 0; k + 1 < m; ++k) {
                const T vk = __shfl_sync(0xffffffffu, v, k);
                if (lane > k && lane < m) {
                    s = fma(M[lane][k], vk, s);
                    v = v0 - s;
                }
            }
        } else {
            for (int k = m - 1; k > 0; --k) {
                const T vk = __shfl_sync(0xffffffffu, v, k);
                if (lane < k) {
                    s = fma(M[k][lane], vk, s);
                    v = v0 - s;
                }
            }
        }
        return v;
    };
    if (tr && on && a) {  // x_tip = L_T^{-T} B_tip
        t = lane < a ? quotient(t, S.td[lane], S.trd[lane]) : T(0);
        t = substitute(t, S.tm, a);
        if (lane < a) Bc[(n * b + lane) * A.ldb] = t;
    }
    T prev = T(0);  // backward: the block solved before
    for (int64_t s = 0; s < n; ++s) {
        const int p = (int)(s & 1);
        const int64_t i = blk(s);
        if (w >= 4) {  // the next block into the other buffer, the one after on its way
            park(p ^ 1);
            fetch(s + 2);
        } else if (on) {
            if (s + 1 < n && lane < b) xn = Bc[(blk(s + 1) * b + lane) * A.ldb];
            if (!tr) {
                x = substitute(x, S.M[p], b);
                x = lane < b ? quotient(x, S.d[p][lane], S.rd[p][lane]) : T(0);
                if (lane < b) Bc[(i * b + lane) * A.ldb] = x;
                T sl = T(0), sa = T(0);
                for (int k = 0; k < b; ++k) {
                    const T xk = __shfl_sync(0xffffffffu, x, k);
                    if (lane < b) sl = fma(S.Lo[p][lane][k], xk, sl);
                }
                if (a)
                    for (int k = 0; k < b; ++k) {
                        const T xk = __shfl_sync(0xffffffffu, x, k);
                        if (lane < a) sa = fma(S.Ar[p][lane][k], xk, sa);
                    }
                t -= sa;
                x = xn - sl;
            } else {
                T sa = T(0);
                for (int k = 0; k < a; ++k) {
                    const T tk = __shfl_sync(0xffffffffu, t, k);
                    if (lane < b) sa = fma(S.Ar[p][k][lane], tk, sa);
                }
                if (i < n - 1)
                    for (int k = 0; k < b; ++k) {
                        const T yk = __shfl_sync(0xffffffffu, prev, k);
                        if (lane < b) sa = fma(S.Lo[p][k][lane], yk, sa);
                    }
                x = lane < b ? quotient(x - sa, S.d[p][lane], S.rd[p][lane]) : T(0);
                x = substitute(x, S.M[p], b);
                if (lane < b) Bc[(i * b + lane) * A.ldb] = x;
                prev = x;
                x = xn;
            }
        }
        __syncthreads();
    }
    if (!tr && on && a) {  // B_tip = L_T^{-1} B_tip
        t = substitute(t, S.tm, a);
        if (lane < a) Bc[(n * b + lane) * A.ldb] = quotient(t, S.td[lane], S.trd[lane]);
    }
}

}  // namespace

template <typename T>
bool small_factor_ok(const sgb_bta* m) {
    return m->b <= (sizeof(T) == 8 ? 16 : 32) && m->a <= kMaxTip && m->n * m->b < (int64_t)1 << 30;
}

template <typename T>
cudaError_t small_factor(const sgb_bta* m, int last, int32_t* info, int32_t* status, cudaStream_t s) {
    SmallArgs<T> A;
    A.D = (T*)m->diag;
    A.Lo = (T*)m->lower;
    A.Ar = (T*)m->arrow;
    A.Tp = (T*)m->tip;
    A.n = m->n;
    A.b = (int32_t)m->b;
    A.a = (int32_t)m->a;
    A.last = last != 0;
    A.info = info;
    A.status = status;
    prof_before(s, SGB_KCLASS_PANEL);
    if (m->b <= 16) k_small_factor<T, 16><<<1, NT, 0, s>>>(A);
    else k_small_factor<T, 32><<<1, NT, 0, s>>>(A);
    const double b = (double)m->b, a = (double)m->a;
    prof_after(SGB_KCLASS_PANEL, s, (double)m->n * (7.0 / 3.0 * b * b * b + 3.0 * a * b * b + a * a * b));
    return cudaGetLastError();
}

template <typename T>
bool small_inverse_ok(const sgb_bta* m) {
    const bool few = m->n <= 8;
    return m->b <= (sizeof(T) == 8 ? (few ? 16 : 8) : (few ? 32 : 16)) && m->a <= kMaxTip;
}

template <typename T, int MB>
cudaError_t launch_inverse(const SmallArgs<T>& A, cudaStream_t s) {
    constexpr size_t bytes = sizeof(InvSmem<T, MB>);
    if (bytes > 48 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_small_inverse<T, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
    }
    k_small_inverse<T, MB><<<1, NT, bytes, s>>>(A);
    return cudaGetLastError();
}

template <typename T>
cudaError_t small_inverse(const sgb_bta* m, int last, int32_t* status, cudaStream_t s) {
    SmallArgs<T> A;
    A.D = (T*)m->diag;
    A.Lo = (T*)m->lower;
    A.Ar = (T*)m->arrow;
    A.Tp = (T*)m->tip;
    A.n = m->n;
    A.b = (int32_t)m->b;
    A.a = (int32_t)m->a;
    A.last = last != 0;
    A.info = nullptr;
    A.status = status;
    prof_before(s, SGB_KCLASS_GEMM);
    const cudaError_t e = m->b <= 16 ? launch_inverse<T, 16>(A, s) : launch_inverse<T, 32>(A, s);
    const double b = (double)m->b, a = (double)m->a;
    prof_after(SGB_KCLASS_GEMM, s, (double)m->n * (19.0 / 3.0 * b * b * b + 7.0 * a * b * b + 2.0 * a * a * b));
    return e;
}

// Any number of right-hand sides: a CTA takes kSolveCols of them, and many still gain
// over the batched inverses and products (ms, L and then L^T, so / with those: FP64
// n=128 b=8 1024 columns 0.74 / 5.65, 4096 2.40 / 6.71; n=16 b=16 4096 0.64 / 0.96;
// FP32 n=128 b=32 1024 0.76 / 4.29, 4096 2.31 / 4.39).
template <typename T>
bool small_solve_ok(const sgb_bta* m, int64_t nrhs) {
    return m->b <= (sizeof(T) == 4 ? 32 : m->n <= 16 ? 16 : 8) && m->a <= kMaxTip && nrhs >= 1 && nrhs <= (int64_t)1 << 20;
}

template <typename T, int MB>
cudaError_t launch_solve(const SmallSolve<T>& A, cudaStream_t s) {
    constexpr size_t bytes = sizeof(SolveSmem<T, MB>);
    if (bytes > 48 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_small_solve<T, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
    }
    k_small_solve<T, MB><<<(unsigned)ceil_div(A.nrhs, kSolveCols), 256, bytes, s>>>(A);
    return cudaGetLastError();
}

template <typename T>
cudaError_t small_solve(const sgb_bta* m, T* B, int64_t nrhs, int64_t ldb, bool trans, int32_t* status,
                        cudaStream_t s) {
    SmallSolve<T> A;
    A.D = (const T*)m->diag;
    A.Lo = (const T*)m->lower;
    A.Ar = (const T*)m->arrow;
    A.Tp = (const T*)m->tip;
    A.B = B;
    A.n = m->n;
    A.ldb = ldb;
    A.nrhs = nrhs;
    A.b = (int32_t)m->b;
    A.a = (int32_t)m->a;
    A.trans = trans;
    A.status = status;
    prof_before(s, SGB_KCLASS_GEMM);
    const cudaError_t e = m->b <= 16 ? launch_solve<T, 16>(A, s) : launch_solve<T, 32>(A, s);
    const double b = (double)m->b, a = (double)m->a;
    prof_after(SGB_KCLASS_GEMM, s, (double)nrhs * ((double)m->n * (3.0 * b * b + 2.0 * a * b) + a * a));
    return e;
}

#define SGB_INST(T)                                   \
    template bool small_solve_ok<T>(const sgb_bta*, int64_t);                                         \
    template cudaError_t small_solve<T>(const sgb_bta*, T*, int64_t, int64_t, bool, int32_t*, cudaStream_t); \
    template bool small_factor_ok<T>(const sgb_bta*);  \
    template bool small_inverse_ok<T>(const sgb_bta*); \
    template cudaError_t small_inverse<T>(const sgb_bta*, int, int32_t*, cudaStream_t); \
    template cudaError_t small_factor<T>(const sgb_bta*, int, int32_t*, int32_t*, cudaStream_t);
SGB_INST(double)
SGB_INST(float)

}  // namespace sgb
