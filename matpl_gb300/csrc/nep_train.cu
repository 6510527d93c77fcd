// NEP training operators: the descriptor of one neighbor list with its first and second
// derivatives, the drop-in for CalcOps calculateNepFeat (radial, src/op/src/CalcOps.cpp:385-680)
// and calculateNepMbFeat (3-/4-/5-body, CalcOps.cpp:680-1023) with their Grad functions.
//
// For a descriptor q(c, d12) of one list (d12 [N, NN, 4] = (r, x, y, z) of every slot, c the
// coefficients [T, T, n, K]) and the features' gradient G = dL/dq [N, F]:
//   FWD   q [N, F]
//   BWD   grad_d12 = G . dq/dd12 [N, NN, 4] and W (either may be skipped), from which dL/dc
//         follows by a sum over the atoms of each centre type (matpl_nep_cgrad):
//           radial   W [N, T, K] = sum over neighbors j of type t of f_k(r_ij),
//                    dL/dc[ti, t, n, k] = sum_i G[i, n] W[i, t, k];
//           angular  W [N, T, n, K] = sum_j of type t of f_k(r_ij) sum_m Sbar_nm b_m(r_ij),
//                    Sbar = G . dq/ds (s_nm = sum_j g_n b_m), dL/dc[ti] = sum_i W[i].
//   BWD2  for H = dL/d(grad_d12) [N, NN, 4] (the second backward of the Grad function):
//         gso = dq/dd12 . H [N, F] (the gradient of L with respect to G) and W2 [N, T, n, K]
//         with dL/dc[ti] = sum_i W2[i] (radial: W2 [N, T, K] = sum_j H_r f_k'(r), times G).
// The derivatives are those of the reference's CPU descriptor (nep_net.py:651-870) under
// autograd, i.e. partial derivatives in the four columns of d12 taken as independent inputs:
// f_k depends on r, b_lm on (x, y, z) / r.
// One warp per centre atom, lanes over its slots 32 at a time; per-pair values are staged in
// shared memory and lanes switch to (n, lm) or (t, n, k) entries for the sums over pairs.
#include <algorithm>

#include "common.cuh"
#include "nep_math.cuh"

namespace matpl {
namespace {

constexpr int kFeatWarps = 4;
constexpr size_t kTableBytes = 16 * 1024;   // see matpl_nep_feat_grad_workspace_bytes
enum { kFwd = 0, kBwd = 1, kBwd2 = 2 };

struct FeatArgs {
    int natoms, nn, ntypes, nmax, nbase;
    double rc;
    const void *coeff;          // [T, T, nmax, nbase]
    const void *d12;            // [N, nn, 4]
    const long long *NL;        // [N, nn], -1 = empty
    const long long *type;      // [N]
    const void *G;              // [N, ldG] dL/dq (BWD, BWD2)
    long long ldG;
    const void *H;              // [N, nn, 4] (BWD2)
    void *q;                    // [N, ldQ] (FWD) or gso (BWD2)
    long long ldQ;
    void *grad_d12;             // [N, nn, 4] (BWD), written whole
    void *W;                    // partial c-gradient per atom, zero-filled by the caller
    void *dc;                   // or the c-gradient [T, T, nmax, nbase] itself
    double *sum;                // and its FP64 sums over the blocks, followed by the count of blocks
                                // that have added theirs (zero-filled)
    bool vec;                   // d12, H, grad_d12 on 16-byte boundaries
    int l3, four, five;         // angular: l_max of the 3-body part, 4-/5-body present
    int *err;
};

template <typename T>
__device__ __forceinline__ T ld(const void *p, long long k) { return static_cast<const T *>(p)[k]; }

// the four values of slot ps of a [N, nn, 4] array, one or two wide accesses where it is aligned
template <typename T>
__device__ __forceinline__ void ld4(const void *p, long long ps, bool vec, T *v) {
    const T *a = static_cast<const T *>(p) + 4 * ps;
    if (!vec) {
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = a[c];
    } else if (sizeof(T) == 4) {
        const float4 f = *reinterpret_cast<const float4 *>(a);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
        const double2 f = reinterpret_cast<const double2 *>(a)[0],
                      g = reinterpret_cast<const double2 *>(a)[1];
        v[0] = f.x; v[1] = f.y; v[2] = g.x; v[3] = g.y;
    }
}
template <typename T>
__device__ __forceinline__ void st4(void *p, long long ps, bool vec, T a, T b, T c, T d) {
    T *o = static_cast<T *>(p) + 4 * ps;
    if (vec) {
        store4(o, a, b, c, d);
    } else {
        o[0] = a; o[1] = b; o[2] = c; o[3] = d;
    }
}
// zeros for slots s0, s0 + 1, ... of atom i's row (empty slots have no gradient)
template <typename T>
__device__ __forceinline__ void zero_slots(const FeatArgs &A, long long i, int s0, int lane) {
    for (int s = s0 + lane; s < A.nn; s += 32)
        st4<T>(A.grad_d12, i * A.nn + s, A.vec, T(0), T(0), T(0), T(0));
}

// The c-gradient without a per-atom table in memory: every warp adds its atoms' terms to a table
// [T, T, nmax, nbase] of its own in shared memory, a block adds its four to FP64 sums and the last
// block rounds those.  (A table per atom is 14 MB written, zeroed before and read again for 20,000 atoms
// of four types; FP32 sums over this many blocks would round more than those over its 313.)
template <typename T>
__device__ __forceinline__ void flush_tables(const T *tab, int E, const FeatArgs &A) {
    __shared__ bool last;
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        double v = 0.0;
        for (int w = 0; w < kFeatWarps; ++w) v += (double)tab[w * E + e];
        if (v != 0.0) atomicAdd(A.sum + e, v);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        last = atomicAdd(reinterpret_cast<unsigned *>(A.sum + E), 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int e = threadIdx.x; e < E; e += blockDim.x) static_cast<T *>(A.dc)[e] = (T)__ldcg(A.sum + e);
}

// ---------------------------------------------------------------- radial (calculateNepFeat)
// Blocks an SM that the registers have to leave room for.  The large form (n up to 8) takes 152 registers
// in FP32 and 197 in FP64 unless it is told, half the warps it had in its earlier shape: backward
// of 15,000 atoms, one type of n 5 / K 13, 36 + 36 pairs: radial 129 us so, 80 before; angular 611 (255
// registers), 472 before.  With the bounds here the three passes of 10,000 such atoms take 724 us
// (880 without, 814 before).
template <typename T, int NM>
constexpr int radial_blocks() { return NM > 5 ? (sizeof(T) == 8 ? 4 : 6) : sizeof(T) == 8 ? 1 : 8; }
template <typename T, int MODE, int NM>
constexpr int angular_blocks() {
    return sizeof(T) == 8 ? (MODE == kFwd && NM > 5 ? 5 : 1) : NM <= 5 ? 5 : MODE == kBwd2 ? 4 : 3;
}

// Bound by issue: the sums over pairs of one type (W) take as long as basis and features.  Empty slots
// are written here, so no caller clears grad_d12.
template <typename T, int MODE, int NM, int KM>
__global__ void __launch_bounds__(32 * kFeatWarps, radial_blocks<T, NM>()) nep2b_op(FeatArgs A) {
    __shared__ T s_st[kFeatWarps][32][KM + 1];
    __shared__ __align__(16) int s_tj[kFeatWarps][32];
    extern __shared__ __align__(16) unsigned char mb_raw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int T_ = A.ntypes, n_ = A.nmax, K = A.nbase;
    const T rc = (T)A.rc, rcinv = T(1) / rc;
    const T *c = static_cast<const T *>(A.coeff);
    const long long gw = (long long)blockIdx.x * kFeatWarps + wib;
    const long long nw = (long long)gridDim.x * kFeatWarps;
    const bool want_c = MODE == kBwd2 || (MODE == kBwd && (A.W || A.dc));
    const int E = T_ * T_ * n_ * K;
    T *tab = reinterpret_cast<T *>(mb_raw) + wib * E;
    T *wsum = reinterpret_cast<T *>(mb_raw) + kFeatWarps * E + wib * T_ * K;   // W of one atom
    if (want_c && A.dc) {
        for (int e = lane; e < E; e += 32) tab[e] = T(0);
        for (int e = lane; e < T_ * K; e += 32) wsum[e] = T(0);
        __syncwarp();
    }
    for (long long i = gw; i < A.natoms; i += nw) {
        const int ti = (int)A.type[i];
        if (ti < 0 || ti >= T_) {
            if (lane == 0) atomicMax(A.err, MATPL_KERR_BAD_TYPE);
            if (MODE != kBwd && lane < n_) static_cast<T *>(A.q)[i * A.ldQ + lane] = T(0);
            if (MODE == kBwd && A.grad_d12) zero_slots<T>(A, i, 0, lane);
            continue;
        }
        T *w = A.dc ? wsum : static_cast<T *>(A.W) + i * (long long)T_ * K;
        T G[NM], acc[NM];
#pragma unroll
        for (int n = 0; n < NM; ++n) {
            acc[n] = T(0);
            G[n] = (MODE != kFwd && n < n_) ? ld<T>(A.G, i * A.ldG + n) : T(0);
        }
        for (int base = 0; base < A.nn; base += 32) {
            const int slot = base + lane;
            const long long ps = i * A.nn + slot;
            const long long j = slot < A.nn ? A.NL[ps] : -1;
            const bool ok = j >= 0 && j < A.natoms;
            if (j >= A.natoms) atomicMax(A.err, MATPL_KERR_BAD_COUNT);
            if (!__any_sync(0xffffffffu, ok)) {
                if (MODE == kBwd && A.grad_d12) zero_slots<T>(A, i, base, lane);
                break;
            }
            T f[KM], df[KM];
            int tj = -1;
            if (ok) {
                tj = (int)A.type[j];
                if (tj < 0 || tj >= T_) {
                    atomicMax(A.err, MATPL_KERR_BAD_TYPE);
                    tj = -1;
                }
            }
            const bool use = ok && tj >= 0;
            const T r = use ? ld<T>(A.d12, ps * 4) : T(0);
            basis<T, KM>(r, rc, rcinv, K, f, df);
            const T *cr = c + ((long long)(ti * T_ + (tj < 0 ? 0 : tj)) * n_) * K;
            if (MODE == kFwd) {
                if (use)
#pragma unroll
                    for (int n = 0; n < NM; ++n) {
                        if (n >= n_) break;
                        T g = T(0);
#pragma unroll
                        for (int k = 0; k < KM; ++k)
                            if (k < K) g += cr[n * K + k] * f[k];
                        acc[n] += g;
                    }
            } else if (MODE == kBwd) {
                if (A.grad_d12 && slot < A.nn) {
                    T gp = T(0);
                    if (use)
#pragma unroll
                    for (int n = 0; n < NM; ++n) {
                        if (n >= n_) break;
                        T d = T(0);
#pragma unroll
                        for (int k = 0; k < KM; ++k)
                            if (k < K) d += cr[n * K + k] * df[k];
                        gp += G[n] * d;
                    }
                    st4<T>(A.grad_d12, ps, A.vec, gp, T(0), T(0), T(0));
                }
#pragma unroll
                for (int k = 0; k < KM; ++k) s_st[wib][lane][k] = use ? f[k] : T(0);
            } else {
                const T h0 = use ? ld<T>(A.H, ps * 4) : T(0);
                if (use)
#pragma unroll
                    for (int n = 0; n < NM; ++n) {
                        if (n >= n_) break;
                        T d = T(0);
#pragma unroll
                        for (int k = 0; k < KM; ++k)
                            if (k < K) d += cr[n * K + k] * df[k];
                        acc[n] += h0 * d;
                    }
#pragma unroll
                for (int k = 0; k < KM; ++k) s_st[wib][lane][k] = use ? h0 * df[k] : T(0);
            }
            if (want_c) {
                s_tj[wib][lane] = use ? tj : -1;
                __syncwarp();
                if (sizeof(T) == 8) {
                    // few additions, for the FP64 pipe: the slots of one type after another, lane k (and
                    // k + 16, on the upper slots) sums column k
                    for (unsigned rem = __ballot_sync(0xffffffffu, use); rem;) {
                        const int t = __shfl_sync(0xffffffffu, tj, __ffs(rem) - 1);
                        const unsigned mine = __ballot_sync(0xffffffffu, use && tj == t);
                        rem &= ~mine;
                        const int k0 = lane & 15;
                        T sum = T(0);
                        for (unsigned m = mine & (lane < 16 ? 0xffffu : 0xffff0000u); m; m &= m - 1)
                            if (k0 < K) sum += s_st[wib][__ffs(m) - 1][k0];
                        __syncwarp();
                        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
                        if (lane < K) w[t * K + lane] += sum;
                    }
                } else {
                    // FP32: every lane an entry (t, k), a loop without branches
                    for (int e = lane; e < T_ * K; e += 32) {
                        const int t = e / K, k = e - t * K;
                        T sum = T(0);
#pragma unroll
                        for (int p = 0; p < 32; p += 4) {
                            const int4 j4 = *reinterpret_cast<const int4 *>(s_tj[wib] + p);
                            if (j4.x == t) sum += s_st[wib][p][k];
                            if (j4.y == t) sum += s_st[wib][p + 1][k];
                            if (j4.z == t) sum += s_st[wib][p + 2][k];
                            if (j4.w == t) sum += s_st[wib][p + 3][k];
                        }
                        w[e] += sum;
                    }
                }
                __syncwarp();
            }
        }
        if (want_c && A.dc) {
            T *tt = tab + ti * T_ * n_ * K;
            for (int e = lane; e < T_ * n_ * K; e += 32) {
                const int t = e / (n_ * K), n = e / K - t * n_, k = e % K;
                tt[e] += ld<T>(A.G, i * A.ldG + n) * w[t * K + k];
            }
            __syncwarp();
            for (int e = lane; e < T_ * K; e += 32) w[e] = T(0);
            __syncwarp();
        }
        if (MODE != kBwd) {
#pragma unroll
            for (int n = 0; n < NM; ++n) {
                const T v = warp_sum(acc[n]);
                if (lane == 0 && n < n_) static_cast<T *>(A.q)[i * A.ldQ + n] = v;
            }
        }
    }
    if (want_c && A.dc) flush_tables<T>(reinterpret_cast<T *>(mb_raw), E, A);
}

// ---------------------------------------------------------------- angular (calculateNepMbFeat)
// feature index of the 3-body (l, n), the 4-body n and the 5-body n (l-major, then n)
__device__ __forceinline__ int f3(int l, int n, int nmax) { return l * nmax + n; }

// dq_f / ds_m for the features of one n (3-body of l(m), 4-body, 5-body) contracted with G:
// returns sum_f G_f dq_f/ds_m.  sv = s_n[0..23] of this atom; c3 = the 3-body constants in
// shared memory (lanes index them by their own m).
template <typename T>
__device__ __forceinline__ T sbar_of(const T *c3, int m, const T *sv, T g3, T g4, T g5, bool four,
                                     bool five) {
    T v = g3 * T(2) * c3[m] * sv[m];
    if (four && m >= 3 && m <= 7) {
        const T s3 = sv[3], s4 = sv[4], s5 = sv[5], s6 = sv[6], s7 = sv[7];
        T d;
        if (m == 3) d = T(3) * C4<T>(0) * s3 * s3 + C4<T>(1) * (s4 * s4 + s5 * s5) +
                        C4<T>(2) * (s6 * s6 + s7 * s7);
        else if (m == 4) d = T(2) * C4<T>(1) * s3 * s4 - T(2) * C4<T>(3) * s6 * s4 + C4<T>(4) * s5 * s7;
        else if (m == 5) d = T(2) * C4<T>(1) * s3 * s5 + T(2) * C4<T>(3) * s6 * s5 + C4<T>(4) * s4 * s7;
        else if (m == 6) d = T(2) * C4<T>(2) * s3 * s6 + C4<T>(3) * (s5 * s5 - s4 * s4);
        else d = T(2) * C4<T>(2) * s3 * s7 + C4<T>(4) * s4 * s5;
        v += g4 * d;
    }
    if (five && m <= 2) {
        const T a0 = sv[0] * sv[0], a12 = sv[1] * sv[1] + sv[2] * sv[2];
        const T da = m == 0 ? T(2) * C5<T>(0) * a0 + C5<T>(1) * a12 : C5<T>(1) * a0 + T(2) * C5<T>(2) * a12;
        v += g5 * da * T(2) * sv[m];
    }
    return v;
}

// the derivative of sbar_of along sd (Hessian of q in s times sd, contracted with G)
template <typename T>
__device__ __forceinline__ T sbar_dot(const T *c3, int m, const T *sv, const T *sd, T g3, T g4,
                                      T g5, bool four, bool five) {
    T v = g3 * T(2) * c3[m] * sd[m];
    if (four && m >= 3 && m <= 7) {
        const T s3 = sv[3], s4 = sv[4], s5 = sv[5], s6 = sv[6], s7 = sv[7];
        const T d3 = sd[3], d4 = sd[4], d5 = sd[5], d6 = sd[6], d7 = sd[7];
        T d;
        if (m == 3) d = T(6) * C4<T>(0) * s3 * d3 + T(2) * C4<T>(1) * (s4 * d4 + s5 * d5) +
                        T(2) * C4<T>(2) * (s6 * d6 + s7 * d7);
        else if (m == 4) d = T(2) * C4<T>(1) * (d3 * s4 + s3 * d4) - T(2) * C4<T>(3) * (d6 * s4 + s6 * d4) +
                             C4<T>(4) * (d5 * s7 + s5 * d7);
        else if (m == 5) d = T(2) * C4<T>(1) * (d3 * s5 + s3 * d5) + T(2) * C4<T>(3) * (d6 * s5 + s6 * d5) +
                             C4<T>(4) * (d4 * s7 + s4 * d7);
        else if (m == 6) d = T(2) * C4<T>(2) * (d3 * s6 + s3 * d6) + T(2) * C4<T>(3) * (s5 * d5 - s4 * d4);
        else d = T(2) * C4<T>(2) * (d3 * s7 + s3 * d7) + C4<T>(4) * (d4 * s5 + s4 * d5);
        v += g4 * d;
    }
    if (five && m <= 2) {
        const T a0 = sv[0] * sv[0], a12 = sv[1] * sv[1] + sv[2] * sv[2];
        const T a0d = T(2) * sv[0] * sd[0], a12d = T(2) * (sv[1] * sd[1] + sv[2] * sd[2]);
        T da, dad;
        if (m == 0) {
            da = T(2) * C5<T>(0) * a0 + C5<T>(1) * a12;
            dad = T(2) * C5<T>(0) * a0d + C5<T>(1) * a12d;
        } else {
            da = C5<T>(1) * a0 + T(2) * C5<T>(2) * a12;
            dad = C5<T>(1) * a0d + T(2) * C5<T>(2) * a12d;
        }
        v += g5 * (dad * T(2) * sv[m] + da * T(2) * sd[m]);
    }
    return v;
}

// per warp shared memory of the angular operator; the tangents (sd, sbd, gb, bb, fb) exist in BWD2
// only and pass 2's f_k take the place of pass 1's b_m: 5.4 KB a warp in BWD, 10.1 in BWD2 (FP32, n 5)
template <typename T, int MODE, int NM, int KM>
struct alignas(16) MbSmem {
    static constexpr int NP = (NM + 3) / 4 * 4, D = MODE == kBwd2 ? 1 : 0, G = MODE == kFwd ? 0 : 1;
    static constexpr int F0 = KM + 1 > 25 ? KM + 1 : 25;
    T ga[32][NP], gb[D ? 32 : 1][NP];      // pass 1: g_n, g_n dot; pass 2: B_n / P_n, Q_n
    T ba[32][F0], bb[D ? 32 : 1][F0];      // pass 1: b_m, b_m dot; pass 2: f_k, f_k'
    T s[NM][24], sd[D ? NM : 1][24], sb[G ? NM : 1][24], sbd[D ? NM : 1][24];
};

// a row of NP values in shared memory, 16 bytes at a time
template <int NP>
__device__ __forceinline__ void row_of(const float *p, float *v) {
#pragma unroll
    for (int q = 0; q < NP; q += 4) {
        const float4 f = *reinterpret_cast<const float4 *>(p + q);
        v[q] = f.x; v[q + 1] = f.y; v[q + 2] = f.z; v[q + 3] = f.w;
    }
}
template <int NP>
__device__ __forceinline__ void row_of(const double *p, double *v) {
#pragma unroll
    for (int q = 0; q < NP; q += 2) {
        const double2 f = *reinterpret_cast<const double2 *>(p + q);
        v[q] = f.x; v[q + 1] = f.y;
    }
}

// pair quantities of slot ps: f, f' (K), g_n, g_n' (n), the unit vector and 1/r (0 outside
// (1e-5, rc), where b_lm is zero)
template <typename T, int NM, int KM>
__device__ __forceinline__ void mb_pair(const FeatArgs &A, const T *cr, long long ps, T *f, T *df, T *g,
                                        T *gp, T &ux, T &uy, T &uz, T &ri) {
    const T rc = (T)A.rc, rcinv = T(1) / rc;
    T d4[4];
    ld4<T>(A.d12, ps, A.vec, d4);
    const T r = d4[0];
    basis<T, KM>(r, rc, rcinv, A.nbase, f, df);
#pragma unroll
    for (int n = 0; n < NM; ++n) {
        T a = T(0), d = T(0);
        if (n < A.nmax)
#pragma unroll
            for (int k = 0; k < KM; ++k)
                if (k < A.nbase) {
                    a += cr[n * A.nbase + k] * f[k];
                    d += cr[n * A.nbase + k] * df[k];
                }
        g[n] = a;
        gp[n] = d;
    }
    const bool in = r < rc && r > T(1e-5);
    ri = in ? T(1) / r : T(0);
    ux = d4[1] * ri;
    uy = d4[2] * ri;
    uz = d4[3] * ri;
}

// b_m and its partials in r and in (x, y, z) (= grad_u b / r; d/dr = -(u . grad_u b) / r)
template <typename T>
__device__ __forceinline__ void harm_d(int m, T ux, T uy, T uz, T ri, T &b, T &br, T &bx, T &by,
                                       T &bz) {
    T v, gx, gy, gz;
    harmonic<T>(m, ux, uy, uz, v, gx, gy, gz);
    b = ri != T(0) ? v : T(0);
    bx = gx * ri;
    by = gy * ri;
    bz = gz * ri;
    br = -(gx * ux + gy * uy + gz * uz) * ri;
}

// Bound by issue and shared loads (FP64: by the FP64 pipe).  Pass 1 has lanes over m with all n in
// registers, so a pair's b_m is read once instead of once per n; the c-terms walk the pairs of one type
// instead of testing every pair for every entry.  20,000 atoms, four types, 22 pairs each, FP32, with the
// c-gradient: backward 167 -> 108 us, second backward 209 -> 162; 100,000: 786 -> 508, 1119 -> 791.  Five
// blocks an SM in FP32 (96 registers): with 128 the backward takes 117 us.  (Shared memory leaves the
// second backward of four types four: 41 KB a block and 11 of tables.)
template <typename T, int MODE, int NM, int KM>
__global__ void __launch_bounds__(32 * kFeatWarps, angular_blocks<T, MODE, NM>()) nepmb_op(FeatArgs A) {
    extern __shared__ __align__(16) unsigned char mb_raw[];
    using Sm = MbSmem<T, MODE, NM, KM>;
    constexpr int NP = Sm::NP;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    Sm &S = reinterpret_cast<Sm *>(mb_raw)[wib];
    const int T_ = A.ntypes, n_ = A.nmax, K = A.nbase;
    const bool four = A.four, five = A.five;
    const T *c = static_cast<const T *>(A.coeff);
    const long long gw = (long long)blockIdx.x * kFeatWarps + wib;
    const long long nw = (long long)gridDim.x * kFeatWarps;
    const int nlm = n_ * 24;
    // the 3-body constants in shared memory: lane-varying indices into __constant__ memory are
    // served one address at a time
    __shared__ T c3s[24];
    if (threadIdx.x < 24) c3s[threadIdx.x] = C3<T>(threadIdx.x);
    const bool want_c = MODE == kBwd2 || (MODE == kBwd && (A.W || A.dc));
    const int E = T_ * T_ * n_ * K;
    T *tabs = reinterpret_cast<T *>(mb_raw + sizeof(Sm) * kFeatWarps), *tab = tabs + wib * E;
    if (want_c && A.dc)
        for (int e = lane; e < E; e += 32) tab[e] = T(0);
    __syncthreads();
    for (long long i = gw; i < A.natoms; i += nw) {
        const int ti = (int)A.type[i];
        if (ti < 0 || ti >= T_) {
            if (lane == 0) atomicMax(A.err, MATPL_KERR_BAD_TYPE);
            if (MODE != kBwd)
                for (int e = lane; e < n_ * (A.l3 + four + five); e += 32)
                    static_cast<T *>(A.q)[i * A.ldQ + e] = T(0);
            if (MODE == kBwd && A.grad_d12) zero_slots<T>(A, i, 0, lane);
            continue;
        }
        // ---- pass 1: s_nm (and its tangent along H)
        T sacc[NP], sdacc[NP];   // lane m < 24 has column m
#pragma unroll
        for (int n = 0; n < NP; ++n) sacc[n] = sdacc[n] = T(0);
        int nvalid = 0;
        for (int base = 0; base < A.nn; base += 32) {
            const int slot = base + lane;
            const long long ps = i * A.nn + slot;
            const long long j = slot < A.nn ? A.NL[ps] : -1;
            bool ok = j >= 0 && j < A.natoms;
            if (j >= A.natoms) atomicMax(A.err, MATPL_KERR_BAD_COUNT);
            if (!__any_sync(0xffffffffu, ok)) break;
            nvalid = base + 32;
            int tj = ok ? (int)A.type[j] : -1;
            if (ok && (tj < 0 || tj >= T_)) {
                atomicMax(A.err, MATPL_KERR_BAD_TYPE);
                ok = false;
            }
            T f[KM], df[KM], g[NM], gp[NM], ux, uy, uz, ri;
            const T *cr = c + ((long long)(ti * T_ + (ok ? tj : 0)) * n_) * K;
            mb_pair<T, NM, KM>(A, cr, ok ? ps : 0, f, df, g, gp, ux, uy, uz, ri);
            T h[4] = {T(0), T(0), T(0), T(0)};
            if (MODE == kBwd2 && ok) ld4<T>(A.H, ps, A.vec, h);
#pragma unroll
            for (int n = 0; n < NP; ++n) {
                const int q = n < NM ? n : 0;
                S.ga[lane][n] = ok && n < NM ? g[q] : T(0);
                if (MODE == kBwd2) S.gb[lane][n] = ok && n < NM ? gp[q] * h[0] : T(0);
            }
#pragma unroll
            for (int m = 0; m < 24; ++m) {
                T b, br, bx, by, bz;
                harm_d<T>(m, ux, uy, uz, ri, b, br, bx, by, bz);
                S.ba[lane][m] = ok ? b : T(0);
                if (MODE == kBwd2)
                    S.bb[lane][m] = ok ? br * h[0] + bx * h[1] + by * h[2] + bz * h[3] : T(0);
            }
            __syncwarp();
            // lanes over m, all n in registers: the pairs' g_n are read as broadcast rows
            const int np = 32 - __clz(__ballot_sync(0xffffffffu, ok)), m = lane < 24 ? lane : 0;
            T a[NP], d[NP];
#pragma unroll
            for (int n = 0; n < NP; ++n) a[n] = d[n] = T(0);
            for (int p = 0; p < np; ++p) {
                T ga[NP], gb[NP];
                row_of<NP>(S.ga[p], ga);
                const T b = S.ba[p][m];
#pragma unroll
                for (int n = 0; n < NM; ++n) a[n] += ga[n] * b;
                if (MODE == kBwd2) {
                    row_of<NP>(S.gb[p], gb);
                    const T bd = S.bb[p][m];
#pragma unroll
                    for (int n = 0; n < NM; ++n) d[n] += gb[n] * b + ga[n] * bd;
                }
            }
#pragma unroll
            for (int n = 0; n < NM; ++n) {
                sacc[n] += a[n];
                sdacc[n] += d[n];
            }
            __syncwarp();
        }
        if (lane < 24)
#pragma unroll
            for (int n = 0; n < NM; ++n) {
                S.s[n][lane] = sacc[n];
                if (MODE == kBwd2) S.sd[n][lane] = sdacc[n];
            }
        __syncwarp();
        // ---- features (FWD) / their tangent (BWD2); Sbar, Sbar dot (BWD, BWD2)
        if (MODE == kFwd || MODE == kBwd2) {
            T *out = static_cast<T *>(A.q) + i * A.ldQ;
            for (int e = lane; e < n_ * (A.l3 + four + five); e += 32) {
                const int blk = e / n_, n = e - blk * n_;
                const T *sv = S.s[n];
                const T *sd = S.sd[MODE == kBwd2 ? n : 0];
                T v = T(0);
                if (blk < A.l3) {
                    const int m0 = blk == 0 ? 0 : blk == 1 ? 3 : blk == 2 ? 8 : 15;
                    const int m1 = blk == 0 ? 3 : blk == 1 ? 8 : blk == 2 ? 15 : 24;
                    for (int m = m0; m < m1; ++m)
                        v += MODE == kFwd ? c3s[m] * sv[m] * sv[m] : T(2) * c3s[m] * sv[m] * sd[m];
                } else if (four && blk == A.l3) {
                    if (MODE == kFwd) {
                        const T s3 = sv[3], s4 = sv[4], s5 = sv[5], s6 = sv[6], s7 = sv[7];
                        v = C4<T>(0) * s3 * s3 * s3 + C4<T>(1) * s3 * (s4 * s4 + s5 * s5) +
                            C4<T>(2) * s3 * (s6 * s6 + s7 * s7) + C4<T>(3) * s6 * (s5 * s5 - s4 * s4) +
                            C4<T>(4) * s4 * s5 * s7;
                    } else {
                        for (int m = 3; m <= 7; ++m)
                            v += sbar_of<T>(c3s, m, sv, T(0), T(1), T(0), true, false) * sd[m];
                    }
                } else {
                    if (MODE == kFwd) {
                        const T a0 = sv[0] * sv[0], a12 = sv[1] * sv[1] + sv[2] * sv[2];
                        v = C5<T>(0) * a0 * a0 + C5<T>(1) * a0 * a12 + C5<T>(2) * a12 * a12;
                    } else {
                        for (int m = 0; m <= 2; ++m)
                            v += sbar_of<T>(c3s, m, sv, T(0), T(0), T(1), false, true) * sd[m];
                    }
                }
                out[blk * n_ + n] = v;
            }
        }
        if (MODE == kFwd) continue;
        const T *Gr = static_cast<const T *>(A.G) + i * A.ldG;
        for (int e = lane; e < nlm; e += 32) {
            const int n = e / 24, m = e - n * 24;
            const int l = l_of(m);
            const T g3 = l < A.l3 ? Gr[f3(l, n, n_)] : T(0);
            const T g4 = four ? Gr[A.l3 * n_ + n] : T(0);
            const T g5 = five ? Gr[(A.l3 + four) * n_ + n] : T(0);
            S.sb[n][m] = sbar_of<T>(c3s, m, S.s[n], g3, g4, g5, four, five);
            if (MODE == kBwd2)
                S.sbd[n][m] = sbar_dot<T>(c3s, m, S.s[n], S.sd[n], g3, g4, g5, four, five);
        }
        __syncwarp();
        // ---- pass 2: grad_d12 (BWD) and the per-atom c-gradient table W (either may be
        // skipped in BWD: null pointer)
        T *W = A.W ? static_cast<T *>(A.W) + i * (long long)T_ * n_ * K : nullptr;
        if (MODE == kBwd && A.grad_d12) zero_slots<T>(A, i, nvalid, lane);
        for (int base = 0; base < nvalid; base += 32) {
            const int slot = base + lane;
            const long long ps = i * A.nn + slot;
            const long long j = slot < A.nn ? A.NL[ps] : -1;
            int tj = (j >= 0 && j < A.natoms) ? (int)A.type[j] : -1;
            const bool ok = tj >= 0 && tj < T_;
            T f[KM], df[KM], g[NM], gp[NM], ux, uy, uz, ri;
            const T *cr = c + ((long long)(ti * T_ + (ok ? tj : 0)) * n_) * K;
            mb_pair<T, NM, KM>(A, cr, ok ? ps : 0, f, df, g, gp, ux, uy, uz, ri);
            if (MODE == kBwd && !A.grad_d12) {
                // c-gradient only: B_n = sum_m Sbar_nm b_m
                T Bn[NM];
#pragma unroll
                for (int n = 0; n < NM; ++n) Bn[n] = T(0);
#pragma unroll
                for (int m = 0; m < 24; ++m) {
                    T b, br, bx, by, bz;
                    harm_d<T>(m, ux, uy, uz, ri, b, br, bx, by, bz);
#pragma unroll
                    for (int n = 0; n < NM; ++n) Bn[n] += (n < n_ ? S.sb[n][m] : T(0)) * b;
                }
#pragma unroll
                for (int n = 0; n < NM; ++n) S.ga[lane][n] = ok ? Bn[n] : T(0);
            } else if (MODE == kBwd) {
                T Bn[NM], Br[NM], Bx[NM], By[NM], Bz[NM];
#pragma unroll
                for (int n = 0; n < NM; ++n) Bn[n] = Br[n] = Bx[n] = By[n] = Bz[n] = T(0);
#pragma unroll
                for (int m = 0; m < 24; ++m) {
                    T b, br, bx, by, bz;
                    harm_d<T>(m, ux, uy, uz, ri, b, br, bx, by, bz);
#pragma unroll
                    for (int n = 0; n < NM; ++n) {
                        const T w = n < n_ ? S.sb[n][m] : T(0);
                        Bn[n] += w * b;
                        Br[n] += w * br;
                        Bx[n] += w * bx;
                        By[n] += w * by;
                        Bz[n] += w * bz;
                    }
                }
                T c0 = T(0), cx = T(0), cy = T(0), cz = T(0);
#pragma unroll
                for (int n = 0; n < NM; ++n) {
                    c0 += gp[n] * Bn[n] + g[n] * Br[n];
                    cx += g[n] * Bx[n];
                    cy += g[n] * By[n];
                    cz += g[n] * Bz[n];
                    S.ga[lane][n] = ok ? Bn[n] : T(0);
                }
                if (slot < A.nn)
                    st4<T>(A.grad_d12, ps, A.vec, ok ? c0 : T(0), ok ? cx : T(0), ok ? cy : T(0),
                           ok ? cz : T(0));
            } else {
                T h[4] = {T(0), T(0), T(0), T(0)};
                if (ok) ld4<T>(A.H, ps, A.vec, h);
                T P[NM], Q[NM];
#pragma unroll
                for (int n = 0; n < NM; ++n) P[n] = Q[n] = T(0);
#pragma unroll
                for (int m = 0; m < 24; ++m) {
                    T b, br, bx, by, bz;
                    harm_d<T>(m, ux, uy, uz, ri, b, br, bx, by, bz);
                    const T bd = br * h[0] + bx * h[1] + by * h[2] + bz * h[3];
#pragma unroll
                    for (int n = 0; n < NM; ++n) {
                        const T w = n < n_ ? S.sb[n][m] : T(0);
                        const T wd = n < n_ ? S.sbd[n][m] : T(0);
                        P[n] += w * b;
                        Q[n] += w * bd + wd * b;
                    }
                }
#pragma unroll
                for (int n = 0; n < NM; ++n) {
                    S.ga[lane][n] = ok ? P[n] * h[0] : T(0);
                    S.gb[lane][n] = ok ? Q[n] : T(0);
                }
            }
            if (!want_c) continue;     // grad_d12 only
#pragma unroll
            for (int k = 0; k < KM; ++k) {
                S.ba[lane][k] = ok ? f[k] : T(0);
                if (MODE == kBwd2) S.bb[lane][k] = ok ? df[k] : T(0);
            }
            __syncwarp();
            // the pairs of one neighbor type after another, lanes over the (n, k) entries
            constexpr int Q = (NM * KM + 31) / 32;
            int en[Q], ek[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int e = min(lane + 32 * q, n_ * K - 1);
                en[q] = e / K;
                ek[q] = e - en[q] * K;
            }
            for (unsigned rem = __ballot_sync(0xffffffffu, ok); rem;) {
                const int t = __shfl_sync(0xffffffffu, tj, __ffs(rem) - 1);
                unsigned mine = __ballot_sync(0xffffffffu, ok && tj == t);
                rem &= ~mine;
                T sum[Q];
#pragma unroll
                for (int q = 0; q < Q; ++q) sum[q] = T(0);
                for (; mine; mine &= mine - 1) {
                    const int p = __ffs(mine) - 1;
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        if (MODE == kBwd2)
                            sum[q] += S.ga[p][en[q]] * S.bb[p][ek[q]] + S.gb[p][en[q]] * S.ba[p][ek[q]];
                        else
                            sum[q] += S.ga[p][en[q]] * S.ba[p][ek[q]];
                    }
                }
                T *o = A.dc ? tab + (ti * T_ + t) * n_ * K : W + t * n_ * K;
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    if (lane + 32 * q < n_ * K) o[lane + 32 * q] += sum[q];
            }
            __syncwarp();
        }
    }
    if (want_c && A.dc) flush_tables<T>(tabs, E, A);
}

// Blocks: enough for every atom's warp, but where each leaves a table behind, one wave of them in FP32
// (5,000 atoms, n 5, K 13: 398 us for first and second backward with forward, 421 in two waves) and
// up to four in FP64, whose blocks run long enough for the last of a single wave to show (2,000 such
// atoms: 3152 us in one wave, 2952 in four).
template <typename T, typename K>
int feat_blocks(const FeatArgs &A, K k, size_t smem) {
    const long long need = (A.natoms + kFeatWarps - 1) / kFeatWarps;
    int per_sm = 32;
    if (A.dc && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * kFeatWarps, smem) != cudaSuccess)
        per_sm = 1;
    const int waves = A.dc && sizeof(T) == 8 ? 4 : 1;
    return (int)std::max<long long>(1, std::min<long long>(need, (long long)device_sms() * waves * std::max(per_sm, 1)));
}

template <typename T>
size_t table_bytes(const FeatArgs &A) {
    return A.dc ? sizeof(T) * kFeatWarps * A.ntypes * A.ntypes * A.nmax * A.nbase : 0;
}

template <typename T, int MODE, int NM, int KM>
int launch_mb(const FeatArgs &A, cudaStream_t s) {
    const size_t smem = sizeof(MbSmem<T, MODE, NM, KM>) * kFeatWarps + table_bytes<T>(A);
    auto k = nepmb_op<T, MODE, NM, KM>;
    if (allow_smem(k, smem) != cudaSuccess) {
        set_error("matpl_nep_feat: shared-memory attribute rejected");
        return MATPL_ERR_CUDA;
    }
    k<<<feat_blocks<T>(A, k, smem), 32 * kFeatWarps, smem, s>>>(A);
    return check_launch("matpl_nep_feat");
}

template <typename T, int MODE, int NM, int KM>
int launch_2b(const FeatArgs &A, cudaStream_t s) {
    const size_t smem = A.dc ? table_bytes<T>(A) + sizeof(T) * kFeatWarps * A.ntypes * A.nbase : 0;
    auto k = nep2b_op<T, MODE, NM, KM>;
    if (smem && allow_smem(k, smem) != cudaSuccess) {
        set_error("matpl_nep_feat: shared-memory attribute rejected");
        return MATPL_ERR_CUDA;
    }
    k<<<feat_blocks<T>(A, k, smem), 32 * kFeatWarps, smem, s>>>(A);
    return check_launch("matpl_nep_feat");
}

template <typename T, int MODE>
int dispatch(bool angular, const FeatArgs &A, cudaStream_t s) {
    if (angular) {
        if (A.nmax <= 5 && A.nbase <= 9) return launch_mb<T, MODE, 5, 9>(A, s);
        return launch_mb<T, MODE, 8, 16>(A, s);
    }
    if (A.nmax <= 5 && A.nbase <= 9) return launch_2b<T, MODE, 5, 9>(A, s);
    return launch_2b<T, MODE, 8, 16>(A, s);
}

}  // namespace
}  // namespace matpl

using namespace matpl;

namespace matpl {
namespace {

// dL/dc [T, T, n, K] from the per-atom tables of the backward modes.  A block takes kCgAtoms
// consecutive atoms; for each centre type t present among them it compacts their indices
// (warp ballots, list order kept), its 8 warps split those atoms, and each lane sums kCols
// columns (a 256-column pass: lane + 32 c) of their rows - radial G[i, nn] * W[i, tt, k],
// angular W[i, tt, nn, k] - with the loads of all its columns in flight together.  The warps'
// partial sums meet in shared memory and each column leaves with one atomic into dc[t] per
// block.  The work of a block does not depend on how the types are mixed (sorted or
// interleaved atoms cost the same).
constexpr int kCgWarps = 8;
constexpr int kCgAtoms = 64;
constexpr int kCols = 8;
constexpr int kPass = 32 * kCols;

template <typename T>
__global__ void __launch_bounds__(32 * kCgWarps)
nep_cgrad_kernel(int part, int natoms, int ntypes, int nmax, int K,
                 const long long *__restrict__ type_map, const T *__restrict__ G, long long ldG,
                 const T *__restrict__ W, T *__restrict__ dc, int *__restrict__ err) {
    __shared__ int tsh[kCgAtoms];
    __shared__ int idx[kCgAtoms];
    __shared__ int wbase[kCgAtoms / 32];
    __shared__ int cnt;
    __shared__ T part_sum[kCgWarps][kPass];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long base = (long long)blockIdx.x * kCgAtoms;
    if (threadIdx.x < kCgAtoms) {
        const long long a = base + threadIdx.x;
        int ta = -1;
        if (a < natoms) {
            const long long v = type_map[a];
            if (v < 0 || v >= ntypes) atomicMax(err, MATPL_KERR_BAD_TYPE);
            else ta = (int)v;
        }
        tsh[threadIdx.x] = ta;
    }
    __syncthreads();
    const int E = ntypes * nmax * K;
    for (int t = 0; t < ntypes; ++t) {
        if (threadIdx.x < kCgAtoms) {
            const bool mine = tsh[threadIdx.x] == t;
            const unsigned bal = __ballot_sync(0xffffffffu, mine);
            if (lane == 0) wbase[warp] = __popc(bal);
            __syncwarp();
            if (mine) idx[32 * warp + __popc(bal & ((1u << lane) - 1u))] = threadIdx.x;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            // close the gap between the warps' runs (list order kept)
            int n0 = wbase[0];
            for (int w = 1; w < kCgAtoms / 32; ++w) {
                for (int k = 0; k < wbase[w]; ++k) idx[n0 + k] = idx[32 * w + k];
                n0 += wbase[w];
            }
            cnt = n0;
        }
        __syncthreads();
        const int n = cnt;
        if (n == 0) continue;
        for (int e0 = 0; e0 < E; e0 += kPass) {
            T acc[kCols];
            long long goff[kCols], woff[kCols];
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                acc[c] = 0;
                const int e = e0 + lane + 32 * c;
                const int tt = e / (nmax * K), nn = (e / K) % nmax, k = e % K;
                goff[c] = nn;
                woff[c] = part == 0 ? (long long)tt * K + k : e;
            }
            for (int j = warp; j < n; j += kCgWarps) {
                const long long i = base + idx[j];
                if (part == 0) {
                    const T *g = G + i * ldG;
                    const T *w = W + i * ntypes * K;
#pragma unroll
                    for (int c = 0; c < kCols; ++c)
                        if (e0 + lane + 32 * c < E) acc[c] += g[goff[c]] * w[woff[c]];
                } else {
                    const T *w = W + i * E;
#pragma unroll
                    for (int c = 0; c < kCols; ++c)
                        if (e0 + lane + 32 * c < E) acc[c] += w[woff[c]];
                }
            }
#pragma unroll
            for (int c = 0; c < kCols; ++c) part_sum[warp][lane + 32 * c] = acc[c];
            __syncthreads();
            const int e = e0 + threadIdx.x;
            if (threadIdx.x < kPass && e < E) {
                T v = 0;
#pragma unroll
                for (int w = 0; w < kCgWarps; ++w) v += part_sum[w][threadIdx.x];
                atomicAdd(dc + (long long)t * E + e, v);
            }
            __syncthreads();
        }
    }
}

// Forces and per-image virial of one NEP list from dE = dE/d(r, x, y, z) [N, NN, 4] and the
// rows Ri = (r, x, y, z) themselves (the expanded d(r, x, y, z)/d(x, y, z) of nep_net.py:440-468
// has x_a / r in row 0 and the identity below, so it is formed in registers): per slot
// f_a = dE_0 x_a / r + dE_(1+a) (empty slots, |r| <= 1e-5, give 0), the centre gets -f, the
// neighbor NL +f, and the slot adds f_a r_b to the virial of the centre's image.  A block takes
// kFvAtoms consecutive atoms, each warp kFvAtoms / 8 of them (lanes over slots, warp sums of the
// centre force); the virial is summed per warp and then per block in shared memory, runs of one
// image (frames are contiguous) leaving with 9 atomics, so the atomics on the few virial
// addresses stay at one set per block.
constexpr int kFvWarps = 8;
constexpr int kFvAtoms = 32;

template <typename T>
__global__ void __launch_bounds__(32 * kFvWarps)
nep_force_virial_kernel(int natoms, int nn, int nimages, const long long *__restrict__ NL,
                        const long long *__restrict__ image_of, const T *__restrict__ dE,
                        const T *__restrict__ Ri, T *__restrict__ force, T *__restrict__ virial,
                        int *__restrict__ err) {
    __shared__ T vsh[kFvWarps][9];
    __shared__ long long bsh[kFvWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int per_warp = kFvAtoms / kFvWarps;
    const long long a0 = (long long)blockIdx.x * kFvAtoms + (long long)warp * per_warp;
    T v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    long long cur = -1;
    for (int k = 0; k < per_warp; ++k) {
        const long long i = a0 + k;
        if (i >= natoms) break;
        const long long b = image_of[i];
        if (b < 0 || b >= nimages) {
            if (lane == 0) atomicMax(err, MATPL_KERR_BAD_COUNT);
            continue;
        }
        if (b != cur) {                 // a frame boundary inside the warp's atoms
            if (cur >= 0 && lane < 9) atomicAdd(virial + 9 * cur + lane, v[0]);
#pragma unroll
            for (int c = 0; c < 9; ++c) v[c] = 0;
            cur = b;
        }
        T fc[3] = {0, 0, 0}, vi[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int s = lane; s < nn; s += 32) {
            const long long q = i * nn + s;
            const T r = Ri[4 * q];
            if (!(fabs(r) > T(1e-5))) continue;
            const T x[3] = {Ri[4 * q + 1], Ri[4 * q + 2], Ri[4 * q + 3]};
            const T e0 = dE[4 * q];
            T f[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c] = e0 * (x[c] / r) + dE[4 * q + 1 + c];
            const long long j = NL[q];
            if (j >= natoms) {
                atomicMax(err, MATPL_KERR_BAD_COUNT);
            } else if (j >= 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) atomicAdd(force + 3 * j + c, f[c]);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                fc[c] -= f[c];
#pragma unroll
                for (int d = 0; d < 3; ++d) vi[3 * c + d] += f[c] * x[d];
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) fc[c] = warp_sum(fc[c]);
        if (lane < 3) atomicAdd(force + 3 * i + lane, lane == 0 ? fc[0] : lane == 1 ? fc[1] : fc[2]);
        // the warp's 9 virial sums, lane c < 9 keeping term c in v[0]
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const T t = warp_sum(vi[c]);
            if (lane == c) v[0] += t;
        }
    }
    if (lane < 9) vsh[warp][lane] = v[0];
    if (lane == 0) bsh[warp] = cur;
    __syncthreads();
    if (threadIdx.x < 9) {
        long long run = -1;
        T acc = 0;
        for (int w = 0; w < kFvWarps; ++w) {
            const long long b = bsh[w];
            if (b < 0) continue;
            if (b != run) {
                if (run >= 0) atomicAdd(virial + 9 * run + threadIdx.x, acc);
                run = b;
                acc = 0;
            }
            acc += vsh[w][threadIdx.x];
        }
        if (run >= 0) atomicAdd(virial + 9 * run + threadIdx.x, acc);
    }
}

// The gradient of the kernel above (linear in dE): per slot u_a = gF[NL]_a - gF[i]_a +
// sum_b gV[image(i)][a][b] r_b, then gdE = (sum_a u_a x_a / r, u_0, u_1, u_2); empty slots 0.
// One thread per slot; gF or gV may be absent (zero).
template <typename T>
__global__ void __launch_bounds__(256)
nep_force_virial_grad_kernel(int natoms, int nn, int nimages, const long long *__restrict__ NL,
                             const long long *__restrict__ image_of, const T *__restrict__ Ri,
                             const T *__restrict__ gF, const T *__restrict__ gV,
                             T *__restrict__ gdE, int *__restrict__ err) {
    const long long total = (long long)natoms * nn;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const long long i = q / nn;
        const T r = Ri[4 * q];
        T g[4] = {0, 0, 0, 0};
        if (fabs(r) > T(1e-5)) {
            const T x[3] = {Ri[4 * q + 1], Ri[4 * q + 2], Ri[4 * q + 3]};
            T u[3] = {0, 0, 0};
            if (gF) {
                const long long j = NL[q];
#pragma unroll
                for (int a = 0; a < 3; ++a) u[a] = -gF[3 * i + a];
                if (j >= natoms) {
                    atomicMax(err, MATPL_KERR_BAD_COUNT);
                } else if (j >= 0) {
#pragma unroll
                    for (int a = 0; a < 3; ++a) u[a] += gF[3 * j + a];
                }
            }
            if (gV) {
                const long long b = image_of[i];
                if (b < 0 || b >= nimages) {
                    atomicMax(err, MATPL_KERR_BAD_COUNT);
                } else {
#pragma unroll
                    for (int a = 0; a < 3; ++a)
#pragma unroll
                        for (int c = 0; c < 3; ++c) u[a] += gV[9 * b + 3 * a + c] * x[c];
                }
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                g[0] += u[a] * (x[a] / r);
                g[1 + a] = u[a];
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) gdE[4 * q + c] = g[c];
    }
}

}  // namespace
}  // namespace matpl

extern "C" int matpl_nep_cgrad(int dtype, int part, int natoms, int ntypes, int n_max, int n_base,
                               const long long *type_map, const void *G, long long ldG,
                               const void *W, void *dc, int *err_dev, void *stream) {
    MATPL_REQUIRE(dtype == MATPL_F32 || dtype == MATPL_F64, MATPL_ERR_DTYPE,
                  "matpl_nep_cgrad: dtype is MATPL_F32 or MATPL_F64");
    MATPL_REQUIRE(part == 0 || part == 1, MATPL_ERR_INVALID, "part: 0 radial, 1 angular");
    MATPL_REQUIRE(natoms >= 0 && ntypes >= 1 && n_max >= 1 && n_base >= 1, MATPL_ERR_INVALID,
                  "bad sizes");
    MATPL_REQUIRE(part == 1 || ldG >= n_max, MATPL_ERR_INVALID, "radial: ldG >= n_max");
    MATPL_REQUIRE(dc && err_dev && (natoms == 0 || (type_map && W && (part == 1 || G))),
                  MATPL_ERR_INVALID, "null pointer argument");
    MATPL_REQUIRE_ON_DEVICE(dc, "matpl_nep_cgrad");
    cudaStream_t s = as_stream(stream);
    const size_t esz = dtype == MATPL_F64 ? sizeof(double) : sizeof(float);
    const size_t nout = (size_t)ntypes * ntypes * n_max * n_base;
    if (cudaMemsetAsync(dc, 0, esz * nout, s) != cudaSuccess) {
        set_error("matpl_nep_cgrad: memset failed");
        return MATPL_ERR_CUDA;
    }
    if (natoms == 0) return MATPL_OK;
    ProfScope ps("nep_cgrad", s);
    const int grid = (int)((natoms + kCgAtoms - 1) / kCgAtoms);
    if (dtype == MATPL_F64)
        nep_cgrad_kernel<double><<<grid, 32 * kCgWarps, 0, s>>>(
            part, natoms, ntypes, n_max, n_base, type_map, (const double *)G, ldG,
            (const double *)W, (double *)dc, err_dev);
    else
        nep_cgrad_kernel<float><<<grid, 32 * kCgWarps, 0, s>>>(
            part, natoms, ntypes, n_max, n_base, type_map, (const float *)G, ldG,
            (const float *)W, (float *)dc, err_dev);
    return check_launch("matpl_nep_cgrad");
}

extern "C" int matpl_nep_force_virial(int dtype, int natoms, int max_nn, int nimages,
                                      const long long *NL, const long long *image_of,
                                      const void *dE, const void *Ri, void *force, void *virial,
                                      int *err_dev, void *stream) {
    MATPL_REQUIRE(dtype == MATPL_F32 || dtype == MATPL_F64, MATPL_ERR_DTYPE,
                  "matpl_nep_force_virial: dtype is MATPL_F32 or MATPL_F64");
    MATPL_REQUIRE(natoms >= 0 && max_nn >= 0 && nimages >= 1, MATPL_ERR_INVALID, "bad sizes");
    MATPL_REQUIRE(force && virial && err_dev &&
                      (natoms * (long long)max_nn == 0 || (NL && image_of && dE && Ri)),
                  MATPL_ERR_INVALID, "null pointer argument");
    MATPL_REQUIRE_ON_DEVICE(force, "matpl_nep_force_virial");
    cudaStream_t s = as_stream(stream);
    const size_t esz = dtype == MATPL_F64 ? sizeof(double) : sizeof(float);
    if (cudaMemsetAsync(force, 0, esz * 3 * (size_t)natoms, s) != cudaSuccess ||
        cudaMemsetAsync(virial, 0, esz * 9 * (size_t)nimages, s) != cudaSuccess) {
        set_error("matpl_nep_force_virial: memset failed");
        return MATPL_ERR_CUDA;
    }
    if (natoms == 0 || max_nn == 0) return MATPL_OK;
    ProfScope ps("nep_force_virial", s);
    const int grid = (int)((natoms + kFvAtoms - 1) / kFvAtoms);
    if (dtype == MATPL_F64)
        nep_force_virial_kernel<double><<<grid, 32 * kFvWarps, 0, s>>>(
            natoms, max_nn, nimages, NL, image_of, (const double *)dE, (const double *)Ri,
            (double *)force, (double *)virial, err_dev);
    else
        nep_force_virial_kernel<float><<<grid, 32 * kFvWarps, 0, s>>>(
            natoms, max_nn, nimages, NL, image_of, (const float *)dE, (const float *)Ri,
            (float *)force, (float *)virial, err_dev);
    return check_launch("matpl_nep_force_virial");
}

extern "C" int matpl_nep_force_virial_grad(int dtype, int natoms, int max_nn, int nimages,
                                           const long long *NL, const long long *image_of,
                                           const void *Ri, const void *g_force,
                                           const void *g_virial, void *g_dE, int *err_dev,
                                           void *stream) {
    MATPL_REQUIRE(dtype == MATPL_F32 || dtype == MATPL_F64, MATPL_ERR_DTYPE,
                  "matpl_nep_force_virial_grad: dtype is MATPL_F32 or MATPL_F64");
    MATPL_REQUIRE(natoms >= 0 && max_nn >= 0 && nimages >= 1, MATPL_ERR_INVALID, "bad sizes");
    MATPL_REQUIRE(err_dev && (natoms * (long long)max_nn == 0 || (NL && image_of && Ri && g_dE)),
                  MATPL_ERR_INVALID, "null pointer argument");
    const long long total = (long long)natoms * max_nn;
    if (total == 0) return MATPL_OK;
    MATPL_REQUIRE_ON_DEVICE(g_dE, "matpl_nep_force_virial_grad");
    cudaStream_t s = as_stream(stream);
    ProfScope ps("nep_force_virial_grad", s);
    const int grid = (int)std::min<long long>((total + 255) / 256, (long long)device_sms() * 16);
    if (dtype == MATPL_F64)
        nep_force_virial_grad_kernel<double><<<grid, 256, 0, s>>>(
            natoms, max_nn, nimages, NL, image_of, (const double *)Ri, (const double *)g_force,
            (const double *)g_virial, (double *)g_dE, err_dev);
    else
        nep_force_virial_grad_kernel<float><<<grid, 256, 0, s>>>(
            natoms, max_nn, nimages, NL, image_of, (const float *)Ri, (const float *)g_force,
            (const float *)g_virial, (float *)g_dE, err_dev);
    return check_launch("matpl_nep_force_virial_grad");
}

static int feat_op(int dtype, int part, int mode, int natoms, int max_nn, int ntypes, int n_max,
                   int n_base, int l_max_3b, int l_max_4b, int l_max_5b, double cutoff,
                   const void *coeff, const void *d12, const long long *NL,
                   const long long *type_map, const void *G, long long ldG, const void *H, void *q,
                   long long ldQ, void *grad_d12, void *W, void *dc, void *sum, int *err_dev,
                   void *stream) {
    MATPL_REQUIRE(dtype == MATPL_F32 || dtype == MATPL_F64, MATPL_ERR_DTYPE,
                  "matpl_nep_feat_op: dtype is MATPL_F32 or MATPL_F64");
    MATPL_REQUIRE(part == 0 || part == 1, MATPL_ERR_INVALID, "part: 0 radial, 1 angular");
    MATPL_REQUIRE(mode >= 0 && mode <= 2, MATPL_ERR_INVALID, "mode: 0 fwd, 1 bwd, 2 bwd2");
    MATPL_REQUIRE(natoms >= 0 && max_nn >= 0 && ntypes >= 1 && cutoff > 0, MATPL_ERR_INVALID,
                  "bad sizes");
    MATPL_REQUIRE(n_max >= 1 && n_max <= 8 && n_base >= 1 && n_base <= 16, MATPL_ERR_UNSUPPORTED,
                  "compiled for n_max <= 8 and basis size <= 16 (coefficient dims 2, 3)");
    MATPL_REQUIRE(part == 0 || (l_max_3b >= 0 && l_max_3b <= 4 && (l_max_4b == 0 || l_max_4b == 2) &&
                                (l_max_5b == 0 || l_max_5b == 1)),
                  MATPL_ERR_UNSUPPORTED, "angular l_max (<= 4, 2 or 0, 1 or 0)");
    MATPL_REQUIRE(err_dev && coeff && type_map && (natoms == 0 || (d12 && NL)), MATPL_ERR_INVALID,
                  "null pointer argument");
    MATPL_REQUIRE(mode != 0 || q, MATPL_ERR_INVALID, "fwd needs q");
    MATPL_REQUIRE(mode != 1 || (G && (W || dc || grad_d12)), MATPL_ERR_INVALID,
                  "bwd needs G and grad_d12 or W");
    MATPL_REQUIRE(mode != 2 || (G && H && q && (W || dc)), MATPL_ERR_INVALID, "bwd2 needs G, H, gso, W");
    if (natoms == 0 || max_nn == 0) return MATPL_OK;
    MATPL_REQUIRE_ON_DEVICE(d12, "matpl_nep_feat_op");
    FeatArgs A{};
    A.natoms = natoms;
    A.nn = max_nn;
    A.ntypes = ntypes;
    A.nmax = n_max;
    A.nbase = n_base;
    A.rc = cutoff;
    A.coeff = coeff;
    A.d12 = d12;
    A.NL = NL;
    A.type = type_map;
    A.G = G;
    A.ldG = ldG;
    A.H = H;
    A.q = q;
    A.ldQ = ldQ;
    A.grad_d12 = grad_d12;
    A.W = W;
    A.dc = dc;
    A.sum = static_cast<double *>(sum);
    A.vec = (((uintptr_t)d12 | (uintptr_t)H | (uintptr_t)grad_d12) & 15u) == 0;
    A.l3 = l_max_3b;
    A.four = l_max_4b > 0;
    A.five = l_max_5b > 0;
    A.err = err_dev;
    cudaStream_t s = as_stream(stream);
    ProfScope ps(part ? "nep_mb_op" : "nep_2b_op", s);
    const bool ang = part == 1;
    if (dtype == MATPL_F64) {
        if (mode == 0) return dispatch<double, kFwd>(ang, A, s);
        if (mode == 1) return dispatch<double, kBwd>(ang, A, s);
        return dispatch<double, kBwd2>(ang, A, s);
    }
    if (mode == 0) return dispatch<float, kFwd>(ang, A, s);
    if (mode == 1) return dispatch<float, kBwd>(ang, A, s);
    return dispatch<float, kBwd2>(ang, A, s);
}

extern "C" int matpl_nep_feat_op(int dtype, int part, int mode, int natoms, int max_nn,
                                 int ntypes, int n_max, int n_base, int l_max_3b, int l_max_4b,
                                 int l_max_5b, double cutoff, const void *coeff, const void *d12,
                                 const long long *NL, const long long *type_map, const void *G,
                                 long long ldG, const void *H, void *q, long long ldQ,
                                 void *grad_d12, void *W, int *err_dev, void *stream) {
    return feat_op(dtype, part, mode, natoms, max_nn, ntypes, n_max, n_base, l_max_3b, l_max_4b,
                   l_max_5b, cutoff, coeff, d12, NL, type_map, G, ldG, H, q, ldQ, grad_d12, W,
                   nullptr, nullptr, err_dev, stream);
}

// Tables in shared memory up to 16 KB a block (four types of n 5, K 9 in FP32 take 11.5): the backward of
// 20,000 atoms takes 65 us radial and 108 angular, by a per-atom table in W 72 and 123.  Beyond that the
// tables cost more blocks on an SM than the passes over W (eight types, 46 KB: 149 and 183 us against
// 105 and 157), except in a batch of no more blocks than fit side by side anyway: up to 1,024 atoms
// eight types take 36 and 40 us against 53 and 42, so there 48 KB is allowed.
static bool feat_tabled(int dtype, int natoms, int ntypes, int n_max, int n_base) {
    const size_t esz = dtype == MATPL_F64 ? sizeof(double) : sizeof(float);
    const size_t tables = esz * kFeatWarps * ntypes * ntypes * n_max * n_base;
    return tables <= kTableBytes || (tables <= 3 * kTableBytes && natoms <= 1024);
}

extern "C" size_t matpl_nep_feat_grad_workspace_bytes(int dtype, int part, int natoms, int ntypes,
                                                      int n_max, int n_base) {
    const size_t row = (size_t)ntypes * n_max * n_base;
    if (feat_tabled(dtype, natoms, ntypes, n_max, n_base)) return 8 * (row * ntypes + 1);
    return (dtype == MATPL_F64 ? sizeof(double) : sizeof(float)) * natoms *
           (part == 0 ? (size_t)ntypes * n_base : row);
}

extern "C" int matpl_nep_feat_grad(int dtype, int part, int mode, int natoms, int max_nn,
                                   int ntypes, int n_max, int n_base, int l_max_3b, int l_max_4b,
                                   int l_max_5b, double cutoff, const void *coeff,
                                   const void *d12, const long long *NL,
                                   const long long *type_map, const void *G, long long ldG,
                                   const void *H, void *gso, long long ldQ, void *grad_d12,
                                   void *dc, void *workspace, size_t workspace_bytes,
                                   int *err_dev, void *stream) {
    MATPL_REQUIRE(dtype == MATPL_F32 || dtype == MATPL_F64, MATPL_ERR_DTYPE,
                  "matpl_nep_feat_grad: dtype is MATPL_F32 or MATPL_F64");
    MATPL_REQUIRE(part == 0 || part == 1, MATPL_ERR_INVALID, "part: 0 radial, 1 angular");
    MATPL_REQUIRE(mode == kBwd || mode == kBwd2, MATPL_ERR_INVALID, "mode: 1 bwd, 2 bwd2");
    MATPL_REQUIRE(natoms >= 0 && max_nn >= 0 && ntypes >= 1, MATPL_ERR_INVALID, "bad sizes");
    MATPL_REQUIRE(n_max >= 1 && n_max <= 8 && n_base >= 1 && n_base <= 16, MATPL_ERR_UNSUPPORTED,
                  "compiled for n_max <= 8 and basis size <= 16 (coefficient dims 2, 3)");
    MATPL_REQUIRE(dc, MATPL_ERR_INVALID, "null pointer argument");
    const size_t need =
        matpl_nep_feat_grad_workspace_bytes(dtype, part, natoms, ntypes, n_max, n_base);
    MATPL_REQUIRE(need == 0 || (workspace && workspace_bytes >= need), MATPL_ERR_INVALID,
                  "workspace too small");
    MATPL_REQUIRE_ON_DEVICE(dc, "matpl_nep_feat_grad");
    cudaStream_t s = as_stream(stream);
    const size_t esz = dtype == MATPL_F64 ? sizeof(double) : sizeof(float);
    const bool tabled = feat_tabled(dtype, natoms, ntypes, n_max, n_base);
    if ((need && cudaMemsetAsync(workspace, 0, need, s) != cudaSuccess) ||
        ((natoms == 0 || max_nn == 0) &&
         cudaMemsetAsync(dc, 0, esz * ntypes * ntypes * n_max * n_base, s) != cudaSuccess)) {
        set_error("matpl_nep_feat_grad: memset failed");
        return MATPL_ERR_CUDA;
    }
    const int st = feat_op(dtype, part, mode, natoms, max_nn, ntypes, n_max, n_base, l_max_3b,
                           l_max_4b, l_max_5b, cutoff, coeff, d12, NL, type_map, G, ldG, H, gso,
                           ldQ, grad_d12, tabled ? nullptr : workspace, tabled ? dc : nullptr,
                           workspace, err_dev, stream);
    if (st != MATPL_OK || tabled || natoms == 0 || max_nn == 0) return st;
    return matpl_nep_cgrad(dtype, part, natoms, ntypes, n_max, n_base, type_map, G, ldG, workspace,
                           dc, err_dev, stream);
}
