// Mixed-precision DP fitting net (and its adjoint) on the tcgen05 tensor cores.
//
// Same math as dp_fused.cu's dp_fit (src/model/dp_embedding.py:140-163 and dp_dp.py:304-342 plus
// the autograd adjoint down to dE/dA): per atom D = A^T A[:, :16] (400), Ei = fit(D), dE/dA.
// Atoms are first sorted by element (fit_order, a stable counting sort), so that a CTA owns a
// tile of 128 atoms of one element (MMA M = 128) and runs that element's net only.  Two threads
// share an atom: thread (r, half) forms one of the two D columns of a chunk, holds 32 of the 64
// (padded) hidden columns and two of the four rows of dE/dA.  A tile is one chain of 24 dependent
// steps, so its length is what the kernel takes at any batch up to two tiles per SM.  One thread
// per atom, weights copied in front of each step and dE/dA added up in global memory took 84 us
// per tile and 122 us for 250 tiles (32,000 atoms); two threads, weights copied behind the step
// before and dE/dA kept on chip take 37 and 53 us.
//
//   layer 1  h1 = D W0: 13 K-chunks of 32; each chunk of D is built on the SIMT cores from the
//            atom's A (kept in shared memory) and double-buffered into the MMA (N = 64, the 50
//            outputs padded), FP32 accumulator in 64 TMEM columns.
//   layers 2, 3 (50 x 50 padded to 64 x 64) and the two transposed GEMMs of the adjoint run as
//            single MMAs (K = 64); tanh / residual / bias on SIMT; the three layers' tanh
//            outputs are stashed in TMEM (tcgen05.st) for the adjoint.
//   dE/dD = g1 W0^T (N = 400) in 7 chunks of 64 columns, each consumed straight from TMEM into
//            dE/dA = sum_q dD[p][q] A[c][q] + sum_p' dD[p'][p] A[c][p'].
// BF16x3 (hi/lo split) operands keep FP32-level accuracy; weight tiles are prepared once per
// call in global memory (prep_fit_tiles).  Every mbarrier wait is bounded (MATPL_KERR_TIMEOUT).
#include "common.cuh"
#include "dp_layout.cuh"
#include "tc.cuh"

namespace matpl {
namespace {

using namespace dp;
constexpr int FM = 128;                   // atoms per tile
constexpr int FT = 2 * FM;                // threads
constexpr int HC = 32;                    // hidden columns per thread
constexpr int FN = 64;                    // padded fitting width
constexpr int K1C = 13;                   // K chunks of layer 1 (32 each; 400 padded to 416)
constexpr int NDC = 7;                    // N chunks of dE/dD (64 each; 400 padded to 448)
constexpr int XKS = FM / 8 * 128;         // K-chunk stride of a 128-row activation tile (2048 B)
constexpr int BKS = FN / 8 * 128;         // K-chunk stride of a 64-row weight tile (1024 B)
constexpr int X32 = FM * 32 * 2;          // 128 x 32 bf16 tile (8 KB)
constexpr int X64 = FM * 64 * 2;          // 128 x 64 bf16 tile (16 KB)
constexpr int W32 = FN * 32 * 2;          // 64 x 32 bf16 weight tile (4 KB)
constexpr int W64 = FN * 64 * 2;          // 64 x 64 bf16 weight tile (8 KB)
constexpr int ASTR = NA + 1;              // A row stride in shared memory (floats)
constexpr int kWait = 1 << 24;

// Per-net tile offsets in the prepared buffer (each entry is a hi tile followed by a lo tile).
constexpr size_t OFF_F0 = 0;                                  // [13] 64 x 32: B[n=o][k] = W0[32c+k][o]
constexpr size_t OFF_F1 = OFF_F0 + (size_t)K1C * 2 * W32;     // 64 x 64: B[n=o][k=i] = W1[i][o]
constexpr size_t OFF_F2 = OFF_F1 + 2 * W64;                   // W2 likewise
constexpr size_t OFF_B2 = OFF_F2 + 2 * W64;                   // B[n=i][k=o] = W2[i][o]
constexpr size_t OFF_B1 = OFF_B2 + 2 * W64;                   // B[n=i][k=o] = W1[i][o]
constexpr size_t OFF_B0 = OFF_B1 + 2 * W64;                   // [7] 64 x 64: B[n=kD][k=o] = W0[64c+n][o]
constexpr size_t FIT_TILE_BYTES = OFF_B0 + (size_t)NDC * 2 * W64;

__device__ __forceinline__ void put_hilo(unsigned char *hi, unsigned char *lo, uint32_t off,
                                         float v) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    *reinterpret_cast<__nv_bfloat16 *>(hi + off) = h;
    *reinterpret_cast<__nv_bfloat16 *>(lo + off) = __float2bfloat16_rn(v - __bfloat162float(h));
}

__global__ void prep_fit_tiles(const float *__restrict__ params, unsigned char *__restrict__ out,
                               int ntypes) {
    const long long woff = (long long)ntypes * ntypes * EmbOff::SIZE;
    // work items: per net, (13 + 7) chunks x 64 x 64 elements + 4 matrices x 64 x 64
    const int per_net = (K1C * 32 + NDC * 64 + 4 * 64) * FN;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
         q < (long long)ntypes * per_net; q += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(q / per_net);
        int r = (int)(q - (long long)t * per_net);
        const float *fw = params + woff + (long long)t * FitOff::SIZE;
        unsigned char *base = out + (size_t)t * FIT_TILE_BYTES;
        const int n = r % FN;                 // weight-tile row
        int k = r / FN;                       // running K index over all tiles of the net
        if (k < K1C * 32) {                   // layer-1 chunks (K = 32 each)
            const int c = k / 32, kk = k % 32, kD = 32 * c + kk;
            const float v = (kD < DIN && n < F) ? fw[FitOff::W0 + kD * F + n] : 0.f;
            unsigned char *hi = base + OFF_F0 + (size_t)c * 2 * W32;
            put_hilo(hi, hi + W32, tc::tile_off(n, kk, BKS), v);
            continue;
        }
        k -= K1C * 32;
        if (k < 4 * 64) {                     // the four 64 x 64 hidden-layer tiles
            const int mat = k / 64, kk = k % 64;
            float v = 0.f;
            if (n < F && kk < F) {
                switch (mat) {
                    case 0: v = fw[FitOff::W1 + kk * F + n]; break;   // F1: W1[i=kk][o=n]
                    case 1: v = fw[FitOff::W2 + kk * F + n]; break;   // F2
                    case 2: v = fw[FitOff::W2 + n * F + kk]; break;   // B2: W2[i=n][o=kk]
                    default: v = fw[FitOff::W1 + n * F + kk]; break;  // B1
                }
            }
            const size_t offs[4] = {OFF_F1, OFF_F2, OFF_B2, OFF_B1};
            unsigned char *hi = base + offs[mat];
            put_hilo(hi, hi + W64, tc::tile_off(n, kk, BKS), v);
            continue;
        }
        k -= 4 * 64;                          // dE/dD chunks: N = 64 rows of D index, K = o
        const int c = k / 64, kk = k % 64, kD = 64 * c + n;
        const float v = (kD < DIN && kk < F) ? fw[FitOff::W0 + kD * F + kk] : 0.f;
        unsigned char *hi = base + OFF_B0 + (size_t)c * 2 * W64;
        put_hilo(hi, hi + W64, tc::tile_off(n, kk, BKS), v);
    }
}

// Asynchronous 16-byte global -> shared copies (cp.async), waited for with cp_async_wait_all.
__device__ __forceinline__ void copy_tiles_async(const unsigned char *__restrict__ src,
                                                 unsigned char *dst, int bytes) {
    for (int q = threadIdx.x; q < bytes / 16; q += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(dst + 16 * q)),
                     "l"(src + 16 * q)
                     : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Row r of a 128-row K-major tile: NK values from column 8 c0 as BF16 hi and lo halves.
template <int NK>
__device__ __forceinline__ void store_row_hilo(unsigned char *hi, unsigned char *lo, int r, int c0,
                                               const float *v) {
#pragma unroll
    for (int c = 0; c < NK / 8; ++c) {
        float h[8], l[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            h[q] = v[8 * c + q];
            l[q] = v[8 * c + q] - __bfloat162float(__float2bfloat16_rn(v[8 * c + q]));
        }
        tc::store_row8(hi, r, c0 + c, XKS, h);
        tc::store_row8(lo, r, c0 + c, XKS, l);
    }
}

// Shared memory written by the threads becomes visible to the tensor core, and prior TMEM
// reads are ordered before the next MMA.
__device__ __forceinline__ void mma_sync_point() {
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
}

// D[128 x 64] (+)= X W with BF16x3 operands; KCH K-steps of 16.
template <int KCH>
__device__ __forceinline__ void issue_split3(uint32_t tmem, const unsigned char *xh,
                                             const unsigned char *xl, const unsigned char *wh,
                                             const unsigned char *wl, bool accumulate) {
    const uint32_t id = tc::idesc_bf16(FM, FN);
    const uint32_t a[2] = {tc::smem_u32(xh), tc::smem_u32(xl)};
    const uint32_t b[2] = {tc::smem_u32(wh), tc::smem_u32(wl)};
    uint32_t acc = accumulate ? 1u : 0u;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const uint32_t xa = a[p == 2 ? 1 : 0], wb = b[p == 1 ? 1 : 0];
#pragma unroll
        for (int kk = 0; kk < KCH; ++kk) {
            tc::mma_bf16(tmem, tc::desc_kmajor(xa + kk * 2 * XKS, XKS, 128),
                         tc::desc_kmajor(wb + kk * 2 * BKS, BKS, 128), id, acc);
            acc = 1u;
        }
    }
}

template <bool FAST>
__device__ __forceinline__ float fit_act(float x) {
    if (FAST) return tc::tanh_fast(x);
    return tanhf(x);
}

constexpr size_t FIT_SMEM = sizeof(float) * (FM * ASTR) + 2 * X64 + 2 * W64;
constexpr int FIT_TCOLS = 256;   // TMEM: [0, 64) accumulator, [64 + 64 l, 128 + 64 l) tanh of layer l

// Stable counting sort of the atoms of one image by model type into order[natoms], with
// type_start[0..ntypes+1] (bucket ntypes: atoms whose type is not evaluated), in two launches
// over 1024-atom blocks: per-block bucket counts, then per-block offsets (previous blocks'
// counts) and the ranks inside the block (warp match + a prefix over the block's warps).
constexpr int kOrderBlock = 1024;

__device__ __forceinline__ int fit_bucket(const int32_t *__restrict__ type_map, int i, int ntypes,
                                          int present_mask) {
    const int t = type_map[i];
    return (t >= 0 && t < ntypes && ((present_mask >> t) & 1)) ? t : ntypes;
}

__global__ void fit_order_count(const int32_t *__restrict__ type_map, int natoms, int ntypes,
                                int present_mask, int *__restrict__ blk_count) {
    __shared__ int cnt[17];
    if (threadIdx.x < 17) cnt[threadIdx.x] = 0;
    __syncthreads();
    const int i = blockIdx.x * kOrderBlock + threadIdx.x;
    if (i < natoms) atomicAdd(&cnt[fit_bucket(type_map, i, ntypes, present_mask)], 1);
    __syncthreads();
    if (threadIdx.x <= ntypes) blk_count[blockIdx.x * 17 + threadIdx.x] = cnt[threadIdx.x];
}

__global__ void fit_order_scatter(const int32_t *__restrict__ type_map, int natoms, int ntypes,
                                  int present_mask, const int *__restrict__ blk_count,
                                  int *__restrict__ order, int *__restrict__ type_start) {
    __shared__ int base[17];                   // global start of this block's atoms per bucket
    __shared__ int wcnt[kOrderBlock / 32][17];
    __shared__ int before_s[17], total_s[17];  // per bucket: earlier blocks' atoms, all atoms
    const int T = ntypes + 1, nblk = gridDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // every block's bucket counts, summed by one warp per bucket (lanes over blocks, then a
    // shuffle tree), instead of one thread walking them serially
    for (int q = warp; q < T; q += kOrderBlock / 32) {
        int bef = 0, tot = 0;
        for (int b = lane; b < nblk; b += 32) {
            const int v = blk_count[b * 17 + q];
            tot += v;
            if (b < (int)blockIdx.x) bef += v;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            bef += __shfl_xor_sync(0xffffffffu, bef, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if (lane == 0) {
            before_s[q] = bef;
            total_s[q] = tot;
        }
    }
    __syncthreads();
    if (threadIdx.x < T) {
        const int q = threadIdx.x;
        int total_lower = 0;
        for (int p = 0; p < q; ++p) total_lower += total_s[p];
        base[q] = total_lower + before_s[q];
        if (blockIdx.x == 0) type_start[q] = total_lower;
        if (blockIdx.x == 0 && q == T - 1) type_start[T] = natoms;
    }
    const int i = blockIdx.x * kOrderBlock + threadIdx.x;
    const int q = i < natoms ? fit_bucket(type_map, i, ntypes, present_mask) : 17;
    const unsigned peers = __match_any_sync(0xffffffffu, q);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (lane < 17) wcnt[warp][lane] = 0;
    __syncwarp();
    if (q < 17 && rank == 0) wcnt[warp][q] = __popc(peers);
    __syncthreads();
    if (q < 17) {
        int off = base[q] + rank;
        for (int w = 0; w < warp; ++w) off += wcnt[w][q];
        order[off] = i;
    }
}

// 4-byte asynchronous copy, or a zero where !ok
__device__ __forceinline__ void copy4_async(const float *src, float *dst, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tc::smem_u32(dst)), "l"(src),
                 "r"(ok ? 4 : 0)
                 : "memory");
}

template <bool FAST>
__global__ void __launch_bounds__(FT, 2)
dp_fit_tc(const float *__restrict__ Ain, const int *__restrict__ order,
          const int *__restrict__ type_start, const float *__restrict__ params,
          const unsigned char *__restrict__ ftiles, float *__restrict__ Ei,
          float *__restrict__ dAout, int32_t *__restrict__ err, int batch, int natoms,
          int ntypes) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t tmem_base;
    __shared__ long long ratom[FM];
    __shared__ float vec[6 * FN + 4];
    __shared__ float esum[FM];
    float *As = reinterpret_cast<float *>(smem_raw);
    unsigned char *XB = reinterpret_cast<unsigned char *>(As + FM * ASTR);
    unsigned char *WB = XB + 2 * X64;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int r = tid & (FM - 1), half = tid >> 7, col0 = HC * half;
    if (tid == 0) {
        tc::mbar_init(&mbar[0], 1);
        tc::mbar_init(&mbar[1], 1);
    }
    if (warp == 0) tc::tmem_alloc(&tmem_base, FIT_TCOLS);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    // this thread's row and columns of the accumulator and of the stashes (warp w reaches the
    // TMEM lanes of quarter w % 4)
    const uint32_t tmine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col0;
    uint32_t ph[2] = {0u, 0u};
    bool ok = true;
    const long long woff = (long long)ntypes * ntypes * EmbOff::SIZE;
    const int vsrc[6] = {FitOff::B0, FitOff::B1, FitOff::DT1, FitOff::B2, FitOff::DT2, FitOff::W3};
    // tiles: per image, ceil(n_t / 128) tiles of each element t (an upper bound of their number
    // per image is ceil(natoms / 128) + ntypes; the surplus indices have no work)
    const long long tiles_b = (natoms + FM - 1) / FM + ntypes;
    for (long long v = blockIdx.x; v < (long long)batch * tiles_b; v += gridDim.x) {
        const long long b = v / tiles_b;
        int rem = (int)(v - b * tiles_b), tt = -1, chunk = 0;
        for (int q = 0; q < ntypes; ++q) {
            const int nq = (type_start[q + 1] - type_start[q] + FM - 1) / FM;
            if (rem < nq) {
                tt = q;
                chunk = rem;
                break;
            }
            rem -= nq;
        }
        if (tt < 0) continue;                      // the same for every thread of the CTA
        const int idx = type_start[tt] + chunk * FM + r;
        const bool valid = idx < type_start[tt + 1];
        const long long t = valid ? b * natoms + order[idx] : -1;
        const unsigned char *tw = ftiles + (size_t)tt * FIT_TILE_BYTES;
        __syncthreads();                           // the previous tile's buffers are free
        copy_tiles_async(tw + OFF_F0, WB, 2 * W32);
        if (half == 0) ratom[r] = t;
        {
            const float *fw = params + woff + (long long)tt * FitOff::SIZE;
            for (int q = tid; q < 6 * FN; q += FT) {
                const int part = q / FN, o = q - part * FN;
                vec[q] = o < F ? fw[vsrc[part] + o] : 0.f;
            }
            if (tid == 0) vec[6 * FN] = fw[FitOff::B3];
        }
        __syncthreads();
        for (int q = tid; q < FM * NA; q += FT) {
            const int row = q / NA, e = q - row * NA;
            const long long tr = ratom[row];
            copy4_async(Ain + (tr >= 0 ? tr * NA + e : 0), As + row * ASTR + e, tr >= 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        cp_async_wait_all();
        __syncthreads();
        float *a = As + r * ASTR;
        // ---- layer 1: 13 double-buffered K chunks of D W0.  The weights of chunk c + 1
        // are copied asynchronously while chunk c is formed and multiplied; buffer b of
        // chunk c is free once the MMA of chunk c - 2 is done (waited at the end of the
        // previous chunk, before that chunk's prefetch).
        {
            float aq[4][M2];                      // A[c][q], q < M2: every chunk's right factor
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4)
#pragma unroll
                for (int q = 0; q < M2; ++q) aq[c4][q] = a[c4 * E + q];
            for (int c = 0; c < K1C; ++c) {
                const int b = c & 1;
                const int p = 2 * c + half;
                float d[16];
                const float ap0 = p < E ? a[p] : 0.f, ap1 = p < E ? a[E + p] : 0.f,
                            ap2 = p < E ? a[2 * E + p] : 0.f, ap3 = p < E ? a[3 * E + p] : 0.f;
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    d[q] = p < E ? ap0 * aq[0][q] + ap1 * aq[1][q] + ap2 * aq[2][q] + ap3 * aq[3][q]
                                 : 0.f;
                unsigned char *xh = XB + b * 2 * X32;
                store_row_hilo<16>(xh, xh + X32, r, 2 * half, d);
                cp_async_wait_all();
                mma_sync_point();
                if (tid == 0) {
                    issue_split3<2>(tmem, xh, xh + X32, WB + b * 2 * W32, WB + b * 2 * W32 + W32, c > 0);
                    tc::commit(&mbar[b]);
                }
                if (c + 1 < K1C) {
                    if (c >= 1) {                     // the MMA of chunk c - 1 read buffer b ^ 1
                        ok &= tc::mbar_wait(&mbar[b ^ 1], ph[b ^ 1], kWait);
                        ph[b ^ 1] ^= 1u;
                    }
                    copy_tiles_async(tw + OFF_F0 + (size_t)(c + 1) * 2 * W32,
                                     WB + (b ^ 1) * 2 * W32, 2 * W32);
                }
            }
        }
        ok &= tc::mbar_wait(&mbar[1], ph[1], kWait);
        ph[1] ^= 1u;
        ok &= tc::mbar_wait(&mbar[0], ph[0], kWait);
        ph[0] ^= 1u;
        tc::fence_after_sync();
        // from here on every step's weights are copied while the step before it is finished on
        // the SIMT cores (the MMA that read the buffer is done).  real(o): hidden column, not
        // padding (those stay zero whatever an overflown row holds).
        auto real = [&](int o) { return o < F - HC || half == 0; };
        copy_tiles_async(tw + OFF_F1, WB, 2 * W64);
        float h[HC], x[HC];
        tc::tmem_ld32(tmine, h);
#pragma unroll
        for (int o = 0; o < HC; ++o) x[o] = real(o) ? fit_act<FAST>(h[o] + vec[col0 + o]) : 0.f;
        tc::tmem_st32(tmine + 64, x);
        auto run_mma64 = [&]() {                      // accumulator = X W of the staged tiles
            cp_async_wait_all();
            mma_sync_point();
            if (tid == 0) {
                issue_split3<4>(tmem, XB, XB + X64, WB, WB + W64, false);
                tc::commit(&mbar[0]);
            }
            ok &= tc::mbar_wait(&mbar[0], ph[0], kWait);
            ph[0] ^= 1u;
            tc::fence_after_sync();
        };
        // ---- layers 2, 3
#pragma unroll 1
        for (int l = 1; l <= 2; ++l) {
            store_row_hilo<HC>(XB, XB + X64, r, 4 * half, x);
            run_mma64();
            copy_tiles_async(tw + (l == 1 ? OFF_F2 : OFF_B2), WB, 2 * W64);
            tc::tmem_ld32(tmine, h);
            const float *bias = vec + (l == 1 ? FN : 3 * FN) + col0;
            const float *dt = vec + (l == 1 ? 2 * FN : 4 * FN) + col0;
#pragma unroll
            for (int o = 0; o < HC; ++o) {
                h[o] = real(o) ? fit_act<FAST>(h[o] + bias[o]) : 0.f;
                x[o] = fmaf(h[o], dt[o], x[o]);
            }
            tc::tmem_st32(tmine + 64 + 64 * l, h);
        }
        // Ei in column order: the first half's sum, then the second half's terms
        if (half == 0) {
            float e = vec[6 * FN];
#pragma unroll
            for (int o = 0; o < HC; ++o) e += x[o] * vec[5 * FN + o];
            esum[r] = e;
        }
        __syncthreads();
        if (half == 1 && valid) {
            float e = esum[r];
#pragma unroll
            for (int o = 0; o < F - HC; ++o) e += x[o] * vec[5 * FN + HC + o];
            Ei[t] = e;
        }
        // ---- adjoint: dx3 = W3; through layers 3 and 2
#pragma unroll
        for (int o = 0; o < HC; ++o) x[o] = vec[5 * FN + col0 + o];
#pragma unroll 1
        for (int l = 2; l >= 1; --l) {
            const float *dt = vec + (l == 2 ? 4 * FN : 2 * FN) + col0;
            tc::tmem_ld32(tmine + 64 + 64 * l, h);    // tanh outputs of layer l
#pragma unroll
            for (int o = 0; o < HC; ++o) h[o] = real(o) ? x[o] * dt[o] * (1.f - h[o] * h[o]) : 0.f;
            store_row_hilo<HC>(XB, XB + X64, r, 4 * half, h);
            run_mma64();
            copy_tiles_async(tw + (l == 2 ? OFF_B1 : OFF_B0), WB, 2 * W64);
            tc::tmem_ld32(tmine, h);
#pragma unroll
            for (int o = 0; o < HC; ++o) x[o] += h[o];     // padding: masked when it is used
        }
        tc::tmem_ld32(tmine + 64, h);                 // tanh outputs of layer 1
#pragma unroll
        for (int o = 0; o < HC; ++o) h[o] = real(o) ? x[o] * (1.f - h[o] * h[o]) : 0.f;
        store_row_hilo<HC>(XB, XB + X64, r, 4 * half, h);
        // ---- dE/dD = g1 W0^T in 7 chunks of 64 D entries (columns p = 4c + j, q), folded into
        // rows 2 half and 2 half + 1 of dE/dA:
        //   dA[c4][p] = sum_q dD[p][q] A[c4][q] (+ sum_p' dD[p'][p] A[c4][p'] for p < 16).
        // Column p of A is used by chunk c only when p >= 16, so dA[p] replaces it in shared
        // memory; the first 16 columns wait in registers for their second sum.
        float acc2[2][16], first[2][16];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int q = 0; q < 16; ++q) acc2[k][q] = 0.f;
        float *ah = a + 2 * half * E;
#pragma unroll
        for (int c = 0; c < NDC; ++c) {
            run_mma64();
            if (c + 1 < NDC) copy_tiles_async(tw + OFF_B0 + (size_t)(c + 1) * 2 * W64, WB, 2 * W64);
#pragma unroll
            for (int jp = 0; jp < 4; jp += 2) {       // two D columns at a time
                if (4 * c + jp >= E) break;
                tc::tmem_ld32(tmine - col0 + 16 * jp, h);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    float sj[2] = {0.f, 0.f};
#pragma unroll
                    for (int q = 0; q < M2; ++q) {
                        const float aqv = ah[k * E + q];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            if (4 * c + jp + j >= E) break;
                            sj[j] += h[16 * j + q] * aqv;
                            acc2[k][q] += h[16 * j + q] * ah[k * E + 4 * c + jp + j];
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        if (4 * c + jp + j >= E) break;
                        if (4 * c + jp + j < 16) first[k][(4 * c + jp + j) & 15] = sj[j];
                        else ah[k * E + 4 * c + jp + j] = sj[j];
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int q = 0; q < 16; ++q) ah[k * E + q] = first[k][q] + acc2[k][q];
        __syncthreads();
        for (int q = tid; q < FM * NA; q += FT) {
            const int row = q / NA, e = q - row * NA;
            const long long tr = ratom[row];
            if (tr >= 0) dAout[tr * NA + e] = As[row * ASTR + e];
        }
    }
    // atoms whose element is not evaluated: Ei = 0, dE/dA = 0
    const int nskip = type_start[ntypes + 1] - type_start[ntypes];
    for (long long q = (long long)blockIdx.x * FT + tid; q < (long long)batch * nskip;
         q += (long long)gridDim.x * FT) {
        const long long b = q / nskip;
        const long long t = b * natoms + order[type_start[ntypes] + (int)(q - b * nskip)];
        Ei[t] = 0.f;
        for (int e = 0; e < NA; ++e) dAout[t * NA + e] = 0.f;
    }
    if (!ok) atomicMax(err, MATPL_KERR_TIMEOUT);
    // nothing issued may still run when the TMEM is freed: one more commit after all of this
    // thread's MMAs, waited for (bounded) by every thread
    __shared__ __align__(8) uint64_t mbar_drain;
    if (tid == 0) {
        tc::mbar_init(&mbar_drain, 1);
        tc::commit(&mbar_drain);
    }
    __syncthreads();
    tc::mbar_wait(&mbar_drain, 0u, kWait);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, FIT_TCOLS);
}

}  // namespace

// Prepared tiles of every element, then the element order of the atoms (order [natoms],
// type_start [ntypes + 2], per-block bucket counts of the sort).
size_t fit_tile_bytes(int ntypes, int natoms) {
    const size_t nblk = ((size_t)natoms + kOrderBlock - 1) / kOrderBlock;
    return align_up((size_t)ntypes * FIT_TILE_BYTES, 256) + align_up(sizeof(int) * natoms, 256) +
           sizeof(int) * (32 + 17 * nblk);
}

// Prepares the BF16 fitting tiles of every type into `tiles`, then runs the fitting kernel.
int launch_fit_tc(bool fast, const float *A, const int32_t *type_map, const float *params,
                  unsigned char *tiles, float *Ei, float *dA, int32_t *err, int batch, int natoms,
                  int ntypes, int present_mask, cudaStream_t s) {
    {
        ProfScope ps("prep_fit_tiles", s);
        const long long n = (long long)ntypes * (K1C * 32 + NDC * 64 + 4 * 64) * FN;
        prep_fit_tiles<<<(int)((n + 255) / 256), 256, 0, s>>>(params, tiles, ntypes);
    }
    int *order = reinterpret_cast<int *>(tiles + align_up((size_t)ntypes * FIT_TILE_BYTES, 256));
    int *type_start = order + align_up(sizeof(int) * natoms, 256) / sizeof(int);
    int *blk_count = type_start + 32;
    const int nblk = (natoms + kOrderBlock - 1) / kOrderBlock;
    if (nblk > 0) {
        ProfScope ps("fit_order", s);
        fit_order_count<<<nblk, kOrderBlock, 0, s>>>(type_map, natoms, ntypes, present_mask,
                                                    blk_count);
        fit_order_scatter<<<nblk, kOrderBlock, 0, s>>>(type_map, natoms, ntypes, present_mask,
                                                      blk_count, order, type_start);
    }
    const long long tiles_b = (natoms + FM - 1) / FM + ntypes;
    const long long ntiles = (long long)batch * tiles_b;
    const long long cap = 2LL * device_sms();            // two resident CTAs per SM
    const int grid = (int)(ntiles < cap ? ntiles : cap);
    auto k = fast ? dp_fit_tc<true> : dp_fit_tc<false>;
    allow_smem(k, FIT_SMEM);
    ProfScope ps("dp_fit_tc", s);
    k<<<grid, FT, FIT_SMEM, s>>>(A, order, type_start, params, tiles, Ei, dA, err, batch, natoms,
                                 ntypes);
    return check_launch("dp_fit_tc");
}

}  // namespace matpl
