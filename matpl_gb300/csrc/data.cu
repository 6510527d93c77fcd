// Data-path statistics: the sums behind davg / dstd, replacing the per-image calc_stat +
// smooth of src/pre_data/dpuni_data_loader.py:422-563 (called from calculate_davg_dstd,
// :377-420, for the images set_davg_dstd picks, :180-215).
//
// For every configuration b and centre type t it accumulates over all slots of the atoms of
// type t the smoothed environment rows Ri = vv(r) * (1/r, x/r^2, y/r^2, z/r^2), r and r^2
// from the pair vector (x, y, z) of image_dr as calc_stat forms them (vv the
// switching function of smooth with the model's Rmin / Rmax): sums of Ri_0, Ri_0^2 and of the
// three angular channels and their squares, in FP64.  The caller turns them into davg / dstd
// (the slot count per type is known on the host).  One warp per atom, lanes over slots, warp
// reduction, one FP64 atomic per (b, t, channel) and warp.
#include <algorithm>

#include "common.cuh"

namespace matpl {
namespace {

__global__ void __launch_bounds__(128)
env_stats_kernel(int batch, int natoms, int nslots, int ntypes, const int32_t *__restrict__ type_map,
                 const int32_t *__restrict__ list_neigh, const double *__restrict__ image_dr,
                 double rmin, double rmax, double *__restrict__ sums, int32_t *__restrict__ err) {
    const int lane = threadIdx.x & 31;
    const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
    const long long total = (long long)batch * natoms;
    for (long long ba = gw; ba < total; ba += nw) {
        const int b = (int)(ba / natoms), a = (int)(ba - (long long)b * natoms);
        const int t = type_map[a];
        if (t < 0 || t >= ntypes) {
            if (lane == 0) atomicMax(err, MATPL_KERR_BAD_TYPE);
            continue;
        }
        double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int s = lane; s < nslots; s += 32) {
            const long long q = ba * nslots + s;
            if (list_neigh[q] <= 0) continue;
            // the reference's order: dR2 from the pair vector, Rij = sqrt(dR2), r = dR2 / Rij
            const double x = image_dr[4 * q + 1], y = image_dr[4 * q + 2], z = image_dr[4 * q + 3];
            const double r2 = x * x + y * y + z * z;
            const double r = r2 / sqrt(r2);
            double vv;
            if (r < rmin) vv = 1.0;
            else if (r < rmax) {
                const double u = (r - rmin) / (rmax - rmin);
                vv = u * u * u * (-6.0 * u * u + 15.0 * u - 10.0) + 1.0;
            } else vv = 0.0;
            const double c[4] = {vv / r, vv * x / r2, vv * y / r2, vv * z / r2};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[2 * k] += c[k];
                acc[2 * k + 1] += c[k] * c[k];
            }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = warp_sum(acc[k]);
        if (lane < 8) {
            double v = acc[0];
#pragma unroll
            for (int k = 1; k < 8; ++k) v = lane == k ? acc[k] : v;
            atomicAdd(&sums[((long long)b * ntypes + t) * 8 + lane], v);
        }
    }
}

// Bound: latency.  One block: a type map is some kilobytes (16,000 int32: four loads a thread).
__global__ void __launch_bounds__(1024)
bytes_differ_kernel(const unsigned char *__restrict__ a, const unsigned char *__restrict__ b,
                    size_t n, int32_t *answer) {
    const uintptr_t at = (uintptr_t)a | (uintptr_t)b;
    size_t done = 0;
    bool d = false;
    if ((at & 15u) == 0) {
        const uint4 *x = reinterpret_cast<const uint4 *>(a), *y = reinterpret_cast<const uint4 *>(b);
        for (size_t q = threadIdx.x; q < n / 16; q += blockDim.x) {
            const uint4 u = x[q], v = y[q];
            d |= ((u.x ^ v.x) | (u.y ^ v.y) | (u.z ^ v.z) | (u.w ^ v.w)) != 0u;
        }
        done = n / 16 * 16;
    } else if ((at & 3u) == 0) {
        const unsigned *x = reinterpret_cast<const unsigned *>(a), *y = reinterpret_cast<const unsigned *>(b);
        for (size_t q = threadIdx.x; q < n / 4; q += blockDim.x) d |= x[q] != y[q];
        done = n / 4 * 4;
    }
    for (size_t q = done + threadIdx.x; q < n; q += blockDim.x) d |= a[q] != b[q];
    const int any = __syncthreads_or(d);
    if (threadIdx.x == 0) *answer = any != 0;
}

}  // namespace
}  // namespace matpl

using namespace matpl;

extern "C" int matpl_bytes_differ(const void *a, const void *b, size_t bytes, int32_t *answer,
                                  void *stream) {
    MATPL_REQUIRE(answer && (bytes == 0 || (a && b)), MATPL_ERR_INVALID, "null pointer argument");
    MATPL_REQUIRE_ON_DEVICE(a, "matpl_bytes_differ");
    bytes_differ_kernel<<<1, 1024, 0, as_stream(stream)>>>(
        static_cast<const unsigned char *>(a), static_cast<const unsigned char *>(b), bytes, answer);
    return check_launch("matpl_bytes_differ");
}

extern "C" int matpl_env_stats(int batch, int natoms, int nslots, int ntypes,
                               const int32_t *type_map, const int32_t *list_neigh,
                               const double *image_dr, double rmin, double rmax, double *sums,
                               int32_t *err_dev, void *stream) {
    MATPL_REQUIRE(batch >= 0 && natoms >= 0 && nslots >= 0 && ntypes >= 1, MATPL_ERR_INVALID,
                  "bad sizes");
    MATPL_REQUIRE(rmax > rmin && rmin >= 0, MATPL_ERR_INVALID, "need 0 <= rmin < rmax");
    MATPL_REQUIRE(sums && err_dev && (batch * (long long)natoms == 0 ||
                                      (type_map && list_neigh && image_dr)),
                  MATPL_ERR_INVALID, "null pointer argument");
    cudaStream_t s = as_stream(stream);
    MATPL_REQUIRE_ON_DEVICE(sums, "matpl_env_stats");
    if (cudaMemsetAsync(sums, 0, sizeof(double) * 8 * (size_t)batch * ntypes, s) != cudaSuccess) {
        set_error("matpl_env_stats: memset failed");
        return MATPL_ERR_CUDA;
    }
    const long long total = (long long)batch * natoms;
    if (total == 0 || nslots == 0) return MATPL_OK;
    ProfScope ps("env_stats", s);
    const long long grid = std::min<long long>((total + 3) / 4, (long long)device_sms() * 16);
    env_stats_kernel<<<(int)grid, 128, 0, s>>>(batch, natoms, nslots, ntypes, type_map,
                                               list_neigh, image_dr, rmin, rmax, sums, err_dev);
    return check_launch("matpl_env_stats");
}
