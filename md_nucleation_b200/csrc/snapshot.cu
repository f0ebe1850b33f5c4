/*
 * snapshot.cu -- the output path: every replica's in-domain atoms (what
 * MD::export_dump_close writes, src/output/output.cpp:133-170) and energies
 * gathered on the device into one packed staging buffer and copied to the
 * host with one asynchronous copy per array.
 *
 * Layout of a snapshot: replica r owns rows [offset[r], offset[r+1]); inside
 * a replica the ion atoms come first, then the gas atoms of the in-domain
 * molecules (ascending molecule index), then the vapor atoms -- the order of
 * the reference's dump loop over molecules with region[i] set.
 */
#include <cuda_runtime.h>

#include "mdn.h"
#include "mdn_types.h"

namespace {

/* Row offsets: one block, kCountThreads replicas at a time, a prefix sum over
 * the block (one thread that walked the replicas, two dependent loads each,
 * took 160 us for 256 of them). */
constexpr int kCountThreads = 1024;
__global__ void __launch_bounds__(kCountThreads) snapshot_counts(const RepParams* P, const RepDyn* D, int R,
                                                                  long long* offset) {
  __shared__ long long warp_sum[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  long long base = 0;
  for (int r0 = 0; r0 < R; r0 += blockDim.x) {
    const int r = r0 + (int)threadIdx.x;
    long long n = 0;
    if (r < R)
      n = P[r].n_ion + (long long)D[r].n_gas_in * P[r].a_g +
          (long long)D[r].n_vap_in * (P[r].n_vap > 0 ? P[r].a_v : 0);
    long long v = n;
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) warp_sum[wid] = v;
    __syncthreads();
    if (wid == 0) {
      long long w = lane < nw ? warp_sum[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
      }
      warp_sum[lane] = w;
    }
    __syncthreads();
    if (r < R) offset[r] = base + (wid > 0 ? warp_sum[wid - 1] : 0) + v - n;
    base += warp_sum[nw - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) offset[R] = base;
}

/* blocks per replica: a replica holds 500 to 20,000 rows */
constexpr int kGatherBlocks = 8;

/* Rows of replica blockIdx.y, a component (x or v, three per row) per thread,
 * so that a warp's stores and, within a molecule's slab rows, its loads are
 * contiguous. */
__global__ void snapshot_gather(const RepParams* P, const RepDyn* D, const int* iblob, const long long* offset,
                                long long capacity, const double* ion_x, const double* ion_v, const double* slab_x,
                                const double* slab_v, const double* vslab_x, const double* vslab_v, int* type,
                                double* x, double* v) {
  const int r = blockIdx.y;
  const RepParams& p = P[r];
  const RepDyn& d = D[r];
  const long long base = offset[r];
  const int* ib = iblob + p.iblob_off;
  const int ni = p.n_ion, ag = p.a_g, av = p.a_v;
  const long long ng = (long long)d.n_gas_in * ag;
  const long long nv = p.n_vap > 0 ? (long long)d.n_vap_in * av : 0;
  /* a replica's gas rows and vapor rows lie one after another in its slabs,
   * in the order of the snapshot */
  const size_t gas0 = (size_t)p.slab_off + (size_t)d.parity * p.slab_cap * ag;
  const size_t vap0 = (size_t)p.vslab_off + (size_t)d.parity * p.vcap * av;
  const long long n = min(ni + ng + nv, capacity - base);
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < 3 * n;
       q += (long long)gridDim.x * blockDim.x) {
    const long long t = q / 3;
    const int k = (int)(q - 3 * t);
    const double *sx, *sv;
    size_t g;
    int ty;
    if (t < ni) {
      sx = ion_x, sv = ion_v;
      g = (size_t)p.ion_off + t;
      ty = p.o_ion_type + (int)t;
    } else if (t < ni + ng) {
      sx = slab_x, sv = slab_v;
      g = gas0 + (t - ni);
      ty = p.o_gas_type + (int)((t - ni) % ag);
    } else {
      sx = vslab_x, sv = vslab_v;
      g = vap0 + (t - ni - ng);
      ty = p.o_vap_type + (int)((t - ni - ng) % av);
    }
    x[3 * base + q] = sx[3 * g + k];
    v[3 * base + q] = sv[3 * g + k];
    if (k == 0) type[base + t] = ib[ty];
  }
}

}  // namespace

/* Host side, called from engine.cu and snapshot_noalloc.cu with the
 * handle's device pointers.  Returns the launch error it read (and thereby
 * cleared), cudaSuccess when both kernels were queued. */
cudaError_t mdn_snapshot_device(const RepParams* dP, const RepDyn* dD, const int* d_iblob, int R,
                                const double* ion_x, const double* ion_v, const double* slab_x,
                                const double* slab_v, const double* vslab_x, const double* vslab_v,
                                long long* d_offset, int* d_type, double* d_x, double* d_v, long long d_capacity,
                                cudaStream_t stream) {
  snapshot_counts<<<1, R <= 32 ? 32 : kCountThreads, 0, stream>>>(dP, dD, R, d_offset);
  /* replicas in y: at most 65,535 to a launch */
  for (int r0 = 0; r0 < R; r0 += 65535)
    snapshot_gather<<<dim3(kGatherBlocks, R - r0 < 65535 ? R - r0 : 65535), 256, 0, stream>>>(
        dP + r0, dD + r0, d_iblob, d_offset + r0, d_capacity, ion_x, ion_v, slab_x, slab_v, vslab_x, vslab_v, d_type,
        d_x, d_v);
  return cudaGetLastError();
}

/* Loads the snapshot kernels on the current device (under lazy module
 * loading a kernel's module is loaded, and its code memory allocated, when
 * the kernel is first named), so that a later snapshot loads nothing. */
__attribute__((visibility("hidden"))) cudaError_t mdn_snapshot_load_kernels() {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, snapshot_counts);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, snapshot_gather);
  return e;
}
