// Read-back of a field: the padded device rows as one dense array in pinned
// host memory (phono_download).
//
// A strided copy moves a row (nz elements, 260 bytes to 1 KB) at a time.  Here
// a thread gathers 16 bytes of the dense array, whichever rows they lie in, and
// stores them to the host array through its device address, so that a warp
// writes 512 contiguous bytes.  Bound by the link to the host: 190 GB/s, the
// rate of a contiguous copy (191).  us a field, strided copy / here: 160x128x64
// cells FP32 117 to 135 / 47, 256x256x128 420 / 196, 512x512x256 2000 / 1420,
// 149x130x46 FP64 133 / 59; fields of a few kilobytes 20 either way.  (uz of a
// mesh of 2^n cells has the rows the strided copy likes and takes the same.)
#include <cstdint>
#include <cuda_runtime.h>

namespace phono {

// Vector v holds elements [v * VE - lead, + VE) of the n = ex * ey * ez dense
// ones; `lead` elements lie between the 16-byte boundary at or before out and
// out itself, so that whole vectors are aligned and only the two ends are not.
template <class T>
__global__ void __launch_bounds__(256) readback_kernel(const T* __restrict__ in, long long sx, long long sy, unsigned ey,
                                                       unsigned ez, unsigned n, int lead, T* __restrict__ out) {
  constexpr int VE = 16 / sizeof(T);
  const long long e0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * VE - lead;
  if (e0 >= n) return;
  const unsigned first = e0 < 0 ? 0u : (unsigned)e0;
  const int count = (int)((e0 + VE < n ? e0 + VE : (long long)n) - first);
  unsigned row = first / ez, k = first - row * ez, i = row / ey, j = row - i * ey;
  const T* p = in + i * sx + j * sy;
  T x[VE];
#pragma unroll
  for (int q = 0; q < VE; q++) {
    if (q < count) x[q] = p[k];
    if (++k == ez) {
      k = 0;
      if (++j == ey) j = 0, i++;
      p = in + i * sx + j * sy;
    }
  }
  if (count == VE) {
    int4 w;
    memcpy(&w, x, 16);
    *reinterpret_cast<int4*>(out + first) = w;
    return;
  }
#pragma unroll
  for (int q = 0; q < VE; q++)
    if (q < count) out[first + q] = x[q];
}

template <class T>
static cudaError_t launch(const void* in, long long sx, long long sy, int ex, int ey, int ez, void* out, cudaStream_t st) {
  constexpr long long VE = 16 / sizeof(T);
  const long long n = (long long)ex * ey * ez;
  const int lead = (int)((uintptr_t)out % 16 / sizeof(T));
  const long long blocks = ((n + lead + VE - 1) / VE + 255) / 256;
  readback_kernel<T><<<(unsigned)blocks, 256, 0, st>>>((const T*)in, sx, sy, (unsigned)ey, (unsigned)ez, (unsigned)n, lead,
                                                     (T*)out);
  return cudaGetLastError();
}

// in: element (0, 0, 0) on the device; out: device address of ex * ey * ez < 2^32
// dense elements of es bytes, aligned to es
cudaError_t launch_readback(const void* in, long long sx, long long sy, int ex, int ey, int ez, int es, void* out,
                            cudaStream_t st) {
  return es == 4 ? launch<float>(in, sx, sy, ex, ey, ez, out, st) : launch<double>(in, sx, sy, ex, ey, ez, out, st);
}

}  // namespace phono
