// Copies of several fields in one launch: a handle's fields to and from its
// pinned host mirrors, and a batch's packed fields to and from its members.
#include <algorithm>

#include "fg_internal.cuh"

namespace fg {

namespace {

// Every item a linear array of rows x width floats on one side and the same
// rows at a pitch on the other (a batch's slices: width = pitch).  Linear
// storage is walked in 16-byte pieces, so writes to a host mirror leave the
// chip as whole lines whatever the width; the pitched side is addressed in
// 16-byte pieces where the width allows it.  Bound by the host link for mirrors
// (185 GB/s; small ones by the launch: 4 fields of 130 x 130 in 10 us with the
// synchronisation, 17 by four copies) and by HBM for a batch's slices (147
// slices of 21 scenes in 33 us with both synchronisations, 640 by copies).
template <bool TO_LINEAR>
__global__ void __launch_bounds__(256) k_copy_list(const __grid_constant__ CopyList l) {
  const CopyItem c = l.it[blockIdx.y];
  const unsigned W = c.width, n = c.rows * W, n4 = n / 4;
  const bool vec = (W & 3) == 0 && (c.pitch & 3) == 0 &&
                   (reinterpret_cast<uintptr_t>(c.pitched) & 15) == 0;
  for (unsigned k = blockIdx.x * 256 + threadIdx.x; k < n4; k += gridDim.x * 256) {
    unsigned i = 4 * k / W, j = 4 * k - i * W;
    float4* lin = reinterpret_cast<float4*>(c.linear) + k;
    if (vec) {
      float4* p = reinterpret_cast<float4*>(c.pitched + (size_t)i * c.pitch + j);
      if (TO_LINEAR) *lin = *p;
      else *p = *lin;
      continue;
    }
    float v[4];
    if (!TO_LINEAR) {
      const float4 x = *lin;
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float* p = c.pitched + (size_t)i * c.pitch + j;
      if (TO_LINEAR) v[q] = *p;
      else *p = v[q];
      if (++j == W) {
        j = 0;
        ++i;
      }
    }
    if (TO_LINEAR) *lin = make_float4(v[0], v[1], v[2], v[3]);
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const unsigned e = 4 * n4 + threadIdx.x, i = e / W, j = e - i * W;
    float* p = c.pitched + (size_t)i * c.pitch + j;
    if (TO_LINEAR) c.linear[e] = *p;
    else *p = c.linear[e];
  }
}

}  // namespace

cudaError_t launch_copy_list(fg_fluid* f, const CopyList& l, bool to_linear) {
  if (l.n == 0) return cudaSuccess;
  unsigned most = 0;
  for (int k = 0; k < l.n; ++k) most = std::max(most, l.it[k].rows * l.it[k].width);
  // Two 16-byte pieces a thread, up to 128 blocks an item.
  const dim3 gr(std::min(128u, most / (8 * 256) + 1), l.n);
  count(f);
  if (to_linear) k_copy_list<true><<<gr, 256, 0, f->stream>>>(l);
  else k_copy_list<false><<<gr, 256, 0, f->stream>>>(l);
  return cudaGetLastError();
}

}  // namespace fg
