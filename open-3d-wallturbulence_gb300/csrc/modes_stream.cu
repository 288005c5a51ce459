// Mode-kernel variants on packed factor streams (see modes_stream.cuh), and the
// packing.
#include "modes_stream.cuh"

#include <algorithm>

namespace owt {

namespace {
// rs[p] of the listed rows, in their order
__global__ void k_str_row_scales(double *__restrict__ out, const double *__restrict__ rs, const StrRow *__restrict__ rows,
                                 int U) {
  const double *src = rs + (size_t)rows[blockIdx.y].p * U;
  for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < U; u += gridDim.x * blockDim.x)
    out[(size_t)blockIdx.y * U + u] = src[u];
}

struct Variant {
  const char *name;
  void (*kernel)(ModeArgs), (*sixth)(ModeArgs);
  void (*batch)(BatchTable<ModeArgs>, int *);
};
// seven blocks an SM fill the FP64 pipe of a large channel; where an SM has
// fewer blocks anyway the larger register budget of six is a little faster
const Variant kVariants[] = {
    {"stream/64/r128", k_modes_stream<7, VMasks>, k_modes_stream<7, VMasks6>, k_modes_stream_batch<7>},
    {"stream/64/r168", k_modes_stream<6, VMasks>, k_modes_stream<6, VMasks6>, k_modes_stream_batch<6>},
};
}  // namespace

int modes_stream_count() { return (int)(sizeof(kVariants) / sizeof(kVariants[0])); }
const char *modes_stream_name(int v) { return kVariants[v].name; }
void modes_stream_launch(int v, const ModeArgs &a, bool sixth, cudaStream_t st) {
  const int blocks = 2 * ((a.u1 + kStrModes - 1) / kStrModes - a.u0 / kStrModes);
  if (blocks > 0) (sixth ? kVariants[v].sixth : kVariants[v].kernel)<<<blocks, 64, 0, st>>>(a);
}
ModeBatchShape modes_stream_batch_shape(int v) { return {64, kMapStream, resident_blocks(kVariants[v].batch, 64, 0)}; }
void modes_stream_batch_launch(int v, const BatchTable<ModeArgs> &t, int *work, int grid, cudaStream_t st) {
  kVariants[v].batch<<<grid, 64, 0, st>>>(t, work);
}

int str_groups(int U) { return (U + kStrModes - 1) / kStrModes; }
size_t str_scratch_values(int U) { return (size_t)2 * str_groups(U) * 16; }

StrSizes str_sizes(int n_v, int n_g, bool sixth) {
  StrSizes z;
  z.vf = sixth ? StrLayout<StrV<VMasks6>>::fwd_size(n_v) : StrLayout<StrV<VMasks>>::fwd_size(n_v);
  z.vb = sixth ? StrLayout<StrV<VMasks6>>::bwd_size(n_v) : StrLayout<StrV<VMasks>>::bwd_size(n_v);
  z.gf = StrLayout<StrG>::fwd_size(n_g);
  z.gb = StrLayout<StrG>::bwd_size(n_g);
  return z;
}

void launch_str_pack(const ModeArgs &a, bool sixth, const StrBuffers &s, int nvrows, int ngrows, cudaStream_t st) {
  const int groups = str_groups(a.U);
  const dim3 b(16, 16), gv(groups, (a.n_v + 15) / 16), gg(groups, (a.n_g + 15) / 16);
  if (sixth) k_str_pack<StrV<VMasks6>><<<gv, b, 0, st>>>(a.ab_v, a.piv_v, a.n_v, a.U, s.vf, s.vb);
  else k_str_pack<StrV<VMasks>><<<gv, b, 0, st>>>(a.ab_v, a.piv_v, a.n_v, a.U, s.vf, s.vb);
  k_str_pack<StrG><<<gg, b, 0, st>>>(a.ab_g, a.piv_g, a.n_g, a.U, s.gf, s.gb);
  const unsigned bx = (unsigned)std::min((a.U + 127) / 128, 64);
  k_str_row_scales<<<dim3(bx, nvrows), 128, 0, st>>>(s.vrs, a.rs_v, a.vrows, a.U);
  k_str_row_scales<<<dim3(bx, ngrows), 128, 0, st>>>(s.grs, a.rs_gi, a.grows, a.U);
}

}  // namespace owt
