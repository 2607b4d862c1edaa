// Mixed-precision RHS kernels of the euler equation on the CUDA cores
// (dg_mixed.cuh) and the launch that fills their node records.
#include "mixed_instantiate.cuh"

namespace dg {
namespace {
// Node records (rho, E, m_x, m_y), (m_z, p, 1/rho, |u| + c) with the pressure
// recovered from total energy in FP64 (the mixed kernels' reciprocal: FP32
// estimate refined by one Newton step).
__global__ void __launch_bounds__(256)
    dg_nodes_f32_kernel(const double* __restrict__ q, float4* __restrict__ rec, int64_t nelnp,
                        double gamma) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < nelnp; n += stride) {
    const double rho = __ldg(q + n), en = __ldg(q + nelnp + n), m0 = __ldg(q + 2 * nelnp + n),
                 m1 = __ldg(q + 3 * nelnp + n), m2 = __ldg(q + 4 * nelnp + n);
    // rcp64_fast with its conversions on the integer ALU (the FP64 pipe bounds
    // this launch)
    const float f[5] = {d2f_alu(rho), d2f_alu(en), d2f_alu(m0), d2f_alu(m1), d2f_alu(m2)};
    const double r0 = f2d_alu(__frcp_rn(f[0]));
    double rinv = fma(r0, fma(-rho, r0, 1.0), r0);
    // these conversions know normal floats only: 2^-126 <= |rho| < 2^126
    if (((uint32_t)__double2hiint(rho) & 0x7fffffffu) - (897u << 20) >= (252u << 20))
      rinv = rcp64_fast(rho);
    const float p = d2f_alu((gamma - 1.0) * (en - 0.5 * (m0 * m0 + m1 * m1 + m2 * m2) * rinv));
    const mix::Trace s = mix::euler_trace(f, p, (float)gamma);
    rec[2 * n] = make_float4(f[0], f[1], f[2], f[3]);
    rec[2 * n + 1] = make_float4(f[4], s.p, s.rinv, s.lam);
  }
}
}  // namespace

cudaError_t mixed_shape_euler(int order, bool stage, LaunchShape* out) {
  return mixed_shape_any<DG_EULER>(order, stage, out);
}
cudaError_t mixed_launch_euler(int order, bool stage, const RhsArgs& a, int grid,
                             cudaStream_t s) {
  return mixed_launch_any<DG_EULER>(order, stage, a, grid, s);
}
cudaError_t mixed_nodes_euler(const double* q, float4* rec, int64_t nelnp, double gamma, int grid,
                              cudaStream_t s) {
  dg_nodes_f32_kernel<<<grid, 256, 0, s>>>(q, rec, nelnp, gamma);
  return cudaGetLastError();
}
}  // namespace dg
