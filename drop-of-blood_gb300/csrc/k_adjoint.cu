// k_adjoint.cu — discrete adjoint (transpose of the Jacobian) of every stage
// of the closed-box step, FP32 and mixed precision.
//
// Each kernel is the exact transpose of the linearisation of one forward
// kernel at the forward state it is given (the "tape"):
//   advection        transpose of the trilinear interpolation of the face
//                    values at the departure point, plus the chain through
//                    the RK2 departure point into the centre velocity
//                    (scattered with atomics: several cells can sample the
//                    same texel)
//   centre average   transpose of the face -> centre average
//   Casson viscosity explicit Laplacian with coefficient alpha(|grad u|, c):
//                    transpose of the stencil plus the alpha chain (two
//                    passes: per-cell coefficients, then a gather)
//   divergence / projection  D^T and G^T with the wall masks
//   pressure solve   FP32 (a fixed number of V-cycles): the transposed cycles
//                    (launch_transposed_cycles); mixed (solved to a
//                    tolerance): the adjoint of an exact solve, the same
//                    solver on the adjoint right-hand side
//   dye predict / MacCormack resolve  transposed samples; the limiter passes
//                    the adjoint through, or to the neighbourhood tap that
//                    supplied the clamped value
// Where the forward is not differentiable (clamps at their bounds, the
// limiter's min/max selection, |grad u| = 0) the adjoint takes the branch the
// forward took, i.e. the one-sided derivative of the executed expression.
//
// Adjoint arrays are FP32, natural layout except the pressure / right-hand
// side / multigrid ones (red-black split like their forward arrays).
#include <cuda_runtime.h>

#include "dob_kernels.cuh"

namespace dob {

// ---- trilinear helpers --------------------------------------------------------------------
__device__ __forceinline__ void tri_w(const Taps& t, float w[8]) {
  const float gx = 1.0f - t.fx, gy = 1.0f - t.fy, gz = 1.0f - t.fz;
  w[0] = gx * gy * gz; w[1] = t.fx * gy * gz; w[2] = gx * t.fy * gz; w[3] = t.fx * t.fy * gz;
  w[4] = gx * gy * t.fz; w[5] = t.fx * gy * t.fz; w[6] = gx * t.fy * t.fz; w[7] = t.fx * t.fy * t.fz;
}
__device__ __forceinline__ uint32_t tap_at(const Taps& t, int k) {
  return t.base + ((k & 1) ? t.ox : 0u) + ((k & 2) ? t.oy : 0u) + ((k & 4) ? t.oz : 0u);
}
// d lerp8 / d(fx, fy, fz) of a scalar field.  Linear interpolation has a
// slope kink at every grid node; where a sample sits on a node along an axis
// (e.g. a departure point of fluid at rest) the slope along that axis is the
// mean of the slopes on either side, the value central differences see.  "On
// a node" means a fraction of exactly 0 (kNodeBand = 0; a positive band would
// also catch samples within that many texel units of a node from either side).
// NodeLo gives the element offsets from the base node to the node below it
// and from the node above the base to the next one (0 where clamp-to-edge
// makes the function flat).
constexpr float kNodeBand = 0.0f;
struct NodeLo {
  uint32_t lx, ly, lz;  // base -> base - 1
  uint32_t hx, hy, hz;  // base + 1 -> base + 2
};
__device__ __forceinline__ NodeLo node_lo(const Grid& g, float u, float v, float w) {
  const int ix = dob_clampi((int)floorf(texel(u, g.nx)), 0, g.nx - 1);  // as make_taps forms it
  const int iy = dob_clampi((int)floorf(texel(v, g.ny)), 0, g.ny - 1);
  const int iz = dob_clampi((int)floorf(texel(w, g.nz)), 0, g.nz - 1);
  const uint32_t sy = (uint32_t)g.nx, sz = (uint32_t)g.nx * (uint32_t)g.ny;
  NodeLo n;
  n.lx = ix > 0 ? 1u : 0u;
  n.ly = iy > 0 ? sy : 0u;
  n.lz = iz > 0 ? sz : 0u;
  n.hx = ix + 2 <= g.nx - 1 ? 1u : 0u;
  n.hy = iy + 2 <= g.ny - 1 ? sy : 0u;
  n.hz = iz + 2 <= g.nz - 1 ? sz : 0u;
  return n;
}
template <class F>
__device__ __forceinline__ dob_v3 dfrac_core(const Taps& t, const NodeLo& n, F val) {
  const uint32_t b = t.base;
  const float c0 = val(b), c1 = val(b + t.ox), c2 = val(b + t.oy), c3 = val(b + t.oy + t.ox);
  const float c4 = val(b + t.oz), c5 = val(b + t.oz + t.ox), c6 = val(b + t.oz + t.oy);
  const float c7 = val(b + t.oz + t.oy + t.ox);
  const float x00 = dob_mix(c0, c1, t.fx), x10 = dob_mix(c2, c3, t.fx);
  const float x01 = dob_mix(c4, c5, t.fx), x11 = dob_mix(c6, c7, t.fx);
  float dfx = dob_mix(dob_mix(c1 - c0, c3 - c2, t.fy), dob_mix(c5 - c4, c7 - c6, t.fy), t.fz);
  float dfy = dob_mix(x10 - x00, x11 - x01, t.fz);
  const float y0 = dob_mix(x00, x10, t.fy), y1 = dob_mix(x01, x11, t.fy);
  float dfz = y1 - y0;
  if (t.fx <= kNodeBand) {  // node at the base: slope below it from base - 1
    const uint32_t o = b - n.lx;
    const float l0 = val(o), l2 = val(o + t.oy), l4 = val(o + t.oz), l6 = val(o + t.oz + t.oy);
    dfx = 0.5f * (dfx + dob_mix(dob_mix(c0 - l0, c2 - l2, t.fy), dob_mix(c4 - l4, c6 - l6, t.fy), t.fz));
  } else if (t.fx >= 1.0f - kNodeBand) {  // node at base + 1: slope above it to base + 2
    const uint32_t o = b + t.ox + n.hx;
    const float h0 = val(o), h2 = val(o + t.oy), h4 = val(o + t.oz), h6 = val(o + t.oz + t.oy);
    dfx = 0.5f * (dfx + dob_mix(dob_mix(h0 - c1, h2 - c3, t.fy), dob_mix(h4 - c5, h6 - c7, t.fy), t.fz));
  }
  if (t.fy <= kNodeBand) {
    const uint32_t o = b - n.ly;
    const float l00 = dob_mix(val(o), val(o + t.ox), t.fx);
    const float l01 = dob_mix(val(o + t.oz), val(o + t.oz + t.ox), t.fx);
    dfy = 0.5f * (dfy + dob_mix(x00 - l00, x01 - l01, t.fz));
  } else if (t.fy >= 1.0f - kNodeBand) {
    const uint32_t o = b + t.oy + n.hy;
    const float h00 = dob_mix(val(o), val(o + t.ox), t.fx);
    const float h01 = dob_mix(val(o + t.oz), val(o + t.oz + t.ox), t.fx);
    dfy = 0.5f * (dfy + dob_mix(h00 - x10, h01 - x11, t.fz));
  }
  if (t.fz <= kNodeBand) {
    const uint32_t o = b - n.lz;
    const float m0 = dob_mix(val(o), val(o + t.ox), t.fx);
    const float m1 = dob_mix(val(o + t.oy), val(o + t.oy + t.ox), t.fx);
    dfz = 0.5f * (dfz + (y0 - dob_mix(m0, m1, t.fy)));
  } else if (t.fz >= 1.0f - kNodeBand) {
    const uint32_t o = b + t.oz + n.hz;
    const float m0 = dob_mix(val(o), val(o + t.ox), t.fx);
    const float m1 = dob_mix(val(o + t.oy), val(o + t.oy + t.ox), t.fx);
    dfz = 0.5f * (dfz + (dob_mix(m0, m1, t.fy) - y1));
  }
  return v3(dfx, dfy, dfz);
}
template <class S>
__device__ __forceinline__ dob_v3 lerp8_dfrac(const Taps& t, const NodeLo& n, const S* a) {
  return dfrac_core(t, n, [&](uint32_t k) { return ldv(a + k); });
}
// sum over the xyz channels of a float4 field: sum_ch g_ch * d lerp8_ch / d(fx, fy, fz)
// (the derivative is linear in the values, so the channels are contracted first)
__device__ __forceinline__ dob_v3 lerp8x3_dfrac(const Taps& t, const NodeLo& n, const float4* a, dob_v3 g) {
  return dfrac_core(t, n, [&](uint32_t k) {
    const float4 c = a[k];
    return g.x * c.x + g.y * c.y + g.z * c.z;
  });
}
// transpose of lerp8: a[tap k] += g * w_k
__device__ __forceinline__ void scatter8(float* a, const Taps& t, float g) {
  if (g == 0.0f) return;
  float w[8];
  tri_w(t, w);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (w[k] != 0.0f) atomicAdd(a + tap_at(t, k), g * w[k]);
}
__device__ __forceinline__ void scatter8v(float4* a, const Taps& t, dob_v3 g) {
  if (g.x == 0.0f && g.y == 0.0f && g.z == 0.0f) return;
  float w[8];
  tri_w(t, w);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (w[k] != 0.0f) atomicAdd(a + tap_at(t, k), make_float4(g.x * w[k], g.y * w[k], g.z * w[k], 0.0f));
}
// derivative mask of dob_clampf(v, lo, hi): 1 where the value passed through
__device__ __forceinline__ float pass(float v, float lo, float hi) { return (v > lo && v < hi) ? 1.0f : 0.0f; }
__device__ __forceinline__ dob_v3 pass3(dob_v3 v, float lo, float hi) {
  return v3(pass(v.x, lo, hi), pass(v.y, lo, hi), pass(v.z, lo, hi));
}

#define ADJ_CELL                                     \
  const int x = blockIdx.x * blockDim.x + threadIdx.x; \
  const int y = blockIdx.y * blockDim.y + threadIdx.y; \
  const int z = blockIdx.z;                          \
  if (x >= g.nx || y >= g.ny) return;                \
  const size_t i = g.at(x, y, z);

// ---- FLUID_ADVECT_MAC (closed box) ------------------------------------------------------------
// Forward per face: B = trace_back(cen, F) (RK2 with clamps), value =
// damp * lerp8(u_k, clamp(B - half-cell offset)).  Adjoint of the output
// au2 -> au (face values) and acen (centre velocity).
__device__ __forceinline__ void adj_face(const Grid& g, const float* uk, const float4* cen, float4* acen, float* auk,
                                         dob_v3 F, int comp, float gout, float dtv, const Recip3& dom,
                                         dob_v3 dims) {
  if (gout == 0.0f) return;
  // forward recompute
  const dob_v3 F0 = clamp3(F, 0.002f, 0.998f);
  const Taps t0 = make_taps_exact(g, F0.x, F0.y, F0.z);  // as trace_back forms it
  const dob_v3 v0 = lerp8x3_fixed(t0, cen);
  const dob_v3 M = F - (0.5f * (v0 * dtv)) / dom;
  const dob_v3 Mc = clamp3(M, 0.002f, 0.998f);
  const Taps tM = make_taps_in(g, Mc.x, Mc.y, Mc.z);
  const float4 vmr = lerp8xn<3>(tM, cen);
  const dob_v3 vMid = v3(vmr.x, vmr.y, vmr.z);
  const dob_v3 B = F - (vMid * dtv) / dom;
  const dob_v3 Bc = clamp3(B, 0.002f, 0.998f);
  dob_v3 S = Bc;
  if (comp == 0) S.x = S.x - 0.5f * g.rx;
  if (comp == 1) S.y = S.y - 0.5f * g.ry;
  if (comp == 2) S.z = S.z - 0.5f * g.rz;
  const dob_v3 Sc = clamp3(S, 0.001f, 0.999f);
  const Taps tS = make_taps_in(g, Sc.x, Sc.y, Sc.z);
  // backward
  scatter8(auk, tS, gout);
  const dob_v3 gS = (gout * lerp8_dfrac(tS, node_lo(g, Sc.x, Sc.y, Sc.z), uk)) * dims * pass3(S, 0.001f, 0.999f);
  const dob_v3 gB = gS * pass3(B, 0.002f, 0.998f);
  const dob_v3 gvMid = -(gB * dtv) / dom;
  scatter8v(acen, tM, gvMid);
  const dob_v3 gM = lerp8x3_dfrac(tM, node_lo(g, Mc.x, Mc.y, Mc.z), cen, gvMid) * dims * pass3(M, 0.002f, 0.998f);
  const dob_v3 gv0 = -(0.5f * (gM * dtv)) / dom;
  scatter8v(acen, t0, gv0);
}

// One thread per face (grid z = 3 nz: the face's axis is blockIdx.z % 3,
// uniform over the block), so a thread holds one face's trace; capped at 64
// registers (4 blocks per SM, a 12-byte spill): the kernel is bound by the
// latency of its gathers, and twice the resident warps of the uncapped
// three-face thread hide more of it.
__global__ void __launch_bounds__(256, 4) k_adj_advect_mac(Grid g, const StepParams* __restrict__ Pp,
                                                        const float* __restrict__ u, const float* __restrict__ v,
                                                        const float* __restrict__ w, const float4* __restrict__ cen,
                                                        const float* __restrict__ au2, const float* __restrict__ av2,
                                                        const float* __restrict__ aw2, float* au, float* av, float* aw,
                                                        float4* acen) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int comp = blockIdx.z % 3, z = blockIdx.z / 3;
  if (x >= g.nx || y >= g.ny) return;
  const size_t i = g.at(x, y, z);
  const StepParams& P = *Pp;
  const dob_v3 dims = v3((float)g.nx, (float)g.ny, (float)g.nz);
  const Recip3 dimr = grid_recip(g), dom = dom_recip(P);
  const float dtv = P.dt;
  const float damp = P.damp;
  const bool wall = comp == 0 ? x >= g.nx - 1 : comp == 1 ? y >= g.ny - 1 : z >= g.nz - 1;
  const float* ga = comp == 0 ? au2 : comp == 1 ? av2 : aw2;
  const float gout = wall ? 0.0f : ga[i] * damp;
  const dob_v3 F = v3((float)x + (comp == 0 ? 1.0f : 0.5f), (float)y + (comp == 1 ? 1.0f : 0.5f),
                      (float)z + (comp == 2 ? 1.0f : 0.5f)) / dimr;
  adj_face(g, comp == 0 ? u : comp == 1 ? v : w, cen, acen, comp == 0 ? au : comp == 1 ? av : aw, F, comp, gout, dtv,
           dom, dims);
}

// ---- FLUID_MAC_TO_CENTER (closed box): au += C^T acen ---------------------------------------
__global__ void __launch_bounds__(256) k_adj_mac_to_center(Grid g, const float4* __restrict__ acen, float* au,
                                                           float* av, float* aw) {
  ADJ_CELL
  const float4 c = acen[i];
  if (x < g.nx - 1) au[i] += 0.5f * c.x + 0.5f * acen[i + 1].x;
  if (y < g.ny - 1) av[i] += 0.5f * c.y + 0.5f * acen[i + g.nx].y;
  if (z < g.nz - 1) aw[i] += 0.5f * c.z + 0.5f * acen[i + (size_t)g.nx * g.ny].z;
}

// ---- FLUID_CASSON_FORCES (closed box) ----------------------------------------------------------
__device__ __forceinline__ dob_v3 ldm(const Grid& g, const float* u, const float* v, const float* w, int x, int y,
                                      int z) {
  const size_t j = g.at(dob_clampi(x, 0, g.nx - 1), dob_clampi(y, 0, g.ny - 1), dob_clampi(z, 0, g.nz - 1));
  return v3(u[j], v[j], w[j]);
}
__device__ __forceinline__ dob_v3 out_adj(const Grid& g, const float* au2, const float* av2, const float* aw2, int x,
                                          int y, int z) {
  const size_t j = g.at(x, y, z);
  return v3(x >= g.nx - 1 ? 0.0f : au2[j], y >= g.ny - 1 ? 0.0f : av2[j], z >= g.nz - 1 ? 0.0f : aw2[j]);
}
// Pass 1: per cell, alpha and G = 2 dL/dQ (Q = |grad u|^2 of the Casson
// shear rate); the dye adjoint of the cell.
template <class DS>
__global__ void __launch_bounds__(256, 5) k_adj_casson1(Grid g, const StepParams* __restrict__ Pp,
                                                     const float* __restrict__ u, const float* __restrict__ v,
                                                     const float* __restrict__ w, const DS* __restrict__ dye,
                                                     const float* __restrict__ au2, const float* __restrict__ av2,
                                                     const float* __restrict__ aw2, float* __restrict__ alpha_out,
                                                     float* __restrict__ gq_out, float* ac) {
  ADJ_CELL
  const StepParams& P = *Pp;
  const float dtv = P.dt;
  const dob_v3 mac = v3(u[i], v[i], w[i]);
  const dob_v3 mXp = ldm(g, u, v, w, x + 1, y, z), mXn = ldm(g, u, v, w, x - 1, y, z);
  const dob_v3 mYp = ldm(g, u, v, w, x, y + 1, z), mYn = ldm(g, u, v, w, x, y - 1, z);
  const dob_v3 mZp = ldm(g, u, v, w, x, y, z + 1), mZn = ldm(g, u, v, w, x, y, z - 1);
  const dob_v3 du = mXp - mXn, dv = mYp - mYn, dw = mZp - mZn;
  const dob_v3 lap = (mXp + mXn + mYp + mYn + mZp + mZn) - 6.0f * mac;
  const float cval = ldv(dye + i);
  const float c = dob_clampf(cval, 0.0f, 1.5f);
  const float dxv = P.dx;
  const float Q = dot3(du, du) + dot3(dv, dv) + dot3(dw, dw);
  const float gdot = dob_sqrt(Q) / (2.0f * dxv);
  const float sqrtMu = dob_sqrt(P.mu_p);
  const float S = dob_sqrt(P.tau_y * c * c / (gdot + 0.4f));
  const float nu = (sqrtMu + S) * (sqrtMu + S);
  const float araw = nu * dtv / (dxv * dxv);
  const float alpha = dob_minf(araw, 0.125f);
  alpha_out[i] = alpha;
  float G = 0.0f;
  if (araw < 0.125f) {
    const dob_v3 o = out_adj(g, au2, av2, aw2, x, y, z);
    const float ab = dot3(o, lap);
    const float nub = ab * dtv / (dxv * dxv);
    const float Sb = nub * 2.0f * (sqrtMu + S);
    const float K = dob_sqrt(P.tau_y / (gdot + 0.4f));
    ac[i] += Sb * K * pass(cval, 0.0f, 1.5f);
    const float gb = Sb * (-S / (2.0f * (gdot + 0.4f)));
    if (Q > 0.0f) G = 2.0f * (gb / (2.0f * dxv)) / (2.0f * dob_sqrt(Q));
  }
  gq_out[i] = G;
}
// Pass 2: gather the adjoint of each face value from the cells whose
// (clamped) stencils read it.
__global__ void __launch_bounds__(256) k_adj_casson2(Grid g, const float* __restrict__ u, const float* __restrict__ v,
                                                     const float* __restrict__ w, const float* __restrict__ au2,
                                                     const float* __restrict__ av2, const float* __restrict__ aw2,
                                                     const float* __restrict__ alpha, const float* __restrict__ gq,
                                                     float* au, float* av, float* aw) {
  ADJ_CELL
  const int n[3] = {g.nx, g.ny, g.nz};
  const int jc[3] = {x, y, z};
  const dob_v3 o = out_adj(g, au2, av2, aw2, x, y, z);
  const float aj = alpha[i], Gj = gq[i];
  const dob_v3 mj = v3(u[i], v[i], w[i]);
  int ncl = 0;
  dob_v3 acc = v3(0.0f, 0.0f, 0.0f);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    int e[3] = {0, 0, 0};
    e[d] = 1;
    if (jc[d] > 0) {  // i = j - e_d: j is its + neighbour
      const int ix = x - e[0], iy = y - e[1], iz = z - e[2];
      const size_t ii = g.at(ix, iy, iz);
      const dob_v3 oi = out_adj(g, au2, av2, aw2, ix, iy, iz);
      const dob_v3 mm = ldm(g, u, v, w, x - 2 * e[0], y - 2 * e[1], z - 2 * e[2]);
      acc = acc + alpha[ii] * oi + gq[ii] * (mj - mm);
    } else {
      ++ncl;  // the - neighbour of j clamps onto j
      const dob_v3 mp = ldm(g, u, v, w, x + e[0], y + e[1], z + e[2]);
      acc = acc - Gj * (mp - mj);
    }
    if (jc[d] < n[d] - 1) {  // i = j + e_d: j is its - neighbour
      const int ix = x + e[0], iy = y + e[1], iz = z + e[2];
      const size_t ii = g.at(ix, iy, iz);
      const dob_v3 oi = out_adj(g, au2, av2, aw2, ix, iy, iz);
      const dob_v3 mp = ldm(g, u, v, w, x + 2 * e[0], y + 2 * e[1], z + 2 * e[2]);
      acc = acc + alpha[ii] * oi - gq[ii] * (mp - mj);
    } else {
      ++ncl;  // the + neighbour of j clamps onto j
      const dob_v3 mm = ldm(g, u, v, w, x - e[0], y - e[1], z - e[2]);
      acc = acc + Gj * (mj - mm);
    }
  }
  const float self = 1.0f - 6.0f * aj + aj * (float)ncl;
  acc = acc + self * o;
  au[i] += acc.x;
  av[i] += acc.y;
  aw[i] += acc.z;
}

// ---- FLUID_MAC_RHS (closed box): au += D^T arhs (arhs already mean-free) -----------------------
__global__ void __launch_bounds__(256) k_adj_mac_rhs(Grid g, const float* __restrict__ arhs, float* au, float* av,
                                                     float* aw) {
  ADJ_CELL
  const float bj = arhs[rb_index(g, x, y, z)];
  if (x < g.nx - 1) au[i] += bj - arhs[rb_index(g, x + 1, y, z)];
  if (y < g.ny - 1) av[i] += bj - arhs[rb_index(g, x, y + 1, z)];
  if (z < g.nz - 1) aw[i] += bj - arhs[rb_index(g, x, y, z + 1)];
}

// ---- FLUID_MAC_PROJECT (closed box): au <- W au, ap += D(W au) --------------------------------
__global__ void __launch_bounds__(256) k_adj_project(Grid g, float* au, float* av, float* aw, float* ap) {
  ADJ_CELL
  const float ox = x < g.nx - 1 ? au[i] : 0.0f;
  const float oy = y < g.ny - 1 ? av[i] : 0.0f;
  const float oz = z < g.nz - 1 ? aw[i] : 0.0f;
  const float oxm = x > 0 ? au[i - 1] : 0.0f;
  const float oym = y > 0 ? av[i - g.nx] : 0.0f;
  const float ozm = z > 0 ? aw[i - (size_t)g.nx * g.ny] : 0.0f;
  ap[rb_index(g, x, y, z)] += (ox - oxm) + (oy - oym) + (oz - ozm);
  // wall faces are zeroed by the forward; no neighbour reads them
  if (x == g.nx - 1) au[i] = 0.0f;
  if (y == g.ny - 1) av[i] = 0.0f;
  if (z == g.nz - 1) aw[i] = 0.0f;
}

// ---- CONC_PREDICT (closed box) ------------------------------------------------------------------
// The per-cell adjoints below (dye predictor and resolve, the Casson
// coefficients) are capped at 4-5 blocks of 256
// per SM (a few spilled bytes): latency-bound, they gain more from the
// resident warps.
template <class DS>
__global__ void __launch_bounds__(256, 4) k_adj_conc_predict(Grid gc, Grid g, const StepParams* __restrict__ Pp,
                                                          const float4* __restrict__ cen, const DS* __restrict__ dye,
                                                          const float* __restrict__ apred, float* ac, float4* acen) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int z = blockIdx.z;
  if (x >= gc.nx || y >= gc.ny) return;
  const size_t i = gc.at(x, y, z);
  const float gout = apred[i];
  if (gout == 0.0f) return;
  const StepParams& P = *Pp;
  const dob_v3 dimsc = v3((float)gc.nx, (float)gc.ny, (float)gc.nz);
  const dob_v3 dimsg = v3((float)g.nx, (float)g.ny, (float)g.nz);
  const float dtv = P.dt;
  const Recip3 dom = dom_recip(P);
  const dob_v3 uvw = (v3((float)x, (float)y, (float)z) + v3(0.5f, 0.5f, 0.5f)) / grid_recip(gc);
  const Taps t0 = make_taps_exact(g, uvw.x, uvw.y, uvw.z);  // the forward's cell-centre sample (dye on the velocity grid)
  const dob_v3 v0 = lerp8x3_fixed(t0, cen);
  const dob_v3 M = uvw - (0.5f * (v0 * dtv)) / dom;
  const dob_v3 Mc = clamp3(M, 0.001f, 0.999f);
  const Taps tM = make_taps_in(g, Mc.x, Mc.y, Mc.z);
  const float4 vmr = lerp8xn<3>(tM, cen);
  const dob_v3 vMid = v3(vmr.x, vmr.y, vmr.z);
  const dob_v3 B = uvw - (vMid * dtv) / dom;
  const dob_v3 Bc = clamp3(B, 0.001f, 0.999f);
  const Taps tB = make_taps_in(gc, Bc.x, Bc.y, Bc.z);
  scatter8(ac, tB, gout);
  const dob_v3 gB = (gout * lerp8_dfrac(tB, node_lo(gc, Bc.x, Bc.y, Bc.z), dye)) * dimsc * pass3(B, 0.001f, 0.999f);
  const dob_v3 gvMid = -(gB * dtv) / dom;
  scatter8v(acen, tM, gvMid);
  const dob_v3 gM = lerp8x3_dfrac(tM, node_lo(g, Mc.x, Mc.y, Mc.z), cen, gvMid) * dimsg * pass3(M, 0.001f, 0.999f);
  const dob_v3 gv0 = -(0.5f * (gM * dtv)) / dom;
  scatter8v(acen, t0, gv0);
}

// ---- CONC_RESOLVE (closed box: MacCormack with the 8-tap limiter) -----------------------------
template <class DS>
__global__ void __launch_bounds__(256, 5) k_adj_dye_resolve(Grid gc, Grid g, const StepParams* __restrict__ Pp,
                                                         const float4* __restrict__ cen, const DS* __restrict__ dye,
                                                         const DS* __restrict__ pred, const float* __restrict__ ac2,
                                                         float* ac, float* apred, float4* acen) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int z = blockIdx.z;
  if (x >= gc.nx || y >= gc.ny) return;
  const size_t i = gc.at(x, y, z);
  const float gout = ac2[i];
  if (gout == 0.0f) return;
  const StepParams& P = *Pp;
  const dob_v3 dims = v3((float)gc.nx, (float)gc.ny, (float)gc.nz);
  const float dtv = P.dt;
  const Recip3 dom = dom_recip(P);
  const dob_v3 uvw = (v3((float)x, (float)y, (float)z) + v3(0.5f, 0.5f, 0.5f)) / grid_recip(gc);
  const Taps t0 = make_taps_exact(g, uvw.x, uvw.y, uvw.z);  // the forward's cell-centre sample (dye on the velocity grid)
  const dob_v3 v0 = lerp8x3_fixed(t0, cen);
  const dob_v3 uvwMid = clamp3(uvw - (0.5f * (v0 * dtv)) / dom, 0.001f, 0.999f);
  const float4 vmr = lerp8xn<3>(make_taps_in(g, uvwMid.x, uvwMid.y, uvwMid.z), cen);
  const dob_v3 vMid = v3(vmr.x, vmr.y, vmr.z);
  const dob_v3 uvwBack = clamp3(uvw - (vMid * dtv) / dom, 0.001f, 0.999f);
  const dob_v3 Fw = uvw + (v0 * dtv) / dom;
  const dob_v3 uvwFwd = clamp3(Fw, 0.001f, 0.999f);
  const Taps tF = make_taps_in(gc, uvwFwd.x, uvwFwd.y, uvwFwd.z);
  const float gBackEst = lerp8(tF, pred);
  const float kap = 0.45f * P.sharp;
  const float gCorr = __fmaf_rn(kap, ldv(dye + i) - gBackEst, ldv(pred + i));  // as the forward rounds it
  // the limiter's taps: the forward predictor's (make_taps at the departure point)
  const int bx = (int)floorf(texel(uvwBack.x, gc.nx)), by = (int)floorf(texel(uvwBack.y, gc.ny));
  const int bz = (int)floorf(texel(uvwBack.z, gc.nz));
  size_t id[8];
  float s[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    id[k] = gc.at(dob_clampi(bx + (k & 1), 0, gc.nx - 1), dob_clampi(by + ((k >> 1) & 1), 0, gc.ny - 1),
                  dob_clampi(bz + ((k >> 2) & 1), 0, gc.nz - 1));
    s[k] = ldv(dye + id[k]);
  }
  // the forward's min/max trees (dob_minf/dob_maxf keep the second operand on ties)
  auto pick_min = [&](int a, int b) { return s[a] < s[b] ? a : b; };
  auto pick_max = [&](int a, int b) { return s[a] > s[b] ? a : b; };
  const int kmin = pick_min(pick_min(pick_min(0, 1), pick_min(2, 3)), pick_min(pick_min(4, 5), pick_min(6, 7)));
  const int kmax = pick_max(pick_max(pick_max(0, 1), pick_max(2, 3)), pick_max(pick_max(4, 5), pick_max(6, 7)));
  const float minG = s[kmin], maxG = s[kmax];
  if (!(gCorr > minG)) {
    atomicAdd(ac + id[kmin], gout);
  } else if (!(gCorr < maxG)) {
    atomicAdd(ac + id[kmax], gout);
  } else {
    atomicAdd(apred + i, gout);
    atomicAdd(ac + i, kap * gout);
    const float gE = -kap * gout;
    scatter8(apred, tF, gE);
    const dob_v3 gF = (gE * lerp8_dfrac(tF, node_lo(gc, uvwFwd.x, uvwFwd.y, uvwFwd.z), pred)) * dims *
                      pass3(Fw, 0.001f, 0.999f);
    const dob_v3 gv0 = (gF * dtv) / dom;
    scatter8v(acen, t0, gv0);
  }
}

// ---- launchers ----------------------------------------------------------------------------------
static inline dim3 cgrid(const Grid& g) { return dim3((g.nx + 31) / 32, (g.ny + 7) / 8, g.nz); }
static inline dim3 cblock() { return dim3(32, 8, 1); }

void launch_adj_advect_mac(const DevState& s, const AdjState& a, cudaStream_t st) {
  const dim3 g3(cgrid(s.g).x, cgrid(s.g).y, 3 * s.g.nz);
  k_adj_advect_mac<<<g3, cblock(), 0, st>>>(s.g, s.params, (const float*)s.u, (const float*)s.v,
                                                    (const float*)s.w, (const float4*)s.cen, a.au2, a.av2, a.aw2, a.au,
                                                    a.av, a.aw, a.acen);
}
void launch_adj_mac_to_center(const DevState& s, const AdjState& a, cudaStream_t st) {
  k_adj_mac_to_center<<<cgrid(s.g), cblock(), 0, st>>>(s.g, a.acen, a.au, a.av, a.aw);
}
// The dye and the predictor are read at their storage width: binary16 in
// the mixed mode (the adjoint of the rounding store is the identity, so the
// adjoint arrays stay FP32).
#define ADJ_DYE_DISPATCH(prec, ...)                                \
  do {                                                             \
    if ((prec) == DOB_PREC_MIXED) { using DS = __half; __VA_ARGS__; } \
    else { using DS = float; __VA_ARGS__; }                        \
  } while (0)

void launch_adj_casson(const DevState& s, const AdjState& a, cudaStream_t st) {
  ADJ_DYE_DISPATCH(s.prec, {
    k_adj_casson1<DS><<<cgrid(s.g), cblock(), 0, st>>>(s.g, s.params, (const float*)s.u, (const float*)s.v,
                                                       (const float*)s.w, (const DS*)s.conc, a.au2, a.av2, a.aw2,
                                                       a.alpha, a.gq, a.ac);
  });
  k_adj_casson2<<<cgrid(s.g), cblock(), 0, st>>>(s.g, (const float*)s.u, (const float*)s.v, (const float*)s.w, a.au2,
                                                 a.av2, a.aw2, a.alpha, a.gq, a.au, a.av, a.aw);
}
void launch_adj_mac_rhs(const DevState& s, const AdjState& a, cudaStream_t st) {
  // transpose of the mean removal (a symmetric projection), then D^T
  launch_sum(a.arhs, s.g.n(), a.part, s.num_sms, st);
  launch_sub_mean(a.arhs, s.g.n(), a.part, s.num_sms, st);
  k_adj_mac_rhs<<<cgrid(s.g), cblock(), 0, st>>>(s.g, a.arhs, a.au, a.av, a.aw);
}
void launch_adj_project(const DevState& s, const AdjState& a, cudaStream_t st) {
  k_adj_project<<<cgrid(s.g), cblock(), 0, st>>>(s.g, a.au, a.av, a.aw, a.ap);
}

// rhs += lam + lamlo (the adjoint of the right-hand side through an exact
// solve); the solution's adjoint is consumed
__global__ void __launch_bounds__(256) k_adj_take_solution(const float* __restrict__ lam,
                                                           const float* __restrict__ lamlo, float* arhs, float* ap,
                                                           size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    arhs[i] += lam[i] + lamlo[i];
    ap[i] = 0.0f;
  }
}
void launch_adj_pressure_solve(const DevState& s, const AdjState& a, cudaStream_t st) {
  const size_t n = s.g.n();
  if (!s.ref) {
    launch_sum(a.ap, n, a.part + kSumBlocks, s.num_sms, st);
    launch_sub_mean(a.ap, n, a.part + kSumBlocks, s.num_sms, st);
  }
  if (s.prec == DOB_PREC_MIXED) {
    // The mixed forward solves to a tolerance, not a fixed number of cycles:
    // its pressure is A^+ b up to that tolerance, whatever the warm start, so
    // its adjoint is the same solve: A lam = ap (A symmetric, ap zero-mean),
    // by the mixed solver itself to ||ap - A lam|| <= kAdjRelTol ||ap||, then
    // rhs adjoint += lam and no adjoint reaches the warm start.  The solve
    // starts from the previous (later) step's lam, which the reverse sweep
    // leaves in place: the adjoint pressures of neighbouring steps are close,
    // so fewer V-cycles reach the tolerance.
    DevState t = s;
    t.p = a.lam;
    t.plo = a.lamlo;
    t.rhs = a.ap;
    t.rel_tol = kAdjRelTol;
    t.div_tol_r = 0.0f;
    t.max_outer = kMixedMaxRounds;
    t.cycles = 0;
    launch_pressure_solve(t, st);
    k_adj_take_solution<<<s.num_sms * 4, 256, 0, st>>>(a.lam, a.lamlo, a.arhs, a.ap, n);
    return;
  }
  // the Casson adjoint's scratch arrays hold the cycle's iterate and residual
  launch_transposed_cycles(s, a.ap, a.arhs, a.alpha, a.gq, a.lr, st);
}
void launch_adj_conc_predict(const DevState& s, const AdjState& a, cudaStream_t st) {
  ADJ_DYE_DISPATCH(s.prec, {
    k_adj_conc_predict<DS><<<cgrid(s.gc), cblock(), 0, st>>>(s.gc, s.g, s.params, (const float4*)s.cen,
                                                             (const DS*)s.conc, a.apred, a.ac, a.acen);
  });
}
void launch_adj_conc_resolve(const DevState& s, const AdjState& a, cudaStream_t st) {
  ADJ_DYE_DISPATCH(s.prec, {
    k_adj_dye_resolve<DS><<<cgrid(s.gc), cblock(), 0, st>>>(s.gc, s.g, s.params, (const float4*)s.cen,
                                                            (const DS*)s.conc, (const DS*)s.pred, a.ac2, a.ac,
                                                            a.apred, a.acen);
  });
}

}  // namespace dob
