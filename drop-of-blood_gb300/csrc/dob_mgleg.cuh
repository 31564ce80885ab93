// dob_mgleg.cuh — one leg of a multigrid level in one launch: the
// pre-smoothing with the residual and restriction after it (k_leg_down), and
// the prolongation with the post-smoothing after it (k_leg_up).
//
// A small level is bound by its launches: a half-sweep of 48x64x48 takes
// 2.3 us whatever it does, and a level of a 2+2 V-cycle is nine of them.
// Here a block holds a region of the level as deep around its tile as the
// leg's dependence (one cell per half-sweep, one for the residual) and runs
// the half-sweeps on it, so blocks never wait for one another.  The halo's
// cells are computed by several blocks; every one of them forms the same
// value (same operations in the same order as the half-sweep kernel of the
// level's rows, k_rbgs_v4 or k_rbgs_split, k_residual_restrict2 and
// k_prolong_add2, rounded to the level's storage type after each
// half-sweep), so the results are the bits of the launch chain.
// A block reads its neighbours' cells, so the leg's result goes to another
// array than its input.
//
// Layout: the region is 2 KW x 16 x 16 cells; thread (k, yy, zh) owns the
// lower (zh = 0) or upper half of the z column of word k of row yy in both
// colours (cells x = X0 + 2 k and + 1) in registers, values and right-hand
// sides, index 0 at the region's outermost plane.  Of a cell's neighbours,
// both z ones (but at the halves' seam) and one x one are then the thread's
// own, the other x one is the next or previous lane's (a shuffle), and the
// two y ones come through shared memory: three shared-memory accesses and a
// shuffle per update.  The z range shrinks by one cell per half-sweep; in x
// and y the whole region is updated and the outermost cells, which miss
// neighbours, hold values that nothing needed reads.  Cells outside the grid
// are zeros that nothing updates, so absent neighbours add an exact zero.
//
// Measured (four 2+2 cycles): 48x64x48 234 -> 185 us a step in the graph (the
// solve as a stage 184 -> 135); 192x256x192, whose levels 2 and 3 run this way,
// 1326 -> 1289.  One thread per cell and half-sweep with index
// arithmetic (263 us a step) and one thread per whole z column (209) were
// slower: the legs are bound by the instruction latency of their few warps.
#pragma once

#include "dob_kernels.cuh"

namespace dob {

constexpr int kLegR = 16;         // rows and planes of the region
constexpr int kLegZ = kLegR / 2;  // planes of a thread

// S: sweeps of the leg; the halo is 2 S cells
template <int KW_, int S_>
struct LegTile {
  static constexpr int KW = KW_, S = S_, H = 2 * S, PL = KW * kLegR, NT = 2 * PL;
  static constexpr int TX = 2 * KW - 2 * H, TY = kLegR - 2 * H, TZ = kLegR - 2 * H;
  static constexpr int CX = KW + 2, CY = kLegR / 2 + 2, CZ = kLegR / 2 + 2;  // k_leg_up: coarse taps
};

// One thread's half columns of the region.
template <class L>
struct LegCol {
  int k, y, yy, kk;      // global word and row, row and word in the region
  int zb, zs;            // plane of index i: zb + zs i (zs = 1 or -1)
  int pos;               // position of (k, yy) in a plane of the region
  bool up;               // the upper half (zs = -1)
  bool in;               // the word and row are inside the grid
  unsigned q;            // x parity of colour 0's cell at index 0
  int lane[2];           // the lane of the outer x neighbour of a cell of x parity 0, 1
  // diagonal of the cells of x parity 0, 1 away from the z walls and next to
  // one, with the reciprocals, and these again or 0 where the half-sweep
  // multiplies by 1/6 instead of dividing: k_rbgs_v4 (rows of a multiple of 8)
  // at every diagonal of 6, k_rbgs_split at interior cells only, so that it
  // divides by the 6 of the row below the Dirichlet top
  float d0[2], r0[2], c0[2], d1[2], r1[2], c1[2];
  uint32_t at, sz;       // offset of (k, y, plane zb) in a colour's half, plane stride
  __device__ __forceinline__ LegCol(const Grid& d, int ref) {
    const int tid = (int)threadIdx.x;
    pos = tid % L::PL;
    up = tid >= L::PL;
    kk = pos % L::KW;
    yy = pos / L::KW;
    k = (int)blockIdx.x * (L::TX / 2) - L::H / 2 + kk;
    y = (int)blockIdx.y * L::TY - L::H + yy;
    const int Z0 = (int)blockIdx.z * L::TZ - L::H;
    zb = up ? Z0 + kLegR - 1 : Z0;
    zs = up ? -1 : 1;
    const int hx = d.nx >> 1;
    in = (unsigned)k < (unsigned)hx && (unsigned)y < (unsigned)d.ny;
    q = (unsigned)(y + zb) & 1u;
    lane[0] = (tid & 31) - 1;
    lane[1] = (tid & 31) + 1;
    const float dy = 6.0f - (y == 0 ? 1.0f : 0.0f) - (y == d.ny - 1 && !ref ? 1.0f : 0.0f);
    const bool divides = ref && y == d.ny - 1 && d.nx % 8 != 0;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      d0[p] = dy - (k == (p ? hx - 1 : 0) ? 1.0f : 0.0f);
      d1[p] = d0[p] - 1.0f;
      r0[p] = d0[p] == 6.0f ? 1.0f / 6.0f : d0[p] == 5.0f ? 1.0f / 5.0f : d0[p] == 4.0f ? 1.0f / 4.0f : 1.0f / 3.0f;
      r1[p] = d1[p] == 5.0f ? 1.0f / 5.0f : d1[p] == 4.0f ? 1.0f / 4.0f : d1[p] == 3.0f ? 1.0f / 3.0f : 1.0f / 2.0f;
      c0[p] = d0[p] == 6.0f && !divides ? 0.0f : r0[p];
      c1[p] = r1[p];
    }
    sz = (uint32_t)d.ny * hx;
    at = (uint32_t)zb * sz + (uint32_t)y * hx + (uint32_t)k;  // modulo 2^32 outside the grid (not used there)
  }
  __device__ __forceinline__ int z(int i) const { return zb + zs * i; }
  __device__ __forceinline__ uint32_t off(int i) const { return up ? at - i * sz : at + i * sz; }
  __device__ __forceinline__ bool has_z(const Grid& d, int i) const { return (unsigned)z(i) < (unsigned)d.nz; }
  __device__ __forceinline__ bool wall_z(const Grid& d, int i) const { return z(i) == 0 || z(i) == d.nz - 1; }
  // x parity of colour c's cell at index i
  __device__ __forceinline__ unsigned par(int c, int i) const { return q ^ (unsigned)((i ^ c) & 1); }
};

// shared copies of both colours' values: plane of the region, position;
// padded by a row on both sides for the region's outermost rows
template <class L> struct LegShared {
  float pad0[L::KW];
  float v[2][kLegR][L::PL];
  float pad1[L::KW];
};

template <class T, class L>
__device__ __forceinline__ void leg_load(const Grid& d, const LegCol<L>& t, const T* __restrict__ a, int c,
                                         float (&v)[kLegZ]) {
  const T* h = a + (c ? (uint32_t)(d.n() >> 1) : 0u);
#pragma unroll
  for (int i = 0; i < kLegZ; ++i) v[i] = t.in && t.has_z(d, i) ? ldv(h + t.off(i)) : 0.0f;
}
template <class L>
__device__ __forceinline__ float* leg_at(LegShared<L>& sh, const LegCol<L>& t, int c, int i) {
  return &sh.v[c][0][0] + ((t.up ? kLegR - 1 - i : i) * L::PL + t.pos);
}
template <class L>
__device__ __forceinline__ void leg_share(LegShared<L>& sh, const LegCol<L>& t, int c, const float (&v)[kLegZ]) {
#pragma unroll
  for (int i = 0; i < kLegZ; ++i) *leg_at<L>(sh, t, c, i) = v[i];
}
// neighbour sum of colour c's cell at index i >= 1, in the order x, y-, y+,
// z-, z+ (the two x neighbours' sum does not depend on their order)
template <class L>
__device__ __forceinline__ float leg_sum(const LegCol<L>& t, LegShared<L>& sh, const float (&e)[2][kLegZ], int c,
                                         int i) {
  const float* o = e[1 - c];
  const float ext = __shfl_sync(0xffffffffu, o[i], t.par(c, i) ? t.lane[1] : t.lane[0]);
  const float* s = leg_at<L>(sh, t, 1 - c, i);
  const float inner = i + 1 < kLegZ ? o[i + 1 < kLegZ ? i + 1 : 0] : (t.up ? s[-L::PL] : s[L::PL]);
  const float outer = o[i - 1];
  const float zm = t.up ? inner : outer, zp = t.up ? outer : inner;
  return ((((o[i] + ext) + s[-L::KW]) + s[L::KW]) + zm) + zp;
}
// t / diag as the half-sweep kernels form it at colour c's cell of index i:
// the product with 1/6, else the IEEE quotient (from the correctly rounded
// reciprocal and one exact remainder, see div_by; an infinite quotient as it
// is), rounded to the storage type; 0 outside the grid
template <class T, class L>
__device__ __forceinline__ float leg_value(const Grid& d, const LegCol<L>& t, int c, int i, float num) {
  if (!t.has_z(d, i)) return 0.0f;  // uniform over the half block
  const bool w = t.wall_z(d, i);
  const bool p = t.par(c, i) != 0;
  const float dg = w ? (p ? t.d1[1] : t.d1[0]) : (p ? t.d0[1] : t.d0[0]);
  const float r = w ? (p ? t.r1[1] : t.r1[0]) : (p ? t.r0[1] : t.r0[0]);
  const float rc = w ? (p ? t.c1[1] : t.c1[0]) : (p ? t.c0[1] : t.c0[0]);
  const float qv = __fmul_rn(num, r);
  const float v = __fmaf_rn(__fmaf_rn(-qv, dg, num), rc, qv);
  return t.in ? as_stored<T>(fabsf(qv) <= 3.4028234e38f ? v : qv) : 0.0f;
}
// half-sweep of colour c on the planes within D of the tile
template <class T, class L, int D>
__device__ __forceinline__ void leg_half(const Grid& d, float h2, const LegCol<L>& t, LegShared<L>& sh, int c,
                                         float (&e)[2][kLegZ], const float (&b)[2][kLegZ]) {
#pragma unroll
  for (int i = L::H - D; i < kLegZ; ++i) {
    const float sumN = leg_sum<L>(t, sh, e, c, i);
    e[c][i] = leg_value<T, L>(d, t, c, i, sumN - h2 * b[c][i]);
    *leg_at<L>(sh, t, c, i) = e[c][i];
  }
  __syncthreads();
}
// the tile's cells to the split array
template <class T, class L>
__device__ __forceinline__ void leg_store(const Grid& d, const LegCol<L>& t, const float (&e)[2][kLegZ],
                                          T* __restrict__ a) {
  if (!t.in || t.kk < L::H / 2 || t.kk >= L::H / 2 + L::TX / 2 || t.yy < L::H || t.yy >= L::H + L::TY) return;
  const uint32_t half = (uint32_t)(d.n() >> 1);
#pragma unroll
  for (int i = L::H; i < kLegZ; ++i)
    if (t.has_z(d, i)) {
      stf(a + t.off(i), e[0][i]);
      stf(a + (half + t.off(i)), e[1][i]);
    }
}

// S red-black sweeps against b into out, then the residual of the result
// averaged into the coarse right-hand side bc.  ZERO: the sweeps start from
// zero; else the preceding launch was the first red half-sweep on a, whose red
// cells are read, and the loads of b, which it did not write, issue ahead of
// the wait for it.
// TR (with ZERO; the transposed cycle): the colours change places, and the
// residual of the black cells goes to res (the red ones, updated last, have
// none but rounding).
// sixth (with ZERO): the first half-sweep multiplies by 1/6 at every diagonal of
// 6, as the restriction forms it in the FP32 cycle's chain (restrict_pair); in
// the mixed one's chain the half-sweep kernel forms it.
template <class T, class TC, class L, bool ZERO, bool TR>
__global__ void __launch_bounds__(L::NT) k_leg_down(Grid d, Grid dc, float h2, float inv_h2, int ref, int sixth,
                                                    const T* __restrict__ a, const T* __restrict__ b,
                                                    T* __restrict__ out, TC* __restrict__ bc, T* __restrict__ res,
                                                    const unsigned int* __restrict__ skip) {
  static_assert(ZERO || !TR, "the transposed cycle starts from zero");
  constexpr int c0 = TR ? 1 : 0;  // the colour of the first half-sweep
  __shared__ LegShared<L> sh;
  const LegCol<L> t(d, ref);
  float e[2][kLegZ], bb[2][kLegZ];
  if (!ZERO) {
    leg_load<T, L>(d, t, b, 0, bb[0]);
    leg_load<T, L>(d, t, b, 1, bb[1]);
  }
  pdl_wait();
  pdl_trigger();
  if (skip_now(skip)) return;
  if (ZERO) {
    leg_load<T, L>(d, t, b, 0, bb[0]);
    leg_load<T, L>(d, t, b, 1, bb[1]);
    LegCol<L> first = t;
#pragma unroll
    for (int p = 0; p < 2; ++p)
      if (sixth && t.d0[p] == 6.0f) first.c0[p] = 0.0f;
#pragma unroll
    for (int i = 0; i < kLegZ; ++i) e[c0][i] = leg_value<T, L>(d, first, c0, i, 0.0f - h2 * bb[c0][i]);
  } else {
    leg_load<T, L>(d, t, a, c0, e[c0]);
  }
  leg_share<L>(sh, t, c0, e[c0]);
  __syncthreads();
  if constexpr (L::S == 2) {
    leg_half<T, L, 3>(d, h2, t, sh, 1 - c0, e, bb);
    leg_half<T, L, 2>(d, h2, t, sh, c0, e, bb);
  }
  leg_half<T, L, 1>(d, h2, t, sh, 1 - c0, e, bb);
  leg_store<T, L>(d, t, e, out);
  auto residual = [&](int c, int i) {
    const float sumN = leg_sum<L>(t, sh, e, c, i);
    const bool w = t.wall_z(d, i), p = t.par(c, i) != 0;
    const float dg = w ? (p ? t.d1[1] : t.d1[0]) : (p ? t.d0[1] : t.d0[0]);
    const float lap = (sumN - dg * e[c][i]) * inv_h2;
    return bb[c][i] - lap;
  };
  const bool mine = t.in && t.kk >= L::H / 2 && t.kk < L::H / 2 + L::TX / 2 && t.yy >= L::H && t.yy < L::H + L::TY;
  if constexpr (TR) {
    T* r = res + (uint32_t)(d.n() >> 1);
#pragma unroll
    for (int i = L::H; i < kLegZ; ++i) {
      const float v = residual(1, i);
      if (mine && t.has_z(d, i)) stf(r + t.off(i), v);
    }
    return;
  }
  // the residuals of a coarse cell: x = 2k, 2k + 1 and both planes are this
  // thread's, the row above the next row's thread's
  const bool put = mine && (t.yy & 1) == 0;
#pragma unroll
  for (int i = L::H; i < kLegZ; i += 2) {
    float r[2][2], u[2][2];  // [index][x] of this row and the next
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float rc[2] = {residual(0, i + j), residual(1, i + j)};
      const bool sw = t.par(0, i + j) != 0;  // colour 0's cell is x = 2k + 1
      r[j][0] = sw ? rc[1] : rc[0];
      r[j][1] = sw ? rc[0] : rc[1];
#pragma unroll
      for (int x = 0; x < 2; ++x) u[j][x] = __shfl_down_sync(0xffffffffu, r[j][x], L::KW);
    }
    float sum = 0.0f;  // z, then y, then x ascending: index j is plane j, or 1 - j in the upper half
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float a0 = t.up ? r[1 - j][0] : r[j][0], a1 = t.up ? r[1 - j][1] : r[j][1];
      const float b0 = t.up ? u[1 - j][0] : u[j][0], b1 = t.up ? u[1 - j][1] : u[j][1];
      sum = (((sum + a0) + a1) + b0) + b1;
    }
    const int Z = (t.up ? t.z(i + 1) : t.z(i)) >> 1;
    if (put && Z < dc.nz) stf(bc + rb_index(dc, t.k, t.y >> 1, Z), sum * 0.125f);
  }
}

// a + the prolonged coarse correction ec, then S red-black sweeps against b,
// into out.  Only the black cells take the correction (the first half-sweep
// overwrites the red ones without reading them).  a and b were not written
// by the preceding launch: their loads issue ahead of the wait for it.
// TR (the transposed cycle): the colours change places, and the correction is
// an eighth of ec's cell (the transpose of the restriction's average).
template <class T, class TC, class L, bool TR>
__global__ void __launch_bounds__(L::NT) k_leg_up(Grid d, Grid dc, float h2, int ref, const T* __restrict__ a,
                                                  const T* __restrict__ b, const TC* __restrict__ ec,
                                                  T* __restrict__ out, const unsigned int* __restrict__ skip) {
  __shared__ LegShared<L> sh;
  // coarse taps, clamped at the grid (0 above a Dirichlet top)
  __shared__ float C[TR ? 1 : L::CZ][L::CY][L::CX];
  const LegCol<L> t(d, ref);
  float e[2][kLegZ], bb[2][kLegZ];
  leg_load<T, L>(d, t, b, 0, bb[0]);
  leg_load<T, L>(d, t, b, 1, bb[1]);
  constexpr int c0 = TR ? 0 : 1;  // the colour that takes the correction
  leg_load<T, L>(d, t, a, c0, e[c0]);
  if constexpr (TR) {
    pdl_wait();
    pdl_trigger();
    if (skip_now(skip)) return;
    const uint32_t hc = (uint32_t)(dc.nx >> 1), halfc = (uint32_t)(dc.n() >> 1);
#pragma unroll
    for (int i = 0; i < kLegZ; i += 2) {  // planes i and i + 1 have one parent
      const int Y = t.y >> 1, Z = t.z(i) >> 1;
      const bool on = t.in && t.has_z(d, i);
      const float v =
          on ? 0.125f * ldv(ec + ((((t.k + Y + Z) & 1) ? halfc : 0u) + ((uint32_t)Z * dc.ny + Y) * hc + (t.k >> 1)))
             : 0.0f;
      e[c0][i] = on ? as_stored<T>(e[c0][i] + v) : 0.0f;
      e[c0][i + 1] = on ? as_stored<T>(e[c0][i + 1] + v) : 0.0f;
    }
  } else {
    // first coarse tap: the region's corner is even, so fine cell i of an axis
    // interpolates taps (i + 1) / 2 and (i + 1) / 2 + 1
    const int Z0 = (int)blockIdx.z * L::TZ - L::H;
    const int XC = t.k - t.kk - 1, YC = ((int)blockIdx.y * L::TY - L::H) / 2 - 1, ZC = Z0 / 2 - 1;
    auto frac = [](int i, int n, float r, int m) {
      const float u = __fmaf_rn(div_by((float)i + 0.5f, (float)n, r), (float)m, -0.5f);
      return u - floorf(u);
    };
    const float fx0 = frac(2 * t.k, d.nx, d.rx, dc.nx), fx1 = frac(2 * t.k + 1, d.nx, d.rx, dc.nx);
    const float fy = frac(t.y, d.ny, d.ry, dc.ny);
    pdl_wait();
    pdl_trigger();
    if (skip_now(skip)) return;
#pragma unroll
    for (int i0 = 0; i0 < L::CX * L::CY * L::CZ; i0 += L::NT) {
      const int i = i0 + (int)threadIdx.x;
      if (i < L::CX * L::CY * L::CZ) {
        const int xi = i % L::CX, yi = (i / L::CX) % L::CY, zi = i / (L::CX * L::CY);
        const int X = dob_clampi(XC + xi, 0, dc.nx - 1), Y = dob_clampi(YC + yi, 0, dc.ny - 1),
                  Z = dob_clampi(ZC + zi, 0, dc.nz - 1);
        const uint32_t j = (((X + Y + Z) & 1) ? (uint32_t)(dc.n() >> 1) : 0u) +
                           ((uint32_t)Z * dc.ny + (uint32_t)Y) * (uint32_t)(dc.nx >> 1) + (uint32_t)(X >> 1);
        const float v = ldv(ec + j);
        C[zi][yi][xi] = ref && YC + yi >= dc.ny ? 0.0f : v;
      }
    }
    __syncthreads();
    // coarse plane m interpolated in x and y at this row's cells x = 2k (s0)
    // and 2k + 1 (s1); region plane zz interpolates coarse planes (zz + 1) / 2
    // and the next: going inwards from index 0, the lower half meets planes
    // 0, 1, .. with (zz + 1) / 2 = (i + 1) / 2, the upper half planes 9, 8, ..
    // with (zz + 1) / 2 + 1 = 9 - (i + 1) / 2
    auto plane = [&](int m, float& s0, float& s1) {
      const float* c0 = &C[t.up ? L::CZ - 1 - m : m][(t.yy + 1) >> 1][t.kk];
      const float* c1 = c0 + L::CX;
      s0 = dob_mix(dob_mix(c0[0], c0[1], fx0), dob_mix(c1[0], c1[1], fx0), fy);
      s1 = dob_mix(dob_mix(c0[1], c0[2], fx1), dob_mix(c1[1], c1[2], fx1), fy);
    };
    float lo0, lo1;
    plane(0, lo0, lo1);
#pragma unroll
    for (int m = 0; m <= kLegZ / 2; ++m) {
      float hi0, hi1;
      plane(m + 1, hi0, hi1);
#pragma unroll
      for (int i = 2 * m - 1; i <= 2 * m; ++i) {
        if (i < 0 || i >= kLegZ) continue;
        const bool p = t.par(1, i) != 0;
        const float fz = frac(t.z(i), d.nz, d.rz, dc.nz);
        const float u = p ? lo1 : lo0, v = p ? hi1 : hi0;  // the outer and the inner plane
        const float corr = dob_mix(t.up ? v : u, t.up ? u : v, fz);
        e[1][i] = t.in && t.has_z(d, i) ? as_stored<T>(e[1][i] + corr) : 0.0f;
      }
      lo0 = hi0;
      lo1 = hi1;
    }
  }
  leg_share<L>(sh, t, c0, e[c0]);
  __syncthreads();
  if constexpr (L::S == 2) {
    leg_half<T, L, 3>(d, h2, t, sh, 1 - c0, e, bb);
    leg_half<T, L, 2>(d, h2, t, sh, c0, e, bb);
  }
  leg_half<T, L, 1>(d, h2, t, sh, 1 - c0, e, bb);
  leg_half<T, L, 0>(d, h2, t, sh, c0, e, bb);
  leg_store<T, L>(d, t, e, out);
}

}  // namespace dob
