// rhs_fp32.cuh -- fused DG Maxwell right-hand side on the CUDA cores, in FP32
// (rhs_fp32_kernel, the FP32 engine and the Arnoldi matvec) or FP64
// (rhs_fp64_kernel, the FP64 path: f64 operators, element records and state).
//
// One persistent CTA per SM slot walks tiles of E elements.  Per tile:
//   1. the y tile (E*6*Np floats, contiguous in the SoA layout) and the element
//      records are copied to shared memory with 16-byte vector loads;
//   2. the numerical flux of all 4*Nfp face nodes of every element is formed
//      (rhs.rs:1370-1441): the neighbour trace comes from shared memory when
//      the neighbour is in the tile, else from L2/HBM;
//   3. each thread owns one (element, node), at order 4 two: 18 reference derivatives
//      D_k * F_c (rhs.rs:39-85), combined with J^-1 into curl H / -curl E;
//   4. the LIFT sum over the 4*Nfp flux values (rhs.rs:1433-1439), the
//      material scaling (rhs.rs:1443-1454), and the mode's epilogue:
//      plain dy, the fused LSERK4 stage update (explicit.rs:122-133, so dy
//      never reaches HBM), or the Krylov matvec output (scaled dy plus the
//      augmented source column).
// D and LIFT live in shared memory for the whole kernel.
#pragma once
#include <cstdint>
#include <type_traits>

#include "dgtd_common.cuh"
#include "tc_util.cuh"

namespace dgtd {

// One node per thread: every order but 4 (PairCfg, below).
template <int N, class R = float, int TD = 1>
struct Fp32Cfg {
  static_assert(N != 4, "order 4 has two nodes per thread");
  static constexpr int NP = np_of(N);
  static constexpr int NFP = nfp_of(N);
  static constexpr int NF = 4 * NFP;
  // Elements per tile: ~256 threads (TD = 1) or half as many (TD = 2, the
  // small-tile engine), E even so the tile start stays 16B aligned.
  static constexpr int E = (N == 1 ? 64 : N == 2 ? 24 : N == 3 ? 12 : 4) / TD;
  static_assert(TD == 1 || TD == 2, "tile divisor");
  static constexpr int THREADS = ((E * NP + 31) / 32) * 32;
  static constexpr int TILE = E * 6 * NP;  // values of state per tile
  // shared memory layout (in R); every region starts on a 16-byte boundary
  // because the state tile and the element records are filled with 16-byte
  // vectors (4 floats or 2 doubles).
  static constexpr int PER16 = 16 / (int)sizeof(R);
  static constexpr int al4(int x) { return (x + PER16 - 1) / PER16 * PER16; }
  static constexpr int OFF_D = 0;
  static constexpr int OFF_L = al4(OFF_D + 3 * NP * NP);
  static constexpr int OFF_Y = al4(OFF_L + NF * NP);
  static constexpr int OFF_F = al4(OFF_Y + TILE);
  static constexpr int OFF_M = al4(OFF_F + E * 6 * NF);
  static constexpr int OFF_B = al4(OFF_M + E * kMetaWords);  // byte tables start (in R)
  static constexpr int BYTES_TAB = 4 * NFP + kMaxGather * NFP;
  static constexpr int SMEM = OFF_B * (int)sizeof(R) + ((BYTES_TAB + 15) / 16) * 16;
  static_assert(OFF_Y % PER16 == 0 && OFF_M % PER16 == 0, "vector regions must be 16-byte aligned");
  static_assert(((E * 6 * NP) % PER16) == 0, "consecutive tiles must start 16-byte aligned");
  static_assert((kMetaWords % PER16) == 0, "element records are whole 16-byte vectors");
};

template <class R> struct Vec16;
template <> struct Vec16<float> { using T = float4; };
template <> struct Vec16<double> { using T = double2; };

// Integer words of an element record: bit patterns in the f32 records, exact
// values in the f64 records.
__device__ __forceinline__ int rec_int(float v) { return __float_as_int(v); }
__device__ __forceinline__ int rec_int(double v) { return (int)v; }
__device__ __forceinline__ uint32_t rec_uint(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t rec_uint(double v) { return (uint32_t)v; }

template <class R>
__device__ __forceinline__ void cross3f(R ax, R ay, R az, R bx, R by, R bz, R& ox, R& oy, R& oz) {
  ox = ay * bz - az * by;
  oy = az * bx - ax * bz;
  oz = ax * by - ay * bx;
}

template <int N, int MODE, class R, int TD = 1>
__device__ __forceinline__ void rhs_cc_body(const RhsParamsT<R>& P, const OpTablesT<R>& T) {
  using C = Fp32Cfg<N, R, TD>;
  using V = typename Vec16<R>::T;
  constexpr int NP = C::NP, NFP = C::NFP, NF = C::NF, E = C::E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* smem = reinterpret_cast<R*>(smem_raw);
  R* sD = smem + C::OFF_D;
  R* sL = smem + C::OFF_L;
  R* sY = smem + C::OFF_Y;
  R* sF = smem + C::OFF_F;
  R* sM = smem + C::OFF_M;
  uint8_t* sFn = reinterpret_cast<uint8_t*>(smem + C::OFF_B);
  uint8_t* sG = sFn + 4 * NFP;
  const int tid = threadIdx.x;

  for (int i = tid; i < 3 * NP * NP; i += blockDim.x) sD[i] = T.dT[i];
  for (int i = tid; i < NF * NP; i += blockDim.x) sL[i] = T.liftT[i];
  for (int i = tid; i < 4 * NFP; i += blockDim.x) sFn[i] = T.fnodes[i];
  for (int i = tid; i < T.n_gather * NFP; i += blockDim.x) sG[i] = T.gtab[i];

  pdl_wait();
  if (P.skip != nullptr && *P.skip) return;  // uniform: nothing to do for this launch
  R kry_sig = 1, kry_g = 0;
  if (MODE == kModeKrylov) {
    kry_sig = (R)P.kry[0];
    kry_g = (R)P.kry[1];
  }

  const int64_t n_tiles = (P.n_elem - P.e_begin + E - 1) / E;
  const int le_me = tid / NP;
  const int i_me = tid - le_me * NP;
  const bool owns = tid < E * NP;

  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t e0 = P.e_begin + tile * E;
    const int ne = (int)((P.n_elem - e0) < E ? (P.n_elem - e0) : E);
    __syncthreads();  // previous tile fully consumed (and tables loaded on the first pass)
    // ---- 1. state tile and element records -> shared memory
    const int nfloat = ne * 6 * NP;
    {
      const R* src = P.y_in + e0 * 6 * NP;
      if ((nfloat % C::PER16) == 0) {
        const V* s4 = reinterpret_cast<const V*>(src);
        V* d4 = reinterpret_cast<V*>(sY);
        for (int i = tid; i < nfloat / C::PER16; i += blockDim.x) d4[i] = s4[i];
      } else {
        for (int i = tid; i < nfloat; i += blockDim.x) sY[i] = src[i];
      }
    }
    {
      const V* m4 = reinterpret_cast<const V*>(P.meta + e0 * kMetaWords);
      V* d4 = reinterpret_cast<V*>(sM);
      for (int i = tid; i < ne * kMetaWords / C::PER16; i += blockDim.x) d4[i] = __ldg(m4 + i);
    }
    __syncthreads();

    // ---- 2. numerical flux at the 4*Nfp face nodes of each element
    for (int q = tid; q < ne * NF; q += blockDim.x) {
      const int le = q / NF;
      const int s = q - le * NF;
      const int f = s / NFP;
      const int m = s - f * NFP;
      const R* M = sM + le * kMetaWords;
      const R nx = M[9 + 3 * f], ny = M[10 + 3 * f], nz = M[11 + 3 * f];
      const R coef = R(0.5) * M[21 + f];
      const int nbr = rec_int(M[37 + f]);
      const uint32_t codes = rec_uint(M[41 + (f >> 1)]);
      const uint32_t code = (f & 1) ? (codes >> 16) : (codes & 0xffffu);
      const int kind = (code >> 8) & 3;
      const int vi = sFn[f * NFP + m];
      const R* Y = sY + le * 6 * NP;
      const R ex = Y[0 * NP + vi], ey = Y[1 * NP + vi], ez = Y[2 * NP + vi];
      const R hx = Y[3 * NP + vi], hy = Y[4 * NP + vi], hz = Y[5 * NP + vi];
      R jex, jey, jez, jhx, jhy, jhz;
      R a = P.alpha;
      if (kind == kPort) {
        // characteristic boundary against a zero incident field (rhs.rs:1380-1386)
        jex = ex; jey = ey; jez = ez; jhx = hx; jhy = hy; jhz = hz;
        a = R(1);
      } else if (kind == kPec) {
        // PEC ghost: [E] = 2 E_tan, [H] = 2 H_n (rhs.rs:1387-1402)
        const R edn = nx * ex + ny * ey + nz * ez;
        const R hdn = nx * hx + ny * hy + nz * hz;
        jex = R(2) * (ex - edn * nx); jey = R(2) * (ey - edn * ny); jez = R(2) * (ez - edn * nz);
        jhx = R(2) * (hdn * nx); jhy = R(2) * (hdn * ny); jhz = R(2) * (hdn * nz);
      } else {
        const int vj = sG[(code & 0xff) * NFP + m];
        const int64_t lo = (int64_t)nbr - e0;
        R px, py, pz, qx, qy, qz;
        if (lo >= 0 && lo < ne) {
          const R* Z = sY + lo * 6 * NP;
          px = Z[0 * NP + vj]; py = Z[1 * NP + vj]; pz = Z[2 * NP + vj];
          qx = Z[3 * NP + vj]; qy = Z[4 * NP + vj]; qz = Z[5 * NP + vj];
        } else {
          const R* Z = P.y_in + (int64_t)nbr * 6 * NP;
          px = Z[0 * NP + vj]; py = Z[1 * NP + vj]; pz = Z[2 * NP + vj];
          qx = Z[3 * NP + vj]; qy = Z[4 * NP + vj]; qz = Z[5 * NP + vj];
        }
        jex = ex - px; jey = ey - py; jez = ez - pz;
        jhx = hx - qx; jhy = hy - qy; jhz = hz - qz;
      }
      // n x [H], n x [E], n x (n x [E]), n x (n x [H])   (rhs.rs:1420-1432)
      R nhx, nhy, nhz, nex, ney, nez, pex, pey, pez, phx, phy, phz;
      cross3f(nx, ny, nz, jhx, jhy, jhz, nhx, nhy, nhz);
      cross3f(nx, ny, nz, jex, jey, jez, nex, ney, nez);
      cross3f(nx, ny, nz, nex, ney, nez, pex, pey, pez);
      cross3f(nx, ny, nz, nhx, nhy, nhz, phx, phy, phz);
      R* F = sF + le * 6 * NF;
      F[0 * NF + s] = coef * (-nhx + a * pex);
      F[1 * NF + s] = coef * (-nhy + a * pey);
      F[2 * NF + s] = coef * (-nhz + a * pez);
      F[3 * NF + s] = coef * (nex + a * phx);
      F[4 * NF + s] = coef * (ney + a * phy);
      F[5 * NF + s] = coef * (nez + a * phz);
    }

    // ---- 3. volume term: reference derivatives of E and H at my node
    R dex = 0, dey = 0, dez = 0, dhx = 0, dhy = 0, dhz = 0;
    const bool active = owns && le_me < ne;
    if (active) {
      const R* Y = sY + le_me * 6 * NP;
      R r[3][6];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < 6; ++c) r[k][c] = 0;
      if constexpr (N == 5 && sizeof(R) == 4) {
        // the element's state rows are 16-byte aligned (Np = 56): four nodes of
        // all six components per float4 (broadcast) load, same accumulation
        // order (order 5: 14 % faster; order 3 measured no gain)
#pragma unroll 2
        for (int j0 = 0; j0 < NP; j0 += 4) {
          float4 yv[6];
#pragma unroll
          for (int c = 0; c < 6; ++c) yv[c] = *reinterpret_cast<const float4*>(Y + c * NP + j0);
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const int j = j0 + jj;
            const float d0 = sD[(0 * NP + j) * NP + i_me];
            const float d1 = sD[(1 * NP + j) * NP + i_me];
            const float d2 = sD[(2 * NP + j) * NP + i_me];
#pragma unroll
            for (int c = 0; c < 6; ++c) {
              const float v = jj == 0 ? yv[c].x : jj == 1 ? yv[c].y : jj == 2 ? yv[c].z : yv[c].w;
              r[0][c] = fmaf(d0, v, r[0][c]);
              r[1][c] = fmaf(d1, v, r[1][c]);
              r[2][c] = fmaf(d2, v, r[2][c]);
            }
          }
        }
      } else {
#pragma unroll 5
        for (int j = 0; j < NP; ++j) {
          const R d0 = sD[(0 * NP + j) * NP + i_me];
          const R d1 = sD[(1 * NP + j) * NP + i_me];
          const R d2 = sD[(2 * NP + j) * NP + i_me];
#pragma unroll
          for (int c = 0; c < 6; ++c) {
            const R v = Y[c * NP + j];
            r[0][c] = fma(d0, v, r[0][c]);
            r[1][c] = fma(d1, v, r[1][c]);
            r[2][c] = fma(d2, v, r[2][c]);
          }
        }
      }
      // physical derivatives pd[p][c] = sum_k Jinv[k][p] r[k][c] (rhs.rs:62-75)
      const R* M = sM + le_me * kMetaWords;
      R pd[3][6];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const R j0 = M[0 * 3 + p], j1 = M[1 * 3 + p], j2 = M[2 * 3 + p];
#pragma unroll
        for (int c = 0; c < 6; ++c) pd[p][c] = j0 * r[0][c] + j1 * r[1][c] + j2 * r[2][c];
      }
      // dE = curl H, dH = -curl E (rhs.rs:78-84, :1365-1368)
      dex = pd[1][5] - pd[2][4];
      dey = pd[2][3] - pd[0][5];
      dez = pd[0][4] - pd[1][3];
      dhx = -(pd[1][2] - pd[2][1]);
      dhy = -(pd[2][0] - pd[0][2]);
      dhz = -(pd[0][1] - pd[1][0]);
    }
    __syncthreads();  // flux complete

    // ---- 4. LIFT, materials, epilogue
    if (active) {
      const R* F = sF + le_me * 6 * NF;
      // order 5: the element's flux rows (NF = 4 Nfp values each) are 16-byte
      // aligned, so four face nodes of all six components come per float4
      // (broadcast) load; same accumulation order
      static_assert(NF % 4 == 0, "flux rows are whole float4s");
      if constexpr (N == 5 && sizeof(R) == 4) {
#pragma unroll 2
      for (int s0 = 0; s0 < NF; s0 += 4) {
        float4 fv[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) fv[c] = *reinterpret_cast<const float4*>(F + c * NF + s0);
#pragma unroll
        for (int ss = 0; ss < 4; ++ss) {
          const float w = sL[(s0 + ss) * NP + i_me];
          const auto pick = [ss](const float4& q) { return ss == 0 ? q.x : ss == 1 ? q.y : ss == 2 ? q.z : q.w; };
          dex = fmaf(w, pick(fv[0]), dex);
          dey = fmaf(w, pick(fv[1]), dey);
          dez = fmaf(w, pick(fv[2]), dez);
          dhx = fmaf(w, pick(fv[3]), dhx);
          dhy = fmaf(w, pick(fv[4]), dhy);
          dhz = fmaf(w, pick(fv[5]), dhz);
        }
      }
      } else {
#pragma unroll 4
        for (int s = 0; s < NF; ++s) {
          const R w = sL[s * NP + i_me];
          dex = fma(w, F[0 * NF + s], dex);
          dey = fma(w, F[1 * NF + s], dey);
          dez = fma(w, F[2 * NF + s], dez);
          dhx = fma(w, F[3 * NF + s], dhx);
          dhy = fma(w, F[4 * NF + s], dhy);
          dhz = fma(w, F[5 * NF + s], dhz);
        }
      }
      const R* M = sM + le_me * kMetaWords;
      const R* Y = sY + le_me * 6 * NP;
      R dy[6];
      dy[0] = M[25] * dex - M[31] * Y[0 * NP + i_me];
      dy[1] = M[26] * dey - M[32] * Y[1 * NP + i_me];
      dy[2] = M[27] * dez - M[33] * Y[2 * NP + i_me];
      dy[3] = M[28] * dhx - M[34] * Y[3 * NP + i_me];
      dy[4] = M[29] * dhy - M[35] * Y[4 * NP + i_me];
      dy[5] = M[30] * dhz - M[36] * Y[5 * NP + i_me];
      const int64_t base = (e0 + le_me) * 6 * NP + i_me;
      if (MODE == kModeApply) {
#pragma unroll
        for (int c = 0; c < 6; ++c) P.out[base + c * NP] = dy[c];
      } else if (MODE == kModeLserk) {
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          const int64_t g = base + c * NP;
          R k = dy[c];
          if (P.src_vec != nullptr) k = fma(P.src_g, P.src_vec[g], k);
          if (g == P.src_idx) k += P.src_g;
          R pv = (P.dt * M[43]) * k;
          if (P.read_p) pv = fma(P.a, P.p[g], pv);
          if (P.write_p) P.p[g] = pv;
          P.out[g] = fma(P.b, pv, Y[c * NP + i_me]);
        }
      } else if (MODE == kModeKcl) {
        // KCL stage (explicit_adaptive.rs:84-152), in the operation order of
        // the separate stage kernel (kcl.cuh k_kcl_stage)
        const R h = (R)*P.kcl_h;
        const R gs = P.kcl_g != nullptr ? (R)P.kcl_g[*P.kcl_frame] : R(0);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          const int64_t g = base + c * NP;
          R kk = dy[c];
          if (P.src_vec != nullptr) kk += P.src_vec[g] * gs;
          if (g == P.src_idx) kk += gs;
          const R f = h * kk;
          const R yn = P.kcl_y[g] + P.kcl_b * f;
          P.kcl_y[g] = yn;
          P.kcl_e[g] = P.kcl_stage == 0 ? P.kcl_ew * f : P.kcl_e[g] + P.kcl_ew * f;
          if (P.kcl_next != nullptr) P.kcl_next[g] = yn + P.kcl_amb * f;
        }
      } else {
        // Krylov matvec of a stored basis vector: its scale and the source
        // coefficient of the augmented system come from device memory
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          const int64_t g = base + c * NP;
          R w = kry_sig * dy[c];
          if (P.src_vec != nullptr) w = fma(kry_g, P.src_vec[g], w);
          if (g == P.src_idx) w += kry_g;
          P.out[g] = w;
        }
      }
    }
  }
  // Several of these CTAs share an SM: a next launch let in earlier is placed
  // wherever there is room, unevenly (the f64 kernel: 13 % slower).
  pdl_launch();
}

// The numerical flux (rhs.rs:1370-1441) at the face nodes of a tile's `ne` elements
// from e0 on, by all threads: states sY and fluxes sF with element strides YS, FS.
// (As in rhs_cc_body, which keeps its own copy: called from there it cost order 5
// 18 %, and as long as order 5 needs the copy, calling it at the other orders
// would spare no code.)
template <int N, int YS, int FS, class R>
__device__ __forceinline__ void rhs_cc_flux(const RhsParamsT<R>& P, int64_t e0, int ne, const R* sY, const R* sM,
                                            const uint8_t* sFn, const uint8_t* sG, R* sF) {
  constexpr int NP = np_of(N), NFP = nfp_of(N), NF = 4 * NFP;
  for (int q = threadIdx.x; q < ne * NF; q += blockDim.x) {
    const int le = q / NF;
    const int s = q - le * NF;
    const int f = s / NFP;
    const int m = s - f * NFP;
    const R* M = sM + le * kMetaWords;
    const R nx = M[9 + 3 * f], ny = M[10 + 3 * f], nz = M[11 + 3 * f];
    const R coef = R(0.5) * M[21 + f];
    const int nbr = rec_int(M[37 + f]);
    const uint32_t codes = rec_uint(M[41 + (f >> 1)]);
    const uint32_t code = (f & 1) ? (codes >> 16) : (codes & 0xffffu);
    const int kind = (code >> 8) & 3;
    const int vi = sFn[f * NFP + m];
    const R* Y = sY + le * YS;
    const R ex = Y[0 * NP + vi], ey = Y[1 * NP + vi], ez = Y[2 * NP + vi];
    const R hx = Y[3 * NP + vi], hy = Y[4 * NP + vi], hz = Y[5 * NP + vi];
    R jex, jey, jez, jhx, jhy, jhz;
    R a = P.alpha;
    if (kind == kPort) {
      // characteristic boundary against a zero incident field (rhs.rs:1380-1386)
      jex = ex; jey = ey; jez = ez; jhx = hx; jhy = hy; jhz = hz;
      a = R(1);
    } else if (kind == kPec) {
      // PEC ghost: [E] = 2 E_tan, [H] = 2 H_n (rhs.rs:1387-1402)
      const R edn = nx * ex + ny * ey + nz * ez;
      const R hdn = nx * hx + ny * hy + nz * hz;
      jex = R(2) * (ex - edn * nx); jey = R(2) * (ey - edn * ny); jez = R(2) * (ez - edn * nz);
      jhx = R(2) * (hdn * nx); jhy = R(2) * (hdn * ny); jhz = R(2) * (hdn * nz);
    } else {
      const int vj = sG[(code & 0xff) * NFP + m];
      const int64_t lo = (int64_t)nbr - e0;
      R px, py, pz, qx, qy, qz;
      if (lo >= 0 && lo < ne) {
        const R* Z = sY + lo * YS;
        px = Z[0 * NP + vj]; py = Z[1 * NP + vj]; pz = Z[2 * NP + vj];
        qx = Z[3 * NP + vj]; qy = Z[4 * NP + vj]; qz = Z[5 * NP + vj];
      } else {
        const R* Z = P.y_in + (int64_t)nbr * 6 * NP;
        px = Z[0 * NP + vj]; py = Z[1 * NP + vj]; pz = Z[2 * NP + vj];
        qx = Z[3 * NP + vj]; qy = Z[4 * NP + vj]; qz = Z[5 * NP + vj];
      }
      jex = ex - px; jey = ey - py; jez = ez - pz;
      jhx = hx - qx; jhy = hy - qy; jhz = hz - qz;
    }
    // n x [H], n x [E], n x (n x [E]), n x (n x [H])   (rhs.rs:1420-1432)
    R nhx, nhy, nhz, nex, ney, nez, pex, pey, pez, phx, phy, phz;
    cross3f(nx, ny, nz, jhx, jhy, jhz, nhx, nhy, nhz);
    cross3f(nx, ny, nz, jex, jey, jez, nex, ney, nez);
    cross3f(nx, ny, nz, nex, ney, nez, pex, pey, pez);
    cross3f(nx, ny, nz, nhx, nhy, nhz, phx, phy, phz);
    R* F = sF + le * FS;
    F[0 * NF + s] = coef * (-nhx + a * pex);
    F[1 * NF + s] = coef * (-nhy + a * pey);
    F[2 * NF + s] = coef * (-nhz + a * pez);
    F[3 * NF + s] = coef * (nex + a * phx);
    F[4 * NF + s] = coef * (ney + a * phy);
    F[5 * NF + s] = coef * (nez + a * phz);
  }
}

template <class R> struct Vec2;
template <> struct Vec2<float> { using T = float2; };
template <> struct Vec2<double> { using T = double2; };

// The two nodes of a thread (an f32 pair or two f64): x += a * v for a row of
// operator entries a (one vector load) and one value v.
template <class R> struct Acc;
template <> struct Acc<float> {
  uint64_t p;
  using Row = uint64_t;
  using Val = uint64_t;
  __device__ __forceinline__ void zero() { p = 0ull; }
  __device__ __forceinline__ static Row row(const float* s) { return *reinterpret_cast<const uint64_t*>(s); }
  __device__ __forceinline__ static Val val(float v) { return tc::dup2(v); }
  __device__ __forceinline__ void fma(Row a, Val v) { p = tc::fma2(a, v, p); }
  __device__ __forceinline__ void get(float (&o)[2]) const { tc::unpack2(p, o[0], o[1]); }
  __device__ __forceinline__ void set(const float (&o)[2]) { p = tc::pack2(o[0], o[1]); }
};
template <> struct Acc<double> {
  double p[2];
  using Row = double2;
  using Val = double;
  __device__ __forceinline__ void zero() { p[0] = p[1] = 0.0; }
  __device__ __forceinline__ static Row row(const double* s) { return *reinterpret_cast<const double2*>(s); }
  __device__ __forceinline__ static Val val(double v) { return v; }
  __device__ __forceinline__ void fma(const Row& a, Val v) {
    p[0] = ::fma(a.x, v, p[0]);
    p[1] = ::fma(a.y, v, p[1]);
  }
  __device__ __forceinline__ void get(double (&o)[2]) const { o[0] = p[0]; o[1] = p[1]; }
  __device__ __forceinline__ void set(const double (&o)[2]) { p[0] = o[0]; p[1] = o[1]; }
};

// Order 4: two nodes per thread.  The other orders' bodies own one node per thread;
// their contractions wait for shared memory (9 loads per 18 multiply-adds).  Here
// a thread's nodes are NG apart, so neighbouring threads hold neighbouring nodes
// (coalesced global accesses), and next to each other in the shared D and LIFT
// rows: one vector load brings a row entry for both, a state or flux value is
// read once for both, and f32 arithmetic is packed (f32x2).  48,000 elements:
// 220 -> 172 us per f32 stage (TD = 2: 231 -> 178), 364 -> 311 us per f64 stage
// (10,368 elements: 91 -> 64).  Not at the other orders, where the fluxes are the larger part and
// half the threads form them: order 3 76 -> 75 us (1,296 elements: 9.2 -> 13.0),
// order 2 59 -> 66, order 1 32 -> 43, order 5 193 -> 193 (f64: order 3 18.7 ->
// 21.4 ms, order 5 23.7 -> 23.4, orders 1 and 2 the same).
template <int N, class R, int TD>
struct PairCfg {
  static constexpr bool F32 = sizeof(R) == 4;
  static constexpr int NP = np_of(N), NFP = nfp_of(N), NF = 4 * NFP;
  static constexpr int NPT = 2, NG = (NP + 1) / 2, NPAD = NPT * NG;
  // Elements per tile (TD = 2: half as many); all threads form fluxes, the
  // first E * NG own nodes.
  static constexpr int E = F32 ? 14 / TD : 12;
  static constexpr int OWNERS = E * NG;
  static constexpr int THREADS = OWNERS < 256 / TD ? 256 / TD : (OWNERS + 31) / 32 * 32;
  // element strides (in R) of the state and flux tiles: the elements of a warp in
  // different banks, flux rows whole 16-byte vectors
  static constexpr int YS = 6 * NP + (F32 ? 0 : 2), FS = 6 * NF + 4;
  static constexpr int PER16 = 16 / (int)sizeof(R);
  static constexpr int al4(int x) { return (x + PER16 - 1) / PER16 * PER16; }
  static constexpr int OFF_D = 0;
  static constexpr int OFF_L = al4(OFF_D + 3 * NP * NPAD);
  static constexpr int OFF_Y = al4(OFF_L + NF * NPAD);
  static constexpr int OFF_F = al4(OFF_Y + E * YS);
  static constexpr int OFF_M = al4(OFF_F + E * FS);
  static constexpr int OFF_B = al4(OFF_M + E * kMetaWords);
  static constexpr int BYTES_TAB = 4 * NFP + kMaxGather * NFP;
  static constexpr int SMEM = OFF_B * (int)sizeof(R) + ((BYTES_TAB + 15) / 16) * 16;
  static_assert(FS % PER16 == 0 && NF % PER16 == 0, "flux rows are whole vectors");
  static_assert(YS % 2 == 0 && (6 * NP) % 2 == 0, "the state is copied in pairs");
  static_assert((kMetaWords % PER16) == 0, "element records are whole 16-byte vectors");
};

template <int N, int MODE, class R, int TD = 1>
__device__ __forceinline__ void rhs_cc_pair_body(const RhsParamsT<R>& P, const OpTablesT<R>& T) {
  using C = PairCfg<N, R, TD>;
  using V = typename Vec16<R>::T;
  using A = Acc<R>;
  constexpr int NP = C::NP, NFP = C::NFP, NF = C::NF, E = C::E, NPT = C::NPT, NG = C::NG, NPAD = C::NPAD;
  constexpr int YS = C::YS, FS = C::FS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* smem = reinterpret_cast<R*>(smem_raw);
  R* sD = smem + C::OFF_D;
  R* sL = smem + C::OFF_L;
  R* sY = smem + C::OFF_Y;
  R* sF = smem + C::OFF_F;
  R* sM = smem + C::OFF_M;
  uint8_t* sFn = reinterpret_cast<uint8_t*>(smem + C::OFF_B);
  uint8_t* sG = sFn + 4 * NFP;
  const int tid = threadIdx.x;

  // rows of NPAD: entry NPT g + q is node g + NG q (zero past the last node)
  for (int i = tid; i < (3 * NP + NF) * NPAD; i += blockDim.x) {
    const int row = i / NPAD, x = i - row * NPAD, node = x / NPT + NG * (x % NPT);
    const R* src = row < 3 * NP ? T.dT + row * NP : T.liftT + (row - 3 * NP) * NP;
    (row < 3 * NP ? sD + i : sL + i - 3 * NP * NPAD)[0] = node < NP ? src[node] : R(0);
  }
  for (int i = tid; i < 4 * NFP; i += blockDim.x) sFn[i] = T.fnodes[i];
  for (int i = tid; i < T.n_gather * NFP; i += blockDim.x) sG[i] = T.gtab[i];

  pdl_wait();
  if (P.skip != nullptr && *P.skip) return;  // uniform: nothing to do for this launch
  R kry_sig = 1, kry_g = 0;
  if (MODE == kModeKrylov) {
    kry_sig = (R)P.kry[0];
    kry_g = (R)P.kry[1];
  }

  const int64_t n_tiles = (P.n_elem - P.e_begin + E - 1) / E;
  const int le_me = tid / NG;
  const int g_me = tid - le_me * NG;  // nodes g_me + NG q, q < NPT
  const bool owns = tid < C::OWNERS;

  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t e0 = P.e_begin + tile * E;
    const int ne = (int)((P.n_elem - e0) < E ? (P.n_elem - e0) : E);
    __syncthreads();  // previous tile fully consumed (and tables loaded on the first pass)
    // ---- 1. state tile and element records -> shared memory
    {
      using V2 = typename Vec2<R>::T;
      const V2* src = reinterpret_cast<const V2*>(P.y_in + e0 * 6 * NP);
      for (int i = tid; i < ne * (3 * NP); i += blockDim.x) {
        const int el = i / (3 * NP);
        *reinterpret_cast<V2*>(sY + el * YS + 2 * (i - el * (3 * NP))) = src[i];
      }
    }
    {
      const V* m4 = reinterpret_cast<const V*>(P.meta + e0 * kMetaWords);
      V* d4 = reinterpret_cast<V*>(sM);
      for (int i = tid; i < ne * kMetaWords / C::PER16; i += blockDim.x) d4[i] = __ldg(m4 + i);
    }
    __syncthreads();

    // ---- 2. numerical flux at the 4*Nfp face nodes of each element
    rhs_cc_flux<N, YS, FS>(P, e0, ne, sY, sM, sFn, sG, sF);

    // ---- 3. volume term: reference derivatives of E and H at my nodes
    const bool active = owns && le_me < ne;
    A dd[6];  // dE = curl H, dH = -curl E at the thread's nodes
    if (active) {
      const R* Y = sY + le_me * YS;
      A r[3][6];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < 6; ++c) r[k][c].zero();
#pragma unroll 2
      for (int j = 0; j < NP; ++j) {
        typename A::Row d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = A::row(sD + (k * NP + j) * NPAD + NPT * g_me);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          const auto v = A::val(Y[c * NP + j]);
#pragma unroll
          for (int k = 0; k < 3; ++k) r[k][c].fma(d[k], v);
        }
      }
      // physical derivatives pd[p][c] = sum_k Jinv[k][p] r[k][c] (rhs.rs:62-75),
      // dE = curl H, dH = -curl E (rhs.rs:78-84, :1365-1368)
      const R* M = sM + le_me * kMetaWords;
      R rv[3][6][NPT];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < 6; ++c) r[k][c].get(rv[k][c]);
      const auto pd = [&](int p, int c, int q) {
        return M[0 * 3 + p] * rv[0][c][q] + M[1 * 3 + p] * rv[1][c][q] + M[2 * 3 + p] * rv[2][c][q];
      };
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        const int a = (t + 1) % 3, b = (t + 2) % 3;
        R de[NPT], dh[NPT];
#pragma unroll
        for (int q = 0; q < NPT; ++q) {
          de[q] = pd(a, 3 + b, q) - pd(b, 3 + a, q);
          dh[q] = -(pd(a, b, q) - pd(b, a, q));
        }
        dd[t].set(de);
        dd[3 + t].set(dh);
      }
    }
    __syncthreads();  // flux complete

    // ---- 4. LIFT, materials, epilogue
    if (active) {
      const R* F = sF + le_me * FS;
      constexpr int SV = C::PER16;  // face nodes per vector of a flux row
#pragma unroll 1
      for (int s0 = 0; s0 < NF; s0 += SV) {
        typename A::Row w[SV];
#pragma unroll
        for (int ss = 0; ss < SV; ++ss) w[ss] = A::row(sL + (s0 + ss) * NPAD + NPT * g_me);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          const V fv = *reinterpret_cast<const V*>(F + c * NF + s0);
          const R* f = reinterpret_cast<const R*>(&fv);
#pragma unroll
          for (int ss = 0; ss < SV; ++ss) dd[c].fma(w[ss], A::val(f[ss]));
        }
      }
      const R* M = sM + le_me * kMetaWords;
      const R* Y = sY + le_me * YS;
      R kcl_h = 0, kcl_gs = 0;
      if (MODE == kModeKcl) {
        kcl_h = (R)*P.kcl_h;
        kcl_gs = P.kcl_g != nullptr ? (R)P.kcl_g[*P.kcl_frame] : R(0);
      }
      const int64_t base = (e0 + le_me) * 6 * NP;
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        R dv[NPT];
        dd[c].get(dv);
        const R mw = M[25 + c], ms = M[31 + c];
#pragma unroll
        for (int q = 0; q < NPT; ++q) {
          const int i = g_me + NG * q;
          if (i < NP) {
            const int64_t g = base + c * NP + i;
            const R yv = Y[c * NP + i];
            const R dy = mw * dv[q] - ms * yv;
            if (MODE == kModeApply) {
              P.out[g] = dy;
            } else if (MODE == kModeLserk) {
              R k = dy;
              if (P.src_vec != nullptr) k = fma(P.src_g, P.src_vec[g], k);
              if (g == P.src_idx) k += P.src_g;
              R pv = (P.dt * M[43]) * k;
              if (P.read_p) pv = fma(P.a, P.p[g], pv);
              if (P.write_p) P.p[g] = pv;
              P.out[g] = fma(P.b, pv, yv);
            } else if (MODE == kModeKcl) {
              // KCL stage (explicit_adaptive.rs:84-152), in the operation order of
              // the separate stage kernel (kcl.cuh k_kcl_stage)
              R kk = dy;
              if (P.src_vec != nullptr) kk += P.src_vec[g] * kcl_gs;
              if (g == P.src_idx) kk += kcl_gs;
              const R f = kcl_h * kk;
              const R yn = P.kcl_y[g] + P.kcl_b * f;
              P.kcl_y[g] = yn;
              P.kcl_e[g] = P.kcl_stage == 0 ? P.kcl_ew * f : P.kcl_e[g] + P.kcl_ew * f;
              if (P.kcl_next != nullptr) P.kcl_next[g] = yn + P.kcl_amb * f;
            } else {
              // Krylov matvec of a stored basis vector: its scale and the source
              // coefficient of the augmented system come from device memory
              R w = kry_sig * dy;
              if (P.src_vec != nullptr) w = fma(kry_g, P.src_vec[g], w);
              if (g == P.src_idx) w += kry_g;
              P.out[g] = w;
            }
          }
        }
      }
    }
  }
  // Several of these CTAs share an SM: a next launch let in earlier is placed
  // wherever there is room, unevenly (the f64 kernel: 13 % slower).
  pdl_launch();
}

template <int N, class R, int TD = 1>
using CcCfg = std::conditional_t<N == 4, PairCfg<N, R, TD>, Fp32Cfg<N, R, TD>>;

// Order 4 (three blocks per SM in f32, 80 registers).
template <int N, int MODE, int TD = 1>
__global__ void __launch_bounds__(PairCfg<N, float, TD>::THREADS, 3 * TD)
rhs_fp32_pair_kernel(RhsParams P, OpTables T) {
  rhs_cc_pair_body<N, MODE, float, TD>(P, T);
}
template <int N, int MODE>
__global__ void __launch_bounds__(PairCfg<N, double, 1>::THREADS)
rhs_fp64_pair_kernel(RhsParamsT<double> P, OpTablesT<double> T) {
  rhs_cc_pair_body<N, MODE, double, 1>(P, T);
}

// FP32 engine (stage, RHS and the Krylov matvec of an f32 basis); TD = 2 is
// the same engine with half-size element tiles (DGTD_ENGINE_FP32_SMALL_TILES).
template <int N, int MODE, int TD = 1>
__global__ void __launch_bounds__(Fp32Cfg<N, float, TD>::THREADS) rhs_fp32_kernel(RhsParams P, OpTables T) {
  rhs_cc_body<N, MODE, float, TD>(P, T);
}

// FP64 path: the same algorithm with f64 operators, records and state (and
// the Krylov matvec of an f64 basis).
template <int N, int MODE>
__global__ void __launch_bounds__(Fp32Cfg<N, double>::THREADS)
rhs_fp64_kernel(RhsParamsT<double> P, OpTablesT<double> T) {
  rhs_cc_body<N, MODE, double>(P, T);
}

}  // namespace dgtd
