// Mixture-property kernels around the substep (sm_100a): finitechem_W + finitechem_density
// (combustion/finitechem.f90:65-74, :324-345), finitechem_viscosity (:351-406) and
// finitechem_diffusivity (:412-461) with finitechem_omegamu (:467-487).
//
// One cell per lane over the cells of a species-major array (species k of cell c at
// y[k*ldy + c]; the reference's SC(i,j,k,isc_sc+k-1) block with the padded volume as ld), so
// every load and store of a warp is one contiguous segment. The per-cell arithmetic is the
// mechanism's generated code (Mech::mix_w, Mech::transport). Wilke's sum over the pairs of species
// is a product of one constant matrix with three vectors per cell and runs on the FP64 tensor
// cores, 8 cells at a time; its operands u and rho wait in shared memory (16 NS bytes per cell,
// which sets 12 warps per SM for 36 species). Both parts share the FP64 pipe: 8,640 of its cycles per
// warp in the product (16 per m8n8k4 product), about half as many in the species' fits. GRI, 1,064,895
// cells, viscosity and diffusivities: 0.998 ms with three scalar FMAs per pair and matrix entry (8
// warps per SM) -> 0.818 ms -> 0.77 ms with the fits' divisions folded into one rsqrt (and one Newton step
// for eta) and the product's steps unrolled; viscosity alone 0.717 -> 0.595 ms (12.0 TFLOP/s counted, 33 %
// of the pipe).
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace tng {

constexpr int kPropsBlock = 64;

// rows of a warp's shared arrays: the species, padded to the matrix product's steps of four
template <class Mech>
constexpr int props_rows() { return (Mech::NS + 3) / 4 * 4; }

// shared memory of a transport block: per lane u and rho of every species with the viscosity, the
// staged mass fractions for the diffusivities alone
template <class Mech>
constexpr int props_smem(int what) {
  return ((what & TNG_PROPS_VISC) ? 2 : 1) * props_rows<Mech>() * kPropsBlock * (int)sizeof(double);
}

// D += A B on the FP64 tensor cores: A 8 x 4 (lane l: row l/4, column l%4), B 4 x 8 (row l%4,
// column l/4), D 8 x 8 (row l/4, columns 2 (l%4) and the next)
__device__ __forceinline__ void dmma(double (&d)[2], const double a, const double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// Wilke's viscosity of the warp's 32 cells from u and rho in shared memory (Mech::transport's
// layout): eight cells per pass, NS/8 row tiles x {A.u, A.(u rho), A.(u rho^2)} accumulated over the
// species; a fragment of u and rho feeds 3 NS/8 products, u rho and u rho^2 being formed in registers.
// Stored for the lanes set in `live`.
template <class Mech, int LM>
__device__ __forceinline__ void wilke_visc(const double* su, const double* sr, double* visc, const unsigned live,
                                           const int lane) {
  constexpr int NS = Mech::NS, RT = (NS + 7) / 8, KS = (NS + 3) / 4;
  const int r = lane >> 2, q = lane & 3;
  const double* A = Mech::template wilke<LM>() + 8 * q + r;
#pragma unroll 1
  for (int c0 = 0; c0 < 32; c0 += 8) {
    double d[RT][3][2];
#pragma unroll
    for (int t = 0; t < RT; ++t)
#pragma unroll
      for (int i = 0; i < 3; ++i) d[t][i][0] = d[t][i][1] = 0.0;
    const int at = 32 * q + ((c0 + r + 4 * q) & 31);  // species q of cell c0 + r; later steps 128 apart
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      const double u = su[at + 128 * k], rho = sr[at + 128 * k];
      const double v = u * rho, w = v * rho;
#pragma unroll
      for (int t = 0; t < RT; ++t) {
        const double m = (4 * k + 3 < NS || 4 * k + q < NS) ? __ldg(A + (t * NS + 4 * k) * 8) : 0.0;
        dmma(d[t][0], m, u);
        dmma(d[t][1], m, v);
        dmma(d[t][2], m, w);
      }
    }
    double s[2] = {0.0, 0.0};
#pragma unroll
    for (int t = 0; t < RT; ++t) {
      const int k = 8 * t + r;
      if (k < NS) {
        const double q2 = Mech::template wilke_q2<LM>(k);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int p = 32 * k + ((c0 + 2 * q + e + 4 * (k & 3)) & 31);
          const double u = su[p], rho = sr[p];
          // u eta / sum_1 with eta = q^2 / rho^2 (rows with u <= 0 add nothing)
          if (u > 0.0) s[e] += u * q2 / fma(rho * rho, u + d[t][0][e], fma(2.0 * rho, d[t][1][e], d[t][2][e]));
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
      const int c = c0 + 2 * q + e;
      if (r == 0 && (live >> c & 1)) __stcs(visc + c, s[e]);
    }
  }
}

// Viscosity and / or diffusivities (WHAT = TNG_PROPS_VISC / TNG_PROPS_DIFF bits).
template <class Mech, int LM, int WHAT>
__global__ void __launch_bounds__(kPropsBlock) k_props(PropsArgs a) {
  constexpr bool VISC = (WHAT & TNG_PROPS_VISC) != 0, DIFF = (WHAT & TNG_PROPS_DIFF) != 0;
  constexpr int NS = Mech::NS, KP = props_rows<Mech>();
  extern __shared__ double props_sv[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* su = props_sv + warp * (VISC ? 2 : 1) * KP * 32;
  double* sr = su + KP * 32;
  if constexpr (VISC) {
    for (int k = NS; k < KP; ++k) su[32 * k + lane] = 0.0, sr[32 * k + lane] = 0.0;
  }
  const long long stride = (long long)gridDim.x * kPropsBlock;
  for (long long base = (long long)blockIdx.x * kPropsBlock + 32 * warp; base < a.n; base += stride) {
    const long long c = base + lane;
    bool live = c < a.n;
    if (live && a.mask) {
      const long long i = c % a.nxo;
      const long long j = (c / a.nxo) % a.nyo;
      live = __ldg(a.mask + i + (long long)a.nxo * j) != 1;
    }
    const unsigned all = __ballot_sync(0xffffffffu, live);
    if (!all) continue;  // every cell masked (a wall): no work for the warp
    const double T = live ? __ldcs(a.T + c) : 300.0;
    double lc = 0.0;
    Mech::template transport<LM, VISC, DIFF>(a.y + c, a.ldy, live, T, su, sr, lane, &lc);
    if constexpr (VISC) {
      __syncwarp();  // every lane's u and rho are stored
      wilke_visc<Mech, LM>(su, sr, a.visc + base, all, lane);
      __syncwarp();  // u and rho are no longer read
    }
    if constexpr (DIFF) {
      if (!live) continue;
      // DIFF(species k) = (lambda/Cp_mix)/Lewis_k, DIFF(T) = DIFF(ZMIX) = lambda/Cp_mix (:444-451)
#pragma unroll 4
      for (int k = 0; k < NS; ++k) __stcs(a.diff + k * a.ldd + c, lc * __ldg(a.inv_lewis + k));
      __stcs(a.diff_T + c, lc);
      if (a.diff_Z) __stcs(a.diff_Z + c, lc);
    }
  }
}

// Density and W_mix: a streaming kernel (N+1 loads, two stores per cell).
constexpr int kDensityBlock = 256;
template <class Mech, int LM>
__global__ void __launch_bounds__(kDensityBlock) k_density(PropsArgs a) {
  const long long stride = (long long)gridDim.x * kDensityBlock;
  for (long long c = (long long)blockIdx.x * kDensityBlock + threadIdx.x; c < a.n; c += stride) {
    if (a.mask) {
      const long long i = c % a.nxo;
      const long long j = (c / a.nxo) % a.nyo;
      if (__ldg(a.mask + i + (long long)a.nxo * j) == 1) continue;
    }
    const double wm = Mech::template mix_w<LM>(a.y + c, a.ldy);
    // RHO = P_thermo * W_mix / (R_cst * T), R_cst = 8314.34 (finitechem.f90:15, :338)
    if (a.rho) __stcs(a.rho + c, a.p * wm / (8314.34 * __ldcs(a.T + c)));
    if (a.wmix) __stcs(a.wmix + c, wm);
  }
}

// Resident blocks per SM of a kernel, set up once per device (the shared-memory opt-in is a
// per-device attribute); grid = min(blocks needed, SMs x resident blocks) for the grid-stride loop.
template <class K>
cudaError_t launch_grid_stride(K kern, int block, int smem, const PropsArgs& a, int sm_count, cudaStream_t st,
                               int* occ_dev) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  int& occ = occ_dev[dev];
  if (occ == 0) {
    if (smem > 48 * 1024 && (e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) !=
                                cudaSuccess)
      return e;
    int o = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, block, smem);
    if (e != cudaSuccess) return e;
    occ = o < 1 ? 1 : o;
  }
  long long blocks = (a.n + block - 1) / block;
  const long long cap = (long long)sm_count * occ;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  kern<<<(unsigned)blocks, block, smem, st>>>(a);
  return cudaGetLastError();
}

template <class Mech, int LM, int WHAT>
cudaError_t launch_props_w(const PropsArgs& a, int sm_count, cudaStream_t st) {
  static int occ_dev[64] = {};
  if constexpr (WHAT == TNG_PROPS_DENSITY)
    return launch_grid_stride(k_density<Mech, LM>, kDensityBlock, 0, a, sm_count, st, occ_dev);
  else
    return launch_grid_stride(k_props<Mech, LM, WHAT>, kPropsBlock, props_smem<Mech>(WHAT), a, sm_count, st, occ_dev);
}

template <class Mech>
cudaError_t launch_props(int lm, int what, const PropsArgs& a, int sm_count, cudaStream_t st) {
#define TNG_PROPS_CASE(W)                                                                     \
  case W:                                                                                     \
    return lm ? launch_props_w<Mech, 1, W>(a, sm_count, st) : launch_props_w<Mech, 0, W>(a, sm_count, st);
  switch (what) {
    TNG_PROPS_CASE(TNG_PROPS_DENSITY)
    TNG_PROPS_CASE(TNG_PROPS_VISC)
    TNG_PROPS_CASE(TNG_PROPS_DIFF)
    TNG_PROPS_CASE(TNG_PROPS_VISC | TNG_PROPS_DIFF)
    default:
      return cudaErrorInvalidValue;
  }
#undef TNG_PROPS_CASE
}

}  // namespace tng
