// What the march kernels share: the launch parameters of a group of fields, the phase mask, the
// mean-index sums and the propagator, each in one place so that every kernel family forms the
// same bits.
#pragma once

#include "common.cuh"
#include "warp_fft.cuh"

namespace bpmgb {

// sin and cos of a step's phase. The kernels evaluate it up to 32 times per thread in unrolled
// loops, where sincosf brings its reduction of huge arguments along each time; with FFTs of 1024
// points that made the code of a pass too long for the instruction cache. Here: Cody and Waite's
// reduction by pi/2 in three parts, then polynomials fitted to sin r / r and cos r on
// |r| <= pi/4 by iterated reweighted least squares (errors 3.6e-9 and 1e-10), 1 - r^2/2 with the
// rounding errors of its terms, since the magnitude of a march's factors must not drift. Beyond
// 30000 (and for infinities and NaN) sincosf, out of line. Measured on 4 M phases per range against
// FP64, cos_sin / sincosf / correctly rounded values: root mean square error 1.68e-8 / 1.92e-8 /
// 1.45e-8 for |x| up to 3 ... 30000 (1.26e-8 for all three up to 0.3), largest error 6.1e-8 / 8.8e-8 /
// 3.0e-8, mean of |c + i s| - 1 -3.0e-10 / 9.0e-9 / below 4e-11 (up to 0.3: 8e-11 / 1.0e-9 / 1e-11).
static __device__ __noinline__ float2 sincos_far(float x) {
  float2 r;
  sincosf(x, &r.y, &r.x);
  return r;
}
__device__ __forceinline__ float2 cos_sin(float x) {  // (cos x, sin x)
  if (!(fabsf(x) <= 30000.f)) return sincos_far(x);
  const float q = rintf(x * 0.63661977236758134f);
  float r = fmaf(-q, 0x1.921fb6p+0f, x);
  r = fmaf(-q, -0x1.777a5cp-25f, r);
  r = fmaf(-q, -0x1.ee59dap-50f, r);
  const float y = r * r;
  const float s = fmaf(fmaf(fmaf(-0.00019516889f, y, 0.008332175f), y, -0.16666655f), y * r, r);
  const float t = fmaf(-.5f, y, 1.f), w = fmaf(-.5f, fmaf(r, r, -y), fmaf(-.5f, y, 1.f - t));
  const float c = t + fmaf(fmaf(fmaf(2.4437992e-05f, y, -0.0013887364f), y, 0.041666646f), y * y, w);
  const int k = (int)q;
  const float sn = (k & 1) ? c : s, cs = (k & 1) ? s : c;
  return make_float2(((k + 1) & 2) ? -cs : cs, (k & 2) ? -sn : sn);
}

struct RowParams {
  const float2* src;        // group's input planes (u0 + b0*plane, or W)
  long long src_bstride;    // float2 elements between fields
  float2* W;                // group workspace planes
  int nx, ny, nz, z;        // z = plane produced by this pass (dn slice index)
  int do_inv, do_fwd, do_mask;
  const void* dn;           // dn of field 0 of the group
  int dn_dtype;
  long long dn_bstride;     // elements
  float unit_k;
  int absorb;
  const float* taper;
  int mean_mode;
  const float* dn0_field;   // weighted: per group field
  const float* slice_dn0;   // simple: per slice
  void* out;                // output of field 0 of the group
  int out_kind;
  long long out_bstride;    // elements
  int zout0;                // output plane index = z - zout0
  float2* last_plane;       // group's exit planes or NULL
  float2* ckpt;             // group's checkpoint planes (G, n_ckpt, ny, nx) or NULL
  int ckpt_every, n_ckpt;
  const float* scat_part;   // [G][ntiles][2]
  int n_ctiles;
  float* scat_p;            // group's (nz) rows
  float* scat_g;
  float prefac_f;
  const float2* tw;
  const float2* wtw;        // stage-ordered twiddles of the warp FFT
  // adjoint passes only
  const float2* seg;        // forward fields of the current segment (G, planes, ny, nx)
  long long seg_bstride;    // float2 elements between fields
  int seg_z0;               // plane index of the segment's first plane
  float* grad_dn;           // group's (nz, ny, nx) dn gradients
  float2* grad_u0;          // group's (ny, nx) u0 gradients or NULL
  const float2* mask;       // precomputed masks of the shared dn, (nz, ny, nx), or NULL
  // adjoint with the dn gradient summed over the fields (row_adj_shared_kernel, grad_sum 1):
  // block 0 of a row writes its fields' sum to grad_dn, block b >= 1 to grad_part + (b - 1) *
  // grad_part_stride, stored (grad_acc 0, the first group of the request) or added (grad_acc
  // 1, the later groups)
  int grad_sum;
  float* grad_part;
  long long grad_part_stride;
  int grad_acc;
  int carve;                // host: shared-memory partition of the march's launches (percent, 0: the driver's choice)
  int early;                // the next pass may start as soon as this one's inputs are there
};

__device__ __forceinline__ float load_dn_real(const void* dn, int dtype, size_t idx) {
  if (dtype == BPM_DN_F16) return __half2float(reinterpret_cast<const __half*>(dn)[idx]);
  return __ldg(reinterpret_cast<const float*>(dn) + idx);
}

// Phase mask of dn slice z at (x, y): M = taper * exp(-i k0 dz dn) for real dn
// (mult_dn*, bpm_3d_kernels.cl:20-81, 198-262), exp(k0 dz Im dn) * exp(-i k0 dz Re dn) with
// no taper for complex dn (mult_dn*_complex, :84-101, :265-283). The mean-index shift dn0
// enters as the separate factor exp(+i k0 dz dn0) (row_rot), so M depends on dn alone and
// can be computed once per dn volume for a whole batch (bpm_mask_precompute); the on-the-fly
// and precomputed masks are the same FP32 arithmetic, bit for bit.
__device__ __forceinline__ float2 mask_from_complex(float2 d, float unit_k) {
  const float m = expf(unit_k * d.y);
  return cscale(cos_sin((-unit_k) * d.x), m);
}

__device__ __forceinline__ float2 mask_from_real(float dnv, float unit_k, int x, int y, int nx, int ny, int absorb,
                                                 const float* taper) {
  float2 M = cos_sin((-unit_k) * dnv);
  const int dist = min(min(nx - 1 - x, x), min(ny - 1 - y, y));
  if (dist < absorb) {
    const float a = taper[dist];
    M.x *= a;
    M.y *= a;
  }
  return M;
}

__device__ __forceinline__ float2 mask_value(const void* dn, int dtype, size_t idx, float unit_k, int x, int y,
                                             int nx, int ny, int absorb, const float* taper) {
  if (dtype == BPM_DN_C64) return mask_from_complex(__ldg(reinterpret_cast<const float2*>(dn) + idx), unit_k);
  return mask_from_real(load_dn_real(dn, dtype, idx), unit_k, x, y, nx, ny, absorb, taper);
}

// PRE = 1: the masks come precomputed (p.mask); PRE = 0: formed on the fly from dn. The
// two are compiled separately so the precomputed kernel carries no sincosf.
template <int PRE>
__device__ __forceinline__ float2 row_mask(const RowParams& p, int x, int y, int gl, size_t zoff, size_t pix) {
  if constexpr (PRE == 1) {
    return p.mask[zoff + pix];
  } else {
    return mask_value(p.dn, p.dn_dtype, gl * p.dn_bstride + zoff + pix, p.unit_k, x, y, p.nx, p.ny, p.absorb,
                      p.taper);
  }
}

// exp(+i k0 dz dn0), the mean-index shift of the mask (identity when dn0 = 0)
__device__ __forceinline__ float2 row_rot(const RowParams& p, float dn0) {
  return cos_sin(p.unit_k * dn0);
}

struct ColParams {
  float2* W;
  int nx, ny, nz, z;         // z = step index: the field goes from plane z to z+1
  int prop_mode;             // 0 = table H, 1 = FP32 recipe with slice_n[z+1], 2 = weighted
  const float2* H;
  const float2* Ht;          // H transposed (nx, ny): a column's entries are contiguous (cluster march)
  const float* kx2;
  const float* ky2;
  float k0f, dzf, n00f;
  const float* slice_n;
  float scale;               // 1/(nx*ny)
  const void* dn;            // weighted: dn of field 0 of the group (slice 0 is used)
  int dn_dtype;
  long long dn_bstride;
  float* red_part;           // weighted sums: [G][nx][2] per column (tile kernels [G][nx/16][2])
  float* dn0_field;          // [G]
  int scat;
  const float* sw;
  const float* gw;
  float* scat_part;          // [G][ntiles][2]
  double plain_phase;        // k0*n0*dz
  int spi;                   // scattering_plane_ind
  int conj_h;                // adjoint: multiply by conj(H)
  const float2* tw;
  const float2* wtw;         // stage-ordered twiddles of the warp FFT
  int dn_stage;              // weighted: dn rows may be staged with 16-byte cp.async
  int col_block;             // 0: the library's rule; 4, 8 or 16 columns per non-weighted block
  int col_fuse;              // weighted: 1 one fused column pass where available, 0 or 2 two passes
  int carve, early;          // as in RowParams
};

template <int T>
__device__ __forceinline__ void block_sum2(float& a, float& b, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  constexpr int NW = (T + 31) / 32;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    red[2 * w] = a;
    red[2 * w + 1] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f, t = 0.f;
    for (int i = 0; i < NW; i++) {
      s += red[2 * i];
      t += red[2 * i + 1];
    }
    a = s;
    b = t;
  }
}

// plain_wave_dct[z+1] = nx*ny*exp(-i k0 n0 (spi + z+1) dz) of bpm_3d.py:253, FP64 then complex64
__device__ __forceinline__ float2 plain_wave(const ColParams& p) {
  double ph = -p.plain_phase * (double)(p.spi + p.z + 1);
  double s, c;
  sincos(ph, &s, &c);
  double m = (double)p.nx * (double)p.ny;
  return make_float2((float)(m * c), (float)(m * s));
}

// n*n*k0*k0 in the FP32 order of the kernels (bpm_3d_kernels.cl:425), no contraction
__device__ __forceinline__ float prop_nk(const ColParams& p, float n_eff) {
  return __fmul_rn(__fmul_rn(__fmul_rn(n_eff, n_eff), p.k0f), p.k0f);
}

// Weighted-mode sums (sum |u| dn, sum |u|). Every kernel of the sequence-in-registers family
// adds them in one order, so all give the same bits: a lane over its rows t, t + 32, ..., the
// lanes of a column by this tree, and the columns by weighted_total.
__device__ __forceinline__ float2 lane_tree2(float2 a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
  }
  return a;
}

// dn0 = sum |u| dn / sum |u| (mult_dn_mean_buff, bpm_3d_kernels.cl:117) from the column sums
// get(c), c < nx: lane t adds columns t, t + 32, ... (fetched U at a time), then the tree;
// called by whole warps
template <int U, class Get>
__device__ __forceinline__ float weighted_total(int nx, int t, Get get) {
  float2 a = make_float2(0.f, 0.f);
  for (int c = t; c < nx; c += 32 * U) {
    float2 v[U];
#pragma unroll
    for (int k = 0; k < U; k++) v[k] = c + 32 * k < nx ? get(c + 32 * k) : make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < U; k++) {
      a.x += v[k].x;
      a.y += v[k].y;
    }
  }
  a = lane_tree2(a);
  return a.x / a.y;
}

// the propagator on the thread's rows r0 + L i of column x (prop_point's arithmetic): the
// row-major table H (conj(H) for the adjoint; TABLE) or the FP32 recipe with kx^2 of the
// column and the ky^2 table staged in shared memory; with scattering sums
// (bpm_3d.py:335-341) the thread's partials S, G over its rows
template <int N, bool TABLE, bool SCAT, int L>
__device__ __forceinline__ void propagate_rows_t(const ColParams& p, float2 (&v)[N / L], int x, int r0,
                                                 float n_eff, float kx2, const float* sky2, float& S, float& G) {
  const unsigned step = (unsigned)L * (unsigned)p.nx;
  const unsigned off = (unsigned)r0 * (unsigned)p.nx + (unsigned)x;
  const bool cj = p.conj_h;
  const float nkx = TABLE ? 0.f : __fsub_rn(prop_nk(p, n_eff), kx2);
  auto hval = [&](int i) {
    float2 h;
    if constexpr (TABLE) {
      h = __ldg(p.H + off + i * step);
      if (cj) h.y = -h.y;
    } else {
      const float tmp = __fsub_rn(nkx, sky2[r0 + L * i]);
      h = tmp >= 0.f ? cos_sin(__fmul_rn(-p.dzf, __fsqrt_rn(tmp))) : make_float2(0.f, 0.f);
    }
    return h;
  };
  if constexpr (!SCAT) {
#pragma unroll
    for (int i = 0; i < N / L; i++) v[i] = cscale(cmul(v[i], hval(i)), p.scale);
    return;
  }
  const float2 plain = (x == 0 && r0 == 0) ? plain_wave(p) : make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < N / L; i++) {
    const float2 u = cmul(v[i], hval(i));
    float2 d = u;
    if (x == 0 && r0 == 0 && i == 0) d = csub(d, plain);
    const float a2 = cabs2(d);
    S = fmaf(__ldg(p.sw + off + i * step), a2, S);
    G = fmaf(__ldg(p.gw + off + i * step), a2, G);
    v[i] = cscale(u, p.scale);
  }
}
template <int N, bool SCAT, int L>
__device__ __forceinline__ void propagate_rows(const ColParams& p, float2 (&v)[N / L], int x, int r0,
                                               float n_eff, float kx2, const float* sky2, float& S, float& G) {
  if (p.prop_mode == 0)
    propagate_rows_t<N, true, SCAT, L>(p, v, x, r0, n_eff, kx2, sky2, S, G);
  else
    propagate_rows_t<N, false, SCAT, L>(p, v, x, r0, n_eff, kx2, sky2, S, G);
}

// every wait of a march kernel on other blocks gives up after 2 s
constexpr unsigned long long kMarchWaitNs = 2000000000ull;

// records that one did: the sticky device status, and the count of them in the host's word
__device__ __forceinline__ void march_gave_up(int* status, int* count, int* host_word) {
  atomicExch(status, 1);
  const int n = atomicAdd(count, 1) + 1;
  if (host_word) asm volatile("st.relaxed.sys.global.s32 [%0], %1;" ::"l"(host_word), "r"(n) : "memory");
}

}  // namespace bpmgb
