// Whole march of one or a few fields in one cooperative launch (128 <= nx, ny <= 1024).
//
// The row and column passes of a single field leave most of the device idle and pay a kernel
// boundary each, three per step in the weighted mode, whose two column passes also store the
// transformed plane and read it back around the plane-wide sums. Here a team of NB = NX / C
// blocks marches a field through all nz planes: block b owns columns [C b, C b + C) in the
// column phases and R = NY / NB rows in the row phases, the field moves between the phases
// through its workspace plane (L2), and the team meets at a counter after each phase and, in
// the weighted mode, between the forward column transform and the propagator, with the
// transformed tile kept in registers. Constants of the march (twiddles, the block's propagator
// entries or ky^2 and dn slice 0) stay in shared memory; the next plane's masks are fetched and
// the finished plane is written while the team gathers.
//
// The blocks of a grid wait on one another, so it is launched cooperatively (every block
// resident at once) and every wait is bounded in time: a block that gives up one records it for
// bpm_device_status and marches on without waiting, to a wrong result. FFTs, masks, propagator and weighted sums
// are those of the pass kernels, so the fields are the same bits; the scattering sums are added
// per block of C columns, not of 16, and agree to FP32 rounding.
#include <algorithm>
#include <string>

#include "march.cuh"
#include "march_grid.cuh"
#include "tcgen05.cuh"

using namespace bpmgb;

namespace {

__device__ int g_grid_status;    // nonzero once a wait gave up (bpm_device_status)
__device__ int g_grid_timeouts;  // waits that gave up so far (bpm_march_timeouts)

template <int NX, int NY>
struct GridCfg {
  // columns per block: 128 blocks a field (64 at 128 columns, where one-column tiles would read
  // 8 bytes of every 32-byte sector)
  static constexpr int C = NX <= 256 ? 2 : NX / 128;
  static constexpr int NB = NX / C;             // blocks per field
  static constexpr int R = NY / NB;             // rows per block
  static constexpr int W = C > R ? C : R;       // warps
  static constexpr int T = 32 * W;
  static constexpr int TWX = (WarpFft<NX>::TW + 1) & ~1, TWY = (WarpFft<NY>::TW + 1) & ~1;
  // column buffers an offset apart that spreads a half-warp's C columns x 16 / C rows over the
  // banks (16 / C mod 16 float2)
  static constexpr int STRIDE = WarpFft<NY>::BUF + 16 / C;
  static constexpr int FFT_F2 = (std::max(C * STRIDE, R * WarpFft<NX>::BUF) + 1) & ~1;
  static constexpr int RED_F2 = C * 33;         // weighted sums, in the FFT buffers
  static constexpr int CONST_F2 = NY * C;       // H tile, or ky^2 (NY floats) and dn slice 0 (NY x C floats)
  static constexpr int MASK_F2 = R * NX;
  static constexpr size_t SMEM = (size_t)(TWX + TWY + FFT_F2 + CONST_F2 + MASK_F2) * sizeof(float2);
  static_assert(R >= 1 && RED_F2 <= FFT_F2 && SMEM <= 226 * 1024, "grid march shape");
};

template <int NX, int NY>
__global__ void __launch_bounds__(GridCfg<NX, NY>::T) grid_march_kernel(GridMarchArgs a) {
  using Cfg = GridCfg<NX, NY>;
  constexpr int C = Cfg::C, NB = Cfg::NB, R = Cfg::R, T = Cfg::T;
  constexpr int EX = NX / 32, EY = NY / 32;
  const RowParams& p = a.rp;
  const ColParams& q = a.cp;
  extern __shared__ __align__(16) float2 gsm[];
  float2* twx = gsm;
  float2* twy = twx + Cfg::TWX;
  float2* fft = twy + Cfg::TWY;
  float2* cst = fft + Cfg::FFT_F2;
  float2* msk = cst + Cfg::CONST_F2;
  __shared__ float s_dn0;
  __shared__ float2 s_plain;
  __shared__ float red[64];
  const int tid = threadIdx.x, warp = tid >> 5, t = tid & 31;
  const int gl = blockIdx.x / NB, b = blockIdx.x % NB;
  const int r0 = tid / C, cc = tid % C, x0 = b * C, col = x0 + cc;
  const bool in_col = warp < C, in_row = warp < R;
  const int y = b * R + warp;  // the warp's row
  const size_t plane = (size_t)NX * NY;
  float2* Wp = p.W + gl * plane;
  float2* colbuf = fft + cc * Cfg::STRIDE;
  float2* colmid = fft + warp * Cfg::STRIDE;
  float2* rowbuf = fft + warp * WarpFft<NX>::BUF;
  float2* mrow = msk + (size_t)warp * NX;
  float2* colsums = reinterpret_cast<float2*>(q.red_part) + (size_t)gl * NX;
  const bool table = q.prop_mode == 0, weighted = q.prop_mode == 2;
  const float* sky2 = reinterpret_cast<const float*>(cst);
  const float* sdn = sky2 + NY;
  const int nz = a.nz;
  unsigned* counter = a.counter + gl * kGridCounterStride;
  // The blocks' partial scattering sums of plane z, two copies by the parity of z: block 0 adds
  // plane z's behind the gathering of its row phase, when the other blocks may already be storing
  // those of plane z + 1. They store plane z + 2's only after block 0 has arrived once more.
  auto scat_part = [&](int z) { return q.scat_part + ((size_t)(2 * gl + (z & 1)) * NB) * 2; };
  unsigned target = a.starve;
  bool dead = false;

  auto arrive = [&] {
    __syncthreads();
    if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    target += NB;
  };
  auto gather = [&] {
    if (tid == 0 && !dead) {
      const uint64_t t0 = tc::global_ns();
      for (unsigned n = 1;; n++) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
        if ((int)(v - target) >= 0) break;
        if (n % 64 == 0 && tc::global_ns() - t0 > a.wait_ns) {
          dead = true;
          march_gave_up(&g_grid_status, &g_grid_timeouts, a.timeouts);
          break;
        }
      }
    }
    __syncthreads();
  };
  // the warp's row of plane z's masks (or of dn) into shared memory, each lane the elements it
  // will use, asynchronously (half values by ordinary loads)
  auto stage_mask = [&](int z) {
    if (!in_row || !p.do_mask || z >= nz) return;
    const size_t off = (size_t)z * plane + (size_t)y * NX + t;
    if (p.mask || p.dn_dtype == BPM_DN_C64) {
      const float2* src = p.mask ? p.mask + off : reinterpret_cast<const float2*>(p.dn) + gl * p.dn_bstride + off;
#pragma unroll
      for (int m = 0; m < EX; m++) cp_async8(mrow + t + 32 * m, src + 32 * m);
    } else if (p.dn_dtype == BPM_DN_F32) {
      const float* src = reinterpret_cast<const float*>(p.dn) + gl * p.dn_bstride + off;
#pragma unroll
      for (int m = 0; m < EX; m++) cp_async4(mrow + t + 32 * m, src + 32 * m);
    } else {
      const __half* src = reinterpret_cast<const __half*>(p.dn) + gl * p.dn_bstride + off;
#pragma unroll
      for (int m = 0; m < EX; m++) mrow[t + 32 * m].x = __half2float(src[32 * m]);
    }
    cp_async_commit();
  };
  // the masks of the staged dn row in its place
  auto form_mask = [&] {
    if (!in_row || !p.do_mask || p.mask) return;
    cp_async_wait<0>();
#pragma unroll 4
    for (int m = 0; m < EX; m++) {
      float2& e = mrow[t + 32 * m];
      e = p.dn_dtype == BPM_DN_C64 ? mask_from_complex(e, p.unit_k)
                                   : mask_from_real(e.x, p.unit_k, t + 32 * m, y, NX, NY, p.absorb, p.taper);
    }
  };
  auto store_plane = [&](int z, const float2 (&u)[EX]) {
    const size_t pix = (size_t)y * NX + t, o = (size_t)z * plane + pix;
    if (p.out_kind == BPM_OUT_FIELD) {
      float2* out = reinterpret_cast<float2*>(p.out) + gl * p.out_bstride + o;
#pragma unroll
      for (int m = 0; m < EX; m++) __stcs(out + 32 * m, u[m]);
    } else if (p.out_kind == BPM_OUT_INTENSITY) {
      float* out = reinterpret_cast<float*>(p.out) + gl * p.out_bstride + o;
#pragma unroll
      for (int m = 0; m < EX; m++) __stcs(out + 32 * m, cabs2(u[m]));
    }
    if (z == nz - 1 && p.last_plane) {
      float2* last = p.last_plane + gl * plane + pix;
#pragma unroll
      for (int m = 0; m < EX; m++) last[32 * m] = u[m];
    }
  };
  // plain_wave of the step that produces plane z, by a thread of block 0 that waits otherwise
  auto plain_next = [&](int z) {
    if (!q.scat || b != 0 || tid != T - 1 || z >= nz) return;
    ColParams w = q;
    w.z = z - 1;
    s_plain = plain_wave(w);
  };

  for (int k = tid; k < WarpFft<NX>::TW; k += T) twx[k] = p.wtw[k];
  for (int k = tid; k < WarpFft<NY>::TW; k += T) twy[k] = q.wtw[k];
  if (table) {
    for (int k = tid; k < NY * C; k += T) cst[k] = q.H[(size_t)(k / C) * NX + x0 + k % C];
  } else {
    float* f = reinterpret_cast<float*>(cst);
    for (int k = tid; k < NY; k += T) f[k] = q.ky2[k];
    if (weighted)
      for (int k = tid; k < NY * C; k += T)
        f[NY + k] = q.dn ? load_dn_real(q.dn, q.dn_dtype, gl * q.dn_bstride + (size_t)(k / C) * NX + x0 + k % C) : 0.f;
  }
  const float kx2 = __ldg(q.kx2 + col % NX);
  __syncthreads();

  float dn0 = 0.f;
  for (int z = 0; z < nz; z++) {
    // ---- row phase: [inverse FFT, mask], forward FFT. Both transforms of the phase run one copy
    // of the code (an inverse one between two conjugations, which change no bit of it), as do
    // the column phase's: unrolled twice, a step of 1024-point transforms stalled on
    // instruction fetches more than on anything else ----
    float2 u[EX], v[EX];
    if (z > 0) gather();
    if (in_row) {
      const float2* src = (z > 0 ? Wp : a.u0 + gl * plane) + (size_t)y * NX + t;
#pragma unroll
      for (int m = 0; m < EX; m++) {
        v[m] = __ldcg(src + 32 * m);
        if (z > 0) v[m].y = -v[m].y;
      }
      const float2 rot = row_rot(p, dn0);
#pragma unroll 1
      for (int pass = z == 0; pass < 2; pass++) {
        if (pass == 1) {
#pragma unroll
          for (int m = 0; m < EX; m++) u[m] = v[m];
          if (z + 1 == nz) break;
        }
        warp_fft<NX, false>(v, rowbuf, twx, t);
        if (pass == 0) {
          cp_async_wait<0>();
#pragma unroll
          for (int m = 0; m < EX; m++) {
            v[m].y = -v[m].y;
            if (p.do_mask) {
              v[m] = cmul(v[m], mrow[t + 32 * m]);
              if (dn0 != 0.f) v[m] = cmul(v[m], rot);
            }
          }
        }
      }
      if (z + 1 < nz) {
#pragma unroll
        for (int m = 0; m < EX; m++) Wp[(size_t)y * NX + t + 32 * m] = v[m];
      }
    }
    if (z + 1 < nz) arrive();
    // behind the team's gathering: the plane's output, the scattering sums, the next masks
    if (in_row) store_plane(z, u);
    if (p.scat_p && b == 0 && warp == 0) {
      float2 s = make_float2(0.f, 0.f);
      if (z > 0) {
        const float2* part = reinterpret_cast<const float2*>(scat_part(z));
        for (int k = t; k < NB; k += 32) {
          const float2 w = __ldcg(part + k);
          s.x += w.x;
          s.y += w.y;
        }
        s = lane_tree2(s);
      }
      if (t == 0) {
        const float pv = p.prefac_f * s.x;
        p.scat_p[(size_t)gl * p.nz + z] = pv;
        if (p.scat_g) p.scat_g[(size_t)gl * p.nz + z] = __fdiv_rn(p.prefac_f * s.y, pv);
      }
    }
    if (z + 1 == nz) break;
    stage_mask(z + 1);
    plain_next(z + 1);

    // ---- column phase, plane z to plane z + 1: forward FFT, propagator, inverse FFT ----
    gather();
    float2 k[EY];
    if (in_col) {
      const float2* src = Wp + (size_t)r0 * NX + col;
#pragma unroll
      for (int i = 0; i < EY; i++) k[i] = __ldcg(src + (size_t)(32 * i) * NX);
    }
    float n_eff = q.prop_mode == 1 ? q.slice_n[z + 1] : q.n00f;
    dn0 = (p.mean_mode == BPM_MEAN_SIMPLE && p.slice_dn0) ? p.slice_dn0[z + 1] : 0.f;
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
      if (in_col) colsplit_first<NY, false>(k, colbuf, r0);
      __syncthreads();
      if (in_col) colsplit_middle<NY, false>(colmid, twy, t);
      __syncthreads();
      if (in_col) colsplit_last<NY, false>(k, colbuf, twy, r0);
      if (pass == 1) break;
      __syncthreads();  // the column buffers are free
      if (weighted) {
        if (in_col) {
          float sd = 0.f, su = 0.f;
#pragma unroll
          for (int i = 0; i < EY; i++) {
            const float aa = __fsqrt_rn(cabs2(k[i]));
            su += aa;
            sd = fmaf(aa, sdn[(r0 + 32 * i) * C + cc], sd);
          }
          fft[cc * 33 + r0] = make_float2(sd, su);
        }
        __syncthreads();
        if (in_col) {
          const float2 cs = lane_tree2(fft[warp * 33 + t]);
          if (t == 0) colsums[x0 + warp] = cs;
        }
        arrive();
        gather();
        if (warp == 0) {
          const float d =
              weighted_total<(NX / 32 < 16 ? NX / 32 : 16)>(NX, t, [&](int c) { return __ldcg(colsums + c); });
          if (t == 0) s_dn0 = d;
        }
        __syncthreads();
        dn0 = s_dn0;
        n_eff = q.n00f + dn0;  // mult_propagator_buff, bpm_3d_kernels.cl:482
      }
      if (in_col) {
        const float nkx = table ? 0.f : __fsub_rn(prop_nk(q, n_eff), kx2);
        float S = 0.f, G = 0.f;
#pragma unroll
        for (int i = 0; i < EY; i++) {
          const int r = r0 + 32 * i;
          float2 h;
          if (table) {
            h = cst[r * C + cc];
          } else {
            const float tmp = __fsub_rn(nkx, sky2[r]);
            h = tmp >= 0.f ? cos_sin(__fmul_rn(-q.dzf, __fsqrt_rn(tmp))) : make_float2(0.f, 0.f);
          }
          const float2 w = cmul(k[i], h);
          if (q.scat) {
            float2 d = w;
            if (col == 0 && r == 0) d = csub(d, s_plain);
            const float a2 = cabs2(d);
            const size_t o = (size_t)r * NX + col;
            S = fmaf(__ldg(q.sw + o), a2, S);
            G = fmaf(__ldg(q.gw + o), a2, G);
          }
          k[i] = make_float2(w.x * q.scale, -(w.y * q.scale));  // conjugated for the inverse
        }
        if (q.scat) {
          const float2 s = lane_tree2(make_float2(S, G));
          if (t == 0) red[2 * warp] = s.x, red[2 * warp + 1] = s.y;
        }
      }
    }
    if (in_col) {
      float2* dst = Wp + (size_t)r0 * NX + col;
#pragma unroll
      for (int i = 0; i < EY; i++) dst[(size_t)(32 * i) * NX] = make_float2(k[i].x, -k[i].y);
    }
    if (q.scat && tid == 0) {  // red: written before the second transform's barriers
      float S = 0.f, G = 0.f;
      for (int w = 0; w < C; w++) S += red[2 * w], G += red[2 * w + 1];
      float* o = scat_part(z + 1) + 2 * b;
      o[0] = S;
      o[1] = G;
    }
    arrive();
    form_mask();
  }
  cp_async_wait<0>();
}

template <int NX, int NY>
struct GridK {
  using Cfg = GridCfg<NX, NY>;
  // fields whose teams are resident at once (0: the kernel does not fit this device)
  static int capacity() {
    static PerDevice st;
    return st.get([] {
      int dev = 0, nsm = 0, coop = 0, occ = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
      if (!coop || cudaFuncSetAttribute(grid_march_kernel<NX, NY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)Cfg::SMEM) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, grid_march_kernel<NX, NY>, Cfg::T, Cfg::SMEM) !=
              cudaSuccess)
        occ = 0;
      cudaGetLastError();
      return occ * nsm / Cfg::NB;
    });
  }
  static int launch(const GridMarchArgs& a, int nfields, cudaStream_t s) {
    BPM_CUDA_TRY(cudaMemsetAsync(a.counter, 0, (size_t)nfields * kGridCounterStride * sizeof(unsigned), s));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nfields * Cfg::NB);
    cfg.blockDim = dim3(Cfg::T);
    cfg.dynamicSmemBytes = Cfg::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    BPM_CUDA_TRY(cudaLaunchKernelEx(&cfg, grid_march_kernel<NX, NY>, a));
    BPM_LAUNCH_CHECK("grid_march_kernel");
    return BPM_OK;
  }
};

#define GRID_CASES(X) \
  X(128, 128) X(128, 256) X(128, 512) X(128, 1024) X(256, 128) X(256, 256) X(256, 512) X(256, 1024) \
  X(512, 128) X(512, 256) X(512, 512) X(512, 1024) X(1024, 128) X(1024, 256) X(1024, 512) X(1024, 1024)

}  // namespace

int bpmgb::grid_march_capacity(int nx, int ny) {
#define CASE(NX, NY) \
  if (nx == NX && ny == NY) return GridK<NX, NY>::capacity();
  GRID_CASES(CASE)
#undef CASE
  return 0;
}

int bpmgb::grid_march_launch(int nx, int ny, const GridMarchArgs& a, int nfields, cudaStream_t s) {
#define CASE(NX, NY) \
  if (nx == NX && ny == NY) return GridK<NX, NY>::launch(a, nfields, s);
  GRID_CASES(CASE)
#undef CASE
  set_error("grid march: no kernel for this size");
  return BPM_ERR_SHAPE;
}

int bpmgb::grid_march_status(int clear, int* v) {
  BPM_CUDA_TRY(cudaMemcpyFromSymbol(v, g_grid_status, sizeof(int)));
  if (clear && *v) {
    const int zero = 0;
    BPM_CUDA_TRY(cudaMemcpyToSymbol(g_grid_status, &zero, sizeof(int)));
  }
  return BPM_OK;
}
