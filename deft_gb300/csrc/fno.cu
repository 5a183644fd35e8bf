// Learned warm start: a 3-D Fourier neural operator (FNO) that maps the
// constraint mask of a problem (hard walls / solutes) and its bulk packing
// fraction to an initial density, trained on converged solutions.
//
// Network (C channels, L Fourier layers, m retained modes per axis):
//   h0 = P [mask, eta] + p                                  (lift, 2 -> C)
//   h_{l+1} = act(K_l h_l + Wp_l h_l + b_l)                  (l < L; no act on the last)
//   K_l h = Finv( W_l . F(h) )                               (spectral convolution)
//   y = Q2 . gelu(Q1 h_L + q1) + q2                          (projection, C -> C -> 1)
// The density estimate is n = nb * y on free points (0 in the walls).
// F keeps kx, ky in {0..m-1} U {N-m..N-1} and kz in {0..m-1}; it and its
// inverse are truncated DFTs done as three small dense contractions (z, then
// y, then x), which on 24 x 24 x 12 retained modes costs far less than a
// full multi-channel FFT.  Finv(U)(r) = N^-3 sum_kz c_kz Re[sum U e^{+i k.r}]
// with c_0 = 1, c_kz = 2 (the real synthesis from a half spectrum).
//
// Weights: FP32 master copies updated by Adam; every forward and backward
// pass reads BF16 copies (round-to-nearest-even of the masters) and
// accumulates in FP32.
#include "../../include/deft_gb300.h"
#include "dev_mem.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

namespace deft {
void set_last_error_message(const std::string &m);
void fmt_shape(const deft_fmt *f, int N[3]);
}

namespace {

constexpr int kT = 256;

__device__ __forceinline__ float gelu(float x) {
  return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_d(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) +
         x * expf(-0.5f * x * x) * 0.39894228040143268f;
}

__device__ __forceinline__ float bf(const __nv_bfloat16 *w, size_t i) {
  return __bfloat162float(w[i]);
}

// ---------------------------------------------------------------------------
// Truncated DFT along z (contiguous lines of length N), as two small dense
// contractions per block in registers.
// fwd: out[l][k] = s_k sum_z in[l][z] e^{-2 pi i k z / N}   (k < Kz <= kMaxKz)
// with E[z*Kz + k] = s_k (cos, -sin) precomputed.  A block of 128 threads
// stages 128 lines (16-byte loads, eight in flight per thread) with row
// stride N + 4 floats (16-byte rows; the eight rows one load instruction
// touches fall in distinct banks).  Lane (lg = lane / 4,
// mg = lane % 4) of warp w accumulates lines 32 w + lg + 8 r (r < 4) and
// modes mg + 4 j (j < KB / 4): per z, four row values and KB / 4 table
// entries feed 2 KB multiply-adds.  KB is Kz rounded up to a multiple of 4.
constexpr int kMaxKz = 16;
constexpr int kZfLines = 128;

template <int KB>
__global__ void __launch_bounds__(128) k_dft_z_fwd(const float *__restrict__ in,
                                                   float2 *__restrict__ out,
                                                   const float2 *__restrict__ E, int L, int N,
                                                   int Kz) {
  constexpr int J = KB / 4;
  extern __shared__ __align__(16) float sm[];
  const int S = N + 4;
  float *tile = sm;                                                   // [128][N+4]
  float2 *Es = reinterpret_cast<float2 *>(tile + kZfLines * S);      // [N][Kz]
  const int l0 = blockIdx.x * kZfLines;
  for (int i = threadIdx.x; i < N * Kz; i += blockDim.x) Es[i] = E[i];
  // N is a multiple of 4 (the network's grids are): float4 rows
  const int N4 = N >> 2;
  const int nl = L - l0 < kZfLines ? L - l0 : kZfLines;
  const float4 *src = reinterpret_cast<const float4 *>(in + (size_t)l0 * N);
#pragma unroll 8
  for (int i = threadIdx.x; i < kZfLines * N4; i += blockDim.x) {
    const int ll = i / N4, q = i - ll * N4;
    const float4 v = ll < nl ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4 *>(tile + ll * S + 4 * q) = v;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int lg = lane >> 2, mg = lane & 3;
  float2 acc[4][J];
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int j = 0; j < J; j++) acc[r][j] = make_float2(0.f, 0.f);
  const float *rows = tile + (32 * w + lg) * S;
#pragma unroll 2
  for (int z = 0; z < N; z++) {
    float a[4];
#pragma unroll
    for (int r = 0; r < 4; r++) a[r] = rows[8 * r * S + z];
    float2 e[J];
#pragma unroll
    for (int j = 0; j < J; j++) {
      const int k = mg + 4 * j;
      e[j] = k < Kz ? Es[z * Kz + k] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int j = 0; j < J; j++) {
        acc[r][j].x += a[r] * e[j].x;
        acc[r][j].y += a[r] * e[j].y;
      }
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int l = l0 + 32 * w + lg + 8 * r;
    if (l >= L) continue;
#pragma unroll
    for (int j = 0; j < J; j++) {
      const int k = mg + 4 * j;
      if (k < Kz) out[(size_t)l * Kz + k] = acc[r][j];
    }
  }
}

// inv: out[l][z] (+)= sum_k Re[in[l][k] G[z][k]],  G = c_k s (cos, sin), z-major.
// N is a multiple of 4: a thread keeps the table rows of four consecutive z
// in registers and walks lines of the block's tile, so each 16-byte read of
// two of a line's coefficients (a broadcast) feeds 16 multiply-adds and the
// result leaves as one 16-byte store.  The table's strided reads are paid
// once per tile of kZiLines lines (grids without slab kernels have two such
// tiles an SM or more).  91 us at 96^3 with 16 channels and 12 modes when a thread
// held two z (8-byte reads, 4 multiply-adds each), 73 us with four z and 64
// lines, 44 us with 256.
constexpr int kZiLines = 256;

template <int KB>
__global__ void __launch_bounds__(128) k_dft_z_inv(const float2 *__restrict__ in,
                                                   float *__restrict__ out,
                                                   const float2 *__restrict__ G, int L, int N,
                                                   int Kz, int accumulate) {
  __shared__ __align__(16) float2 cs[kZiLines * KB];  // rows of KB, zero beyond Kz
  const int l0 = blockIdx.x * kZiLines;
  const int nl = L - l0 < kZiLines ? L - l0 : kZiLines;
  for (int i = threadIdx.x; i < nl * KB; i += blockDim.x) {
    const int ll = i / KB, k = i - ll * KB;
    cs[i] = k < Kz ? in[(size_t)(l0 + ll) * Kz + k] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int Q = N >> 2;  // quads of a line
  const int per = Q < (int)blockDim.x ? Q : (int)blockDim.x;
  const int sub = threadIdx.x / per, subs = blockDim.x / per;
  if (sub >= subs) return;
  for (int q = threadIdx.x - sub * per; q < Q; q += per) {
    float2 g[KB][4];
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int k = 0; k < KB; k++)
        g[k][j] = k < Kz ? G[(size_t)(4 * q + j) * Kz + k] : make_float2(0.f, 0.f);
    for (int ll = sub; ll < nl; ll += subs) {
      float4 *o = reinterpret_cast<float4 *>(out + (size_t)(l0 + ll) * N) + q;
      const float4 before = accumulate ? *o : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 *c = reinterpret_cast<const float4 *>(cs + ll * KB);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k2 = 0; k2 < KB / 2; k2++) {
        const float4 a = c[k2];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          v[j] = fmaf(a.x, g[2 * k2][j].x, v[j]);
          v[j] = fmaf(-a.y, g[2 * k2][j].y, v[j]);
          v[j] = fmaf(a.z, g[2 * k2 + 1][j].x, v[j]);
          v[j] = fmaf(-a.w, g[2 * k2 + 1][j].y, v[j]);
        }
      }
      *o = make_float4(before.x + v[0], before.y + v[1], before.z + v[2], before.w + v[3]);
    }
  }
}

// Truncated (complex) DFT along a middle axis:
// out[o][m][i] = sum_n in[o][n][i] * E[m][n],  m < Mout, n < Nin, i < inner.
__global__ void k_dft_axis(const float2 *__restrict__ in, float2 *__restrict__ out,
                           const float2 *__restrict__ E, int outer, int Nin, int Mout,
                           int inner) {
  extern __shared__ float sm[];
  float2 *Es = reinterpret_cast<float2 *>(sm);  // [Mout][Nin]
  for (int i = threadIdx.x; i < Mout * Nin; i += blockDim.x) Es[i] = E[i];
  __syncthreads();
  // 32-bit index arithmetic (the network's tensors hold < 2^31 entries; a
  // 64-bit division costs several times a 32-bit one)
  const int total = outer * Mout * inner;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const int r = t / inner;
    const int i = t - r * inner;
    const int o = r / Mout;
    const int m = r - o * Mout;
    const float2 *src = in + (size_t)o * Nin * inner + i;
    const float2 *e = Es + m * Nin;
    float re = 0.f, im = 0.f;
    int n = 0;
    // eight strided loads in flight before their multiply-adds (same order)
    for (; n + 8 <= Nin; n += 8) {
      float2 a[8];
#pragma unroll
      for (int u = 0; u < 8; u++) a[u] = src[(size_t)(n + u) * inner];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const float2 b = e[n + u];
        re += a[u].x * b.x - a[u].y * b.y;
        im += a[u].x * b.y + a[u].y * b.x;
      }
    }
    for (; n < Nin; n++) {
      const float2 a = src[(size_t)n * inner], b = e[n];
      re += a.x * b.x - a.y * b.y;
      im += a.x * b.y + a.y * b.x;
    }
    out[t] = make_float2(re, im);
  }
}

// The same contraction by tiles: a tile is (o, IC consecutive i), its
// Nin x IC inputs staged in shared memory with the whole table E, staged
// once per block n-major ([n][m], Mout padded with zero rows to a multiple
// of four); a thread forms four outputs m = 4 g .. 4 g + 3 of one column i,
// so per n it reads one staged input and its four table entries as two
// 16-byte words and does sixteen fused multiply-adds.  For the y
// contractions (inner = Kz) a tile is a whole contiguous slab; S tiles go
// through a block at once when one leaves threads idle.
constexpr int kAxMR = 4;
__host__ __device__ constexpr int ax_rows(int Mout) { return (Mout + kAxMR - 1) / kAxMR * kAxMR; }
__device__ __forceinline__ void cmac(float &re, float &im, float2 a, float bx, float by) {
  re = fmaf(a.x, bx, re);
  re = fmaf(-a.y, by, re);
  im = fmaf(a.x, by, im);
  im = fmaf(a.y, bx, im);
}
__global__ void __launch_bounds__(256) k_dft_tile(const float2 *__restrict__ in,
                                                  float2 *__restrict__ out,
                                                  const float2 *__restrict__ E, int outer,
                                                  int Nin, int Mout, int inner, int IC, int S) {
  extern __shared__ __align__(16) float2 smt[];
  const int MS = ax_rows(Mout);
  float2 *Es = smt;             // [Nin][MS]
  float2 *Tb = Es + Nin * MS;   // S x [Nin][IC]
  for (int i = threadIdx.x; i < Nin * MS; i += blockDim.x) {
    const int n = i / MS, m = i - n * MS;
    Es[i] = m < Mout ? E[m * Nin + n] : make_float2(0.f, 0.f);
  }
  const int nch = (inner + IC - 1) / IC;
  const int tiles = outer * nch;
  const int groups = MS / kAxMR;
  const int per = groups * IC;  // work items of one tile
  for (int t0 = blockIdx.x * S; t0 < tiles; t0 += gridDim.x * S) {
    __syncthreads();  // the previous batch's readers are done (and E is in)
    for (int idx = threadIdx.x; idx < S * Nin * IC; idx += blockDim.x) {
      const int s = idx / (Nin * IC), rem = idx - s * Nin * IC;
      const int n = rem / IC, j = rem - n * IC;
      const int tile = t0 + s;
      float2 v = make_float2(0.f, 0.f);
      if (tile < tiles) {
        const int o = tile / nch, i0 = (tile - o * nch) * IC;
        if (i0 + j < inner) v = in[((size_t)o * Nin + n) * inner + i0 + j];
      }
      Tb[idx] = v;
    }
    __syncthreads();
    for (int w = threadIdx.x; w < S * per; w += blockDim.x) {
      const int s = w / per, idx = w - s * per;
      const int tile = t0 + s;
      if (tile >= tiles) continue;
      const int o = tile / nch, i0 = (tile - o * nch) * IC;
      const int ic = inner - i0 < IC ? inner - i0 : IC;
      const int g = idx / IC, j = idx - g * IC;
      if (j >= ic) continue;
      const float2 *pa = Tb + (size_t)s * Nin * IC + j;
      // the group's four table entries of row n: two 16-byte words (MS and
      // 4 g are multiples of four float2, the array is 16-byte aligned)
      const float4 *pe = reinterpret_cast<const float4 *>(Es + g * kAxMR);
      const int ES4 = MS / 2;
      float re[kAxMR], im[kAxMR];
#pragma unroll
      for (int r = 0; r < kAxMR; r++) re[r] = im[r] = 0.f;
#pragma unroll 4
      for (int n = 0; n < Nin; n++) {
        const float2 a = pa[n * IC];
        const float4 b01 = pe[n * ES4], b23 = pe[n * ES4 + 1];
        cmac(re[0], im[0], a, b01.x, b01.y);
        cmac(re[1], im[1], a, b01.z, b01.w);
        cmac(re[2], im[2], a, b23.x, b23.y);
        cmac(re[3], im[3], a, b23.z, b23.w);
      }
#pragma unroll
      for (int r = 0; r < kAxMR; r++) {
        const int m = g * kAxMR + r;
        if (m < Mout) out[((size_t)o * Mout + m) * inner + i0 + j] = make_float2(re[r], im[r]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// z and y transforms of a whole (channel, x) slab in one block, for grids whose
// slab of N x N reals fits in shared memory beside another block's (slab_ok).
// Both axes are folded: with e_n = a_n + a_{N-n}, o_n = a_n - a_{N-n} a
// transform's cosine sums read e and its sine sums o, half the products, and
// along y the sums for +k and -k are the same two.  Yc[n][k] = (cos, sin) of 2
// pi k n / N, k <= m (the last for ky = -m).

// Row stride of the slab tile: 16-byte rows, and the eight rows one load
// instruction touches in distinct banks.
__host__ __device__ inline int slab_stride(int N) { return N + (N % 8 == 0 ? 4 : 8); }
__host__ __device__ inline int slab_chunks(int N) { return (N + 31) / 32; }
__host__ __device__ constexpr int slab_jp(int KB) { return KB / 4 == 3 ? 4 : KB / 4; }
size_t slab_fwd_smem(int N, int m, int KB) {
  return sizeof(float) * 32 * slab_chunks(N) * slab_stride(N) +
         sizeof(float2) * ((size_t)(N / 2 + 1) * (4 * slab_jp(KB) + m + 1));
}
size_t slab_inv_smem(int N, int m, int KB) {
  return sizeof(float2) *
         ((size_t)N * KB + (size_t)KB * N + 2 * (size_t)(m + 1) * KB + (size_t)(N / 2 + 1) * (m + 1));
}
// Two analysis blocks per SM: up to N = 160 with 4 modes, 152 with 8, 144 with 12,
// 136 with 16.  The layer kernel needs more (synth_smem): with 16 channels one
// block fits an SM with 16 modes, and with 12 up to N = 40.
bool slab_ok(int N, int m) { return slab_fwd_smem(N, m, (m + 3) / 4 * 4) <= 110 * 1024; }

// 16-byte asynchronous copies to shared memory.
__device__ __forceinline__ void copy_async16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Analysis: out[slab][ky][kz] = sum_y e^{-i ky y} sum_z E[z][kz] in[slab][y][z].
// Along z two warps share 32 lines, each taking every second quad of z; lane
// (lg = lane / 4, mg = lane % 4) holds lines lg + 8 r (r < 4) and modes mg + 4 j, so
// a quad's three row reads a line and two table words a z feed 96 multiply-adds
// and 32 additions.  The slab's second half
// arrives while the first is transformed.  128^3, 16 channels, 12 modes: 66 us
// against 101 for the z axis and 26 to 55 for the y axis before.
template <int KB>
__global__ void __launch_bounds__(384) k_slab_fwd(const float *__restrict__ in,
                                                  float2 *__restrict__ out,
                                                  const float2 *__restrict__ E,
                                                  const float2 *__restrict__ Yc, int N, int Kz,
                                                  int m) {
  constexpr int J = KB / 4, JP = slab_jp(KB);
  extern __shared__ __align__(16) float sm[];
  const int S = slab_stride(N), rows = 32 * slab_chunks(N), H = N / 2;
  float *tile = sm;                                              // [rows][S]
  float2 *T = reinterpret_cast<float2 *>(tile + rows * S);       // [H + 1][4][JP]
  float2 *Ys = T + (size_t)(H + 1) * 4 * JP;                     // [H + 1][m + 1]
  const float *src = in + (size_t)blockIdx.x * N * N;
  const int N4 = N >> 2, nq = N / 8;  // whole quads below N / 2
  // the quads of z below nq / 2 and their mirrors, then the rest: the first
  // half is transformed while the second is on its way
  const int q1 = nq / 2;
  auto stage = [&](int lo, int count) {  // `count` quads from lo, and nothing else
    const int per = blockDim.x / count, q = threadIdx.x % count, l0 = threadIdx.x / count;
    if (l0 < per) {
      for (int ll = l0; ll < N; ll += per)
        copy_async16(tile + ll * S + 4 * (lo + q), src + (size_t)ll * N + 4 * (lo + q));
    }
  };
  if (q1 > 0) {
    stage(0, q1);
    stage(N4 - q1, q1);
  }
  copy_commit();
  stage(q1, N4 - 2 * q1);
  copy_commit();
  for (int i = threadIdx.x; i < (rows - N) * S; i += blockDim.x) tile[N * S + i] = 0.f;
  for (int i = threadIdx.x; i < (H + 1) * 4 * JP; i += blockDim.x) {
    const int z = i / (4 * JP), r = i - z * 4 * JP, kk = r / JP + 4 * (r % JP);
    T[i] = kk < Kz && r % JP < J ? E[z * Kz + kk] : make_float2(0.f, 0.f);
  }
  for (int i = threadIdx.x; i < (H + 1) * (m + 1); i += blockDim.x) Ys[i] = Yc[i];
  copy_wait<1>();
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, chunk = w >> 1, par = w & 1;
  const int lg = lane >> 2, mg = lane & 3;
  const float *row0 = tile + (32 * chunk + lg) * S;
  float2 acc[4][J];
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int j = 0; j < J; j++) acc[r][j] = make_float2(0.f, 0.f);
  auto load_t = [&](int z, float2(&t)[J]) {
    const float2 *p = T + (z * 4 + mg) * JP;
    if constexpr (J == 1) {
      t[0] = p[0];
    } else {
#pragma unroll
      for (int j = 0; j + 1 < J + 1; j += 2) {
        const float4 v = reinterpret_cast<const float4 *>(p)[j / 2];
        t[j] = make_float2(v.x, v.y);
        if (j + 1 < J) t[j + 1] = make_float2(v.z, v.w);
      }
    }
  };
  auto add = [&](int r, float a, float b, const float2(&t)[J]) {
    const float e = a + b, o = a - b;
#pragma unroll
    for (int j = 0; j < J; j++) {
      acc[r][j].x = fmaf(e, t[j].x, acc[r][j].x);
      acc[r][j].y = fmaf(o, t[j].y, acc[r][j].y);
    }
  };
#pragma unroll 1
  for (int q = par, half = 0; half < 2; q += 2) {
    if (q >= (half ? nq : q1)) {
      if (half++) break;
      copy_wait<0>();
      __syncthreads();
      if (q >= nq) break;
    }
    float4 a[4], b[4];
    float b0[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const float *row = row0 + 8 * r * S;
      a[r] = *reinterpret_cast<const float4 *>(row + 4 * q);
      b[r] = *reinterpret_cast<const float4 *>(row + N - 4 * q - 4);
      b0[r] = q ? row[N - 4 * q] : 0.f;  // z = 0 has no partner
    }
    float2 t[J];
    load_t(4 * q, t);
#pragma unroll
    for (int r = 0; r < 4; r++) add(r, a[r].x, b0[r], t);
    load_t(4 * q + 1, t);
#pragma unroll
    for (int r = 0; r < 4; r++) add(r, a[r].y, b[r].w, t);
    load_t(4 * q + 2, t);
#pragma unroll
    for (int r = 0; r < 4; r++) add(r, a[r].z, b[r].z, t);
    load_t(4 * q + 3, t);
#pragma unroll
    for (int r = 0; r < 4; r++) add(r, a[r].w, b[r].y, t);
  }
  if (par == 0) {
    // what is left below N / 2 (N = 4 mod 8), and z = N / 2 itself
#pragma unroll 1
    for (int z = 4 * nq; z <= H; z++) {
      float2 t[J];
      load_t(z, t);
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float *row = row0 + 8 * r * S;
        add(r, row[z], z > 0 && z < H ? row[N - z] : 0.f, t);
      }
    }
  }
  // the two warps' halves added, as R[y][kz] in the tile's place
  __syncthreads();
  float2 *R = reinterpret_cast<float2 *>(sm);  // [N][KB]
#pragma unroll
  for (int half = 1; half >= 0; half--) {
    if (par == half) {
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int l = 32 * chunk + lg + 8 * r;
        if (l < N) {
#pragma unroll
          for (int j = 0; j < J; j++) {
            float2 &d = R[l * KB + mg + 4 * j];
            const float2 v = acc[r][j];
            d = half ? v : make_float2(d.x + v.x, d.y + v.y);
          }
        }
      }
    }
    __syncthreads();
  }
  // y: a thread takes two k of one kz over a share of n, the shares added up
  // through shared memory (behind R)
  float2 *o = out + (size_t)blockIdx.x * 2 * m * Kz;
  const int kp = (m + 2) / 2, items = kp * Kz;
  int shares = blockDim.x / items;
  const int room = (int)(((size_t)rows * S - (size_t)N * KB * 2) / (8 * (size_t)items));
  shares = shares < 1 || room < 1 ? 1 : (shares < room ? shares : room);
  float4 *part = reinterpret_cast<float4 *>(R + (size_t)N * KB);  // [share][k][item]: (c, s)
  for (int it0 = 0; it0 < items; it0 += blockDim.x) {
    const int sh = threadIdx.x / items;
    const int it = shares > 1 ? (int)threadIdx.x - sh * items : it0 + (int)threadIdx.x;
    const bool on = shares > 1 ? sh < shares : it < items;
    const int k0 = 2 * (it / Kz), kz = it % Kz, k1 = k0 < m ? k0 + 1 : k0;
    float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
    if (on) {
      const float2 *rp = R + kz;
      const int s0 = shares > 1 ? sh : 0;
      auto add2 = [&](float2 e, float2 od, int n) {
        const float2 ya = Ys[n * (m + 1) + k0], yb = Ys[n * (m + 1) + k1];
        v0.x = fmaf(e.x, ya.x, v0.x);
        v0.y = fmaf(e.y, ya.x, v0.y);
        v0.z = fmaf(od.x, ya.y, v0.z);
        v0.w = fmaf(od.y, ya.y, v0.w);
        v1.x = fmaf(e.x, yb.x, v1.x);
        v1.y = fmaf(e.y, yb.x, v1.y);
        v1.z = fmaf(od.x, yb.y, v1.z);
        v1.w = fmaf(od.y, yb.y, v1.w);
      };
      if (s0 == 0) {
        add2(rp[0], make_float2(0.f, 0.f), 0);
        add2(rp[H * KB], make_float2(0.f, 0.f), H);
      }
#pragma unroll 4
      for (int n = 1 + s0; n < H; n += shares) {
        const float2 p = rp[n * KB], q = rp[(N - n) * KB];
        add2(make_float2(p.x + q.x, p.y + q.y), make_float2(p.x - q.x, p.y - q.y), n);
      }
    }
    if (shares > 1) {
      if (on) {
        part[(sh * 2) * items + it] = v0;
        part[(sh * 2 + 1) * items + it] = v1;
      }
      __syncthreads();
      if (sh == 0) {
        for (int u = 1; u < shares; u++) {
          const float4 a = part[(u * 2) * items + it], c = part[(u * 2 + 1) * items + it];
          v0 = make_float4(v0.x + a.x, v0.y + a.y, v0.z + a.z, v0.w + a.w);
          v1 = make_float4(v1.x + c.x, v1.y + c.y, v1.z + c.z, v1.w + c.w);
        }
      }
    }
    if (on && (shares == 1 || sh == 0)) {
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int kk = k0 + u;
        const float4 v = u ? v1 : v0;
        if (kk > m) continue;
        if (kk < m) o[kk * Kz + kz] = make_float2(v.x + v.w, v.y - v.z);
        if (kk > 0) o[(2 * m - kk) * Kz + kz] = make_float2(v.x - v.w, v.y + v.z);
      }
    }
    if (shares > 1) break;
  }
}

// The slab's coefficients B[ky][kz] as the folded pairs P_k = B_k + B_{-k}, Q_k =
// B_k - B_{-k} (k = 0: B_0, 0; k = m: B_{-m}, -B_{-m}), rows of ld.
__device__ __forceinline__ void slab_pairs(const float2 *__restrict__ B, int m, int Kz, float2 &P,
                                           float2 &Q, int k, int kz) {
  const float2 a = k < m ? B[k * Kz + kz] : make_float2(0.f, 0.f);
  const float2 b = k > 0 ? B[(2 * m - k) * Kz + kz] : make_float2(0.f, 0.f);
  P = make_float2(a.x + b.x, a.y + b.y);
  Q = k ? make_float2(a.x - b.x, a.y - b.y) : make_float2(0.f, 0.f);
}

// Synthesis: out[slab][y][z] (+)= sum_kz Re[G[z][kz] sum_ky e^{+i ky y} B[slab][ky][kz]].
// The y sums go to shared memory (y and N - y together), then the z synthesis of
// k_dft_z_inv.  96^3, 16 channels, 12 modes: 47 us against 44 and 25 for the
// two launches.
template <int KB>
__global__ void __launch_bounds__(128) k_slab_inv(const float2 *__restrict__ in,
                                                  float *__restrict__ out,
                                                  const float2 *__restrict__ G,
                                                  const float2 *__restrict__ Yc, int N, int Kz,
                                                  int m, int accumulate) {
  extern __shared__ __align__(16) float sm[];
  const int H = N / 2;
  float2 *A = reinterpret_cast<float2 *>(sm);  // [N][KB]
  float2 *Gs = A + (size_t)N * KB;             // [KB][N]
  float2 *P = Gs + (size_t)KB * N, *Q = P + (m + 1) * KB;
  float2 *Ys = Q + (m + 1) * KB;               // [H + 1][m + 1]
  const float2 *B = in + (size_t)blockIdx.x * 2 * m * Kz;
  for (int i = threadIdx.x; i < N * KB; i += blockDim.x) {
    const int z = i / KB, k = i - z * KB;
    Gs[k * N + z] = k < Kz ? G[z * Kz + k] : make_float2(0.f, 0.f);
  }
  for (int i = threadIdx.x; i < (m + 1) * KB; i += blockDim.x) {
    const int k = i / KB, kz = i - k * KB;
    float2 p = make_float2(0.f, 0.f), q = p;
    if (kz < Kz) slab_pairs(B, m, Kz, p, q, k, kz);
    P[i] = p;
    Q[i] = q;
  }
  for (int i = threadIdx.x; i < (H + 1) * (m + 1); i += blockDim.x) Ys[i] = Yc[i];
  __syncthreads();
  for (int it = threadIdx.x; it < (H + 1) * KB; it += blockDim.x) {
    const int n = it / KB, kz = it - n * KB;
    float2 u = P[kz], v = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int k = 1; k <= m; k++) {
      const float2 p = P[k * KB + kz], q = Q[k * KB + kz], y = Ys[n * (m + 1) + k];
      u.x = fmaf(p.x, y.x, u.x);
      u.y = fmaf(p.y, y.x, u.y);
      v.x = fmaf(-q.y, y.y, v.x);
      v.y = fmaf(q.x, y.y, v.y);
    }
    A[n * KB + kz] = make_float2(u.x + v.x, u.y + v.y);
    if (n > 0 && n < H) A[(N - n) * KB + kz] = make_float2(u.x - v.x, u.y - v.y);
  }
  __syncthreads();
  const int Qd = N >> 2;  // quads of a line
  const int per = Qd < (int)blockDim.x ? Qd : (int)blockDim.x;
  const int sub = threadIdx.x / per, subs = blockDim.x / per;
  if (sub >= subs) return;
  float *base = out + (size_t)blockIdx.x * N * N;
  for (int q = threadIdx.x - sub * per; q < Qd; q += per) {
    float2 g[KB][4];
#pragma unroll
    for (int k = 0; k < KB; k++) {
      const float4 *gp = reinterpret_cast<const float4 *>(Gs + (size_t)k * N + 4 * q);
      const float4 g0 = gp[0], g1 = gp[1];
      g[k][0] = make_float2(g0.x, g0.y);
      g[k][1] = make_float2(g0.z, g0.w);
      g[k][2] = make_float2(g1.x, g1.y);
      g[k][3] = make_float2(g1.z, g1.w);
    }
    for (int ll = sub; ll < N; ll += subs) {
      float4 *o = reinterpret_cast<float4 *>(base + (size_t)ll * N) + q;
      const float4 before = accumulate ? *o : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 *c = reinterpret_cast<const float4 *>(A + ll * KB);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k2 = 0; k2 < KB / 2; k2++) {
        const float4 a = c[k2];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          v[j] = fmaf(a.x, g[2 * k2][j].x, v[j]);
          v[j] = fmaf(-a.y, g[2 * k2][j].y, v[j]);
          v[j] = fmaf(a.z, g[2 * k2 + 1][j].x, v[j]);
          v[j] = fmaf(-a.w, g[2 * k2 + 1][j].y, v[j]);
        }
      }
      *o = make_float4(before.x + v[0], before.y + v[1], before.z + v[2], before.w + v[3]);
    }
  }
}

// Spectral mixing U[o][k] = sum_i W[i][o][k] V[i][k]  (W bf16 complex).
__global__ void k_spec_mix(const float2 *__restrict__ V, const __nv_bfloat16 *__restrict__ W,
                           float2 *__restrict__ U, int C, int K) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= C * K) return;
  const int o = t / K, k = t - o * K;
  float re = 0.f, im = 0.f;
  for (int i = 0; i < C; i++) {
    const size_t w = ((size_t)(i * C + o) * K + k) * 2;
    const float wr = bf(W, w), wi = bf(W, w + 1);
    const float2 v = V[(size_t)i * K + k];
    re += wr * v.x - wi * v.y;
    im += wr * v.y + wi * v.x;
  }
  U[t] = make_float2(re, im);
}

// Adjoint of the mixing: Vbar[i][k] = sum_o conj(W[i][o][k]) Ubar[o][k] and
// Wbar[i][o][k] += Ubar[o][k] conj(V[i][k]).
__global__ void k_spec_mix_bwd(const float2 *__restrict__ V, const __nv_bfloat16 *__restrict__ W,
                               const float2 *__restrict__ Ub, float2 *__restrict__ Vb,
                               float *__restrict__ Wg, int C, int K) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= C * K) return;
  const int i = t / K, k = t - i * K;
  const float2 v = V[(size_t)i * K + k];
  float re = 0.f, im = 0.f;
  for (int o = 0; o < C; o++) {
    const size_t w = ((size_t)(i * C + o) * K + k) * 2;
    const float wr = bf(W, w), wi = bf(W, w + 1);
    const float2 u = Ub[(size_t)o * K + k];
    re += wr * u.x + wi * u.y;
    im += wr * u.y - wi * u.x;
    Wg[w] += u.x * v.x + u.y * v.y;
    Wg[w + 1] += u.y * v.x - u.x * v.y;
  }
  Vb[t] = make_float2(re, im);
}

// Lift: h0[c][r] = P[c][0] mask[r] + P[c][1] eta + p[c].
__global__ void k_lift(const float *__restrict__ mask, float eta, const __nv_bfloat16 *__restrict__ P,
                       const __nv_bfloat16 *__restrict__ p, float *__restrict__ h, int C,
                       long long NR) {
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < NR;
       r += (long long)gridDim.x * blockDim.x) {
    const float m = mask[r];
    for (int c = 0; c < C; c++)
      h[(size_t)c * NR + r] = bf(P, 2 * c) * m + bf(P, 2 * c + 1) * eta + bf(p, c);
  }
}

// Layer output: z[o][r] = spec[o][r] + sum_i Wp[o][i] h[i][r] + b[o];
// hn = act(z).  spec is already in z (from the inverse transform); z is
// written back only when a backward pass will need it (store_z).  A thread
// takes four consecutive points (16-byte loads and stores; N^3 is a
// multiple of 4), so each weight read from shared memory feeds four
// multiply-adds.  The output-channel loop is not unrolled, so the weights
// stay in shared memory instead of C*C registers.
__device__ __forceinline__ float4 gelu4(float4 a) {
  return make_float4(gelu(a.x), gelu(a.y), gelu(a.z), gelu(a.w));
}

template <int C>
__global__ void __launch_bounds__(256) k_layer_pw(const float *__restrict__ h,
                                                  float *__restrict__ z, float *__restrict__ hn,
                                                  const __nv_bfloat16 *__restrict__ Wp,
                                                  const __nv_bfloat16 *__restrict__ b,
                                                  long long NR, int act, int store_z) {
  __shared__ float Ws[C * C], bs[C];
  for (int i = threadIdx.x; i < C * C; i += blockDim.x) Ws[i] = bf(Wp, i);
  for (int i = threadIdx.x; i < C; i += blockDim.x) bs[i] = bf(b, i);
  __syncthreads();
  const long long NR4 = NR >> 2;
  const float4 *h4 = reinterpret_cast<const float4 *>(h);
  float4 *z4 = reinterpret_cast<float4 *>(z);
  float4 *hn4 = reinterpret_cast<float4 *>(hn);
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < NR4;
       q += (long long)gridDim.x * blockDim.x) {
    float4 hv[C];
#pragma unroll
    for (int i = 0; i < C; i++) hv[i] = h4[(size_t)i * NR4 + q];
#pragma unroll 1
    for (int o = 0; o < C; o++) {
      float4 acc = z4[(size_t)o * NR4 + q];
      const float bo = bs[o];
      acc.x += bo;
      acc.y += bo;
      acc.z += bo;
      acc.w += bo;
#pragma unroll
      for (int i = 0; i < C; i++) {
        const float w = Ws[o * C + i];
        acc.x += w * hv[i].x;
        acc.y += w * hv[i].y;
        acc.z += w * hv[i].z;
        acc.w += w * hv[i].w;
      }
      if (store_z) z4[(size_t)o * NR4 + q] = acc;
      hn4[(size_t)o * NR4 + q] = act ? gelu4(acc) : acc;
    }
  }
}

// Inference form of the layer output (no backward pass needs z): the
// z-synthesis of the spectral part fused into the pointwise layer.
// spec[o][r] = sum_k Re[A[o][line][k] G[z][k]] is formed in registers from
// the line's Kz coefficients instead of being written and read back as a
// full C x N^3 field.  A block takes 4 z-lines per pass (two consecutive z
// per thread, so a line is two warps and its coefficients are read as
// broadcasts), the synthesis table transposed to [k][z] in shared memory
// (conflict-free 16-byte reads), the line's coefficients as [k][c] (two
// channels per 16-byte broadcast read), the pointwise weights in shared
// memory (four per 16-byte broadcast read).
template <int C>
__global__ void __launch_bounds__(256) k_layer_synth_pw(const float2 *__restrict__ A,
                                                        const float2 *__restrict__ G,
                                                        const float *__restrict__ h,
                                                        float *__restrict__ hn,
                                                        const __nv_bfloat16 *__restrict__ Wp,
                                                        const __nv_bfloat16 *__restrict__ b, int N,
                                                        int Kz, int act) {
  extern __shared__ __align__(16) float sm[];
  float *Ws = sm;                                                // [C][C]
  float *bs = Ws + C * C;                                        // [C] (padded to 4)
  float2 *Gs = reinterpret_cast<float2 *>(bs + ((C + 3) & ~3));  // [Kz][N]
  float2 *As = Gs + (size_t)Kz * N;                              // [4 lines][Kz][C]
  for (int i = threadIdx.x; i < C * C; i += blockDim.x) Ws[i] = bf(Wp, i);
  for (int i = threadIdx.x; i < C; i += blockDim.x) bs[i] = bf(b, i);
  for (int i = threadIdx.x; i < Kz * N; i += blockDim.x) {
    const int k = i / N, z = i - k * N;
    Gs[i] = G[(size_t)z * Kz + k];
  }
  const int half = N >> 1;                 // threads per line
  const int lines = N * N;                 // z-lines per channel
  const long long NR = (long long)lines * N;
  const int lpb = blockDim.x / half;       // lines per pass (4 at N = 128)
  const int tl = threadIdx.x / half, zp = threadIdx.x - tl * half;
  const int z0 = 2 * zp;
  for (int l0 = blockIdx.x * lpb; l0 < lines; l0 += gridDim.x * lpb) {
    __syncthreads();  // previous pass's readers of As are done (and the tables are in)
    for (int i = threadIdx.x; i < lpb * C * Kz; i += blockDim.x) {
      const int ll = i / (C * Kz), rem = i - ll * C * Kz;
      const int c = rem / Kz, k = rem - c * Kz;
      const int line = l0 + ll;
      As[(size_t)ll * C * Kz + k * C + c] =
          line < lines ? A[((size_t)c * lines + line) * Kz + k] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const int line = l0 + tl;
    if (line >= lines || tl >= lpb) continue;
    const float2 *a = As + (size_t)tl * C * Kz;
    float2 spec[C];
#pragma unroll
    for (int c = 0; c < C; c++) spec[c] = make_float2(0.f, 0.f);
    for (int k = 0; k < Kz; k++) {
      const float4 g = *reinterpret_cast<const float4 *>(Gs + (size_t)k * N + z0);
      const float4 *ak = reinterpret_cast<const float4 *>(a + k * C);
#pragma unroll
      for (int c2 = 0; c2 < C / 2; c2++) {
        const float4 ac = ak[c2];  // channels 2 c2, 2 c2 + 1
        spec[2 * c2].x += ac.x * g.x - ac.y * g.y;
        spec[2 * c2].y += ac.x * g.z - ac.y * g.w;
        spec[2 * c2 + 1].x += ac.z * g.x - ac.w * g.y;
        spec[2 * c2 + 1].y += ac.z * g.z - ac.w * g.w;
      }
    }
    const size_t r = (size_t)line * N + z0;
    float2 hv[C];
#pragma unroll
    for (int i = 0; i < C; i++) hv[i] = *reinterpret_cast<const float2 *>(h + (size_t)i * NR + r);
#pragma unroll
    for (int o = 0; o < C; o++) {
      float2 acc = spec[o];
      acc.x += bs[o];
      acc.y += bs[o];
      const float4 *wr = reinterpret_cast<const float4 *>(Ws + o * C);
#pragma unroll
      for (int i4 = 0; i4 < C / 4; i4++) {
        const float4 w = wr[i4];
        acc.x += w.x * hv[4 * i4].x + w.y * hv[4 * i4 + 1].x + w.z * hv[4 * i4 + 2].x +
                 w.w * hv[4 * i4 + 3].x;
        acc.y += w.x * hv[4 * i4].y + w.y * hv[4 * i4 + 1].y + w.z * hv[4 * i4 + 2].y +
                 w.w * hv[4 * i4 + 3].y;
      }
      if (act) acc = make_float2(gelu(acc.x), gelu(acc.y));
      *reinterpret_cast<float2 *>(hn + (size_t)o * NR + r) = acc;
    }
  }
}

// The inference layer from the x-synthesised coefficients B[c][x][ky][kz]: a
// block holds one x's coefficients of every channel (folded pairs, slab_pairs)
// and walks lines y of a share of that x: per pass the y sums of its lines go
// to shared memory, then a thread synthesises z and N - z together (their
// cosine and sine sums; thread 0 of a line takes z = 0 and N / 2, whose sine
// table is the half difference of the two cosines and multiplies the real part
// again, so its coefficients stand in a second array as (re, re)), adds the
// pointwise layer and activates.  The previous layer's values are loaded before
// the sums, the next pass's y sums are formed while this pass's lines are in
// flight (two buffers).  Bound by issue and
// latency at two blocks per SM (128 registers): 142 us at 128^3, 16 channels, 12
// modes, against 131 without the y sums and 44 for those (packed f32x2
// multiply-adds: 148).
template <int C>
size_t synth_smem(int N, int m, int Kz) {
  const int lpb = 256 / (N / 2);
  return sizeof(float) * (C * C + C) +
         sizeof(float2) * ((size_t)Kz * (N / 2) + (size_t)N * (m + 1) +
                           2 * (size_t)C * (m + 1) * Kz + 4 * (size_t)lpb * C * Kz);
}
template <int C>
__global__ void __launch_bounds__(256, 2) k_layer_synth(const float2 *__restrict__ B,
                                                        const float2 *__restrict__ G,
                                                        const float2 *__restrict__ Yc,
                                                        const float *__restrict__ h,
                                                        float *__restrict__ hn,
                                                        const __nv_bfloat16 *__restrict__ Wp,
                                                        const __nv_bfloat16 *__restrict__ b, int N,
                                                        int Kz, int m, int act) {
  extern __shared__ __align__(16) float sm[];
  const int H = N >> 1, lpb = 256 / H;
  float *Ws = sm;                                       // [C][C]
  float *bs = Ws + C * C;                               // [C]
  float2 *As = reinterpret_cast<float2 *>(bs + C);      // [2][lpb][Kz][C]: (re, im)
  float2 *Ax = As + 2 * (size_t)lpb * Kz * C;           // the same as (re, re)
  float2 *Gs = Ax + 2 * (size_t)lpb * Kz * C;           // [Kz][H]
  float2 *Ys = Gs + (size_t)Kz * H;                     // [N][m + 1]
  float2 *P = Ys + (size_t)N * (m + 1);                 // [m + 1][Kz][C]
  float2 *Q = P + (size_t)(m + 1) * Kz * C;
  const int x = blockIdx.x;
  for (int i = threadIdx.x; i < C * C; i += blockDim.x) Ws[i] = bf(Wp, i);
  for (int i = threadIdx.x; i < C; i += blockDim.x) bs[i] = bf(b, i);
  for (int i = threadIdx.x; i < Kz * H; i += blockDim.x) {
    const int k = i / H, z = i - k * H;
    const float2 g = G[(size_t)z * Kz + k];
    if (z == 0) {
      const float gh = G[(size_t)H * Kz + k].x;
      Gs[i] = make_float2(0.5f * (g.x + gh), 0.5f * (gh - g.x));
    } else {
      Gs[i] = g;
    }
  }
  for (int i = threadIdx.x; i < N * (m + 1); i += blockDim.x) Ys[i] = Yc[i];
  for (int i = threadIdx.x; i < (m + 1) * Kz * C; i += blockDim.x) {
    const int c = i / ((m + 1) * Kz), r = i - c * (m + 1) * Kz, k = r / Kz, kz = r - k * Kz;
    slab_pairs(B + ((size_t)c * N + x) * 2 * m * Kz, m, Kz, P[r * C + c], Q[r * C + c], k, kz);
  }
  const long long NR = (long long)N * N * N;
  const int y0 = (int)((long long)N * blockIdx.y / gridDim.y);
  const int y1 = (int)((long long)N * (blockIdx.y + 1) / gridDim.y);
  // y sums of lines ya .. ya + lpb into buffer `buf`
  auto lines_to = [&](int ya, int buf) {
    for (int i = threadIdx.x; i < lpb * Kz * C; i += blockDim.x) {
      const int ll = i / (Kz * C), r = i - ll * Kz * C, y = ya + ll;
      if (y >= y1) continue;
      const float2 *yp = Ys + (size_t)y * (m + 1);
      float2 u = P[r], v = make_float2(0.f, 0.f);
#pragma unroll 4
      for (int k = 1; k <= m; k++) {
        const float2 p = P[(size_t)k * Kz * C + r], q = Q[(size_t)k * Kz * C + r], cs = yp[k];
        u.x = fmaf(p.x, cs.x, u.x);
        u.y = fmaf(p.y, cs.x, u.y);
        v.x = fmaf(-q.y, cs.y, v.x);
        v.y = fmaf(q.x, cs.y, v.y);
      }
      const float2 a = make_float2(u.x + v.x, u.y + v.y);
      As[(size_t)buf * lpb * Kz * C + i] = a;
      Ax[(size_t)buf * lpb * Kz * C + i] = make_float2(a.x, a.x);
    }
  };
  __syncthreads();
  lines_to(y0, 0);
  __syncthreads();
  const int tl = threadIdx.x / H, zp = threadIdx.x - tl * H, zm = zp ? N - zp : H;
  int buf = 0;
  for (int ya = y0; ya < y1; ya += lpb, buf ^= 1) {
    const int y = ya + tl;
    const bool on = tl < lpb && y < y1;
    const size_t r0 = ((size_t)x * N + (on ? y : y0)) * N;
    float2 hv[C];
#pragma unroll
    for (int i = 0; i < C; i++)
      hv[i] = make_float2(h[(size_t)i * NR + r0 + zp], h[(size_t)i * NR + r0 + zm]);
    if (ya + lpb < y1) lines_to(ya + lpb, buf ^ 1);
    if (on) {
      const float2 *a = (zp ? As : Ax) + ((size_t)buf * lpb + tl) * Kz * C;
      float2 spec[C];  // (cosine, sine) sums
#pragma unroll
      for (int c = 0; c < C; c++) spec[c] = make_float2(0.f, 0.f);
      for (int k = 0; k < Kz; k++) {
        const float2 g = Gs[(size_t)k * H + zp];
        const float4 *ak = reinterpret_cast<const float4 *>(a + k * C);
#pragma unroll
        for (int c2 = 0; c2 < C / 2; c2++) {
          const float4 ac = ak[c2];  // channels 2 c2, 2 c2 + 1
          spec[2 * c2].x = fmaf(ac.x, g.x, spec[2 * c2].x);
          spec[2 * c2].y = fmaf(ac.y, g.y, spec[2 * c2].y);
          spec[2 * c2 + 1].x = fmaf(ac.z, g.x, spec[2 * c2 + 1].x);
          spec[2 * c2 + 1].y = fmaf(ac.w, g.y, spec[2 * c2 + 1].y);
        }
      }
#pragma unroll
      for (int o = 0; o < C; o++) {
        float2 acc = make_float2(spec[o].x - spec[o].y + bs[o], spec[o].x + spec[o].y + bs[o]);
        const float4 *wr = reinterpret_cast<const float4 *>(Ws + o * C);
#pragma unroll
        for (int i4 = 0; i4 < C / 4; i4++) {
          const float4 w = wr[i4];
          acc.x = fmaf(w.x, hv[4 * i4].x, acc.x);
          acc.y = fmaf(w.x, hv[4 * i4].y, acc.y);
          acc.x = fmaf(w.y, hv[4 * i4 + 1].x, acc.x);
          acc.y = fmaf(w.y, hv[4 * i4 + 1].y, acc.y);
          acc.x = fmaf(w.z, hv[4 * i4 + 2].x, acc.x);
          acc.y = fmaf(w.z, hv[4 * i4 + 2].y, acc.y);
          acc.x = fmaf(w.w, hv[4 * i4 + 3].x, acc.x);
          acc.y = fmaf(w.w, hv[4 * i4 + 3].y, acc.y);
        }
        if (act) acc = make_float2(gelu(acc.x), gelu(acc.y));
        hn[(size_t)o * NR + r0 + zp] = acc.x;
        hn[(size_t)o * NR + r0 + zm] = acc.y;
      }
    }
    __syncthreads();
  }
}

// Deterministic block reduction of K floats into partial[block][K].
template <int K>
__device__ void block_sum_store(float (&v)[K], float *partial) {
  __shared__ float red[32 * K];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = 0; k < K; k++) {
    float x = v[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp * K + k] = x;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    float s = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[w * K + threadIdx.x];
    partial[(size_t)blockIdx.x * K + threadIdx.x] = s;
  }
  __syncthreads();
}

// Projection y = Q2 . gelu(Q1 h + q1) + q2 and the masked squared error
// against target; per-block partial loss sums (and weights) in part[2*b].
template <int C>
__global__ void k_project(const float *__restrict__ h, const __nv_bfloat16 *__restrict__ Q1,
                          const __nv_bfloat16 *__restrict__ q1, const __nv_bfloat16 *__restrict__ Q2,
                          const __nv_bfloat16 *__restrict__ q2, float *__restrict__ zq,
                          float *__restrict__ y, const float *__restrict__ target,
                          const float *__restrict__ w, float *__restrict__ part, long long NR) {
  __shared__ float Q1s[C * C], q1s[C], Q2s[C];
  for (int i = threadIdx.x; i < C * C; i += blockDim.x) Q1s[i] = bf(Q1, i);
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    q1s[i] = bf(q1, i);
    Q2s[i] = bf(Q2, i);
  }
  __syncthreads();
  const float q2v = bf(q2, 0);
  float acc[2] = {0.f, 0.f};
  // four consecutive points per thread (16-byte accesses; N^3 is a multiple of 4)
  const long long NR4 = NR >> 2;
  const float4 *h4 = reinterpret_cast<const float4 *>(h);
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < NR4;
       q += (long long)gridDim.x * blockDim.x) {
    float4 hv[C];
#pragma unroll
    for (int i = 0; i < C; i++) hv[i] = h4[(size_t)i * NR4 + q];
    float4 out = make_float4(q2v, q2v, q2v, q2v);
#pragma unroll 1
    for (int c = 0; c < C; c++) {
      const float qc = q1s[c];
      float4 a = make_float4(qc, qc, qc, qc);
#pragma unroll
      for (int i = 0; i < C; i++) {
        const float w = Q1s[c * C + i];
        a.x += w * hv[i].x;
        a.y += w * hv[i].y;
        a.z += w * hv[i].z;
        a.w += w * hv[i].w;
      }
      if (zq) reinterpret_cast<float4 *>(zq)[(size_t)c * NR4 + q] = a;
      const float q2c = Q2s[c];
      out.x += q2c * gelu(a.x);
      out.y += q2c * gelu(a.y);
      out.z += q2c * gelu(a.z);
      out.w += q2c * gelu(a.w);
    }
    reinterpret_cast<float4 *>(y)[q] = out;
    if (target) {
      const float4 t = reinterpret_cast<const float4 *>(target)[q];
      const float4 wv = w ? reinterpret_cast<const float4 *>(w)[q] : make_float4(1.f, 1.f, 1.f, 1.f);
      const float d0 = out.x - t.x, d1 = out.y - t.y, d2 = out.z - t.z, d3 = out.w - t.w;
      acc[0] += wv.x * d0 * d0 + wv.y * d1 * d1 + wv.z * d2 * d2 + wv.w * d3 * d3;
      acc[1] += wv.x + wv.y + wv.z + wv.w;
    }
  }
  if (part) block_sum_store<2>(acc, part);
}

// Weight-gradient reductions over points: a block walks chunks of kChunk
// points, writes the two factors of a chunk to shared memory (point-major
// rows of stride kCS: 16-byte rows, distinct banks for neighbouring rows) and
// each warp adds its eighth of the chunk's points to its own copy of
// sum_p a[o][p] b[i][p].  The outputs are tiled TO x TO over 16 lanes (TO =
// C / 4; a lane's rows lie four apart), the warp's halves taking point quads
// 16 points apart, so the words a load touches fall in distinct banks and
// four points of 2 TO rows feed 4 TO^2 multiply-adds; the copies are added up
// once per block.
constexpr int kChunk = 256;
constexpr int kCS = kChunk + 4;
constexpr int kPwThreads = 128;  // two points a thread

// acc[r][c] += sum over the warp's points of a[lane / 4 % 4 + 4 r] b[lane % 4 + 4 c],
// row[r] += the same rows of a alone.
template <int C>
__device__ __forceinline__ void outer_accumulate(const float (*a)[kCS], const float (*b)[kCS],
                                                 float (&acc)[C / 4][C / 4], float (&row)[C / 4]) {
  constexpr int TO = C / 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4;
  const int o0 = (lane >> 2) & 3, i0 = lane & 3;
  constexpr int kPer = kChunk / (kPwThreads / 32);  // points of a warp
#pragma unroll 2
  for (int j = 0; j < kPer / 8; j++) {
    const int p = warp * kPer + 32 * (j >> 2) + 4 * (j & 3) + 16 * half;
    float4 av[TO], bv[TO];
#pragma unroll
    for (int r = 0; r < TO; r++) {
      av[r] = *reinterpret_cast<const float4 *>(&a[o0 + 4 * r][p]);
      bv[r] = *reinterpret_cast<const float4 *>(&b[i0 + 4 * r][p]);
    }
#pragma unroll
    for (int r = 0; r < TO; r++) {
      row[r] += (av[r].x + av[r].y) + (av[r].z + av[r].w);
#pragma unroll
      for (int c = 0; c < TO; c++) {
        float t = acc[r][c];
        t = fmaf(av[r].x, bv[c].x, t);
        t = fmaf(av[r].y, bv[c].y, t);
        t = fmaf(av[r].z, bv[c].z, t);
        acc[r][c] = fmaf(av[r].w, bv[c].w, t);
      }
    }
  }
}

// Adds the warps' copies (both halves) in a fixed order: out[o * C + i] and
// out[C * C + o].  `red` holds kPwThreads / 32 * (C * C + C) floats and may
// alias the chunk's rows (a barrier is taken first).
template <int C>
__device__ __forceinline__ void outer_store(float (&acc)[C / 4][C / 4], float (&row)[C / 4],
                                            float *red, float *out) {
  constexpr int TO = C / 4, NG = C * C + C, NW = kPwThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int o0 = (lane >> 2) & 3, i0 = lane & 3;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < TO; r++) {
    const float rs = row[r] + __shfl_down_sync(0xffffffffu, row[r], 16);
    if (lane < 16 && (lane & 3) == 0) red[warp * NG + C * C + o0 + 4 * r] = rs;
#pragma unroll
    for (int c = 0; c < TO; c++) {
      const float x = acc[r][c] + __shfl_down_sync(0xffffffffu, acc[r][c], 16);
      if (lane < 16) red[warp * NG + (o0 + 4 * r) * C + i0 + 4 * c] = x;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < NG; t += kPwThreads) {
    float x = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) x += red[w * NG + t];
    out[t] = x;
  }
}

// hb[i] += sum_o W[o][i] zb (two points), W from shared memory.
template <int C>
__device__ __forceinline__ void add_row(const float *Wo, float2 zb, float2 (&hb)[C]) {
#pragma unroll
  for (int i4 = 0; i4 < C / 4; i4++) {
    const float4 w = reinterpret_cast<const float4 *>(Wo)[i4];
    hb[4 * i4].x = fmaf(w.x, zb.x, hb[4 * i4].x);
    hb[4 * i4].y = fmaf(w.x, zb.y, hb[4 * i4].y);
    hb[4 * i4 + 1].x = fmaf(w.y, zb.x, hb[4 * i4 + 1].x);
    hb[4 * i4 + 1].y = fmaf(w.y, zb.y, hb[4 * i4 + 1].y);
    hb[4 * i4 + 2].x = fmaf(w.z, zb.x, hb[4 * i4 + 2].x);
    hb[4 * i4 + 2].y = fmaf(w.z, zb.y, hb[4 * i4 + 2].y);
    hb[4 * i4 + 3].x = fmaf(w.w, zb.x, hb[4 * i4 + 3].x);
    hb[4 * i4 + 3].y = fmaf(w.w, zb.y, hb[4 * i4 + 3].y);
  }
}

template <int C> constexpr size_t pw_bwd_smem() {
  return sizeof(float) * ((size_t)C * C + 2 * C * kCS);
}

// Backward of the projection and loss (loss = sum w (y - t)^2 / sum w).
// hbar[j][r] = sum_c Q1[c][j] zbar_c with zbar_c = ybar Q2[c] gelu'(zq_c),
// ybar = 2 w (y - t) / W.  Per-block partials [Q1 (C*C), q1 (C), Q2 (C), q2].
// N^3 is a multiple of 64, so a thread's two points are both inside or both
// outside.  Bound by its five C x N^3 passes (3 read, 1 written) and the
// activation's arithmetic: 414 -> 81 us at 96^3, C = 16 (a quarter of the
// threads formed the points and each weight product read two shared words).
template <int C>
__global__ void __launch_bounds__(kPwThreads) k_project_bwd(
    const float *__restrict__ h, const float *__restrict__ zq, const float *__restrict__ y,
    const float *__restrict__ target, const float *__restrict__ w,
    const float *__restrict__ invWp, const __nv_bfloat16 *__restrict__ Q1,
    const __nv_bfloat16 *__restrict__ Q2, float *__restrict__ hbar, float *__restrict__ part,
    long long NR) {
  constexpr int NG = C * C + 2 * C + 1;
  extern __shared__ __align__(16) float sm[];
  float *Q1s = sm;
  float(*zbs)[kCS] = reinterpret_cast<float(*)[kCS]>(sm + C * C);
  float(*hs)[kCS] = zbs + C;
  __shared__ float Q2s[C], red2[kPwThreads / 32][C + 1];
  for (int i = threadIdx.x; i < C * C; i += blockDim.x) Q1s[i] = bf(Q1, i);
  for (int i = threadIdx.x; i < C; i += blockDim.x) Q2s[i] = bf(Q2, i);
  const float invW = *invWp;
  float acc[C / 4][C / 4] = {}, row[C / 4] = {}, ga[C] = {}, ya = 0.f;
  const long long nchunks = (NR + kChunk - 1) / kChunk;
  for (long long ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    __syncthreads();
    const int p = 2 * threadIdx.x;
    const long long r = ch * kChunk + p;
    const bool in = r < NR;
    float2 yb = make_float2(0.f, 0.f), hb[C];
    if (in) {
      const float2 wr = w ? *reinterpret_cast<const float2 *>(w + r) : make_float2(1.f, 1.f);
      const float2 yv = *reinterpret_cast<const float2 *>(y + r);
      const float2 tv = *reinterpret_cast<const float2 *>(target + r);
      yb = make_float2(2.f * wr.x * (yv.x - tv.x) * invW, 2.f * wr.y * (yv.y - tv.y) * invW);
    }
    ya += yb.x + yb.y;
#pragma unroll
    for (int i = 0; i < C; i++) {
      hb[i] = make_float2(0.f, 0.f);
      *reinterpret_cast<float2 *>(&hs[i][p]) =
          in ? *reinterpret_cast<const float2 *>(h + (size_t)i * NR + r) : hb[i];
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
      const float2 a = in ? *reinterpret_cast<const float2 *>(zq + (size_t)c * NR + r)
                          : make_float2(0.f, 0.f);
      ga[c] += yb.x * gelu(a.x) + yb.y * gelu(a.y);
      const float2 zb =
          make_float2(yb.x * Q2s[c] * gelu_d(a.x), yb.y * Q2s[c] * gelu_d(a.y));
      *reinterpret_cast<float2 *>(&zbs[c][p]) = zb;
      add_row<C>(Q1s + c * C, zb, hb);
    }
    if (in) {
#pragma unroll
      for (int i = 0; i < C; i++) *reinterpret_cast<float2 *>(hbar + (size_t)i * NR + r) = hb[i];
    }
    __syncthreads();
    outer_accumulate<C>(zbs, hs, acc, row);
  }
  float *out = part + (size_t)blockIdx.x * NG;
  outer_store<C>(acc, row, &zbs[0][0], out);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c <= C; c++) {
    float x = c < C ? ga[c < C ? c : 0] : ya;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red2[warp][c] = x;
  }
  __syncthreads();
  for (int c = threadIdx.x; c <= C; c += blockDim.x) {
    float x = 0.f;
    for (int k = 0; k < kPwThreads / 32; k++) x += red2[k][c];
    out[C * C + C + c] = x;
  }
}

// Backward of a layer's pointwise part: zbar = hbar * act'(z) (written to
// zbar), hprev_bar[i][r] = sum_o Wp[o][i] zbar[o][r] (written), per-block
// partials [Wp (C*C), b (C)].  Bound by its five C x N^3 passes (3 read, 2
// written) and the activation's arithmetic: 464 -> 92 us at 96^3, C = 16.
template <int C>
__global__ void __launch_bounds__(kPwThreads) k_layer_pw_bwd(
    const float *__restrict__ hbar, const float *__restrict__ z, const float *__restrict__ hprev,
    const __nv_bfloat16 *__restrict__ Wp, float *__restrict__ zbar, float *__restrict__ hprev_bar,
    float *__restrict__ part, long long NR, int act) {
  extern __shared__ __align__(16) float sm[];
  float *Ws = sm;
  float(*zbs)[kCS] = reinterpret_cast<float(*)[kCS]>(sm + C * C);
  float(*hs)[kCS] = zbs + C;
  for (int i = threadIdx.x; i < C * C; i += blockDim.x) Ws[i] = bf(Wp, i);
  float acc[C / 4][C / 4] = {}, row[C / 4] = {};
  const long long nchunks = (NR + kChunk - 1) / kChunk;
  for (long long ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    __syncthreads();
    const int p = 2 * threadIdx.x;
    const long long r = ch * kChunk + p;
    const bool in = r < NR;
    float2 hb[C];
#pragma unroll
    for (int i = 0; i < C; i++) {
      hb[i] = make_float2(0.f, 0.f);
      *reinterpret_cast<float2 *>(&hs[i][p]) =
          in ? *reinterpret_cast<const float2 *>(hprev + (size_t)i * NR + r) : hb[i];
    }
#pragma unroll 4
    for (int o = 0; o < C; o++) {
      float2 zb = make_float2(0.f, 0.f);
      if (in) {
        zb = *reinterpret_cast<const float2 *>(hbar + (size_t)o * NR + r);
        if (act) {
          const float2 zv = *reinterpret_cast<const float2 *>(z + (size_t)o * NR + r);
          zb.x *= gelu_d(zv.x);
          zb.y *= gelu_d(zv.y);
        }
        *reinterpret_cast<float2 *>(zbar + (size_t)o * NR + r) = zb;
      }
      *reinterpret_cast<float2 *>(&zbs[o][p]) = zb;
      add_row<C>(Ws + o * C, zb, hb);
    }
    if (in) {
#pragma unroll
      for (int i = 0; i < C; i++)
        *reinterpret_cast<float2 *>(hprev_bar + (size_t)i * NR + r) = hb[i];
    }
    __syncthreads();
    outer_accumulate<C>(zbs, hs, acc, row);
  }
  outer_store<C>(acc, row, &zbs[0][0], part + (size_t)blockIdx.x * (C * C + C));
}

// Lift backward partials: [P (2C), p (C)].
template <int C>
__global__ void k_lift_bwd(const float *__restrict__ hbar, const float *__restrict__ mask, float eta,
                           float *__restrict__ part, long long NR) {
  constexpr int NG = 3 * C;
  float g[NG];
#pragma unroll
  for (int k = 0; k < NG; k++) g[k] = 0.f;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < NR;
       r += (long long)gridDim.x * blockDim.x) {
    const float m = mask[r];
#pragma unroll
    for (int c = 0; c < C; c++) {
      const float hb = hbar[(size_t)c * NR + r];
      g[2 * c] += hb * m;
      g[2 * c + 1] += hb * eta;
      g[2 * C + c] += hb;
    }
  }
  block_sum_store<NG>(g, part);
}

// Sums per-block partials [nblk][K] in a fixed order into grad (+=): a block
// of 32 x 32 threads takes 32 columns, each thread every 32nd row, the 32 row
// sums of a column added in order (one thread per column walking all rows
// was latency-bound: 466 us at 3456 x 272 against 14 us at 608 x 272).
__global__ void __launch_bounds__(1024) k_sum_partials(const float *__restrict__ part, int nblk,
                                                       int K, float *__restrict__ grad) {
  __shared__ double red[32][33];
  const int k = blockIdx.x * 32 + threadIdx.x;
  double s = 0;
  if (k < K) {
#pragma unroll 4
    for (int b = threadIdx.y; b < nblk; b += 32) s += part[(size_t)b * K + k];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && k < K) {
    for (int w = 1; w < 32; w++) s += red[w][threadIdx.x];
    grad[k] += (float)s;
  }
}

// loss[0] = sum w (y - t)^2 / sum w and loss[1] = 1 / sum w from the
// projection's per-block sums (FP64, fixed order; a weight sum of 0 counts
// as 1), left on the device for the backward pass.
__global__ void __launch_bounds__(256) k_loss(const float *__restrict__ part, int nblk,
                                              float *__restrict__ loss) {
  __shared__ double red[2][256];
  double s = 0, w = 0;
  for (int b = threadIdx.x; b < nblk; b += 256) {
    s += part[2 * b];
    w += part[2 * b + 1];
  }
  red[0][threadIdx.x] = s;
  red[1][threadIdx.x] = w;
  for (int o = 128; o > 0; o >>= 1) {
    __syncthreads();
    if (threadIdx.x < o) {
      red[0][threadIdx.x] += red[0][threadIdx.x + o];
      red[1][threadIdx.x] += red[1][threadIdx.x + o];
    }
  }
  if (threadIdx.x == 0) {
    const double W = red[1][0] > 0 ? red[1][0] : 1;
    loss[0] = (float)(red[0][0] / W);
    loss[1] = (float)(1.0 / W);
  }
}

// Adam on the FP32 masters, then the BF16 copies.
__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, __nv_bfloat16 *__restrict__ pb, long long n,
                       float lr, float b1, float b2, float eps, float c1, float c2) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1 - b1) * gi;
    const float vi = b2 * v[i] + (1 - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    p[i] = pi;
    pb[i] = __float2bfloat16_rn(pi);
  }
}

__global__ void k_to_bf16(const float *__restrict__ p, __nv_bfloat16 *__restrict__ pb, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    pb[i] = __float2bfloat16_rn(p[i]);
}

__global__ void k_fill(float *p, float v, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    p[i] = v;
}

// n = nb * max(y, floor) on free points, 0 in the walls (double output).
__global__ void k_density(const float *__restrict__ y, const double *__restrict__ mask, double nb,
                          double floor_rel, double *__restrict__ n, long long NR) {
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < NR;
       r += (long long)gridDim.x * blockDim.x) {
    const double m = mask ? mask[r] : 1.0;
    const double yr = (double)y[r];
    // a NaN estimate stays NaN (the checked warm start then rejects it)
    n[r] = m == 0 ? 0.0 : m * nb * (yr > floor_rel || yr != yr ? yr : floor_rel);
  }
}

constexpr int kNormBlocks = 256;

// Per-block sums of squares (FP64, fixed order) over a strided range.
__global__ void k_norm2_partial(const double *__restrict__ v, long long n, double *__restrict__ out) {
  __shared__ double red[kT / 32];
  double s = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    s += v[i] * v[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    out[blockIdx.x] = t;
  }
}

// Bulk start: nb on free points, 0 in the walls.
__global__ void k_bulk(const double *__restrict__ mask, double nb, double *__restrict__ n,
                       long long NR) {
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < NR;
       r += (long long)gridDim.x * blockDim.x)
    n[r] = mask[r] == 0 ? 0.0 : mask[r] * nb;
}

__global__ void k_d2f(const double *__restrict__ a, float *__restrict__ b, long long n, float s) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    b[i] = (float)(a[i] * s);
}

int grid_for(long long n) {
  long long b = (n + kT - 1) / kT;
  return (int)(b < 4096 ? (b < 1 ? 1 : b) : 4096);
}

}  // namespace

struct deft_fno {
  int device = 0;
  cudaStream_t stream = nullptr;
  int N = 0, C = 0, m = 0, L = 0;
  int Kx = 0, Ky = 0, Kz = 0, K = 0;
  long long NR = 0;
  // parameters (FP32 masters, BF16 copies, grads, Adam moments)
  size_t nparam = 0;
  float *p = nullptr, *g = nullptr, *am = nullptr, *av = nullptr;
  __nv_bfloat16 *pb = nullptr;
  long long adam_t = 0;
  // offsets into the parameter vector
  size_t oP = 0, op = 0, oQ1 = 0, oq1 = 0, oQ2 = 0, oq2 = 0;
  std::vector<size_t> oW, oWp, ob;
  // DFT tables
  float2 *Ezf = nullptr;  // [N][Kz] forward z, scale 1
  float2 *Ezb = nullptr;  // [N][Kz] forward z with the synthesis scale c_k / N^3 (adjoint use)
  float2 *Gzi = nullptr;  // [N][Kz] synthesis c_k / N^3
  float2 *Gza = nullptr;  // [N][Kz] adjoint of the forward z transform (c = 1, s = 1)
  float2 *Eyf = nullptr, *Eyi = nullptr, *Exf = nullptr, *Exi = nullptr;
  float2 *Yc = nullptr;  // [N][m + 1] (cos, sin) of the slab kernels
  bool slab = false;      // slab kernels for the z and y axes
  // activations
  std::vector<float *> h, z;  // h[0..L], z[0..L-1]
  std::vector<float2 *> V;    // V[l] spectral inputs per layer
  float *zq = nullptr, *y = nullptr, *mask = nullptr, *target = nullptr, *wt = nullptr;
  float2 *A = nullptr, *B = nullptr, *S = nullptr, *S2 = nullptr;
  float *hb0 = nullptr, *hb1 = nullptr, *zb = nullptr;
  float *part = nullptr;
  float *loss_d = nullptr;   // loss and 1 / sum of its weights (k_loss)
  double *bulk = nullptr;    // 2 N^3 doubles (bulk start, its gradient), allocated on first use
  double *part_d = nullptr;  // kNormBlocks FP64 partial sums
  long long launches = 0;    // kernel launches queued so far
  int nblk = 0;
  int bwd_blk = 0;           // blocks of the pointwise backward kernels
  std::string err;
};

namespace {

int fno_fail(deft_fno *f, const std::string &m, int code = DEFT_ERR_CUDA) {
  f->err = m;
  deft::set_last_error_message(m);
  return code;
}

int check(deft_fno *f, const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fno_fail(f, std::string(what) + ": " + cudaGetErrorString(e));
  return DEFT_OK;
}

size_t smem_z_fwd(int N, int Kz) {
  return sizeof(float) * kZfLines * (N + 4) + sizeof(float2) * N * Kz;
}

// Kz rounded up to the register tile of the z transforms (4, 8, 12, 16).
int kz_block(int Kz) { return (Kz + 3) / 4 * 4; }

void launch_z_fwd(deft_fno *f, const float *in, float2 *out, const float2 *E) {
  const int L = f->C * f->N * f->N;
  const dim3 grid((L + kZfLines - 1) / kZfLines);
  const size_t sm = smem_z_fwd(f->N, f->Kz);
  switch (kz_block(f->Kz)) {
    case 4: k_dft_z_fwd<4><<<grid, 128, sm, f->stream>>>(in, out, E, L, f->N, f->Kz); break;
    case 8: k_dft_z_fwd<8><<<grid, 128, sm, f->stream>>>(in, out, E, L, f->N, f->Kz); break;
    case 12: k_dft_z_fwd<12><<<grid, 128, sm, f->stream>>>(in, out, E, L, f->N, f->Kz); break;
    default: k_dft_z_fwd<16><<<grid, 128, sm, f->stream>>>(in, out, E, L, f->N, f->Kz); break;
  }
}
void launch_z_inv(deft_fno *f, const float2 *in, float *out, const float2 *G, int acc) {
  const int L = f->C * f->N * f->N;
  const dim3 grid((L + kZiLines - 1) / kZiLines);
  switch (kz_block(f->Kz)) {
    case 4: k_dft_z_inv<4><<<grid, 128, 0, f->stream>>>(in, out, G, L, f->N, f->Kz, acc); break;
    case 8: k_dft_z_inv<8><<<grid, 128, 0, f->stream>>>(in, out, G, L, f->N, f->Kz, acc); break;
    case 12: k_dft_z_inv<12><<<grid, 128, 0, f->stream>>>(in, out, G, L, f->N, f->Kz, acc); break;
    default: k_dft_z_inv<16><<<grid, 128, 0, f->stream>>>(in, out, G, L, f->N, f->Kz, acc); break;
  }
}
void launch_axis(deft_fno *f, const float2 *in, float2 *out, const float2 *E, int outer, int Nin,
                 int Mout, int inner) {
  // tiles of up to 32 columns (a whole slab when inner <= 32) while they fit
  const int IC = inner < 32 ? inner : 32;
  const size_t sm = sizeof(float2) * ((size_t)ax_rows(Mout) * Nin + (size_t)Nin * IC);
  if (sm <= 96 * 1024) {
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    // tiles per block pass: fill the 256 threads when a tile has few items
    const int per = (ax_rows(Mout) / kAxMR) * IC;
    int S = per >= 256 ? 1 : 256 / per;
    while (S > 1 && sm + sizeof(float2) * (size_t)(S - 1) * Nin * IC > 96 * 1024) S--;
    const size_t sm2 = sm + sizeof(float2) * (size_t)(S - 1) * Nin * IC;
    const int tiles = (outer * ((inner + IC - 1) / IC) + S - 1) / S;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // as many resident blocks as shared memory and registers allow: the
    // staging loads of one pass are not overlapped with its multiply-adds,
    // so other resident blocks hide them
    int bps = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_dft_tile, 256, sm2) !=
            cudaSuccess ||
        bps < 1) {
      cudaGetLastError();  // the query's own error, if any, is not the launch's
      bps = 2;
    }
    int grid = bps * (sms > 0 ? sms : 148);
    if (grid > tiles) grid = tiles;
    k_dft_tile<<<grid, 256, sm2, f->stream>>>(in, out, E, outer, Nin, Mout, inner, IC, S);
    return;
  }
  const long long total = (long long)outer * Mout * inner;
  k_dft_axis<<<grid_for(total), kT, sizeof(float2) * Mout * Nin, f->stream>>>(in, out, E, outer,
                                                                              Nin, Mout, inner);
}

// Calls g(std::integral_constant<int, KB>()) with Kz rounded up to the register tile.
template <typename F> void with_kb(int Kz, F &&g) {
  switch (kz_block(Kz)) {
    case 4: g(std::integral_constant<int, 4>()); break;
    case 8: g(std::integral_constant<int, 8>()); break;
    case 12: g(std::integral_constant<int, 12>()); break;
    default: g(std::integral_constant<int, 16>()); break;
  }
}

// z (table E) and y analysis of C fields: f->B [C N Ky Kz].
void analyse_zy(deft_fno *f, const float *in, const float2 *E) {
  const int C = f->C, N = f->N;
  f->launches++;
  if (!f->slab) {
    f->launches++;
    launch_z_fwd(f, in, f->A, E);                                // [C N N Kz]
    launch_axis(f, f->A, f->B, f->Eyf, C * N, N, f->Ky, f->Kz);  // [C N Ky Kz]
    return;
  }
  with_kb(f->Kz, [&](auto kb) {
    constexpr int KB = decltype(kb)::value;
    const size_t sm = slab_fwd_smem(N, f->m, KB);
    k_slab_fwd<KB><<<C * N, 64 * slab_chunks(N), sm, f->stream>>>(in, f->B, E, f->Yc, N, f->Kz,
                                                                  f->m);
  });
}
// y and z (table G) synthesis of f->B into C fields.
void synthesise_yz(deft_fno *f, float *out, const float2 *G, int accumulate) {
  const int C = f->C, N = f->N;
  f->launches++;
  if (!f->slab) {
    f->launches++;
    launch_axis(f, f->B, f->A, f->Eyi, C * N, f->Ky, N, f->Kz);  // [C N N Kz]
    launch_z_inv(f, f->A, out, G, accumulate);
    return;
  }
  with_kb(f->Kz, [&](auto kb) {
    constexpr int KB = decltype(kb)::value;
    const size_t sm = slab_inv_smem(N, f->m, KB);
    k_slab_inv<KB><<<C * N, 128, sm, f->stream>>>(f->B, out, G, f->Yc, N, f->Kz, f->m, accumulate);
  });
}

// Forward through the spectral part of layer l up to the x synthesis: its
// coefficients in f->B.
void spectral_fwd(deft_fno *f, int l, const float *hin) {
  const int C = f->C, N = f->N;
  analyse_zy(f, hin, f->Ezf);
  launch_axis(f, f->B, f->V[l], f->Exf, C, N, f->Kx, f->Ky * f->Kz);  // [C Kx Ky Kz]
  k_spec_mix<<<(C * f->K + kT - 1) / kT, kT, 0, f->stream>>>(f->V[l], f->pb + f->oW[l], f->S, C,
                                                              f->K);
  launch_axis(f, f->S, f->B, f->Exi, C, f->Kx, N, f->Ky * f->Kz);  // [C N Ky Kz]
  f->launches += 3;
}

// The inference layer: y and z synthesis fused with the pointwise layer (slab
// grids), else the z synthesis fused with it.
template <int C>
void launch_layer_synth(deft_fno *f, int l) {
  const int N = f->N, half = N / 2, lpb = 256 / half, act = l < f->L - 1 ? 1 : 0;
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  f->launches++;
  if (f->slab) {
    const size_t sm = synth_smem<C>(N, f->m, f->Kz);
    // blocks per x: the fewest rounds of two blocks per SM (also assumed where
    // only one fits), a round costing its passes and about two more for the
    // block's tables
    const int most = (N + lpb - 1) / lpb;
    int share = 1, best = 0;
    for (int k = 1; k <= most && k <= 16; k++) {
      const int cost = (N * k + 2 * sms - 1) / (2 * sms) * (((N + k - 1) / k + lpb - 1) / lpb + 2);
      if (k == 1 || cost < best) {
        best = cost;
        share = k;
      }
    }
    k_layer_synth<C><<<dim3(N, share), 256, sm, f->stream>>>(
        f->B, f->Gzi, f->Yc, f->h[l], f->h[l + 1], f->pb + f->oWp[l], f->pb + f->ob[l], N, f->Kz,
        f->m, act);
    return;
  }
  f->launches++;
  launch_axis(f, f->B, f->A, f->Eyi, C * N, f->Ky, N, f->Kz);  // [C N N Kz]
  const size_t sm = sizeof(float) * (C * C + ((C + 3) & ~3)) +
                    sizeof(float2) * ((size_t)f->Kz * N + (size_t)lpb * C * f->Kz);
  const int lines = N * N;
  int grid = 4 * sms;
  const int need = (lines + lpb - 1) / lpb;
  if (grid > need) grid = need;
  k_layer_synth_pw<C><<<grid, 256, sm, f->stream>>>(f->A, f->Gzi, f->h[l], f->h[l + 1],
                                                    f->pb + f->oWp[l], f->pb + f->ob[l], N, f->Kz,
                                                    act);
}

// A kernel's shared-memory cap: the device's maximum, whatever this network
// needs.  The cap belongs to the function, which networks of other sizes launch
// too, from other threads.
template <typename K> cudaError_t full_smem(K kernel) {
  cudaFuncAttributes fa;
  int dev = 0, most = 0;
  cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             most - (int)fa.sharedSizeBytes);
  return e;
}
template <int C> cudaError_t synth_caps() {
  const cudaError_t e = full_smem(k_layer_synth<C>);
  return e == cudaSuccess ? full_smem(k_layer_synth_pw<C>) : e;
}
// The caps of the kernels a network launches, for the current device.
cudaError_t kernel_caps(const deft_fno *f) {
  cudaError_t e = full_smem(k_dft_axis);
  if (e == cudaSuccess) e = full_smem(k_dft_tile);
  with_kb(f->Kz, [&](auto kb) {
    constexpr int KB = decltype(kb)::value;
    if (e == cudaSuccess) e = full_smem(k_dft_z_fwd<KB>);
    if (e == cudaSuccess) e = full_smem(k_slab_fwd<KB>);
    if (e == cudaSuccess) e = full_smem(k_slab_inv<KB>);
  });
  if (e != cudaSuccess) return e;
  return f->C == 16 ? synth_caps<16>() : f->C == 8 ? synth_caps<8>() : synth_caps<4>();
}

// Adjoint of the spectral part for upstream zbar: adds K^T zbar to hin_bar and
// accumulates W grads.
void spectral_bwd(deft_fno *f, int l, const float *zbar, float *hin_bar) {
  const int C = f->C, N = f->N;
  analyse_zy(f, zbar, f->Ezb);                                      // B'bar
  launch_axis(f, f->B, f->S, f->Exf, C, N, f->Kx, f->Ky * f->Kz);   // Ubar
  k_spec_mix_bwd<<<(C * f->K + kT - 1) / kT, kT, 0, f->stream>>>(
      f->V[l], f->pb + f->oW[l], f->S, f->S2, f->g + f->oW[l], C, f->K);  // Vbar
  launch_axis(f, f->S2, f->B, f->Exi, C, f->Kx, N, f->Ky * f->Kz);  // Bbar
  synthesise_yz(f, hin_bar, f->Gza, 1);
  f->launches += 3;
}

template <int C>
void launch_layer_pw(deft_fno *f, int l, int store_z) {
  k_layer_pw<C><<<grid_for(f->NR / 4), kT, 0, f->stream>>>(f->h[l], f->z[l], f->h[l + 1],
                                                       f->pb + f->oWp[l], f->pb + f->ob[l], f->NR,
                                                       l < f->L - 1 ? 1 : 0, store_z);
}

template <int C>
void launch_project(deft_fno *f, float *zq, const float *target, const float *w, float *part) {
  k_project<C><<<f->nblk, kT, 0, f->stream>>>(f->h[f->L], f->pb + f->oQ1, f->pb + f->oq1,
                                              f->pb + f->oQ2, f->pb + f->oq2, zq, f->y, target, w,
                                              part, f->NR);
}

void project(deft_fno *f, float *zq, const float *target, const float *w, float *part) {
  f->launches++;
  if (f->C == 16) launch_project<16>(f, zq, target, w, part);
  else if (f->C == 8) launch_project<8>(f, zq, target, w, part);
  else launch_project<4>(f, zq, target, w, part);
}

// Forward through the Fourier layers; `train` keeps the pre-activations the
// backward pass reads.
int forward(deft_fno *f, float eta, bool train) {
  const int C = f->C;
  f->launches++;  // lift
  k_lift<<<grid_for(f->NR), kT, 0, f->stream>>>(f->mask, eta, f->pb + f->oP, f->pb + f->op, f->h[0],
                                               C, f->NR);
  for (int l = 0; l < f->L; l++) {
    spectral_fwd(f, l, f->h[l]);
    if (!train) {
      // inference: no z field for a backward pass
      if (C == 16) launch_layer_synth<16>(f, l);
      else if (C == 8) launch_layer_synth<8>(f, l);
      else launch_layer_synth<4>(f, l);
      continue;
    }
    synthesise_yz(f, f->z[l], f->Gzi, 0);
    f->launches++;
    if (C == 16) launch_layer_pw<16>(f, l, 1);
    else if (C == 8) launch_layer_pw<8>(f, l, 1);
    else launch_layer_pw<4>(f, l, 1);
  }
  return check(f, "fno forward");
}

}  // namespace

extern "C" {

int deft_fno_create(int device, int N, int channels, int modes, int layers, unsigned long long seed,
                    deft_fno **out) {
  if (!out || N < 4 || N % 4 != 0 || (channels != 16 && channels != 4 && channels != 8) || modes < 1 ||
      modes > kMaxKz || 2 * modes > N || layers < 1 || layers > 8)
    return DEFT_ERR_ARG;
  deft_fno *f = new deft_fno();
  f->device = device;
  if (cudaSetDevice(device) != cudaSuccess ||
      cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete f;
    return DEFT_ERR_CUDA;
  }
  f->N = N;
  f->C = channels;
  f->m = modes;
  f->L = layers;
  f->Kx = f->Ky = 2 * modes;
  f->Kz = modes;
  f->K = f->Kx * f->Ky * f->Kz;
  f->NR = (long long)N * N * N;
  const int C = channels;
  // parameter layout
  size_t off = 0;
  f->oP = off; off += 2 * C;
  f->op = off; off += C;
  for (int l = 0; l < layers; l++) {
    f->oW.push_back(off); off += (size_t)2 * C * C * f->K;
    f->oWp.push_back(off); off += (size_t)C * C;
    f->ob.push_back(off); off += C;
  }
  f->oQ1 = off; off += (size_t)C * C;
  f->oq1 = off; off += C;
  f->oQ2 = off; off += C;
  f->oq2 = off; off += 1;
  f->nparam = off;
  // initial weights (seeded): spectral ~ U(0, 1/(C C)) as in the FNO paper,
  // pointwise ~ U(-1/sqrt(fan_in), 1/sqrt(fan_in)), biases 0, q2 = 1 (bulk)
  std::vector<float> hp(off, 0.f);
  std::mt19937_64 rng(seed);
  std::uniform_real_distribution<float> U01(0.f, 1.f);
  auto fill_u = [&](size_t o, size_t n, float a) {
    for (size_t i = 0; i < n; i++) hp[o + i] = (2 * U01(rng) - 1) * a;
  };
  fill_u(f->oP, 2 * C, 1.f / std::sqrt(2.f));
  for (int l = 0; l < layers; l++) {
    const float s = 1.f / (C * C);
    for (size_t i = 0; i < (size_t)2 * C * C * f->K; i++) hp[f->oW[l] + i] = s * U01(rng);
    fill_u(f->oWp[l], (size_t)C * C, 1.f / std::sqrt((float)C));
  }
  fill_u(f->oQ1, (size_t)C * C, 1.f / std::sqrt((float)C));
  fill_u(f->oQ2, C, 0.1f / std::sqrt((float)C));
  hp[f->oq2] = 1.f;
  // DFT tables
  auto cexp = [&](double ang) { return make_float2((float)std::cos(ang), (float)std::sin(ang)); };
  const double tp = 6.283185307179586476925286766559;
  auto kid = [&](int k) { return k < modes ? k : N - 2 * modes + k; };
  const double N3 = (double)N * N * N;
  std::vector<float2> ezf(N * f->Kz), ezb(N * f->Kz), gzi(f->Kz * N), gza(f->Kz * N);
  for (int z = 0; z < N; z++)
    for (int k = 0; k < f->Kz; k++) {
      const double a = tp * k * z / N;
      const double ck = k == 0 ? 1.0 : 2.0;
      ezf[z * f->Kz + k] = cexp(-a);
      const float2 e = cexp(-a);
      ezb[z * f->Kz + k] = make_float2((float)(e.x * ck / N3), (float)(e.y * ck / N3));
      const float2 gg = cexp(a);
      gzi[z * f->Kz + k] = make_float2((float)(gg.x * ck / N3), (float)(gg.y * ck / N3));
      gza[z * f->Kz + k] = gg;
    }
  std::vector<float2> eyf(f->Ky * N), eyi(N * f->Ky), exf(f->Kx * N), exi(N * f->Kx);
  for (int k = 0; k < f->Ky; k++)
    for (int n = 0; n < N; n++) {
      const double a = tp * (double)kid(k) * n / N;
      eyf[k * N + n] = cexp(-a);
      eyi[n * f->Ky + k] = cexp(a);
      exf[k * N + n] = cexp(-a);
      exi[n * f->Kx + k] = cexp(a);
    }
  bool ok = true;
  auto dev = [&](auto **ptr, size_t bytes) {
    if (ok && deft::dev_malloc((void **)ptr, bytes) != cudaSuccess) ok = false;
  };
  const size_t pf = sizeof(float) * off;
  dev(&f->p, pf);
  dev(&f->g, pf);
  dev(&f->am, pf);
  dev(&f->av, pf);
  dev(&f->pb, sizeof(__nv_bfloat16) * off);
  dev(&f->Ezf, sizeof(float2) * ezf.size());
  dev(&f->Ezb, sizeof(float2) * ezb.size());
  dev(&f->Gzi, sizeof(float2) * gzi.size());
  dev(&f->Gza, sizeof(float2) * gza.size());
  dev(&f->Eyf, sizeof(float2) * eyf.size());
  dev(&f->Eyi, sizeof(float2) * eyi.size());
  dev(&f->Exf, sizeof(float2) * exf.size());
  dev(&f->Exi, sizeof(float2) * exi.size());
  f->slab = slab_ok(N, modes);
  std::vector<float2> yc((size_t)N * (modes + 1));
  for (int n = 0; n < N; n++)
    for (int k = 0; k <= modes; k++) yc[(size_t)n * (modes + 1) + k] = cexp(tp * (double)((long long)k * n % N) / N);
  dev(&f->Yc, sizeof(float2) * yc.size());
  const size_t act = sizeof(float) * C * f->NR;
  f->h.resize(layers + 1);
  f->z.resize(layers);
  f->V.resize(layers);
  for (int l = 0; l <= layers; l++) dev(&f->h[l], act);
  for (int l = 0; l < layers; l++) {
    dev(&f->z[l], act);
    dev(&f->V[l], sizeof(float2) * C * f->K);
  }
  dev(&f->zq, act);
  dev(&f->y, sizeof(float) * f->NR);
  dev(&f->mask, sizeof(float) * f->NR);
  dev(&f->target, sizeof(float) * f->NR);
  dev(&f->wt, sizeof(float) * f->NR);
  if (!f->slab) dev(&f->A, sizeof(float2) * C * N * N * f->Kz);  // between the z and y axes
  dev(&f->B, sizeof(float2) * C * N * f->Ky * f->Kz);
  dev(&f->S, sizeof(float2) * C * f->K);
  dev(&f->S2, sizeof(float2) * C * f->K);
  dev(&f->hb0, act);
  dev(&f->hb1, act);
  dev(&f->zb, act);
  f->nblk = grid_for(f->NR);
  dev(&f->part, sizeof(float) * (size_t)f->nblk * (C * C + 2 * C + 1 + 8));
  {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int nch = (int)((f->NR + kChunk - 1) / kChunk);
    f->bwd_blk = 4 * (sms > 0 ? sms : 148);
    if (f->bwd_blk > nch) f->bwd_blk = nch;
    if (f->bwd_blk > f->nblk) f->bwd_blk = f->nblk;
  }
  dev(&f->loss_d, 2 * sizeof(float));
  dev(&f->part_d, sizeof(double) * kNormBlocks);
  if (!ok) {
    deft_fno_destroy(f);
    return DEFT_ERR_NOMEM;
  }
  cudaMemcpy(f->p, hp.data(), pf, cudaMemcpyHostToDevice);
  cudaMemset(f->am, 0, pf);
  cudaMemset(f->av, 0, pf);
  cudaMemset(f->g, 0, pf);
  cudaMemcpy(f->Ezf, ezf.data(), sizeof(float2) * ezf.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(f->Ezb, ezb.data(), sizeof(float2) * ezb.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(f->Gzi, gzi.data(), sizeof(float2) * gzi.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(f->Gza, gza.data(), sizeof(float2) * gza.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(f->Eyf, eyf.data(), sizeof(float2) * eyf.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(f->Eyi, eyi.data(), sizeof(float2) * eyi.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(f->Exf, exf.data(), sizeof(float2) * exf.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(f->Exi, exi.data(), sizeof(float2) * exi.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(f->Yc, yc.data(), sizeof(float2) * yc.size(), cudaMemcpyHostToDevice);
  if (kernel_caps(f) != cudaSuccess) {
    check(f, "fno shared memory");
    deft_fno_destroy(f);
    return DEFT_ERR_CUDA;
  }
  k_to_bf16<<<grid_for((long long)off), kT, 0, f->stream>>>(f->p, f->pb, (long long)off);
  if (check(f, "fno create")) {
    deft_fno_destroy(f);
    return DEFT_ERR_CUDA;
  }
  cudaStreamSynchronize(f->stream);
  *out = f;
  return DEFT_OK;
}

int deft_fno_destroy(deft_fno *f) {
  if (!f) return DEFT_OK;
  cudaSetDevice(f->device);
  if (f->stream) cudaStreamSynchronize(f->stream);
  for (void *q : {(void *)f->p, (void *)f->g, (void *)f->am, (void *)f->av, (void *)f->pb,
                  (void *)f->Ezf, (void *)f->Ezb, (void *)f->Gzi, (void *)f->Gza, (void *)f->Eyf,
                  (void *)f->Eyi, (void *)f->Exf, (void *)f->Exi, (void *)f->Yc, (void *)f->zq, (void *)f->y,
                  (void *)f->mask, (void *)f->target, (void *)f->wt, (void *)f->A, (void *)f->B,
                  (void *)f->S, (void *)f->S2, (void *)f->hb0, (void *)f->hb1, (void *)f->zb,
                  (void *)f->part, (void *)f->loss_d, (void *)f->bulk, (void *)f->part_d})
    deft::dev_free(q);
  for (float *q : f->h) deft::dev_free(q);
  for (float *q : f->z) deft::dev_free(q);
  for (float2 *q : f->V) deft::dev_free(q);
  if (f->stream) cudaStreamDestroy(f->stream);
  delete f;
  return DEFT_OK;
}

size_t deft_fno_param_count(const deft_fno *f) { return f ? f->nparam : 0; }

// Parameters as FP32 masters (host arrays of deft_fno_param_count floats).
int deft_fno_get_params(deft_fno *f, float *host) {
  if (!f || !host) return DEFT_ERR_ARG;
  cudaSetDevice(f->device);
  cudaStreamSynchronize(f->stream);
  return cudaMemcpy(host, f->p, sizeof(float) * f->nparam, cudaMemcpyDeviceToHost) == cudaSuccess
             ? DEFT_OK
             : DEFT_ERR_CUDA;
}

int deft_fno_set_params(deft_fno *f, const float *host) {
  if (!f || !host) return DEFT_ERR_ARG;
  cudaSetDevice(f->device);
  cudaStreamSynchronize(f->stream);
  if (cudaMemcpy(f->p, host, sizeof(float) * f->nparam, cudaMemcpyHostToDevice) != cudaSuccess)
    return DEFT_ERR_CUDA;
  k_to_bf16<<<grid_for((long long)f->nparam), kT, 0, f->stream>>>(f->p, f->pb,
                                                                  (long long)f->nparam);
  f->adam_t = 0;
  cudaMemsetAsync(f->am, 0, sizeof(float) * f->nparam, f->stream);
  cudaMemsetAsync(f->av, 0, sizeof(float) * f->nparam, f->stream);
  if (int s = check(f, "set params")) return s;
  return cudaStreamSynchronize(f->stream) == cudaSuccess ? DEFT_OK : DEFT_ERR_CUDA;
}

}  // extern "C"

namespace {

void sum_partials(deft_fno *f, int nblk, int K, float *grad) {
  k_sum_partials<<<(K + 31) / 32, dim3(32, 32), 0, f->stream>>>(f->part, nblk, K, grad);
}

template <int C> void project_bwd(deft_fno *f) {
  k_project_bwd<C><<<f->bwd_blk, kPwThreads, pw_bwd_smem<C>(), f->stream>>>(
      f->h[f->L], f->zq, f->y, f->target, f->wt, f->loss_d + 1, f->pb + f->oQ1, f->pb + f->oQ2,
      f->hb0, f->part, f->NR);
  sum_partials(f, f->bwd_blk, C * C + 2 * C + 1, f->g + f->oQ1);
}

template <int C> void layer_pw_bwd(deft_fno *f, int l, const float *hb, float *hb_next) {
  k_layer_pw_bwd<C><<<f->bwd_blk, kPwThreads, pw_bwd_smem<C>(), f->stream>>>(
      hb, f->z[l], f->h[l], f->pb + f->oWp[l], f->zb, hb_next, f->part, f->NR,
      l < f->L - 1 ? 1 : 0);
  sum_partials(f, f->bwd_blk, C * C + C, f->g + f->oWp[l]);
}

// Forward pass (and, with want_grad, the backward pass into f->g) on one
// sample; mask / target / y_out are host or device arrays per `kind`.
int eval_impl(deft_fno *f, const float *mask, float eta, const float *target, cudaMemcpyKind kin,
              cudaMemcpyKind kout, float *y_out, float *loss, bool want_grad) {
  const int C = f->C;
  const size_t rb = sizeof(float) * f->NR;
  cudaMemcpyAsync(f->mask, mask, rb, kin, f->stream);
  if (target) {
    cudaMemcpyAsync(f->target, target, rb, kin, f->stream);
    cudaMemcpyAsync(f->wt, mask, rb, kin, f->stream);
  }
  if (int s = forward(f, eta, want_grad)) return s;
  project(f, f->zq, target ? f->target : nullptr, f->wt, target ? f->part : nullptr);
  if (target) {
    f->launches++;
    k_loss<<<1, 256, 0, f->stream>>>(f->part, f->nblk, f->loss_d);
  }
  if (y_out) cudaMemcpyAsync(y_out, f->y, rb, kout, f->stream);
  if (want_grad && target) {
    f->launches += 4 + 2 * f->L;  // projection, lift and pointwise backward passes with their sums
    cudaMemsetAsync(f->g, 0, sizeof(float) * f->nparam, f->stream);
    // projection
    if (C == 16) project_bwd<16>(f);
    else if (C == 8) project_bwd<8>(f);
    else project_bwd<4>(f);
    float *hb = f->hb0, *hb_next = f->hb1;
    for (int l = f->L - 1; l >= 0; l--) {
      if (C == 16) layer_pw_bwd<16>(f, l, hb, hb_next);
      else if (C == 8) layer_pw_bwd<8>(f, l, hb, hb_next);
      else layer_pw_bwd<4>(f, l, hb, hb_next);
      spectral_bwd(f, l, f->zb, hb_next);
      float *t = hb;
      hb = hb_next;
      hb_next = t;
    }
    if (C == 16)
      k_lift_bwd<16><<<f->bwd_blk, kT, 0, f->stream>>>(hb, f->mask, eta, f->part, f->NR);
    else if (C == 8)
      k_lift_bwd<8><<<f->bwd_blk, kT, 0, f->stream>>>(hb, f->mask, eta, f->part, f->NR);
    else
      k_lift_bwd<4><<<f->bwd_blk, kT, 0, f->stream>>>(hb, f->mask, eta, f->part, f->NR);
    sum_partials(f, f->bwd_blk, 3 * C, f->g + f->oP);
    if (int s = check(f, "fno backward")) return s;
  }
  // the copy waits for the stream when its host side is pageable, so it
  // comes after everything is queued
  if (target && loss)
    cudaMemcpyAsync(loss, f->loss_d, sizeof(float), cudaMemcpyDeviceToHost, f->stream);
  return check(f, "fno eval");
}

int adam_impl(deft_fno *f, float lr) {
  f->adam_t++;
  f->launches++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f / (1.f - std::pow(b1, (float)f->adam_t));
  const float c2 = 1.f / (1.f - std::pow(b2, (float)f->adam_t));
  k_adam<<<grid_for((long long)f->nparam), kT, 0, f->stream>>>(
      f->p, f->g, f->am, f->av, f->pb, (long long)f->nparam, lr, b1, b2, 1e-8f, c1, c2);
  return check(f, "adam");
}

}  // namespace

extern "C" {

// Forward pass on arrays of N^3 floats (host, or device with on_device):
// mask (1 free, 0 wall), eta, relative density y (output, may be NULL), and,
// if target != NULL, the masked mean squared error in *loss.  With grad !=
// NULL the parameter gradient of that loss (deft_fno_param_count floats,
// host) is written there.
int deft_fno_eval(deft_fno *f, const float *mask, float eta, const float *target, int on_device,
                  float *y_out, float *loss, float *grad) {
  if (!f || !mask) return DEFT_ERR_ARG;
  cudaSetDevice(f->device);
  const cudaMemcpyKind kin = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  const cudaMemcpyKind kout = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
  if (int s = eval_impl(f, mask, eta, target, kin, kout, y_out, loss, grad && target)) return s;
  if (grad && target)
    cudaMemcpyAsync(grad, f->g, sizeof(float) * f->nparam, cudaMemcpyDeviceToHost, f->stream);
  if (cudaStreamSynchronize(f->stream) != cudaSuccess) return check(f, "fno eval");
  return check(f, "fno eval");
}

// One training step: loss and gradient on one sample, then Adam.
int deft_fno_train_step(deft_fno *f, const float *mask, float eta, const float *target,
                        int on_device, float lr, float *loss) {
  if (!f || !mask || !target) return DEFT_ERR_ARG;
  cudaSetDevice(f->device);
  const cudaMemcpyKind kin = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  if (int s = eval_impl(f, mask, eta, target, kin, kin, nullptr, loss, true)) return s;
  if (int s = adam_impl(f, lr)) return s;
  return cudaStreamSynchronize(f->stream) == cudaSuccess ? DEFT_OK : check(f, "train step");
}

// One Adam step on the gradient of the last deft_fno_eval(..., grad).
int deft_fno_adam(deft_fno *f, float lr) {
  if (!f) return DEFT_ERR_ARG;
  cudaSetDevice(f->device);
  if (int s = adam_impl(f, lr)) return s;
  return cudaStreamSynchronize(f->stream) == cudaSuccess ? DEFT_OK : DEFT_ERR_CUDA;
}

// Warm start for the minimiser: n = nb max(y, floor_rel) on free points,
// 0 where mask == 0.  mask and n_out are DEVICE pointers of N^3 doubles.
}  // extern "C"

namespace {

// The warm start's launches on the network's stream, not waited for.
int warm_start_queue(deft_fno *f, const double *mask_dev, double eta, double nb,
                     double floor_rel, double *n_out_dev) {
  k_d2f<<<grid_for(f->NR), kT, 0, f->stream>>>(mask_dev, f->mask, f->NR, 1.f);
  f->launches += 2;  // this and the density below
  if (int s = forward(f, (float)eta, false)) return s;
  project(f, nullptr, nullptr, nullptr, nullptr);
  k_density<<<grid_for(f->NR), kT, 0, f->stream>>>(f->y, mask_dev, nb, floor_rel, n_out_dev,
                                                   f->NR);
  return check(f, "warm start");
}

}  // namespace

extern "C" {

int deft_fno_warm_start(deft_fno *f, const double *mask_dev, double eta, double nb,
                        double floor_rel, double *n_out_dev) {
  if (!f || !mask_dev || !n_out_dev) return DEFT_ERR_ARG;
  cudaSetDevice(f->device);
  if (int s = warm_start_queue(f, mask_dev, eta, nb, floor_rel, n_out_dev)) return s;
  return cudaStreamSynchronize(f->stream) == cudaSuccess ? DEFT_OK : DEFT_ERR_CUDA;
}

// Checked warm start: the network's density unless it is non-finite or its
// energy under fmt is above the bulk start's, in which case the bulk start
// (nb on free points, 0 in the walls).  *used_network = 1 or 0 says which.
int deft_fno_initial_density(deft_fno *f, deft_fmt *fmt, const double *mask_dev, double eta,
                             double nb, double floor_rel, double *n_out_dev, int *used_network,
                             double *E_out, double *gnorm_bulk_out) {
  if (!f || !fmt || !mask_dev || !n_out_dev) return DEFT_ERR_ARG;
  int shape[3];
  deft::fmt_shape(fmt, shape);
  if (shape[0] != f->N || shape[1] != f->N || shape[2] != f->N)
    return fno_fail(f, "functional grid does not match the network's N^3", DEFT_ERR_ARG);
  cudaSetDevice(f->device);
  if (!f->bulk && deft::dev_malloc((void **)&f->bulk, sizeof(double) * 2 * f->NR) != cudaSuccess) {
    f->bulk = nullptr;
    return fno_fail(f, "bulk start buffer", DEFT_ERR_NOMEM);
  }
  k_bulk<<<grid_for(f->NR), kT, 0, f->stream>>>(mask_dev, nb, f->bulk, f->NR);
  f->launches++;
  if (cudaStreamSynchronize(f->stream) != cudaSuccess) return check(f, "bulk start");
  // the network runs on its own stream while the bulk start is evaluated on
  // the functional's (the forward pass is latency-bound and leaves room)
  if (int s = warm_start_queue(f, mask_dev, eta, nb, floor_rel, n_out_dev)) return s;
  double E0 = 0, E1 = 0;
  if (gnorm_bulk_out) {
    // energy and gradient of the bulk start (gradient in the buffer's upper half)
    double *gb = f->bulk + f->NR;
    if (int s = deft_fmt_energy_grad(fmt, f->bulk, 1, &E0, gb, nullptr)) return s;
    k_norm2_partial<<<kNormBlocks, kT, 0, f->stream>>>(gb, f->NR, f->part_d);
    f->launches++;
    std::vector<double> h(kNormBlocks);
    cudaMemcpyAsync(h.data(), f->part_d, sizeof(double) * kNormBlocks, cudaMemcpyDeviceToHost,
                    f->stream);
    if (cudaStreamSynchronize(f->stream) != cudaSuccess) return check(f, "bulk gradient norm");
    double ss = 0;
    for (double v : h) ss += v;
    *gnorm_bulk_out = std::sqrt(ss);
  } else if (int s = deft_fmt_energy(fmt, f->bulk, 1, &E0, nullptr)) {
    return s;
  }
  if (cudaStreamSynchronize(f->stream) != cudaSuccess) return check(f, "warm start");
  const int s1 = deft_fmt_energy(fmt, n_out_dev, 1, &E1, nullptr);
  const bool use = s1 == DEFT_OK && std::isfinite(E1) && E1 <= E0;
  if (!use) {
    if (cudaMemcpyAsync(n_out_dev, f->bulk, sizeof(double) * f->NR, cudaMemcpyDeviceToDevice,
                        f->stream) != cudaSuccess ||
        cudaStreamSynchronize(f->stream) != cudaSuccess)
      return check(f, "bulk fallback");
  }
  if (used_network) *used_network = use ? 1 : 0;
  if (E_out) *E_out = use ? E1 : E0;
  return DEFT_OK;
}

// Kernel launches this network has queued (forward, backward, Adam and warm
// start kernels; the functional's own evaluations are counted by its grid).
long long deft_fno_launches(const deft_fno *f) { return f ? f->launches : 0; }

}  // extern "C"
