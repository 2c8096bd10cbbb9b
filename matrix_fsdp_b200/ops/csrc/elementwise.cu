// Bandwidth-bound kernels of the model and optimizer path: RMSNorm, RoPE, SwiGLU,
// fused softmax-cross-entropy, flat sharded AdamW/SGD, Muon element-wise stages and the
// segment copy kernels of the flat-buffer runtime.  All use 16-byte vector accesses
// and one pass over HBM per tensor; reductions stay in registers/shared memory.
//
// Counterparts in the reference: the segment copies replace
// matrix_fsdp/kernels/native/matrix_copy_cuda.cu:8-87 (one element per thread there);
// everything else runs as stock PyTorch ops in the reference (torch.optim.AdamW,
// F.layer_norm, ... see test/fsdp/bench_fsdp2_compare.py:305-514).
#include "common.cuh"

namespace mfsdp {

// ============================================================== RMSNorm
// WPR warps per row, 8 / WPR rows per CTA, VPL vectors of 8 per lane: a row's sum needs shuffles and at most one
// barrier, and the rows of a CTA wait for nobody else's memory.  Bound by memory.  One CTA per row -> this: 4096 rows of
// 2048 6.8 -> 5.0 us, 16384 rows of 4096 47.8 -> 41.6 us (6.4 TB/s), of 5120 60.6 -> 54.8, of 12288 174 -> 143.
template <int VPL, int WPR>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_rows_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                        __nv_bfloat16* __restrict__ y, float* __restrict__ rstd_out, long long rows, int H, float eps) {
  __shared__ float part[8];
  pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * (8 / WPR) + warp / WPR;
  const int first = (warp % WPR) * 32 + lane, nvec = H >> 3;
  const bool live = row < rows;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
  uint4 xv[VPL], wv[VPL];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int v = first + i * 32 * WPR;
    const bool in = live && v < nvec;
    xv[i] = in ? xr[v] : make_uint4(0, 0, 0, 0);
    wv[i] = in ? reinterpret_cast<const uint4*>(w)[v] : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const uint32_t u[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = unpack_bf16x2(u[e]);
      ss += f.x * f.x + f.y * f.y;
    }
  }
  ss = warp_sum(ss);
  if (WPR > 1) {
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    ss = 0.f;
#pragma unroll
    for (int i = 0; i < WPR; ++i) ss += part[warp / WPR * WPR + i];
  }
  const float rstd = rsqrtf(ss / (float)H + eps);
  if (!live) return;
  if (first == 0 && rstd_out) rstd_out[row] = rstd;
  uint4* yr = reinterpret_cast<uint4*>(y + row * H);
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int v = first + i * 32 * WPR;
    if (v < nvec) {
      const uint32_t u[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
      const uint32_t ww[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = unpack_bf16x2(u[e]);
        const float2 g = unpack_bf16x2(ww[e]);
        o[e] = pack_bf16x2(f.x * rstd * g.x, f.y * rstd * g.y);
      }
      yr[v] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres);  dw += sum_rows dy * xhat.
// Persistent over rows, WPR warps per row and 8 / WPR rows per CTA at a time: a row's dot product needs shuffles and, for
// WPR > 1, a barrier of its own warps only.  The weight gradient stays in registers until the end, when the warps of a
// CTA add theirs up in shared memory, in a fixed order, into one partial row per CTA.  Bound by memory.  RES: with the
// residual's gradient dres, in a kernel of its own because its registers decide how many CTAs fit.  One CTA per two
// or four rows, barriers of the whole block -> this, residual included: 4096 rows of 2048 18.6 -> 11.5 us, 16384 rows of
// 4096 140 -> 105 us (5.1 TB/s), 4096 rows of 8192 126 -> 66 us; without: 15.0 -> 10.6, 82.9 -> 77.5, 69 -> 57.
template <int VPL, int WPR, int CTAS, bool RES>
__global__ void __launch_bounds__(256, CTAS)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_acc, long long rows, int H) {
  constexpr int RPC = 8 / WPR;
  __shared__ float part[2][8];
  extern __shared__ float dw_smem[];          // [H]
  pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, slot = warp / WPR;
  const int first = (warp % WPR) * 32 + lane, nvec = H >> 3;
  float dwp[VPL][8];
  uint4 wv[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int v = first + i * 32 * WPR;
    wv[i] = v < nvec ? reinterpret_cast<const uint4*>(w)[v] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int e = 0; e < 8; ++e) dwp[i][e] = 0.f;
  }
  int trip = 0;
  for (long long row = (long long)blockIdx.x * RPC + slot; row < rows; row += (long long)gridDim.x * RPC, trip ^= 1) {
    uint4 xv[VPL], dv[VPL], rv[VPL];
    const float rstd = rstd_in[row];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = first + i * 32 * WPR;
      const bool in = v < nvec;
      xv[i] = in ? reinterpret_cast<const uint4*>(x + row * H)[v] : make_uint4(0, 0, 0, 0);
      dv[i] = in ? reinterpret_cast<const uint4*>(dy + row * H)[v] : make_uint4(0, 0, 0, 0);
      if (RES) rv[i] = in ? reinterpret_cast<const uint4*>(dres + row * H)[v] : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const uint32_t xu[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
      const uint32_t du[4] = {dv[i].x, dv[i].y, dv[i].z, dv[i].w};
      const uint32_t wu[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 xf = unpack_bf16x2(xu[e]), df = unpack_bf16x2(du[e]), wf = unpack_bf16x2(wu[e]);
        const float xh0 = xf.x * rstd, xh1 = xf.y * rstd;
        dwp[i][2 * e] += df.x * xh0;
        dwp[i][2 * e + 1] += df.y * xh1;
        dot += df.x * wf.x * xh0 + df.y * wf.y * xh1;
      }
    }
    dot = warp_sum(dot);
    if (WPR > 1) {                            // the warps of a row make the same trips: a barrier of their own
      if (lane == 0) part[trip][warp] = dot;
      asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "n"(WPR * 32) : "memory");
      dot = 0.f;
#pragma unroll
      for (int i = 0; i < WPR; ++i) dot += part[trip][slot * WPR + i];
    }
    const float mean_dot = dot / (float)H;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = first + i * 32 * WPR;
      if (v < nvec) {
        const uint32_t xu[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
        const uint32_t du[4] = {dv[i].x, dv[i].y, dv[i].z, dv[i].w};
        const uint32_t wu[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
        float o[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 xf = unpack_bf16x2(xu[e]), df = unpack_bf16x2(du[e]), wf = unpack_bf16x2(wu[e]);
          o[2 * e] = rstd * (df.x * wf.x - xf.x * rstd * mean_dot);
          o[2 * e + 1] = rstd * (df.y * wf.y - xf.y * rstd * mean_dot);
        }
        if (RES) {
          const uint32_t ru[4] = {rv[i].x, rv[i].y, rv[i].z, rv[i].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 rf = unpack_bf16x2(ru[e]);
            o[2 * e] += rf.x; o[2 * e + 1] += rf.y;
          }
        }
        reinterpret_cast<uint4*>(dx + row * H)[v] =
            make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
      }
    }
  }
  // one partial row per CTA in the scratch matrix [gridDim.x, H]; no atomics
  for (int turn = 0; turn < RPC; ++turn) {
    if (slot == turn) {
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int v = first + i * 32 * WPR;
        if (v < nvec) {
          float4* d = reinterpret_cast<float4*>(turn == RPC - 1 ? dw_acc + (long long)blockIdx.x * H + v * 8 : dw_smem + v * 8);
          float4 a = make_float4(dwp[i][0], dwp[i][1], dwp[i][2], dwp[i][3]), b = make_float4(dwp[i][4], dwp[i][5], dwp[i][6], dwp[i][7]);
          if (turn > 0) {
            const float4 p0 = reinterpret_cast<const float4*>(dw_smem + v * 8)[0], p1 = reinterpret_cast<const float4*>(dw_smem + v * 8)[1];
            a.x += p0.x; a.y += p0.y; a.z += p0.z; a.w += p0.w;
            b.x += p1.x; b.y += p1.y; b.z += p1.z; b.w += p1.w;
          }
          d[0] = a; d[1] = b;
        }
      }
    }
    __syncthreads();
  }
}

// out[c] (bf16) = (accumulate ? out[c] : 0) + sum_r partial[r, c]; one thread per column, rows
// strided over blockIdx.y-less 2-D thread blocks (32 columns x 8 row lanes).
__global__ void colsum_f32_to_bf16_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ out,
                                          int rows, int H, int accumulate) {
  __shared__ float tile[8][33];
  pdl_begin();
  const int col = blockIdx.x * 32 + threadIdx.x;
  float acc = 0.f;
  if (col < H)
    for (int r = threadIdx.y; r < rows; r += 8) acc += partial[(long long)r * H + col];
  tile[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && col < H) {
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) v += tile[j][threadIdx.x];
    if (accumulate) v += __bfloat162float(out[col]);
    out[col] = __float2bfloat16_rn(v);
  }
}

// ============================================================== RoPE
// In-place rotary embedding ("rotate-half" pairing i <-> i + D/2) on `n_heads` heads that
// start at column `col0` of a [T, ld] matrix; cos/sin tables are [S, D/2] fp32, position of
// row t is t % S.  sign = +1 forward, -1 backward (the transpose of a rotation).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ qkv, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, long long T, int S, int ld, int col0,
                            int n_heads, int D, float sign) {
  pdl_begin();
  const int half = D >> 1;
  const int vec_per_head = half >> 3;  // 8 bf16 per vector
  const long long total = T * (long long)n_heads * vec_per_head;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(idx % vec_per_head);
    const int h = (int)((idx / vec_per_head) % n_heads);
    const long long t = idx / ((long long)vec_per_head * n_heads);
    const int pos = (int)(t % S);
    __nv_bfloat16* base = qkv + t * ld + col0 + h * D + v * 8;
    uint4 a = *reinterpret_cast<uint4*>(base);
    uint4 b = *reinterpret_cast<uint4*>(base + half);
    const float4 c0 = *reinterpret_cast<const float4*>(cos_t + (long long)pos * half + v * 8);
    const float4 c1 = *reinterpret_cast<const float4*>(cos_t + (long long)pos * half + v * 8 + 4);
    const float4 s0 = *reinterpret_cast<const float4*>(sin_t + (long long)pos * half + v * 8);
    const float4 s1 = *reinterpret_cast<const float4*>(sin_t + (long long)pos * half + v * 8 + 4);
    const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    uint32_t au[4] = {a.x, a.y, a.z, a.w}, bu[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x1 = unpack_bf16x2(au[e]);
      const float2 x2 = unpack_bf16x2(bu[e]);
      const float s_lo = sign * sn[2 * e], s_hi = sign * sn[2 * e + 1];
      const float o1x = x1.x * cs[2 * e] - x2.x * s_lo;
      const float o1y = x1.y * cs[2 * e + 1] - x2.y * s_hi;
      const float o2x = x2.x * cs[2 * e] + x1.x * s_lo;
      const float o2y = x2.y * cs[2 * e + 1] + x1.y * s_hi;
      au[e] = pack_bf16x2(o1x, o1y);
      bu[e] = pack_bf16x2(o2x, o2y);
    }
    *reinterpret_cast<uint4*>(base) = make_uint4(au[0], au[1], au[2], au[3]);
    *reinterpret_cast<uint4*>(base + half) = make_uint4(bu[0], bu[1], bu[2], bu[3]);
  }
}

// ============================================================== SwiGLU
// gu is [T, 2F]: gate in columns [0,F), up in [F,2F).  h = silu(gate) * up.
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ h,
                                  long long T, int F) {
  pdl_begin();
  const int vpr = F >> 3;
  const long long total = T * vpr;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / vpr;
    const int v = (int)(idx % vpr);
    const uint4 g = *reinterpret_cast<const uint4*>(gu + t * 2 * F + v * 8);
    const uint4 u = *reinterpret_cast<const uint4*>(gu + t * 2 * F + F + v * 8);
    const uint32_t gg[4] = {g.x, g.y, g.z, g.w}, uu[4] = {u.x, u.y, u.z, u.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = unpack_bf16x2(gg[e]);
      const float2 b = unpack_bf16x2(uu[e]);
      const float sx = a.x / (1.f + __expf(-a.x)), sy = a.y / (1.f + __expf(-a.y));
      o[e] = pack_bf16x2(sx * b.x, sy * b.y);
    }
    *reinterpret_cast<uint4*>(h + t * F + v * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// dgu[:, :F] = dh * up * dsilu(gate);  dgu[:, F:] = dh * silu(gate).
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dh,
                                  const __nv_bfloat16* __restrict__ gu,
                                  __nv_bfloat16* __restrict__ dgu, long long T, int F) {
  pdl_begin();
  const int vpr = F >> 3;
  const long long total = T * vpr;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / vpr;
    const int v = (int)(idx % vpr);
    const uint4 g = *reinterpret_cast<const uint4*>(gu + t * 2 * F + v * 8);
    const uint4 u = *reinterpret_cast<const uint4*>(gu + t * 2 * F + F + v * 8);
    const uint4 d = *reinterpret_cast<const uint4*>(dh + t * F + v * 8);
    const uint32_t gg[4] = {g.x, g.y, g.z, g.w}, uu[4] = {u.x, u.y, u.z, u.w},
                   dd[4] = {d.x, d.y, d.z, d.w};
    uint32_t og[4], ou[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = unpack_bf16x2(gg[e]);
      const float2 b = unpack_bf16x2(uu[e]);
      const float2 c = unpack_bf16x2(dd[e]);
      const float sgx = 1.f / (1.f + __expf(-a.x)), sgy = 1.f / (1.f + __expf(-a.y));
      const float silx = a.x * sgx, sily = a.y * sgy;
      const float dsx = sgx * (1.f + a.x * (1.f - sgx)), dsy = sgy * (1.f + a.y * (1.f - sgy));
      og[e] = pack_bf16x2(c.x * b.x * dsx, c.y * b.y * dsy);
      ou[e] = pack_bf16x2(c.x * silx, c.y * sily);
    }
    *reinterpret_cast<uint4*>(dgu + t * 2 * F + v * 8) = make_uint4(og[0], og[1], og[2], og[3]);
    *reinterpret_cast<uint4*>(dgu + t * 2 * F + F + v * 8) = make_uint4(ou[0], ou[1], ou[2], ou[3]);
  }
}

// ============================================================== cross-entropy
// One CTA (128 to 512 threads) per row keeps the whole row in registers, as the bf16 pairs it came in (V <= threads*8*VPT):
// loss[row] = logsumexp - logit[target]; logits are overwritten with
// (softmax - onehot) * grad_scale, i.e. the gradient of the mean loss.  When `grad_scale_dev` is
// given the scale is read from device memory (1 / number of counted targets, computed on the device),
// so a caller that masks targets needs no device-to-host read to launch this.
// A row passes through phases (load, maximum, sum, store) that each leave most of the SM idle, so several rows have to
// share it: packed values and taking the exponentials twice leave room for two blocks of 512 threads, where 1024 threads
// with fp32 values ran alone: 16384 rows of 32000 logits 582 -> 416 us (5.0 TB/s), 3000 117 -> 86 us, 2048 rows of 8192
// 30.7 -> 20.5 us, 16384 rows of 1024 131 -> 20.5 us.
template <int VPT, int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
cross_entropy_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ target,
                             float* __restrict__ loss, int V, long long ld, float grad_scale,
                             const float* __restrict__ grad_scale_dev, long long ignore_index) {
  __shared__ float red[32];
  pdl_begin();
  if (grad_scale_dev != nullptr) grad_scale = *grad_scale_dev;
  const long long row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  const int nvec = V >> 3;
  const long long tgt = target[row];
  const bool valid = (tgt != ignore_index) && tgt >= 0 && tgt < V;
  uint4 x[VPT];
  float mx = -INFINITY;
  // one vector at a time, and nothing unpacked kept for the next phase: the registers have to do for two blocks
  auto in_turn = [&](int i, float& acc) {
    asm volatile("" : "+f"(acc), "+r"(x[i].x), "+r"(x[i].y), "+r"(x[i].z), "+r"(x[i].w));
  };
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * THREADS;
    x[i] = v < nvec ? reinterpret_cast<const uint4*>(lr)[v] : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // -inf
  }
  const float tgt_logit = threadIdx.x == 0 && valid ? __bfloat162float(lr[tgt]) : 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    in_turn(i, mx);
    const uint32_t w[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = unpack_bf16x2(w[e]);
      mx = fmaxf(mx, fmaxf(a.x, a.y));
    }
  }
  mx = block_max(mx, red);      // its barriers also stand between the reading of the target's logit and the first store
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    in_turn(i, sum);
    const uint32_t w[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = unpack_bf16x2(w[e]);
      sum += __expf(a.x - mx) + __expf(a.y - mx);
    }
  }
  sum = block_sum(sum, red);
  if (threadIdx.x == 0) loss[row] = valid ? logf(sum) + mx - tgt_logit : 0.f;
  float inv = valid ? grad_scale / sum : 0.f;
  const int tgt_vec = valid ? (int)(tgt >> 3) : -1, tgt_elem = (int)(tgt & 7);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * THREADS;
    in_turn(i, inv);
    if (v < nvec) {
      const uint32_t w[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
      float o[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 a = unpack_bf16x2(w[e]);
        o[2 * e] = __expf(a.x - mx) * inv;
        o[2 * e + 1] = __expf(a.y - mx) * inv;
      }
      if (v == tgt_vec) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (e == tgt_elem) o[e] -= grad_scale;
      }
      reinterpret_cast<uint4*>(lr)[v] = make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]),
                                                   pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
    }
  }
}

// ============================================================== flat optimizers
// Sharded AdamW over one contiguous flat range.  Master weights and both moments are fp32;
// the gradient arrives as bf16 or fp32 and is scaled by `grad_scale` (1/world, clipping)
// on the fly; the kernel also emits the low-precision copy that the next all-gather
// ships, so no separate cast kernel runs.  Matches torch.optim.AdamW (decoupled decay,
// bias correction, eps outside the sqrt of the corrected second moment).
// Bound by memory: 50 M parameters, bf16 gradients 239 us (5.9 TB/s).  EXACT: four blocks per SM, because with the 72
// registers that the compiler takes for it when it is free to too few loads are in flight (246 us; four blocks 229).
template <typename GradT, bool EXACT>
__global__ void __launch_bounds__(256, EXACT ? 4 : 6) adamw_flat_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                                  const GradT* __restrict__ g, __nv_bfloat16* __restrict__ p_lp,
                                  long long n, const AdamWStep a) {
  const long long nv = n >> 2;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv; i += stride) {
    float4 pp = reinterpret_cast<float4*>(p)[i];
    float4 mm = reinterpret_cast<float4*>(m)[i];
    float4 vv = reinterpret_cast<float4*>(v)[i];
    float gg[4];
    if constexpr (sizeof(GradT) == 2) {
      const uint2 u = reinterpret_cast<const uint2*>(g)[i];
      const float2 a2 = unpack_bf16x2(u.x), b2 = unpack_bf16x2(u.y);
      gg[0] = a2.x; gg[1] = a2.y; gg[2] = b2.x; gg[3] = b2.y;
    } else {
      const float4 g4 = reinterpret_cast<const float4*>(g)[i];
      gg[0] = g4.x; gg[1] = g4.y; gg[2] = g4.z; gg[3] = g4.w;
    }
    float* pa = reinterpret_cast<float*>(&pp);
    float* ma = reinterpret_cast<float*>(&mm);
    float* va = reinterpret_cast<float*>(&vv);
#pragma unroll
    for (int e = 0; e < 4; ++e) adamw_update<EXACT>(pa[e], ma[e], va[e], gg[e], a);
    reinterpret_cast<float4*>(p)[i] = pp;
    reinterpret_cast<float4*>(m)[i] = mm;
    reinterpret_cast<float4*>(v)[i] = vv;
    if (p_lp)
      reinterpret_cast<uint2*>(p_lp)[i] = make_uint2(pack_bf16x2(pa[0], pa[1]), pack_bf16x2(pa[2], pa[3]));
  }
  // scalar tail
  for (long long i = (nv << 2) + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    float gr;
    if constexpr (sizeof(GradT) == 2) gr = __bfloat162float(g[i]);
    else gr = (float)g[i];
    float pv = p[i], mv = m[i], vv = v[i];
    adamw_update<EXACT>(pv, mv, vv, gr, a);
    p[i] = pv; m[i] = mv; v[i] = vv;
    if (p_lp) p_lp[i] = __float2bfloat16_rn(pv);
  }
}

// SGD with optional momentum over a flat fp32 range (same fused low-precision emit).
template <typename GradT>
__global__ void sgd_flat_kernel(float* __restrict__ p, float* __restrict__ mom,
                                const GradT* __restrict__ g, __nv_bfloat16* __restrict__ p_lp,
                                long long n, float lr, float momentum, float weight_decay,
                                float grad_scale, int first_step) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    float gr;
    if constexpr (sizeof(GradT) == 2) gr = __bfloat162float(g[i]) * grad_scale;
    else gr = (float)g[i] * grad_scale;
    float pv = p[i];
    gr += weight_decay * pv;
    if (mom) {
      const float b = first_step ? gr : momentum * mom[i] + gr;
      mom[i] = b;
      gr = b;
    }
    pv -= lr * gr;
    p[i] = pv;
    if (p_lp) p_lp[i] = __float2bfloat16_rn(pv);
  }
}

// ============================================================== Muon element-wise stages
// Stage 1 (per matrix): buf = mu*buf + (1-mu)*g*scale  (torch's lerp form),
// u = nesterov ? lerp(g*scale, buf, mu) : buf; emits u as bf16 and accumulates sum(u^2).
template <typename GradT>
__global__ void muon_momentum_kernel(float* __restrict__ buf, const GradT* __restrict__ g,
                                     __nv_bfloat16* __restrict__ u_out, float* __restrict__ sumsq,
                                     long long n, float mu, float grad_scale, int nesterov) {
  __shared__ float red[32];
  float acc = 0.f;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    float gr;
    if constexpr (sizeof(GradT) == 2) gr = __bfloat162float(g[i]) * grad_scale;
    else gr = (float)g[i] * grad_scale;
    const float b = buf[i] + (1.f - mu) * (gr - buf[i]);
    buf[i] = b;
    const float u = nesterov ? gr + mu * (b - gr) : b;
    const __nv_bfloat16 ub = __float2bfloat16_rn(u);
    u_out[i] = ub;
    const float uf = __bfloat162float(ub);
    acc += uf * uf;
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) atomicAdd(sumsq, acc);
}

// x *= 1 / max(sqrt(sumsq), eps)   (bf16 in place)
__global__ void muon_normalize_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ sumsq,
                                      long long n, float eps) {
  const float inv = 1.f / fmaxf(sqrtf(*sumsq), eps);
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride)
    x[i] = __float2bfloat16_rn(__bfloat162float(x[i]) * inv);
}

// p = p*(1 - lr*wd) - adjusted_lr * o ; o is the orthogonalised update, stored either as
// [rows, cols] (transposed = 0) or as [cols, rows] (transposed = 1).
__global__ void muon_apply_kernel(float* __restrict__ p, const __nv_bfloat16* __restrict__ o,
                                  __nv_bfloat16* __restrict__ p_lp, int rows, int cols,
                                  int transposed, float lr, float weight_decay, float adjusted_lr) {
  const long long n = (long long)rows * cols;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    long long j = i;
    if (transposed) {
      const long long r = i / cols, c = i % cols;
      j = c * rows + r;
    }
    float pv = p[i] * (1.f - lr * weight_decay);
    pv -= adjusted_lr * __bfloat162float(o[j]);
    p[i] = pv;
    if (p_lp) p_lp[i] = __float2bfloat16_rn(pv);
  }
}

// ---- the same stages for up to kMuonBatch matrices of one shape in one launch each
// A step over a few hundred expert matrices was bound by its launches (four per matrix), the element-wise passes by
// their 2- and 4-byte accesses.  Here the matrices' addresses travel in the kernel's parameters, blockIdx.y names the
// matrix and every thread moves 8 elements per access; the updates land directly in the stacked Newton-Schulz operand
// (no copy into it), and the sums of squares are per-block partials that the scaling kernel adds up in a fixed order.
// Bound by memory.  A training step with 16 small experts in each of 4 layers went from 19.1 to 11.8 ms (launches),
// with 64 large ones in each of 2 layers from 71.9 to 65.5 ms, the optimizer step of two 2048-wide blocks from 5.08
// to 4.63 ms.
constexpr int kMuonBatch = 64;
constexpr int kMuonPartials = 256;      // partial sums (= blocks) per matrix at most
struct MuonPtrs {
  void* a[kMuonBatch];
  void* b[kMuonBatch];
};

__device__ __forceinline__ float muon_update(float& buf, float g, float mu, float grad_scale, int nesterov) {
  const float gr = g * grad_scale;
  buf = buf + (1.f - mu) * (gr - buf);
  return nesterov ? gr + mu * (buf - gr) : buf;
}

__device__ __forceinline__ void load8(const float* p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void store8(float* p, const float (&f)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}
__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }

// a = momentum buffers (fp32), b = gradients; u_out is [matrices, n], partial [matrices, gridDim.x].
template <typename GradT>
__global__ void __launch_bounds__(256)
muon_momentum_many_kernel(const __grid_constant__ MuonPtrs ptrs, __nv_bfloat16* __restrict__ u_out,
                          float* __restrict__ partial, long long n, float mu, float grad_scale, int nesterov) {
  __shared__ float red[32];
  float* buf = reinterpret_cast<float*>(ptrs.a[blockIdx.y]);
  const GradT* g = reinterpret_cast<const GradT*>(ptrs.b[blockIdx.y]);
  __nv_bfloat16* u = u_out + (long long)blockIdx.y * n;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(buf) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(u)) & 15) == 0;
  const long long nv = vec ? n >> 3 : 0;
  float acc = 0.f;
#pragma unroll 2
  for (long long i = tid; i < nv; i += stride) {
    float b[8], gr[8], o[8];
    load8(buf + i * 8, b);
    load8(g + i * 8, gr);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = muon_update(b[e], gr[e], mu, grad_scale, nesterov);
    store8(buf + i * 8, b);
    const uint4 packed = pack8(o);
    reinterpret_cast<uint4*>(u)[i] = packed;
    const uint32_t w[4] = {packed.x, packed.y, packed.z, packed.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { const float2 v = unpack_bf16x2(w[e]); acc += v.x * v.x + v.y * v.y; }
  }
  for (long long i = nv * 8 + tid; i < n; i += stride) {
    float b = buf[i];
    const __nv_bfloat16 ub = __float2bfloat16_rn(muon_update(b, to_float(g[i]), mu, grad_scale, nesterov));
    buf[i] = b;
    u[i] = ub;
    const float uf = __bfloat162float(ub);
    acc += uf * uf;
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) partial[(long long)blockIdx.y * gridDim.x + blockIdx.x] = acc;
}

// x[m] *= 1 / max(||x[m]||, eps) for the stacked matrices, ||.||^2 = the sum of the matrix's partials.
__global__ void __launch_bounds__(256)
muon_normalize_many_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ partial, int partials,
                           long long n, float eps) {
  __shared__ float red[32];
  float ss = threadIdx.x < partials ? partial[(long long)blockIdx.y * partials + threadIdx.x] : 0.f;
  ss = block_sum(ss, red);
  const float inv = 1.f / fmaxf(sqrtf(ss), eps);
  __nv_bfloat16* xm = x + (long long)blockIdx.y * n;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const long long nv = (reinterpret_cast<uintptr_t>(xm) & 15) == 0 ? n >> 3 : 0;
#pragma unroll 4
  for (long long i = tid; i < nv; i += stride) {
    float f[8];
    load8(xm + i * 8, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= inv;
    reinterpret_cast<uint4*>(xm)[i] = pack8(f);
  }
  for (long long i = nv * 8 + tid; i < n; i += stride) xm[i] = __float2bfloat16_rn(__bfloat162float(xm[i]) * inv);
}

// p = p * (1 - lr * wd) - adjusted_lr * o for the stacked results; a = parameters (fp32), b = their bf16 copies or null.
__global__ void __launch_bounds__(256)
muon_apply_many_kernel(const __grid_constant__ MuonPtrs ptrs, const __nv_bfloat16* __restrict__ o_all, long long n,
                       float lr, float weight_decay, float adjusted_lr) {
  float* p = reinterpret_cast<float*>(ptrs.a[blockIdx.y]);
  __nv_bfloat16* lp = reinterpret_cast<__nv_bfloat16*>(ptrs.b[blockIdx.y]);
  const __nv_bfloat16* o = o_all + (long long)blockIdx.y * n;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(lp) | reinterpret_cast<uintptr_t>(o)) & 15) == 0;
  const long long nv = vec ? n >> 3 : 0;
  const float keep = 1.f - lr * weight_decay;
#pragma unroll 2
  for (long long i = tid; i < nv; i += stride) {
    float f[8], u[8];
    load8(p + i * 8, f);
    load8(o + i * 8, u);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = f[e] * keep - adjusted_lr * u[e];
    store8(p + i * 8, f);
    if (lp) reinterpret_cast<uint4*>(lp)[i] = pack8(f);
  }
  for (long long i = nv * 8 + tid; i < n; i += stride) {
    const float pv = p[i] * keep - adjusted_lr * __bfloat162float(o[i]);
    p[i] = pv;
    if (lp) lp[i] = __float2bfloat16_rn(pv);
  }
}

// ============================================================== segment copies
struct SegTable {  // device arrays of length nseg
  const long long* src_off;
  const long long* dst_off;
  const long long* len;
};

// Copies nseg (src_off, dst_off, len) element ranges; blockIdx.y walks segments.
// 16-byte vectors when both sides are 16-byte aligned, scalar head/tail otherwise.
template <typename T>
__global__ void copy_segments_kernel(const T* __restrict__ src, T* __restrict__ dst, SegTable tab,
                                     int nseg) {
  for (int s = blockIdx.y; s < nseg; s += gridDim.y) {
    const T* sp = src + tab.src_off[s];
    T* dp = dst + tab.dst_off[s];
    const long long n = tab.len[s];
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    constexpr int kPer = 16 / sizeof(T);
    const uintptr_t sa = reinterpret_cast<uintptr_t>(sp), da = reinterpret_cast<uintptr_t>(dp);
    if ((sa & 15) == (da & 15)) {
      long long head = ((16 - (sa & 15)) & 15) / sizeof(T);
      if (head > n) head = n;
      const long long nvec = (n - head) / kPer;
      for (long long i = tid; i < head; i += stride) dp[i] = sp[i];
      const uint4* sv = reinterpret_cast<const uint4*>(sp + head);
      uint4* dv = reinterpret_cast<uint4*>(dp + head);
      for (long long i = tid; i < nvec; i += stride) dv[i] = sv[i];
      for (long long i = head + nvec * kPer + tid; i < n; i += stride) dp[i] = sp[i];
    } else {
      for (long long i = tid; i < n; i += stride) dp[i] = sp[i];
    }
  }
}

// fp32 -> bf16 cast over segments (mixed-precision shard -> gather staging).
__global__ void cast_f32_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                                     long long n) {
  const long long nv = n >> 2;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const bool aligned = ((reinterpret_cast<uintptr_t>(src) & 15) == 0) &&
                       ((reinterpret_cast<uintptr_t>(dst) & 7) == 0);
  if (aligned) {
    for (long long i = tid; i < nv; i += stride) {
      const float4 a = reinterpret_cast<const float4*>(src)[i];
      reinterpret_cast<uint2*>(dst)[i] = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
    }
    for (long long i = (nv << 2) + tid; i < n; i += stride) dst[i] = __float2bfloat16_rn(src[i]);
  } else {
    for (long long i = tid; i < n; i += stride) dst[i] = __float2bfloat16_rn(src[i]);
  }
}

// bf16 -> fp32, 8 elements per access (reduced gradients into the fp32 shard that the optimizer reads).  Bound by
// memory; the library's converting copy moved 60 M elements in 179 us, 2.0 TB/s.
__global__ void __launch_bounds__(256) cast_bf16_f32_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, long long n) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long nv = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 ? n >> 3 : 0;
#pragma unroll 4
  for (long long i = tid; i < nv; i += stride) {
    float f[8];
    load8(src + i * 8, f);
    store8(dst + i * 8, f);
  }
  for (long long i = nv * 8 + tid; i < n; i += stride) dst[i] = __bfloat162float(src[i]);
}

static inline int grid_for(long long work, int threads, int max_blocks = 148 * 8) {
  long long b = (work + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (int)b;
}

// ============================================================== embedding backward
// dW[v, :] = sum over the positions t with ids[t] == v of dy[t, :], written (or accumulated) straight into
// the gradient bucket.  Count per id, a range of a list for every id, positions dropped into their id's range in
// whatever order the atomics take; then one CTA per vocabulary row puts its few positions into ascending order and
// sums them, so the fp32 sum of a row is the same in every run, and writes the row once, zeros where an id does not
// occur: no separate fill of the V x H gradient, no atomics on values.  (Ranking every position among all earlier ones
// took 290 us for 16384 positions, ranges in the order of the ids by one block's scan 28 us for 32000 ids.)
__global__ void embed_count_kernel(const long long* __restrict__ ids, int T, int V, int* __restrict__ count) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  const long long v = ids[t];
  if (v >= 0 && v < V) atomicAdd(&count[v], 1);
}

// Gives every id a range of `place` as long as its count; which range does not matter, so a block's ids are numbered
// among themselves and one atomic takes their part of the whole.
__global__ void __launch_bounds__(256) embed_range_kernel(const int* __restrict__ count, int* __restrict__ cursor, int V,
                                                          int* __restrict__ taken) {
  __shared__ int warp_total[8];
  __shared__ int block_start;
  const int v = blockIdx.x * 256 + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = v < V ? count[v] : 0;
  int incl = c;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += o;
  }
  if (lane == 31) warp_total[warp] = incl;
  __syncthreads();
  int before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    if (w < warp) before += warp_total[w];
    total += warp_total[w];
  }
  if (threadIdx.x == 0) block_start = total > 0 ? atomicAdd(taken, total) : 0;
  __syncthreads();
  if (v < V) cursor[v] = block_start + before + incl - c;
}

// Afterwards cursor[v] is the end of v's range.
__global__ void __launch_bounds__(256) embed_place_kernel(const long long* __restrict__ ids, int T, int V,
                                                          int* __restrict__ cursor, int* __restrict__ place) {
  const int t = blockIdx.x * 256 + threadIdx.x;
  if (t >= T) return;
  const long long v = ids[t];
  if (v >= 0 && v < V) place[atomicAdd(&cursor[v], 1)] = t;
}

// Up to this many positions of one id are ordered by counting the smaller ones (n^2 comparisons by one block); a more
// frequent id (padding) has its positions collected again, in order, from the ids themselves.
constexpr int kEmbedSortMax = 256;
// Rows of a frequent id in flight.  One block adds them all up, in order, so what counts is how many it has under way:
// as asynchronous copies they cost no registers, and 24 KB leave the SM its eight blocks.
constexpr int kEmbedRing = 6;

__global__ void __launch_bounds__(256, 8) embed_sum_kernel(const __nv_bfloat16* __restrict__ dy, long long lddy,
                                                           __nv_bfloat16* __restrict__ dw, long long lddw, int H,
                                                           const long long* __restrict__ ids, int T,
                                                           const int* __restrict__ count, const int* __restrict__ cursor,
                                                           const int* __restrict__ place, int* __restrict__ order_buf,
                                                           int accumulate) {
  __shared__ int list[kEmbedSortMax];
  __shared__ int sorted[kEmbedSortMax];
  __shared__ int warp_tot[8];
  __shared__ uint4 ring[kEmbedRing][256];
  const int v = blockIdx.x;
  const int n = count[v];
  if (n == 0 && accumulate) return;
  const int first = cursor[v] - n;
  __nv_bfloat16* out = dw + (long long)v * lddw;
  if (n <= kEmbedSortMax) {
    if (threadIdx.x < n) list[threadIdx.x] = place[first + threadIdx.x];
    __syncthreads();
    if (threadIdx.x < n) {
      const int mine = list[threadIdx.x];
      int rank = 0;
      for (int j = 0; j < n; ++j) rank += list[j] < mine;
      sorted[rank] = mine;
    }
    __syncthreads();
    for (int c = threadIdx.x * 8; c < H; c += 256 * 8) {
      float acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
      if (accumulate) load8(out + c, acc);
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
        float f[8];
        load8(dy + (long long)sorted[j] * lddy + c, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += f[e];
      }
      *reinterpret_cast<uint4*>(out + c) = pack8(acc);
    }
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int run = first;
  for (int base = 0; base < T; base += 256) {
    const int t = base + threadIdx.x;
    const bool hit = t < T && ids[t] == v;
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) warp_tot[warp] = __popc(m);
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      if (w < warp) before += warp_tot[w];
      total += warp_tot[w];
    }
    if (hit) order_buf[run + before + __popc(m & ((1u << lane) - 1u))] = t;
    run += total;
    __syncthreads();
  }
  for (int c0 = 0; c0 < H; c0 += 256 * 8) {
    const int c = c0 + threadIdx.x * 8;
    const bool mine = c < H;                            // every thread takes part in the barriers
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    if (mine && accumulate) load8(out + c, acc);
    for (int base = 0; base < n; base += kEmbedSortMax) {
      const int m = min(n - base, kEmbedSortMax);
      __syncthreads();                                  // order_buf is written, the last part of the list used up
      if (threadIdx.x < m) sorted[threadIdx.x] = order_buf[first + base + threadIdx.x];
      __syncthreads();
      if (mine) {
        auto fetch = [&](int j, int slot) {             // a thread reads only what it copied itself
          if (j < m) cp_async16(smem_u32(&ring[slot][threadIdx.x]), dy + (long long)sorted[j] * lddy + c);
          cp_async_commit();
        };
#pragma unroll
        for (int j = 0; j < kEmbedRing; ++j) fetch(j, j);
        int slot = 0;
        for (int j = 0; j < m; ++j) {
          cp_async_wait<kEmbedRing - 1>();
          float f[8];
          load8(reinterpret_cast<const __nv_bfloat16*>(&ring[slot][threadIdx.x]), f);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += f[e];
          fetch(j + kEmbedRing, slot);
          slot = slot + 1 == kEmbedRing ? 0 : slot + 1;
        }
        cp_async_wait<0>();
      }
    }
    if (mine) *reinterpret_cast<uint4*>(out + c) = pack8(acc);
  }
}

__device__ __forceinline__ void put8(float* p, const float (&f)[8]) { store8(p, f); }
__device__ __forceinline__ void put8(__nv_bfloat16* p, const float (&f)[8]) { *reinterpret_cast<uint4*>(p) = pack8(f); }
__device__ __forceinline__ void put1(float* p, float v) { *p = v; }
__device__ __forceinline__ void put1(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// x *= *scale in fp32, 8 elements per access; nothing to do for a scale of one (a loss that is what backward() is called
// on, a gradient below the clipping threshold).  The library's bf16 product with a one-element tensor moved 262 M logits
// in 677 us, 1.5 TB/s.
template <typename T>
__global__ void __launch_bounds__(256) scale_kernel(T* __restrict__ x, long long n, const float* __restrict__ scale) {
  const float f = *scale;
  if (f == 1.f) return;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long nv = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n >> 3 : 0;
#pragma unroll 4
  for (long long i = tid; i < nv; i += stride) {
    float v[8];
    load8(x + i * 8, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] *= f;
    put8(x + i * 8, v);
  }
  for (long long i = nv * 8 + tid; i < n; i += stride) put1(x + i, to_float(x[i]) * f);
}

// partial[block] = sum of squares of the block's share, in fp32; reads bf16 as it is (a widened copy of every gradient
// shard and its norm took 71 us for 34 M elements).
template <typename T>
__global__ void __launch_bounds__(256) sumsq_kernel(const T* __restrict__ x, long long n, float* __restrict__ partial) {
  __shared__ float red[32];
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long nv = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n >> 3 : 0;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (long long i = tid; i < nv; i += stride) {
    float v[8];
    load8(x + i * 8, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e & 3] += v[e] * v[e];
  }
  for (long long i = nv * 8 + tid; i < n; i += stride) acc[0] += to_float(x[i]) * to_float(x[i]);
  const float sum = block_sum((acc[0] + acc[1]) + (acc[2] + acc[3]), red);
  if (threadIdx.x == 0) partial[blockIdx.x] = sum;
}

}  // namespace mfsdp

using namespace mfsdp;

MFSDP_API int mfsdp_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, long long rows,
                                int H, float eps, cudaStream_t st) {
  if (H % 8 || H > 8 * 8 * 256) return -2;    // 16384 columns: a CTA's 256 threads hold a row in 8 vectors each
  if (rows <= 0) return 0;
  const int nvec = H / 8;
  auto X = (const __nv_bfloat16*)x; auto W = (const __nv_bfloat16*)w; auto Y = (__nv_bfloat16*)y;
  // As few warps per row as hold it in four vectors per lane, eight beyond 8192 columns, and no more vectors per lane than
  // that takes: what a lane does not use still costs registers, and with them rows in flight (16384 rows of 5120 columns:
  // 54.8 us with 8 x 3 vectors, 70.3 with 4 x 8; of 4096: 41.6 with 4 x 4, 45.1 with 2 x 8).
  const int wpr = nvec <= 128 ? 1 : nvec <= 256 ? 2 : nvec <= 512 ? 4 : 8;
  const int rpc = 8 / wpr, vpl = (nvec + 32 * wpr - 1) / (32 * wpr);
  const dim3 grid((unsigned)((rows + rpc - 1) / rpc));
#define MFSDP_RMS(VPL, WPR) \
  if (vpl <= VPL && wpr == WPR) return launch_pdl(rmsnorm_fwd_rows_kernel<VPL, WPR>, grid, dim3(256), 0, st, X, W, Y, rstd, rows, H, eps)
  MFSDP_RMS(1, 1); MFSDP_RMS(2, 1); MFSDP_RMS(3, 1); MFSDP_RMS(4, 1);
  MFSDP_RMS(3, 2); MFSDP_RMS(4, 2);
  MFSDP_RMS(3, 4); MFSDP_RMS(4, 4);
  MFSDP_RMS(3, 8); MFSDP_RMS(4, 8); MFSDP_RMS(5, 8); MFSDP_RMS(6, 8); MFSDP_RMS(7, 8); MFSDP_RMS(8, 8);
#undef MFSDP_RMS
  return -2;
}

// Upper bound of the backward kernel's CTAs (= rows of the dw scratch matrix): at most three are resident per SM.
constexpr int kRmsBwdCtas = 3 * 148;
MFSDP_API int mfsdp_rmsnorm_bwd_scratch_rows(long long rows) { return (int)(rows < kRmsBwdCtas ? (rows < 1 ? 1 : rows) : kRmsBwdCtas); }

// Launches the backward kernel on at most `cap` CTAs, each with the same number of trips (up to rounding); returns the
// number of partial rows that it writes to dw_acc.
template <int VPL, int WPR, int CTAS, bool RES>
static int launch_rmsnorm_bwd_as(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w, const float* rstd,
                                 const __nv_bfloat16* dres, __nv_bfloat16* dx, float* dw_acc, long long rows, int H, int cap,
                                 cudaStream_t st) {
  constexpr int RPC = 8 / WPR;
  const long long groups = (rows + RPC - 1) / RPC, trips = (groups + cap - 1) / cap;
  const int grid = (int)((groups + trips - 1) / trips);
  launch_pdl(rmsnorm_bwd_kernel<VPL, WPR, CTAS, RES>, dim3(grid), dim3(256), H * sizeof(float), st, dy, x, w, rstd, dres, dx,
             dw_acc, rows, H);
  return grid;
}

// Which kernel: two or three CTAs per SM, so that one loads while another adds up, where that leaves each six trips or more
// (fewer are not worth the partial rows) and the scratch has room; a lane then has registers for two or three vectors.
// Otherwise one CTA per SM with four, and below 1024 rows with two, whose shorter chain of sums at the end counts there.
// 16384 rows without / with residual, one CTA per SM -> several: of 1024 columns 23.4 / 30.8 -> 21.5 / 27.9 us, of 3072
// 86.2 / 93.6 -> 59.2 / 68.5, of 4096 without 94.3 -> 77.5 (with: 104.8, several 105.3); 64 rows of 1024 6.0 -> 4.0.
static int launch_rmsnorm_bwd(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w, const float* rstd,
                              const __nv_bfloat16* dres, __nv_bfloat16* dx, float* dw_acc, long long rows, int H,
                              int cap, cudaStream_t st) {
  const int nvec = H / 8;
  auto pays = [&](int wpr, int ctas) { return cap >= 148 * ctas && rows * wpr >= 8LL * 6 * 148 * ctas; };
#define MFSDP_RMS(VPL, WPR, CTAS, CAP)                                                                                    \
  return dres ? launch_rmsnorm_bwd_as<VPL, WPR, CTAS, true>(dy, x, w, rstd, dres, dx, dw_acc, rows, H, CAP, st)           \
              : launch_rmsnorm_bwd_as<VPL, WPR, CTAS, false>(dy, x, w, rstd, dres, dx, dw_acc, rows, H, CAP, st)
  if (nvec <= 64) MFSDP_RMS(2, 1, 2, pays(1, 2) ? 2 * 148 : 148);
  if (nvec <= 128 && pays(2, 2)) MFSDP_RMS(2, 2, 2, 2 * 148);
  if (nvec > 128 && nvec <= 192 && pays(2, 2)) MFSDP_RMS(3, 2, 2, 2 * 148);
  if (nvec > 192 && nvec <= 256 && pays(4, 2)) MFSDP_RMS(2, 4, 2, 2 * 148);
  if (nvec > 256 && nvec <= 384 && pays(4, 2)) MFSDP_RMS(3, 4, 2, 2 * 148);
  if (nvec > 384 && nvec <= 512 && !dres && pays(8, 3))
    return launch_rmsnorm_bwd_as<2, 8, 3, false>(dy, x, w, rstd, dres, dx, dw_acc, rows, H, 3 * 148, st);
  if (nvec > 512 && nvec <= 768 && pays(8, 2)) MFSDP_RMS(3, 8, 2, 2 * 148);
  if (nvec <= 128 && rows <= 1024) MFSDP_RMS(2, 2, 2, 148);
  if (nvec <= 256 && rows <= 1024) MFSDP_RMS(2, 4, 2, 148);
  if (nvec <= 128) MFSDP_RMS(4, 1, 1, 148);
  if (nvec <= 256) MFSDP_RMS(4, 2, 1, 148);
  if (nvec <= 512) MFSDP_RMS(4, 4, 1, 148);
  MFSDP_RMS(4, 8, 1, 148);
#undef MFSDP_RMS
}

// dw_acc: fp32 scratch of mfsdp_rmsnorm_bwd_scratch_rows(rows) x H floats (fully overwritten, needs no
// initialisation); dw (bf16) = (accumulate ? dw : 0) + column sums of the scratch.
MFSDP_API int mfsdp_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd,
                                const void* dres, void* dx, float* dw_acc, void* dw,
                                int accumulate_dw, long long rows, int H, cudaStream_t st) {
  if (H % 8 || H > 8 * 4 * 256) return -2;
  if (rows <= 0)                              // no rows: the weight gradient is zero
    return dw && !accumulate_dw ? (int)cudaMemsetAsync(dw, 0, (size_t)H * sizeof(__nv_bfloat16), st) : 0;
  const int grid = launch_rmsnorm_bwd((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, rstd,
                                      (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, dw_acc, rows, H, kRmsBwdCtas, st);
  if (dw) launch_pdl(colsum_f32_to_bf16_kernel, dim3((H + 31) / 32), dim3(32, 8), 0, st, dw_acc, (__nv_bfloat16*)dw, grid, H, accumulate_dw);
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_rope(void* qkv, const float* cos_t, const float* sin_t, long long T, int S, int ld,
                         int col0, int n_heads, int D, float sign, cudaStream_t st) {
  if (D % 16 || ld % 8 || col0 % 8) return -2;
  const long long work = T * (long long)n_heads * (D / 16);
  return launch_pdl(rope_kernel, dim3(grid_for(work, 256, 148 * 16)), dim3(256), 0, st, (__nv_bfloat16*)qkv, cos_t, sin_t, T, S, ld,
                    col0, n_heads, D, sign);
}

MFSDP_API int mfsdp_swiglu_fwd(const void* gu, void* h, long long T, int F, cudaStream_t st) {
  if (F % 8) return -2;
  return launch_pdl(swiglu_fwd_kernel, dim3(grid_for(T * (F / 8), 256, 148 * 16)), dim3(256), 0, st, (const __nv_bfloat16*)gu, (__nv_bfloat16*)h, T, F);
}

// dW[V, H] (row pitch lddw) from dy[T, H] (row pitch lddy) and ids[T]; `work` holds 2 * V + 2 * T + 1 ints.  Ids outside
// [0, V) contribute nothing.  accumulate != 0 adds to what dW holds (rows whose id does not occur stay as they are).
MFSDP_API int mfsdp_embedding_bwd(const void* dy, long long lddy, const long long* ids, void* dw, long long lddw,
                                  int T, int V, int H, int accumulate, int* work, cudaStream_t st) {
  if (T <= 0 || V <= 0 || H <= 0 || (H % 8) || (lddy % 8) || (lddw % 8)) return -2;
  if (((uintptr_t)dy & 15) || ((uintptr_t)dw & 15)) return -2;
  int* count = work;
  int* taken = work + V;
  int* cursor = taken + 1;
  int* place = cursor + V;
  int* order = place + T;
  cudaError_t e = cudaMemsetAsync(count, 0, sizeof(int) * ((size_t)V + 1), st);
  if (e != cudaSuccess) return (int)e;
  embed_count_kernel<<<(T + 255) / 256, 256, 0, st>>>(ids, T, V, count);
  embed_range_kernel<<<(V + 255) / 256, 256, 0, st>>>(count, cursor, V, taken);
  embed_place_kernel<<<(T + 255) / 256, 256, 0, st>>>(ids, T, V, cursor, place);
  embed_sum_kernel<<<V, 256, 0, st>>>((const __nv_bfloat16*)dy, lddy, (__nv_bfloat16*)dw, lddw, H, ids, T, count, cursor,
                                      place, order, accumulate);
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_swiglu_bwd(const void* dh, const void* gu, void* dgu, long long T, int F,
                               cudaStream_t st) {
  if (F % 8) return -2;
  return launch_pdl(swiglu_bwd_kernel, dim3(grid_for(T * (F / 8), 256, 148 * 16)), dim3(256), 0, st, (const __nv_bfloat16*)dh, (const __nv_bfloat16*)gu, (__nv_bfloat16*)dgu, T, F);
}

static int launch_cross_entropy(void* logits, const long long* target, float* loss, long long rows, int V,
                                long long ld, float grad_scale, const float* grad_scale_dev,
                                long long ignore_index, cudaStream_t st) {
  if (V % 8 || ld % 8) return -2;
  // as few threads as hold the row in eight vectors each (twelve above 32768 logits): short rows then share an SM instead
  // of idling most of a block.  Rows through a ring of shared-memory buffers with bulk copies were no faster (16384 rows of
  // 32000: 596 us, against 582 of 1024 threads with their row in fp32 registers).
  const int nvec = V / 8;
  auto L = (__nv_bfloat16*)logits;
  const unsigned g = (unsigned)rows;
#define MFSDP_CE(VPT, THREADS) \
  return launch_pdl(cross_entropy_fwd_bwd_kernel<VPT, THREADS>, dim3(g), dim3(THREADS), 0, st, L, target, loss, V, ld, grad_scale, \
                    grad_scale_dev, ignore_index)
  if (nvec <= 128) MFSDP_CE(1, 128);
  if (nvec <= 256) MFSDP_CE(2, 128);
  if (nvec <= 512) MFSDP_CE(4, 128);
  if (nvec <= 1024) MFSDP_CE(4, 256);
  if (nvec <= 2048) MFSDP_CE(8, 256);
  if (nvec <= 4096) MFSDP_CE(8, 512);
  if (nvec <= 6144) MFSDP_CE(12, 512);
#undef MFSDP_CE
  return -2;
}

MFSDP_API int mfsdp_cross_entropy(void* logits, const long long* target, float* loss, long long rows,
                                  int V, long long ld, float grad_scale, long long ignore_index,
                                  cudaStream_t st) {
  return launch_cross_entropy(logits, target, loss, rows, V, ld, grad_scale, nullptr, ignore_index, st);
}

// Same, with the gradient scale read from device memory at `grad_scale_dev` (one float).
MFSDP_API int mfsdp_cross_entropy_dev_scale(void* logits, const long long* target, float* loss, long long rows,
                                            int V, long long ld, const float* grad_scale_dev,
                                            long long ignore_index, cudaStream_t st) {
  if (grad_scale_dev == nullptr) return -2;
  return launch_cross_entropy(logits, target, loss, rows, V, ld, 0.f, grad_scale_dev, ignore_index, st);
}

MFSDP_API int mfsdp_adamw_flat(float* p, float* m, float* v, const void* g, int grad_is_bf16, void* p_lp,
                               long long n, double lr, double beta1, double beta2, double eps,
                               double weight_decay, long long step, double grad_scale, int exact, cudaStream_t st) {
  if (n <= 0) return 0;
  if (((uintptr_t)p & 15) || ((uintptr_t)m & 15) || ((uintptr_t)v & 15) ||
      ((uintptr_t)g & (grad_is_bf16 ? 7 : 15)) || ((uintptr_t)p_lp & 7))
    return -2;
  const AdamWStep a = adamw_step(lr, beta1, beta2, eps, weight_decay, step, grad_scale);
  const int grid = grid_for(n / 4 + 1, 256, 148 * 8);
  auto kern_bf16 = exact ? adamw_flat_kernel<__nv_bfloat16, true> : adamw_flat_kernel<__nv_bfloat16, false>;
  auto kern_fp32 = exact ? adamw_flat_kernel<float, true> : adamw_flat_kernel<float, false>;
  if (grad_is_bf16) kern_bf16<<<grid, 256, 0, st>>>(p, m, v, (const __nv_bfloat16*)g, (__nv_bfloat16*)p_lp, n, a);
  else kern_fp32<<<grid, 256, 0, st>>>(p, m, v, (const float*)g, (__nv_bfloat16*)p_lp, n, a);
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_sgd_flat(float* p, float* mom, const void* g, int grad_is_bf16, void* p_lp, long long n,
                             float lr, float momentum, float weight_decay, float grad_scale,
                             int first_step, cudaStream_t st) {
  if (n <= 0) return 0;
  const int grid = grid_for(n, 256, 148 * 8);
  if (grad_is_bf16)
    sgd_flat_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(p, mom, (const __nv_bfloat16*)g, (__nv_bfloat16*)p_lp, n, lr,
                                                         momentum, weight_decay, grad_scale, first_step);
  else
    sgd_flat_kernel<float><<<grid, 256, 0, st>>>(p, mom, (const float*)g, (__nv_bfloat16*)p_lp, n, lr, momentum,
                                                 weight_decay, grad_scale, first_step);
  return (int)cudaGetLastError();
}

// sumsq must be zero on entry.
MFSDP_API int mfsdp_muon_momentum(float* buf, const void* g, int grad_is_bf16, void* u_out, float* sumsq,
                                  long long n, float mu, float grad_scale, int nesterov, cudaStream_t st) {
  if (n <= 0) return 0;
  const int grid = grid_for(n, 256, 148 * 4);
  if (grad_is_bf16)
    muon_momentum_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(buf, (const __nv_bfloat16*)g, (__nv_bfloat16*)u_out,
                                                              sumsq, n, mu, grad_scale, nesterov);
  else
    muon_momentum_kernel<float><<<grid, 256, 0, st>>>(buf, (const float*)g, (__nv_bfloat16*)u_out, sumsq, n, mu,
                                                      grad_scale, nesterov);
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_muon_normalize(void* x, const float* sumsq, long long n, float eps, cudaStream_t st) {
  if (n <= 0) return 0;
  muon_normalize_kernel<<<grid_for(n, 256, 148 * 8), 256, 0, st>>>((__nv_bfloat16*)x, sumsq, n, eps);
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_muon_apply(float* p, const void* o, void* p_lp, int rows, int cols, int transposed,
                               float lr, float weight_decay, float adjusted_lr, cudaStream_t st) {
  const long long n = (long long)rows * cols;
  if (n <= 0) return 0;
  muon_apply_kernel<<<grid_for(n, 256, 148 * 8), 256, 0, st>>>(p, (const __nv_bfloat16*)o, (__nv_bfloat16*)p_lp, rows,
                                                              cols, transposed, lr, weight_decay, adjusted_lr);
  return (int)cudaGetLastError();
}

// Stages of `mats` (<= 64) matrices of n elements each; a / b are host arrays of device addresses.  `partial` holds
// mats * mfsdp_muon_partials(mats, n) floats and needs no initialisation.
MFSDP_API int mfsdp_muon_partials(int mats, long long n) {
  // about 8 resident blocks of 256 threads per SM over all matrices, each with at least 4 vectors per thread
  const long long want = (n / 8 + 1023) / 1024, share = (148 * 8 + mats - 1) / (mats > 0 ? mats : 1);
  long long b = want < share ? want : share;
  if (b > kMuonPartials) b = kMuonPartials;
  return b < 1 ? 1 : (int)b;
}

static int muon_ptrs(MuonPtrs* out, const unsigned long long* a, const unsigned long long* b, int mats) {
  if (mats <= 0 || mats > kMuonBatch || !a || !b) return -2;
  for (int i = 0; i < mats; ++i) {
    out->a[i] = reinterpret_cast<void*>(a[i]);
    out->b[i] = reinterpret_cast<void*>(b[i]);
    if (!out->a[i]) return -2;
  }
  return 0;
}

MFSDP_API int mfsdp_muon_prepare_many(const unsigned long long* bufs, const unsigned long long* grads, int mats,
                                      int grad_is_bf16, void* u_out, float* partial, long long n, float mu,
                                      float grad_scale, int nesterov, float eps, cudaStream_t st) {
  MuonPtrs ptrs{};
  if (n <= 0 || muon_ptrs(&ptrs, bufs, grads, mats)) return -2;
  for (int i = 0; i < mats; ++i)
    if (!ptrs.b[i]) return -2;
  const dim3 grid(mfsdp_muon_partials(mats, n), mats);
  auto u = (__nv_bfloat16*)u_out;
  if (grad_is_bf16)
    muon_momentum_many_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(ptrs, u, partial, n, mu, grad_scale, nesterov);
  else
    muon_momentum_many_kernel<float><<<grid, 256, 0, st>>>(ptrs, u, partial, n, mu, grad_scale, nesterov);
  muon_normalize_many_kernel<<<grid, 256, 0, st>>>(u, partial, (int)grid.x, n, eps);
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_muon_apply_many(const unsigned long long* params, const unsigned long long* lps, int mats,
                                    const void* o, long long n, float lr, float weight_decay, float adjusted_lr,
                                    cudaStream_t st) {
  MuonPtrs ptrs{};
  if (n <= 0 || muon_ptrs(&ptrs, params, lps, mats)) return -2;
  muon_apply_many_kernel<<<dim3(mfsdp_muon_partials(mats, n), mats), 256, 0, st>>>(ptrs, (const __nv_bfloat16*)o, n, lr,
                                                                                   weight_decay, adjusted_lr);
  return (int)cudaGetLastError();
}

// elem_size in {1,2,4,8}; offsets/lengths are in elements and live in device memory.
MFSDP_API int mfsdp_copy_segments(const void* src, void* dst, const long long* src_off,
                                  const long long* dst_off, const long long* len, int nseg,
                                  long long max_len, int elem_size, cudaStream_t st) {
  if (nseg <= 0) return 0;
  SegTable tab{src_off, dst_off, len};
  const int per16 = 16 / elem_size;
  int gx = grid_for(max_len / per16 + 1, 256, 148 * 4);
  int gy = nseg < 65535 ? nseg : 65535;
  if ((long long)gx * gy > 148 * 16) gx = (148 * 16 + gy - 1) / gy;
  dim3 grid(gx, gy);
  switch (elem_size) {
    case 1: copy_segments_kernel<uint8_t><<<grid, 256, 0, st>>>((const uint8_t*)src, (uint8_t*)dst, tab, nseg); break;
    case 2: copy_segments_kernel<uint16_t><<<grid, 256, 0, st>>>((const uint16_t*)src, (uint16_t*)dst, tab, nseg); break;
    case 4: copy_segments_kernel<uint32_t><<<grid, 256, 0, st>>>((const uint32_t*)src, (uint32_t*)dst, tab, nseg); break;
    case 8: copy_segments_kernel<uint64_t><<<grid, 256, 0, st>>>((const uint64_t*)src, (uint64_t*)dst, tab, nseg); break;
    default: return -2;
  }
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_cast_f32_bf16(const float* src, void* dst, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  cast_f32_bf16_kernel<<<grid_for(n / 4 + 1, 256, 148 * 8), 256, 0, st>>>(src, (__nv_bfloat16*)dst, n);
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_scale(void* x, int is_bf16, long long n, const float* scale, cudaStream_t st) {
  if (n <= 0) return 0;
  const int grid = grid_for(n / 8 + 1, 256, 148 * 8);
  if (is_bf16) scale_kernel<<<grid, 256, 0, st>>>((__nv_bfloat16*)x, n, scale);
  else scale_kernel<<<grid, 256, 0, st>>>((float*)x, n, scale);
  return (int)cudaGetLastError();
}

// `partial`: kSumsqBlocks floats, all of them written.
constexpr int kSumsqBlocks = 148 * 4;
MFSDP_API int mfsdp_sumsq(const void* x, int is_bf16, long long n, float* partial, cudaStream_t st) {
  if (n < 0) return -2;
  if (is_bf16) sumsq_kernel<<<kSumsqBlocks, 256, 0, st>>>((const __nv_bfloat16*)x, n, partial);
  else sumsq_kernel<<<kSumsqBlocks, 256, 0, st>>>((const float*)x, n, partial);
  return (int)cudaGetLastError();
}

MFSDP_API int mfsdp_cast_bf16_f32(const void* src, float* dst, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  cast_bf16_f32_kernel<<<grid_for(n / 8 + 1, 256, 148 * 8), 256, 0, st>>>((const __nv_bfloat16*)src, dst, n);
  return (int)cudaGetLastError();
}

// ============================================================== allocation-free RMSNorm backward
// Declared and documented in mfsdp_noalloc.h.  The weight-gradient partial sums go to a device
// array that is part of the library image instead of a caller-provided buffer.  In host code the
// array's name is only a handle for the runtime, so its device address is looked up once per device
// with cudaGetSymbolAddress and that pointer is what the kernels receive.
#include "mfsdp_noalloc.h"

namespace mfsdp {
static __device__ __align__(256) float g_noalloc_dw_scratch[MFSDP_NOALLOC_SCRATCH_ROWS * MFSDP_NOALLOC_MAX_HIDDEN];
constexpr int kNoAllocMaxDevices = 64;
static float* g_noalloc_scratch_addr[kNoAllocMaxDevices] = {nullptr};
}  // namespace mfsdp

MFSDP_API int mfsdp_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w, const float* rstd,
                                        const void* dres, void* dx, void* dw, int accumulate_dw, long long rows,
                                        int H, cudaStream_t st) {
  if (rows <= 0 || H <= 0 || H % 8 || H > MFSDP_NOALLOC_MAX_HIDDEN) return -2;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kNoAllocMaxDevices) return -2;
  float* scratch = g_noalloc_scratch_addr[dev];
  if (scratch == nullptr) {
    // set-up, once per device, with that device current
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_dw_scratch);
    if (e != cudaSuccess) return (int)e;
    scratch = static_cast<float*>(p);
    g_noalloc_scratch_addr[dev] = scratch;
  }
  const int grid = launch_rmsnorm_bwd((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, rstd,
                                      (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, scratch, rows, H, MFSDP_NOALLOC_SCRATCH_ROWS, st);
  if (dw) launch_pdl(colsum_f32_to_bf16_kernel, dim3((H + 31) / 32), dim3(32, 8), 0, st, scratch, (__nv_bfloat16*)dw, grid, H, accumulate_dw);
  return (int)cudaGetLastError();
}
