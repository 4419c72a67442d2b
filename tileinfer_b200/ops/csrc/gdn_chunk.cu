// Chunk-parallel gated delta rule for prefill (WY / UT form), on the tensor cores.
//
// Replaces the reference's chunk kernel (kernels/gated_delta_rule_prefill.py:28-120: chunk 32, scalar FMA loops,
// and without the (v - S^T k) correction, i.e. not the delta rule) and the external flash_qla dependency
// (model/qwen_36.py:73-76).  The token-serial recurrence of gdn.cu stays for decode steps and short chunks.
//
// For a chunk of C = 64 tokens of one v-head (g = cumulative log decay inside the chunk, b = beta):
//     L[i][j]  = b_i (k_i . k_j) exp(g_i - g_j)             (i > j)
//     X        = (I + L)^-1                                   (unit lower triangular)
//     u        = X (b v)            w = X (b k exp(g))
//     v_new    = u - w S                                      S: state [dk, dv] before the chunk
//     out      = (q exp(g)) S + ((q k^T) * exp(g_i - g_j), i >= j) v_new
//     S       <- exp(g_C) S + (k exp(g_C - g))^T v_new
// Everything up to u and w does not depend on S: `gdn_chunk_prepare_kernel` computes it for ALL chunks and heads
// in parallel (causal conv + SiLU, q/k norms, gates, the two 64 x 64 Gram products, the blocked triangular inverse,
// u and w), and writes every operand of the scan in the register-fragment order of mma.sync.m16n8k16, so the scan
// fetches a fragment with one coalesced 16-byte load per lane and needs no shared-memory staging or ldmatrix.
// `gdn_chunk_scan_kernel` then walks the chunks of a sequence: one CTA per (v-head, 32 state columns, sequence),
// state slice S^T[32, dk] in fp32 accumulator registers; because the slice is kept TRANSPOSED, the accumulator
// fragment of the update is exactly the B fragment the next chunk's products need (bf16 copy in shared memory).
// `gdn_chunk_finish_kernel` applies the gated RMSNorm * silu(z); `gdn_conv_tail_kernel` writes the conv history.
// Chunks end at the block-aligned positions where a state snapshot is wanted (prefix cache), so snapshots are
// plain copies of the running state.  Matrix products are bf16 x bf16 with fp32 accumulation (u: two terms per operand).
#include <algorithm>

#include "common.cuh"
#include "mma_split.cuh"

namespace ti {

constexpr int kC = 64;   // chunk length
constexpr int kMaxHpc = 8;            // v-heads that one CTA of the prepare kernel takes at most
constexpr int kScale = 4 + 2 * kC;    // floats per (chunk, v-head) in `gamma`

struct GdnChunkParams {
  const __nv_bfloat16* proj;   // [T, ld]: q | k | v | z | b | a columns (per-rank head counts)
  const float* conv_w;         // [2*hk*DK + hv*DV, 4]
  const float* neg_a_exp;      // [hv]
  const float* dt_bias;        // [hv]
  const float* norm_w;         // [DV]
  void* state;                 // [slots, hv, DK, DV] fp32 or bf16
  __nv_bfloat16* conv_state;   // [slots, hv, 3, 2*DK + DV]
  const int* slots;            // [S]
  const int* cu;               // [S+1] token offsets
  __nv_bfloat16* out;          // [T, hv*DV]
  const int* snap_rel;         // [S, NS] snapshot after this many tokens of the step (<= 0: unused), or nullptr
  const int* snap_idx;         // [S, NS] entry of the snapshot buffers
  float* snap_state;           // [entries, hv, DK, DV]
  __nv_bfloat16* snap_conv;    // [entries, hv, 3, 2*DK + DV]
  // chunk table (chunks of a sequence are consecutive and in order)
  const int* ck_seq;           // [nc]
  const int* ck_tok0;          // [nc] first flat token
  const int* ck_ntok;          // [nc] 1..64
  const int* ck_snap;          // [nc] snapshot entry to write after this chunk, or -1
  const int* seq_ck;           // [S+1] chunk range of every sequence; one without chunks is left alone (a one-token sequence
                               // of a mixed step, which the decode kernels of gdn.cu advance)
  // workspace, fragment order (index ch = chunk * hv + v-head, ck = chunk * hk + k-head)
  uint4* wf;                   // [ch][4 m-tiles][DK/16 k-tiles][32 lanes]   A fragments of -w  (64 x DK)
  uint4* qf;                   // [ck][4][DK/16][32]                         A fragments of q DK^-1/2
  uint4* mf;                   // [ch][4][4][32]                             A fragments of the masked q k^T (64 x 64)
  uint2* kf;                   // [ck][4 k-tiles][DK/8 n-tiles][32]          B fragments of k (64 x DK)
  float* u;                    // [ch][64][DV]
  float* gamma;                // [ch][kScale]: exp(g_C), -, -, -, exp(g) of 64 tokens, exp(g_C - g) of 64 tokens
  int ld, hk, hv, num_snap, nc;
  float eps;
};

TI_DEVICE uint32_t lds32(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }
TI_DEVICE float bf(const __nv_bfloat16* p) { return __bfloat162float(*p); }

// ---------------------------------------------------------------------------------------------------------------
// Prepare: one CTA per (chunk, `hpc` v-heads of one k-head), 8 warps.
//
// The v-heads of a k-head share the convolved, normalised q and k and both Gram products; only gates, the triangular
// inverse, u and w are per v-head.  With many chunks a CTA does all v-heads of its k-head one after the other (the shared
// part is computed once: a third of the q / k convolutions and Gram products at 3 v-heads per k-head); with few chunks it
// does one, so that more SMs work (a prompt of 128 tokens is 2 chunks).
// Bound by latency, not by a pipe: chains of loads, shuffles and barriers.  Hence: a warp owns 8 consecutive tokens and
// requests the 11 raw rows that their 4-tap windows span at once (8 bytes per lane; it used to make 48 two-byte loads per
// token and wait for them token by token); tiles stay row-major in shared memory and meet the tensor cores through
// ldmatrix.trans (stores of transposed copies were 16-way bank conflicts); the diagonal blocks of the inverse are solved
// in registers; beta and the decay are folded into the columns of the inverse, and the decays of q and k into the scan, so
// that q and k fragments are written once per k-head.  4096 tokens, 16 k- and 48 v-heads of 128 x 128: 560 -> 203 us.
template <int DK, int DV>
struct PrepSmem {
  static constexpr int QS = DK + 8, VS = DV + 8;   // bf16 row strides (16 bytes modulo 128: conflict-free ldmatrix)
  static constexpr int LS = kC + 8, TS = 36;       // fp32 row strides of the triangular matrix and of its half products
  static constexpr size_t kBytes = (size_t)2 * kC * QS * 2 + (size_t)2 * kC * VS * 2 + (size_t)kC * LS * 4 + 32 * TS * 4 +
                                   kMaxHpc * 3 * kC * 4;
};

// E (2 or 4) adjacent bf16 values, packed in pairs; `vec`: the address is a multiple of 2 E bytes.
template <int E> TI_DEVICE void load_packed(uint32_t (&r)[E / 2], const __nv_bfloat16* p, bool vec) {
  if (vec) {
    if constexpr (E == 4) {
      const uint2 v = *reinterpret_cast<const uint2*>(p);
      r[0] = v.x;
      r[1] = v.y;
    } else {
      r[0] = *reinterpret_cast<const uint32_t*>(p);
    }
  } else {
    const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
    for (int i = 0; i < E / 2; ++i) r[i] = (uint32_t)u[2 * i] | ((uint32_t)u[2 * i + 1] << 16);
  }
}

// The raw inputs of this lane's E channels at flat tokens first .. first + 10 (zero from `last` on); tokens before the
// sequence's first one of this step come from the convolution history (row t + 3 of three).
template <int E>
TI_DEVICE void conv_load(uint32_t (&r)[11][E / 2], const __nv_bfloat16* col, int ld, const __nv_bfloat16* hist, int nch, int first,
                         int last, int seq_t0, bool vec) {
#pragma unroll
  for (int i = 0; i < 11; ++i) {
    const int t = first + i;
#pragma unroll
    for (int e = 0; e < E / 2; ++e) r[i][e] = 0;
    if (t < last) load_packed<E>(r[i], t < seq_t0 ? hist + (size_t)(t - seq_t0 + 3) * nch : col + (size_t)t * ld, vec);
  }
}

// silu(conv) of E channels at the token whose four inputs are rows j .. j + 3
template <int E> TI_DEVICE void conv_silu(float (&y)[E], const uint32_t (&r)[11][E / 2], const float4 (&w)[E], int j) {
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float x0 = e & 1 ? bf16hi(r[j][e / 2]) : bf16lo(r[j][e / 2]), x1 = e & 1 ? bf16hi(r[j + 1][e / 2]) : bf16lo(r[j + 1][e / 2]);
    const float x2 = e & 1 ? bf16hi(r[j + 2][e / 2]) : bf16lo(r[j + 2][e / 2]), x3 = e & 1 ? bf16hi(r[j + 3][e / 2]) : bf16lo(r[j + 3][e / 2]);
    y[e] = silu_f(w[e].x * x0 + w[e].y * x1 + w[e].z * x2 + w[e].w * x3);
  }
}

template <int E> TI_DEVICE void store_packed(__nv_bfloat16* p, const float (&y)[E]) {
  if constexpr (E == 4) *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]));
  else *reinterpret_cast<uint32_t*>(p) = pack_bf16(y[0], y[1]);
}

template <int DK, int DV>
__global__ void __launch_bounds__(256, 2) gdn_chunk_prepare_kernel(const __grid_constant__ GdnChunkParams p, int hpc) {
  using SM = PrepSmem<DK, DV>;
  constexpr int QS = SM::QS, VS = SM::VS, LS = SM::LS, TS = SM::TS, KT = DK / 16, NCH = 2 * DK + DV;
  constexpr int EQ = DK / 32, EV = DV / 32;       // channels per lane in the conv stage
  extern __shared__ __align__(16) uint8_t smem[];
  __nv_bfloat16* qn = reinterpret_cast<__nv_bfloat16*>(smem);     // [64][QS]  q / |q| / sqrt(DK)
  __nv_bfloat16* kn = qn + kC * QS;                               // [64][QS]  k / |k|
  __nv_bfloat16* vs = kn + kC * QS;                               // [2][64][VS]  v of one v-head as two bf16 terms
  float* Lm = reinterpret_cast<float*>(vs + 2 * kC * VS);         // [64][LS]  L, then X
  float* Tm = Lm + kC * LS;                                       // [32][TS]
  float* gates = Tm + 32 * TS;                                    // [hpc][3][64]: cumulative log decay, beta, beta exp(g)

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int ci = blockIdx.x, vh0 = blockIdx.y * hpc, rep = p.hv / p.hk, kh = vh0 / rep;
  const int s = p.ck_seq[ci], tok0 = p.ck_tok0[ci], n = p.ck_ntok[ci];
  const int seq_t0 = p.cu[s];
  const int slot = p.slots[s];
  const int bcol0 = 2 * p.hk * DK + 2 * p.hv * DV;
  // rows of the projection and of the history in vectors of a lane's channels (any other pitch is read value by value)
  const bool vec_q = p.ld % EQ == 0 && (reinterpret_cast<uintptr_t>(p.proj) | reinterpret_cast<uintptr_t>(p.conv_state)) % (2 * EQ) == 0;
  const bool vec_v = p.ld % EV == 0 && (reinterpret_cast<uintptr_t>(p.proj) | reinterpret_cast<uintptr_t>(p.conv_state)) % (2 * EV) == 0;
  const int first = tok0 + 8 * warp - 3, last = tok0 + n;
  float4 wq[EQ], wk[EQ];
#pragma unroll
  for (int e = 0; e < EQ; ++e) {
    wq[e] = *reinterpret_cast<const float4*>(p.conv_w + (size_t)(kh * DK + lane * EQ + e) * 4);
    wk[e] = *reinterpret_cast<const float4*>(p.conv_w + (size_t)(p.hk * DK + kh * DK + lane * EQ + e) * 4);
  }
  pdl_trigger();
  pdl_wait();

  const __nv_bfloat16* hist0 = p.conv_state + (size_t)slot * p.hv * 3 * NCH;
  uint32_t rv[11][EV / 2];
  auto load_v = [&](int vh) {
    conv_load<EV>(rv, p.proj + 2 * p.hk * DK + vh * DV + lane * EV, p.ld, hist0 + (size_t)vh * 3 * NCH + 2 * DK + lane * EV, NCH,
                  first, last, seq_t0, vec_v);
  };
  {
    // ---- B. causal conv + SiLU and norms of q and k: a warp per 8 consecutive tokens
    uint32_t rq[11][EQ / 2], rk[11][EQ / 2];
    const __nv_bfloat16* hist = hist0 + (size_t)vh0 * 3 * NCH + lane * EQ;
    conv_load<EQ>(rq, p.proj + kh * DK + lane * EQ, p.ld, hist, NCH, first, last, seq_t0, vec_q);
    conv_load<EQ>(rk, p.proj + p.hk * DK + kh * DK + lane * EQ, p.ld, hist + DK, NCH, first, last, seq_t0, vec_q);
    load_v(vh0);
    // ---- A. gates of every v-head: log decay, beta, inclusive scan over the chunk (lane -> tokens lane, lane + 32)
    for (int h = warp; h < hpc; h += 8) {
      const int vh = vh0 + h;
      const float neg_a = p.neg_a_exp[vh], dtb = p.dt_bias[vh];
      float gl[2], bb[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = lane + 32 * i;
        gl[i] = 0.f;
        bb[i] = 0.f;
        if (j < n) {
          const __nv_bfloat16* row = p.proj + (size_t)(tok0 + j) * p.ld + bcol0 + vh;
          const float a = bf(row + p.hv) + dtb;
          const float sp = a > 20.f ? a : log1pf(__expf(a));
          gl[i] = neg_a * sp;
          bb[i] = sigmoid_f(bf(row));
        }
      }
      float c0 = gl[0], c1 = gl[1];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float a0 = __shfl_up_sync(0xffffffffu, c0, o), a1 = __shfl_up_sync(0xffffffffu, c1, o);
        if (lane >= o) { c0 += a0; c1 += a1; }
      }
      c1 += __shfl_sync(0xffffffffu, c0, 31);
      const float glast = __shfl_sync(0xffffffffu, c1, 31);
      const float e0 = __expf(c0), e1 = __expf(c1);
      float* gt = gates + h * 3 * kC;
      gt[lane] = c0; gt[lane + 32] = c1;
      gt[kC + lane] = bb[0]; gt[kC + lane + 32] = bb[1];
      gt[2 * kC + lane] = bb[0] * e0; gt[2 * kC + lane + 32] = bb[1] * e1;
      float* sc = p.gamma + ((size_t)ci * p.hv + vh) * kScale;
      if (lane == 0) sc[0] = __expf(glast);
      sc[4 + lane] = e0; sc[4 + lane + 32] = e1;
      sc[4 + kC + lane] = __expf(glast - c0); sc[4 + kC + lane + 32] = __expf(glast - c1);
    }
    const float qscale = rsqrtf((float)DK);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float yq[EQ], yk[EQ], sq = 0.f, sk = 0.f;
      conv_silu<EQ>(yq, rq, wq, j);
      conv_silu<EQ>(yk, rk, wk, j);
#pragma unroll
      for (int e = 0; e < EQ; ++e) {
        sq += yq[e] * yq[e];
        sk += yk[e] * yk[e];
      }
      sq = warp_sum(sq);
      sk = warp_sum(sk);
      const bool live = 8 * warp + j < n;
      const float fq = live ? rsqrtf(sq + 1e-6f) * qscale : 0.f, fk = live ? rsqrtf(sk + 1e-6f) : 0.f;
#pragma unroll
      for (int e = 0; e < EQ; ++e) { yq[e] *= fq; yk[e] *= fk; }
      store_packed<EQ>(qn + (8 * warp + j) * QS + lane * EQ, yq);
      store_packed<EQ>(kn + (8 * warp + j) * QS + lane * EQ, yk);
    }
  }
  __syncthreads();

  // ---- C. k k^T and q k^T (64 x 64 each): warp -> m-tile (warp & 3), four n-tiles (warp >> 2); kept for all v-heads
  const int mtc = warp & 3, half = warp >> 2;
  float akk[4][4], aqk[4][4];
  {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) akk[a][b] = aqk[a][b] = 0.f;
    const __nv_bfloat16* kr0 = kn + (16 * mtc + g) * QS + 2 * t;
    const __nv_bfloat16* qr0 = qn + (16 * mtc + g) * QS + 2 * t;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
      const uint32_t k0 = lds32(kr0 + 16 * kt), k1 = lds32(kr0 + 8 * QS + 16 * kt), k2 = lds32(kr0 + 16 * kt + 8),
                     k3 = lds32(kr0 + 8 * QS + 16 * kt + 8);
      const uint32_t q0 = lds32(qr0 + 16 * kt), q1 = lds32(qr0 + 8 * QS + 16 * kt), q2 = lds32(qr0 + 16 * kt + 8),
                     q3 = lds32(qr0 + 8 * QS + 16 * kt + 8);
      // q as A fragments of the scan, once per k-head
      if (vh0 % rep == 0 && (kt & 1) == half)
        p.qf[((((size_t)ci * p.hk + kh) * 4 + mtc) * KT + kt) * 32 + lane] = make_uint4(q0, q1, q2, q3);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const __nv_bfloat16* br = kn + (8 * (4 * half + c) + g) * QS + 16 * kt + 2 * t;
        const uint32_t b0 = lds32(br), b1 = lds32(br + 8);
        mma_bf16_16816(akk[c], k0, k1, k2, k3, b0, b1);
        mma_bf16_16816(aqk[c], q0, q1, q2, q3, b0, b1);
      }
    }
    // k as B fragments (contraction over the tokens)
    if (vh0 % rep == 0) {
      uint2* kf = p.kf + (((size_t)ci * p.hk + kh) * 4 + mtc) * (DK / 8) * 32 + lane;
#pragma unroll
      for (int c = half; c < DK / 16; c += 2) {
        uint32_t r[4];
        ldsm4t(r, kn + (16 * mtc + (lane & 15)) * QS + 16 * c + (lane >> 4) * 8);
        kf[(2 * c) * 32] = make_uint2(r[0], r[1]);
        kf[(2 * c + 1) * 32] = make_uint2(r[2], r[3]);
      }
    }
  }

  for (int h = 0; h < hpc; ++h) {
    const int vh = vh0 + h;
    const size_t ch = (size_t)ci * p.hv + vh;
    const float *gc = gates + h * 3 * kC, *bet = gc + kC, *bge = bet + kC;
    // ---- v = silu(conv): row-major
    {
      float4 wv[EV];
#pragma unroll
      for (int e = 0; e < EV; ++e) wv[e] = *reinterpret_cast<const float4*>(p.conv_w + (size_t)(2 * p.hk * DK + vh * DV + lane * EV + e) * 4);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float y[EV];
        conv_silu<EV>(y, rv, wv, j);
        if (8 * warp + j >= n)
#pragma unroll
          for (int e = 0; e < EV; ++e) y[e] = 0.f;
        store_packed<EV>(vs + (8 * warp + j) * VS + lane * EV, y);
#pragma unroll
        for (int e = 0; e < EV; ++e) y[e] -= round_bf16(y[e]);
        store_packed<EV>(vs + kC * VS + (8 * warp + j) * VS + lane * EV, y);
      }
      if (h + 1 < hpc) load_v(vh + 1);               // requested ahead: a head's inverse hides the latency
    }
    // ---- L and the masked q k^T of this head
    {
      const int i0 = 16 * mtc + g, i1 = i0 + 8;
      const float g0 = gc[i0], g1 = gc[i1], be0 = bet[i0], be1 = bet[i1];
      uint32_t mpk[4][2];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int j0 = 8 * (4 * half + c) + 2 * t, j1 = j0 + 1;
        const float gj0 = gc[j0], gj1 = gc[j1];
        const float d00 = i0 >= j0 ? __expf(g0 - gj0) : 0.f, d01 = i0 >= j1 ? __expf(g0 - gj1) : 0.f;
        const float d10 = i1 >= j0 ? __expf(g1 - gj0) : 0.f, d11 = i1 >= j1 ? __expf(g1 - gj1) : 0.f;
        *reinterpret_cast<float2*>(Lm + i0 * LS + j0) = make_float2(i0 > j0 ? be0 * akk[c][0] * d00 : 0.f, i0 > j1 ? be0 * akk[c][1] * d01 : 0.f);
        *reinterpret_cast<float2*>(Lm + i1 * LS + j0) = make_float2(i1 > j0 ? be1 * akk[c][2] * d10 : 0.f, i1 > j1 ? be1 * akk[c][3] * d11 : 0.f);
        mpk[c][0] = pack_bf16(aqk[c][0] * d00, aqk[c][1] * d01);
        mpk[c][1] = pack_bf16(aqk[c][2] * d10, aqk[c][3] * d11);
      }
      // accumulator tiles (2kt, 2kt+1) -> A fragment of k-tile kt
#pragma unroll
      for (int kk = 0; kk < 2; ++kk)
        p.mf[((ch * 4 + mtc) * 4 + 2 * half + kk) * 32 + lane] =
            make_uint4(mpk[2 * kk][0], mpk[2 * kk][1], mpk[2 * kk + 1][0], mpk[2 * kk + 1][1]);
    }
    __syncthreads();

    // ---- D. X = (I + L)^-1, fp32, blocked: 16 x 16 diagonal blocks by forward substitution (a column per lane, in
    //         registers), then X21 = -X22 (L21 X11) for the 16- and the 32-blocks.  In place in Lm.
    if (warp < 4 && lane < 16) {
      float* blk = Lm + 16 * warp * LS + 16 * warp;
      float x[16];
#pragma unroll
      for (int ii = 0; ii < 16; ++ii) {
        float acc = ii == lane ? 1.f : 0.f;
#pragma unroll
        for (int m = 0; m < ii; ++m) acc -= blk[ii * LS + m] * x[m];
        x[ii] = acc;
      }
      __syncwarp(0xffffu);
#pragma unroll
      for (int ii = 0; ii < 16; ++ii) blk[ii * LS + lane] = x[ii];
    }
    __syncthreads();
    {
      const int base = 32 * (tid >> 7), r = (tid >> 3) & 15, c = (tid & 7) * 2;
      const float* L21 = Lm + (base + 16 + r) * LS + base;
      float2 a = make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const float2 b = *reinterpret_cast<const float2*>(Lm + (base + m) * LS + base + c);
        a.x += L21[m] * b.x;
        a.y += L21[m] * b.y;
      }
      float* T = Tm + (tid >> 7) * 16 * TS;
      *reinterpret_cast<float2*>(T + r * TS + c) = a;
      __syncthreads();
      a = make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const float2 b = *reinterpret_cast<const float2*>(T + m * TS + c);
        a.x -= L21[16 + m] * b.x;
        a.y -= L21[16 + m] * b.y;
      }
      *reinterpret_cast<float2*>(Lm + (base + 16 + r) * LS + base + c) = a;
    }
    __syncthreads();
    {
      const int r = tid >> 3, c = (tid & 7) * 4;
      const float* L21 = Lm + (32 + r) * LS;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (int m = 0; m < 32; ++m) {
        const float4 b = *reinterpret_cast<const float4*>(Lm + m * LS + c);
        const float l = L21[m];
        a.x += l * b.x; a.y += l * b.y; a.z += l * b.z; a.w += l * b.w;
      }
      *reinterpret_cast<float4*>(Tm + r * TS + c) = a;
      __syncthreads();
      a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (int m = 0; m < 32; ++m) {
        const float4 b = *reinterpret_cast<const float4*>(Tm + m * TS + c);
        const float l = L21[32 + m];
        a.x -= l * b.x; a.y -= l * b.y; a.z -= l * b.z; a.w -= l * b.w;
      }
      *reinterpret_cast<float4*>(Lm + (32 + r) * LS + c) = a;
    }
    __syncthreads();

    // ---- E. u = (X b) v, -w = -(X b exp(g)) k: warp -> m-tile, half of the columns.  X is lower triangular: m-tile mt
    //         meets mt + 1 k-tiles, so the two warps of a scheduler (warp & 3) take m-tiles i and 3 - i.  u is kept in fp32
    //         and is what the state is made of, so X b and v enter as two bf16 terms each (three products): against the
    //         token-by-token rule in 64 bits outputs 0.40 -> 0.33 %, states 0.33 -> 0.23 %, for 18 us in 4096 tokens.
    {
      const int mt = warp < 4 ? warp : 7 - warp;
      uint32_t xu[4][4], xl[4][4], xw[4][4];
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        if (kt > mt) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {                         // fragment order: (row, k), (row + 8, k), (row, k + 8), (row + 8, k + 8)
          const int col = 16 * kt + 2 * t + 8 * (i >> 1);
          const float2 x = *reinterpret_cast<const float2*>(Lm + (16 * mt + g + 8 * (i & 1)) * LS + col);
          const float2 b = *reinterpret_cast<const float2*>(bet + col), be = *reinterpret_cast<const float2*>(bge + col);
          split2(x.x * b.x, x.y * b.y, xu[kt][i], xl[kt][i]);
          xw[kt][i] = pack_bf16(-x.x * be.x, -x.y * be.y);
        }
      }
      float* urow0 = p.u + (ch * kC + 16 * mt + g) * DV;
#pragma unroll 2
      for (int c = 0; c < DV / 32; ++c) {
        const int nt = half * (DV / 16) + 2 * c;
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
          if (kt > mt) continue;
          uint32_t b[4];
          ldsm4t(b, vs + (16 * kt + (lane & 15)) * VS + 8 * nt + (lane >> 4) * 8);
          mma_bf16_16816(acc[0], xu[kt][0], xu[kt][1], xu[kt][2], xu[kt][3], b[0], b[1]);
          mma_bf16_16816(acc[1], xu[kt][0], xu[kt][1], xu[kt][2], xu[kt][3], b[2], b[3]);
          mma_bf16_16816(acc[0], xl[kt][0], xl[kt][1], xl[kt][2], xl[kt][3], b[0], b[1]);
          mma_bf16_16816(acc[1], xl[kt][0], xl[kt][1], xl[kt][2], xl[kt][3], b[2], b[3]);
          ldsm4t(b, vs + kC * VS + (16 * kt + (lane & 15)) * VS + 8 * nt + (lane >> 4) * 8);
          mma_bf16_16816(acc[0], xu[kt][0], xu[kt][1], xu[kt][2], xu[kt][3], b[0], b[1]);
          mma_bf16_16816(acc[1], xu[kt][0], xu[kt][1], xu[kt][2], xu[kt][3], b[2], b[3]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          *reinterpret_cast<float2*>(urow0 + 8 * (nt + i) + 2 * t) = make_float2(acc[i][0], acc[i][1]);
          *reinterpret_cast<float2*>(urow0 + 8 * DV + 8 * (nt + i) + 2 * t) = make_float2(acc[i][2], acc[i][3]);
        }
      }
#pragma unroll 2
      for (int c = 0; c < KT / 2; ++c) {
        const int kt2 = half * (KT / 2) + c;                    // k-tile of w = pair of accumulator n-tiles
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
          if (kt > mt) continue;
          uint32_t b[4];
          ldsm4t(b, kn + (16 * kt + (lane & 15)) * QS + 16 * kt2 + (lane >> 4) * 8);
          mma_bf16_16816(acc[0], xw[kt][0], xw[kt][1], xw[kt][2], xw[kt][3], b[0], b[1]);
          mma_bf16_16816(acc[1], xw[kt][0], xw[kt][1], xw[kt][2], xw[kt][3], b[2], b[3]);
        }
        p.wf[((ch * 4 + mt) * KT + kt2) * 32 + lane] = make_uint4(pack_bf16(acc[0][0], acc[0][1]), pack_bf16(acc[0][2], acc[0][3]),
                                                                 pack_bf16(acc[1][0], acc[1][1]), pack_bf16(acc[1][2], acc[1][3]));
      }
    }
    if (h + 1 < hpc) __syncthreads();                           // the next head overwrites v and L
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Scan: one CTA (4 warps) per (v-head, 32 state columns, sequence).
// A serial chain per chunk: products with the state, barrier, products with v_new, barrier.  The operands come from L2 in
// fragment order straight into registers, and each group is requested one phase ahead (w, q, u of the next chunk while
// v_new is used; M and k of this chunk while the state is used): without that every phase began with a memory round trip.
// The decays of q (rows of the output) and k (rows of v_new) are applied to fp32 accumulators here.  4096 tokens, 48 v-heads
// of 128 x 128 (64 chunks in a row): 427 -> 211 us.
template <typename ST> TI_DEVICE float ldst(const ST* p);
template <> TI_DEVICE float ldst<float>(const float* p) { return *p; }
template <> TI_DEVICE float ldst<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename ST> TI_DEVICE void stst(ST* p, float v);
template <> TI_DEVICE void stst<float>(float* p, float v) { *p = v; }
template <> TI_DEVICE void stst<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

template <int DK, int DV, typename ST>
__global__ void __launch_bounds__(128, 2) gdn_chunk_scan_kernel(const __grid_constant__ GdnChunkParams p) {
  constexpr int DVB = 32, NB = DV / DVB, KT = DK / 16, NTV = DVB / 8, NTW = DK / 32, MTS = DVB / 16;
  constexpr int SS = DK + 8, VS = DVB + 8;                      // 16 bytes modulo 128 (80 for VS): conflict-free ldmatrix
  __shared__ __align__(16) __nv_bfloat16 Sb[DVB * SS];          // S^T (bf16): row = state column, pairs along dk
  __shared__ __align__(16) __nv_bfloat16 vn[2][kC * VS];        // v_new (bf16, row-major), double-buffered by chunk
  __shared__ __align__(16) __nv_bfloat16 ve[2][kC * VS];        // v_new exp(g_C - g)

  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int vh = blockIdx.x / NB, dv0 = (blockIdx.x % NB) * DVB, s = blockIdx.y, kh = vh / (p.hv / p.hk);
  const int c_lo = p.seq_ck[s], c_hi = p.seq_ck[s + 1];
  if (c_lo == c_hi) return;                                      // not this kernel's sequence: its state is not touched
  const int slot = p.slots[s];
  ST* Sp = static_cast<ST*>(p.state) + ((size_t)slot * p.hv + vh) * DK * DV;
  const int dk0 = w * (DK / 4);                                  // this warp's slice of dk in the state update

  // state slice as S^T accumulator fragments: sT[mt][j] covers rows (state columns) 16mt + g (+8), dk = dk0 + 8j + 2t (+1)
  float sT[MTS][NTW][4];
#pragma unroll
  for (int mt = 0; mt < MTS; ++mt)
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
      const int d = dk0 + 8 * j + 2 * t, c = dv0 + 16 * mt + g;
      sT[mt][j][0] = ldst<ST>(Sp + (size_t)d * DV + c);
      sT[mt][j][1] = ldst<ST>(Sp + (size_t)(d + 1) * DV + c);
      sT[mt][j][2] = ldst<ST>(Sp + (size_t)d * DV + c + 8);
      sT[mt][j][3] = ldst<ST>(Sp + (size_t)(d + 1) * DV + c + 8);
    }
  auto publish_state = [&]() {
#pragma unroll
    for (int mt = 0; mt < MTS; ++mt)
#pragma unroll
      for (int j = 0; j < NTW; ++j) {
        const int d = dk0 + 8 * j + 2 * t;
        *reinterpret_cast<uint32_t*>(Sb + (16 * mt + g) * SS + d) = pack_bf16(sT[mt][j][0], sT[mt][j][1]);
        *reinterpret_cast<uint32_t*>(Sb + (16 * mt + g + 8) * SS + d) = pack_bf16(sT[mt][j][2], sT[mt][j][3]);
      }
  };
  publish_state();
  pdl_trigger();
  pdl_wait();                                                    // the operands come from the prepare kernel

  // operands of the products with the state: -w, q, u rows of this warp, decays
  uint4 aw[KT], aq[KT];
  float2 uu[NTV][2];
  float gam, eq0, eq1, ek0, ek1;
  auto load_a = [&](int ci) {
    const size_t ch = (size_t)ci * p.hv + vh, ck = (size_t)ci * p.hk + kh;
    const uint4* wfp = p.wf + ((ch * 4 + w) * KT) * 32 + lane;
    const uint4* qfp = p.qf + ((ck * 4 + w) * KT) * 32 + lane;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
      aw[kt] = __ldg(wfp + kt * 32);
      aq[kt] = __ldg(qfp + kt * 32);
    }
    const float* urow = p.u + (ch * kC + 16 * w + g) * DV + dv0 + 2 * t;
#pragma unroll
    for (int nt = 0; nt < NTV; ++nt) {
      uu[nt][0] = __ldg(reinterpret_cast<const float2*>(urow + 8 * nt));
      uu[nt][1] = __ldg(reinterpret_cast<const float2*>(urow + 8 * DV + 8 * nt));
    }
    const float* sc = p.gamma + ch * kScale;
    gam = __ldg(sc);
    eq0 = __ldg(sc + 4 + 16 * w + g);
    eq1 = __ldg(sc + 4 + 16 * w + g + 8);
    ek0 = __ldg(sc + 4 + kC + 16 * w + g);
    ek1 = __ldg(sc + 4 + kC + 16 * w + g + 8);
  };
  load_a(c_lo);
  __syncthreads();

  for (int ci = c_lo; ci < c_hi; ++ci) {
    const size_t ch = (size_t)ci * p.hv + vh, ck = (size_t)ci * p.hk + kh;
    const int ntok = p.ck_ntok[ci], tok0 = p.ck_tok0[ci];
    __nv_bfloat16 *vb = vn[(ci - c_lo) & 1], *eb = ve[(ci - c_lo) & 1];
    // operands of the products with v_new, wanted after the barrier
    uint4 am[4];
    uint2 kb[4][NTW];
    const uint4* mfp = p.mf + ((ch * 4 + w) * 4) * 32 + lane;
    const uint2* kfp = p.kf + (ck * 4 * (DK / 8)) * 32 + lane;
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      am[kt] = kt <= w ? __ldg(mfp + kt * 32) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < NTW; ++j) kb[kt][j] = __ldg(kfp + (kt * (DK / 8) + w * NTW + j) * 32);
    }
    // ---- v_new rows of this warp = u - w S ; o rows = exp(g) (q S)
    float av[NTV][4], ao[NTV][4];
#pragma unroll
    for (int nt = 0; nt < NTV; ++nt) {
      av[nt][0] = uu[nt][0].x; av[nt][1] = uu[nt][0].y; av[nt][2] = uu[nt][1].x; av[nt][3] = uu[nt][1].y;
      ao[nt][0] = ao[nt][1] = ao[nt][2] = ao[nt][3] = 0.f;
    }
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
#pragma unroll
      for (int nt = 0; nt < NTV; nt += 2) {
        uint32_t b[4];                                          // two n-tiles: rows 8nt.. of S^T, dk 16kt..
        ldsm4(b, Sb + (8 * nt + (lane & 7) + (lane >> 4) * 8) * SS + 16 * kt + ((lane >> 3) & 1) * 8);
        mma_bf16_16816(av[nt], aw[kt].x, aw[kt].y, aw[kt].z, aw[kt].w, b[0], b[1]);
        mma_bf16_16816(av[nt + 1], aw[kt].x, aw[kt].y, aw[kt].z, aw[kt].w, b[2], b[3]);
        mma_bf16_16816(ao[nt], aq[kt].x, aq[kt].y, aq[kt].z, aq[kt].w, b[0], b[1]);
        mma_bf16_16816(ao[nt + 1], aq[kt].x, aq[kt].y, aq[kt].z, aq[kt].w, b[2], b[3]);
      }
    }
    const float gamma = gam;
#pragma unroll
    for (int nt = 0; nt < NTV; ++nt) {
      const int at = (16 * w + g) * VS + 8 * nt + 2 * t;
      *reinterpret_cast<uint32_t*>(vb + at) = pack_bf16(av[nt][0], av[nt][1]);
      *reinterpret_cast<uint32_t*>(vb + at + 8 * VS) = pack_bf16(av[nt][2], av[nt][3]);
      *reinterpret_cast<uint32_t*>(eb + at) = pack_bf16(av[nt][0] * ek0, av[nt][1] * ek0);
      *reinterpret_cast<uint32_t*>(eb + at + 8 * VS) = pack_bf16(av[nt][2] * ek1, av[nt][3] * ek1);
      ao[nt][0] *= eq0; ao[nt][1] *= eq0; ao[nt][2] *= eq1; ao[nt][3] *= eq1;
    }
    if (ci + 1 < c_hi) load_a(ci + 1);
    __syncthreads();
    // ---- o rows += (masked q k^T) v_new : the k-tiles above the diagonal are zero
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      if (kt > w) continue;
#pragma unroll
      for (int nt = 0; nt < NTV; nt += 2) {
        uint32_t b[4];
        ldsm4t(b, vb + (16 * kt + (lane & 15)) * VS + 8 * nt + (lane >> 4) * 8);
        mma_bf16_16816(ao[nt], am[kt].x, am[kt].y, am[kt].z, am[kt].w, b[0], b[1]);
        mma_bf16_16816(ao[nt + 1], am[kt].x, am[kt].y, am[kt].z, am[kt].w, b[2], b[3]);
      }
    }
    {
      const int r0 = 16 * w + g, r1 = r0 + 8;
      __nv_bfloat16* o0 = p.out + (size_t)(tok0 + r0) * p.hv * DV + vh * DV + dv0 + 2 * t;
      __nv_bfloat16* o1 = p.out + (size_t)(tok0 + r1) * p.hv * DV + vh * DV + dv0 + 2 * t;
#pragma unroll
      for (int nt = 0; nt < NTV; ++nt) {
        if (r0 < ntok) *reinterpret_cast<uint32_t*>(o0 + 8 * nt) = pack_bf16(ao[nt][0], ao[nt][1]);
        if (r1 < ntok) *reinterpret_cast<uint32_t*>(o1 + 8 * nt) = pack_bf16(ao[nt][2], ao[nt][3]);
      }
    }
    // ---- S^T slice <- gamma S^T + (v_new exp(g_C - g))^T k
#pragma unroll
    for (int mt = 0; mt < MTS; ++mt)
#pragma unroll
      for (int j = 0; j < NTW; ++j) {
        sT[mt][j][0] *= gamma; sT[mt][j][1] *= gamma; sT[mt][j][2] *= gamma; sT[mt][j][3] *= gamma;
      }
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
#pragma unroll
      for (int mt = 0; mt < MTS; ++mt) {
        uint32_t a[4];                                          // A = v_new^T: 16 state columns x 16 tokens of the row-major tile
        ldsm4t(a, eb + (16 * kt + (lane & 7) + (lane >> 4) * 8) * VS + 16 * mt + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int j = 0; j < NTW; ++j) mma_bf16_16816(sT[mt][j], a[0], a[1], a[2], a[3], kb[kt][j].x, kb[kt][j].y);
      }
    }
    publish_state();
    const int snap = p.ck_snap[ci];
    if (snap >= 0) {
      float* dst = p.snap_state + ((size_t)snap * p.hv + vh) * DK * DV;
#pragma unroll
      for (int mt = 0; mt < MTS; ++mt)
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
          const int d = dk0 + 8 * j + 2 * t, c = dv0 + 16 * mt + g;
          dst[(size_t)d * DV + c] = sT[mt][j][0];
          dst[(size_t)(d + 1) * DV + c] = sT[mt][j][1];
          dst[(size_t)d * DV + c + 8] = sT[mt][j][2];
          dst[(size_t)(d + 1) * DV + c + 8] = sT[mt][j][3];
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int mt = 0; mt < MTS; ++mt)
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
      const int d = dk0 + 8 * j + 2 * t, c = dv0 + 16 * mt + g;
      stst<ST>(Sp + (size_t)d * DV + c, sT[mt][j][0]);
      stst<ST>(Sp + (size_t)(d + 1) * DV + c, sT[mt][j][1]);
      stst<ST>(Sp + (size_t)d * DV + c + 8, sT[mt][j][2]);
      stst<ST>(Sp + (size_t)(d + 1) * DV + c + 8, sT[mt][j][3]);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Finish: gated RMSNorm over the head * silu(z), in place on the un-normalised output.  A warp per kFinish neighbouring
// (token, v-head) items, all of whose rows are requested before the first is used (bound by HBM: three rows of 2 DV bytes
// per item).
constexpr int kFinish = 4;
template <int DV>
__global__ void __launch_bounds__(256) gdn_chunk_finish_kernel(const __grid_constant__ GdnChunkParams p, int T, int DK) {
  constexpr int E = DV / 32;
  const int item0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * kFinish, lane = threadIdx.x & 31, items = T * p.hv;
  const bool vec = p.ld % E == 0 && (reinterpret_cast<uintptr_t>(p.proj) | reinterpret_cast<uintptr_t>(p.out)) % (2 * E) == 0;
  float nw[E];
#pragma unroll
  for (int e = 0; e < E; ++e) nw[e] = p.norm_w[lane * E + e];
  pdl_trigger();
  pdl_wait();
  uint32_t o[kFinish][E / 2], z[kFinish][E / 2];
#pragma unroll
  for (int i = 0; i < kFinish; ++i) {
    const int item = min(item0 + i, items - 1), tok = item / p.hv, vh = item - tok * p.hv;
    load_packed<E>(o[i], p.out + (size_t)item * DV + lane * E, vec);
    load_packed<E>(z[i], p.proj + (size_t)tok * p.ld + 2 * p.hk * DK + p.hv * DV + vh * DV + lane * E, vec);
  }
#pragma unroll
  for (int i = 0; i < kFinish; ++i) {
    if (item0 + i >= items) break;
    float v[E], ss = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      v[e] = e & 1 ? bf16hi(o[i][e / 2]) : bf16lo(o[i][e / 2]);
      ss += v[e] * v[e];
    }
    ss = warp_sum(ss);
    const float rr = rsqrtf(ss / (float)DV + p.eps);
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] *= rr * nw[e] * silu_f(e & 1 ? bf16hi(z[i][e / 2]) : bf16lo(z[i][e / 2]));
    __nv_bfloat16* dst = p.out + (size_t)(item0 + i) * DV + lane * E;
    if (vec) {
      store_packed<E>(dst, v);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) dst[e] = __float2bfloat16_rn(v[e]);
    }
  }
}

// Conv history after the step (z = 0) and at the snapshot points (z = 1 + point): the raw inputs of the last three
// tokens before that position.  Grid (S, hv, 1 + num_snap).  A point in the first two tokens of the step (the rest of a prompt
// that ends a block there) still reads the old history, which the z = 0 block overwrites: that block writes those points itself,
// each thread those of its channels, ahead of the history.
__global__ void __launch_bounds__(128) gdn_conv_tail_kernel(const __grid_constant__ GdnChunkParams p, int DK, int DV) {
  const int s = blockIdx.x, vh = blockIdx.y, z = blockIdx.z;
  const int NCH = 2 * DK + DV;
  const int kh = vh / (p.hv / p.hk);
  if (p.seq_ck[s] == p.seq_ck[s + 1]) return;
  const int t0 = p.cu[s], n = p.cu[s + 1] - t0;
  __nv_bfloat16* hist = p.conv_state + ((size_t)p.slots[s] * p.hv + vh) * 3 * NCH;
  auto point = [&](int j) { return p.snap_rel[s * p.num_snap + j]; };
  auto entry = [&](int j) { return p.snap_conv + ((size_t)p.snap_idx[s * p.num_snap + j] * p.hv + vh) * 3 * NCH; };
  if (z > 0 && (point(z - 1) < 3 || point(z - 1) > n)) return;
  for (int c = threadIdx.x; c < NCH; c += blockDim.x) {
    const int col = c < DK ? kh * DK + c : (c < 2 * DK ? p.hk * DK + kh * DK + (c - DK) : 2 * p.hk * DK + vh * DV + (c - 2 * DK));
    auto write = [&](__nv_bfloat16* dst, int end) {           // the three inputs before token `end` of the step
      __nv_bfloat16 v[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int ti = end - 3 + j;                           // token of the step (negative: older than the step)
        v[j] = ti >= 0 ? p.proj[(size_t)(t0 + ti) * p.ld + col] : hist[(size_t)(3 + ti) * NCH + c];
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) dst[(size_t)j * NCH + c] = v[j];
    };
    if (z > 0) {
      write(entry(z - 1), point(z - 1));
      continue;
    }
    for (int j = 0; p.snap_rel != nullptr && j < p.num_snap; ++j)
      if (point(j) > 0 && point(j) < 3 && point(j) <= n) write(entry(j), point(j));
    write(hist, n);
  }
}

template <int DK, int DV>
static int launch_chunked(const GdnChunkParams& p, int S, int T, int state_bf16, cudaStream_t st) {
  auto prep = gdn_chunk_prepare_kernel<DK, DV>;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PrepSmem<DK, DV>::kBytes);
    configured = true;
  }
  // All v-heads of a k-head in one CTA once that leaves every SM two CTAs, one v-head per CTA otherwise (128 tokens, 16 k-
  // and 48 v-heads: 96 CTAs instead of 32, each a third as long).
  const int rep = p.hv / p.hk, hpc = rep <= kMaxHpc && (long long)p.nc * p.hk >= 2 * 148 ? rep : 1;
  cudaError_t e = launch_kernel(prep, dim3(p.nc, p.hv / hpc), dim3(256), PrepSmem<DK, DV>::kBytes, st, true, p, hpc);
  if (e != cudaSuccess) return (int)e;
  const dim3 sgrid(p.hv * (DV / 32), S);
  if (state_bf16) e = launch_kernel(gdn_chunk_scan_kernel<DK, DV, __nv_bfloat16>, sgrid, dim3(128), 0, st, true, p);
  else e = launch_kernel(gdn_chunk_scan_kernel<DK, DV, float>, sgrid, dim3(128), 0, st, true, p);
  if (e != cudaSuccess) return (int)e;
  e = launch_kernel(gdn_chunk_finish_kernel<DV>, dim3((T * p.hv + 8 * kFinish - 1) / (8 * kFinish)), dim3(256), 0, st, true, p, T, DK);
  if (e != cudaSuccess) return (int)e;
  // not a programmatic launch: it overwrites the conv history the prepare kernel reads
  gdn_conv_tail_kernel<<<dim3(S, p.hv, 1 + (p.snap_rel != nullptr ? p.num_snap : 0)), 128, 0, st>>>(p, DK, DV);
  return (int)cudaGetLastError();
}

}  // namespace ti

extern "C" {

int ti_gdn_chunk_params_size() { return (int)sizeof(ti::GdnChunkParams); }

// Bytes of workspace per (chunk, v-head): wf, qf, mf, kf, u, gamma (in this order, see GdnChunkParams).
int ti_gdn_chunk_ws_bytes(int dk, int dv, int which) {
  switch (which) {
    case 0: case 1: return 4 * (dk / 16) * 32 * 16;
    case 2: return 4 * 4 * 32 * 16;
    case 3: return 4 * (dk / 8) * 32 * 8;
    case 4: return 64 * dv * 4;
    default: return 4 * ti::kScale;
  }
}

// Chunked prefill of the gated DeltaNet mixer for a flattened batch (see the file comment): prepare, scan, finish,
// conv tail.  `num_seqs` sequences, `T` tokens; the chunk table in `p` covers every token of a sequence, or none (its rows of
// `out` are then undefined).
int ti_gdn_chunked(const ti::GdnChunkParams* p, int num_seqs, int T, int dk, int dv, int state_bf16, void* stream) {
  if (num_seqs <= 0 || p->nc <= 0) return 0;
  if (p->hv % p->hk) return -2;
  cudaStream_t st = (cudaStream_t)stream;
  if (dk == 128 && dv == 128) return ti::launch_chunked<128, 128>(*p, num_seqs, T, state_bf16, st);
  if (dk == 64 && dv == 64) return ti::launch_chunked<64, 64>(*p, num_seqs, T, state_bf16, st);
  return -3;
}

}  // extern "C"
