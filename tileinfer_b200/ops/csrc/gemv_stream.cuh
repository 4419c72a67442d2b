// The products of a decode step of one activation row on one GPU, and some bf16 ones of up to 8 rows (stream_rows): weights streamed
// through ONE ring per CTA.
//
// The other form (gemv_body, for packets between ranks and for several rows) gives every warp units of its own, a private
// ring and a lane that schedules and copies.  Its launch of a 27B layer's four products (383 MB, 58.5 us at the measured copy
// rate) took 87.5 us, and as long with weights that stay in L2: 6 shared-memory loads and 8 MMAs per KB of weights, a lane's copy
// and scheduling work in between, warps that end a product up to 15 us apart, and rings (128 KB) that are full long before the
// barrier between two products has been passed.  Here
//   * a CTA's row tiles of a product are fixed (those that do not divide evenly go to other CTAs in each product of a launch), and
//     all 16 consumer warps work on the same two row tiles, a k tile each: they end within a stage of one another;
//   * two warps copy, a row tile's half of a stage of 16 KB (two row tiles x 16 k tiles) each, through all the stages that fit (11
//     at K = 17408); they run on into the next product's weights while that product's row is being waited for and staged.  One
//     warp's wait and two copies a stage took longer than HBM needs for the bytes;
//   * the weights are the MMA's A operand, 16 rows at a time, the activation rows (at most 8) its columns: 4 shared-memory loads
//     and 4 MMAs per KB in int8 (one row: 3 and 2), where lanes without an activation row load nothing;
//   * sums of a unit (two row tiles) of the 16 warps meet in shared memory, as integers for int8 weights (so they are exact
//     whatever the split); one warp adds them up and runs the epilogue, its operands requested ahead;
//   * one row goes to the next product as packets that its consumers poll; several rows, and one that registers do not hold, behind a
//     grid barrier.
// Roles (608 threads): warps 0..15 consume, warps 16 and 18 copy, warp 17 is the epilogue.  Every wait is bounded.
#pragma once

namespace ti {

constexpr int kStreamThreads = kThreads + 96, kStreamCopyB = kWarps + 2;
constexpr int kStreamStage = 2 * kWarps * 512;
// Stages a copying warp has under way at most: 96 KB per SM keep HBM busy, and what goes from one product to the next does not wait
// behind a whole ring of weights (chain of the 27B layer: all 11 under way 74.3 us, 8 69.6, 6 69.2, 4 69.7).
constexpr int kStreamFlight = 6;
constexpr int kStreamMaxRows = 8, kStreamMaxStages = 12, kStreamMinStages = 4, kStreamMaxSlots = 4;
constexpr unsigned long long kStreamWaitNs = 2000000000ull, kStreamDrainNs = 20000000ull;

struct Consumers {
  static TI_DEVICE int threads() { return kThreads; }
  static TI_DEVICE void sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(kThreads) : "memory"); }
};
TI_DEVICE void sync_with_epilogue() { asm volatile("bar.sync 2, %0;\n" ::"n"(kThreads + 32) : "memory"); }
TI_DEVICE void tell_epilogue() { asm volatile("bar.arrive 2, %0;\n" ::"n"(kThreads + 32) : "memory"); }

// A CTA's part of a product: a slice of a pair of left-over row tiles (or none), then row tiles first .. first + count.
// Left-over tiles, one for some of the CTAs, lengthen a product of few row tiles per CTA (N = 5120: 640 tiles, 4.3 for each of 148
// CTAs): the pairs of those are cut along k among the CTAs, and the last CTA of a pair to be done adds the slices up in their order
// (5120 x 17408 19.4 -> 16.6 us).  Taken first, so that the round trips of that are hidden; below 256 KB per CTA they are not.  From
// 16 tiles per CTA on one more is 6 % at most.  Otherwise left-over tiles are dealt whole.
struct StreamPart {
  int first, count, per;                           // whole row tiles; k tiles per stage
  int pair, slice, slices, kt0, kt1, split_per;    // pair of left-over tiles (-1: none), its slice kt0 .. kt1, k tiles per stage
};
constexpr int kStreamSplitBelow = 16, kStreamSplitTiles = 8, kStreamSplitBytes = 256 * 1024;      // row tiles per CTA; k tiles of a slice at least; bytes per CTA
TI_HOST_DEVICE int stream_per(int kts) {
  const int n = (kts + kWarps - 1) / kWarps;
  return (kts + n - 1) / n;
}
TI_HOST_DEVICE int stream_slices(int n_tiles, int KB, int ncta) {
  const int base = n_tiles / ncta, pairs = (n_tiles - base * ncta + 1) / 2;
  if (pairs == 0 || base >= kStreamSplitBelow || (long long)n_tiles * KB * 512 < (long long)kStreamSplitBytes * ncta) return 1;
  const int most = KB / kStreamSplitTiles, s = ncta / pairs < most ? ncta / pairs : most;
  return s < 1 ? 1 : (s < 16 ? s : 16);
}
TI_HOST_DEVICE StreamPart stream_part(int n_tiles, int KB, int slices, int skew, int cta, int ncta) {
  StreamPart q;
  const int base = n_tiles / ncta, rem = n_tiles - base * ncta;
  int i = cta - skew;                    // whole left-over tiles go to the CTAs skew .. skew + rem
  if (i < 0) i += ncta;
  const int extra = slices > 1 ? 0 : rem;
  q.first = i * base + (i < extra ? i : extra);
  q.count = base + (i < extra ? 1 : 0);
  q.per = stream_per(KB);
  q.pair = -1;
  q.slice = q.kt0 = q.kt1 = 0;
  q.split_per = 1;
  q.slices = slices;
  if (slices > 1 && i < (rem + 1) / 2 * slices) {
    q.pair = i / slices;
    q.slice = i - q.pair * slices;
    q.kt0 = q.slice * KB / slices;
    q.kt1 = (q.slice + 1) * KB / slices;
    q.split_per = stream_per(q.kt1 - q.kt0);
  }
  return q;
}
struct StreamUnit { int tile, kt0, kt1, per; bool two, split; };
TI_HOST_DEVICE int stream_units(const StreamPart& q) { return (q.pair >= 0 ? 1 : 0) + (q.count + 1) / 2; }
TI_HOST_DEVICE StreamUnit stream_unit(const StreamPart& q, int n_tiles, int KB, int ncta, int u) {
  StreamUnit x;
  if (q.pair >= 0 && u == 0) {
    x.tile = n_tiles / ncta * ncta + 2 * q.pair;
    x.two = x.tile + 1 < n_tiles;
    x.kt0 = q.kt0;
    x.kt1 = q.kt1;
    x.per = q.split_per;
    x.split = true;
    return x;
  }
  if (q.pair >= 0) --u;
  x.tile = q.first + 2 * u;
  x.two = 2 * u + 1 < q.count;
  x.kt0 = 0;
  x.kt1 = KB;
  x.per = q.per;
  x.split = false;
  return x;
}
TI_HOST_DEVICE int stream_slot_bytes(int wt, int M) { return kWarps * 16 * M * (wt == 0 ? 8 : 4); }

TI_DEVICE void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory"); }
// Whether a poll may go on.  The clock, whose read takes longer than most waits here, is read at every 64th try.
struct PollLimit {
  unsigned long long t0 = 0;
  unsigned spins = 0;
  TI_DEVICE bool more(unsigned* status) {
    if ((++spins & 63u) != 0u) return true;
    if (t0 == 0) t0 = globaltimer_ns();
    if (globaltimer_ns() - t0 < kStreamWaitNs) return true;
    if (status != nullptr) atomicOr(status, kStatusPeerTimeout);
    return false;
  }
};
TI_DEVICE bool stream_wait(uint32_t bar, uint32_t parity, unsigned* status) {
  if (mbar_try_wait(bar, parity)) return true;
  PollLimit limit;
  while (!mbar_try_wait(bar, parity))
    if (!limit.more(status)) return false;
  return true;
}

// Sums of a weight row and an activation row: integers of both limbs, or a float
template <int WT> struct StreamSum;
template <> struct StreamSum<W_INT8> {
  typedef int2 T;
  int hi, lo;
  TI_DEVICE void clear() { hi = lo = 0; }
  TI_DEVICE void add(int2 a) { hi += a.x; lo += a.y; }
  TI_DEVICE void add_other_half() {
    hi += __shfl_xor_sync(0xffffffffu, hi, 16);
    lo += __shfl_xor_sync(0xffffffffu, lo, 16);
  }
  TI_DEVICE int2 bits() const { return make_int2(hi, lo); }
  TI_DEVICE void add_bits(int2 a) { add(a); }
  TI_DEVICE float value(float unit) const { return ((float)hi * 256.f + (float)lo) * unit; }
};
template <> struct StreamSum<W_BF16> {
  typedef float T;
  float v;
  TI_DEVICE void clear() { v = 0.f; }
  TI_DEVICE void add(float a) { v += a; }
  TI_DEVICE void add_other_half() { v += __shfl_xor_sync(0xffffffffu, v, 16); }
  TI_DEVICE int2 bits() const { return make_int2(__float_as_int(v), 0); }
  TI_DEVICE void add_bits(int2 a) { v += __int_as_float(a.x); }
  TI_DEVICE float value(float) const { return v; }
};

// How one row goes from a product to the next of the launch: as packets of 8 bytes, two bf16 values and the launch's tag, which the
// consumers poll.  A grid barrier in between took 2.3 to 2.8 us beside streaming weights (stores acknowledged, an atomic, a poll), the
// load of the row after it another round trip; a packet is one store and the poll that sees it.
struct StreamFlow {
  int8_t emit[kMaxChain];      // the product's results are written as packets too
  int8_t x[kMaxChain];         // the row comes as packets of the product before (otherwise from memory, behind a grid barrier)
  int8_t resid[kMaxChain];     // product whose packets hold the residual row, or -1 (memory)
};
constexpr size_t kStreamPackets = 512 * 1024, kStreamPacketBytes = 128 * 1024;       // in the workspace: start, bytes per product
TI_DEVICE uint2* stream_packets(const GemvParams& p, int op) {
  return reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(p.ws) + kStreamPackets + op * kStreamPacketBytes);
}
TI_DEVICE void packet_store(uint2* dst, uint32_t value, uint32_t tag) {
  asm volatile("st.volatile.global.v2.u32 [%0], {%1,%2};\n" ::"l"(dst), "r"(value), "r"(tag) : "memory");
}
TI_DEVICE uint2 packet_load(const uint2* src) {
  uint2 v;
  asm volatile("ld.volatile.global.v2.u32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "l"(src) : "memory");
  return v;
}
TI_DEVICE uint4 packet_load2(const uint2* src) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(src) : "memory");
  return v;
}
// The launch's tag: odd, so never that of a workspace that has not been written
TI_DEVICE uint32_t stream_tag(const GemvParams& p) { return 2u * (uint32_t)__ldcg(p.sched + 3) + 1u; }

// One activation row of up to 40 * kThreads elements: read once, held in registers.  The norm weights were requested before the
// row is waited for; chunks beyond the row cost nothing (K = 5120 has 1.25 per thread of the 5).
struct RowChunks {
  uint4 nw[5];
  TI_DEVICE void load_norm(const GemvParams& p) {
    if (p.xmode != XNORM) return;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const int c = threadIdx.x + j * kThreads;
      if (c < (p.K >> 3)) nw[j] = ldg_cached16(p.norm_w + (size_t)c * 8);
    }
  }
};
TI_DEVICE float4 lds_f4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// `packets`: where the row comes from, or null (p.x).
template <int WT> TI_DEVICE void stage_row(const GemvParams& p, const RowChunks& r, const uint2* packets, uint32_t tag, uint8_t* dst, int lstride, float* scratch) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, chunks = p.K >> 3;
  const bool norm = p.xmode == XNORM;
  uint4 x[5];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const int c = tid + j * kThreads;
    x[j] = make_uint4(0, 0, 0, 0);
    if (packets == nullptr && c < chunks) x[j] = ld_x16(p.x + (size_t)c * 8);
  }
  if (packets != nullptr) {
    jitter();
    PollLimit limit;
    bool missing = true;
    while (missing) {
      missing = false;
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const int c = tid + j * kThreads;
        if (c >= chunks || !TI_CHECK(c * 4 + 3, kStreamPacketBytes / 8, p.status)) continue;
        const uint4 a = packet_load2(packets + (size_t)c * 4), b = packet_load2(packets + (size_t)c * 4 + 2);
        missing = missing || a.y != tag || a.w != tag || b.y != tag || b.w != tag;
        x[j] = make_uint4(a.x, a.z, b.x, b.z);
      }
      if (missing && !limit.more(p.status)) break;
    }
  }
  if (norm) {
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      if (warp * 32 + j * kThreads >= chunks) continue;
      const uint32_t w4[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) ss += bf16lo(w4[i]) * bf16lo(w4[i]) + bf16hi(w4[i]) * bf16hi(w4[i]);
    }
    ss = warp_sum(ss);
    if (lane == 0) scratch[warp] = ss;
    Consumers::sync();
    float tot = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; w += 4) {
      const float4 f = lds_f4(scratch + w);
      tot = (((tot + f.x) + f.y) + f.z) + f.w;
    }
    const float rr = rsqrtf(tot / (float)p.K + p.eps);
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      if (warp * 32 + j * kThreads >= chunks) continue;
      uint32_t w4[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
      const uint32_t n4[4] = {r.nw[j].x, r.nw[j].y, r.nw[j].z, r.nw[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) w4[i] = pack_bf16(bf16lo(w4[i]) * rr * (1.f + bf16lo(n4[i])), bf16hi(w4[i]) * rr * (1.f + bf16hi(n4[i])));
      x[j] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
    }
  }
  if (WT == W_BF16) {
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const int c = tid + j * kThreads;
      if (c < chunks) *reinterpret_cast<uint4*>(dst + (size_t)c * 16) = x[j];
    }
    Consumers::sync();
    return;
  }
  __nv_bfloat162 m2 = __floats2bfloat162_rn(0.f, 0.f);       // (a maximum with NaN is the other value)
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    if (tid + j * kThreads >= chunks) continue;
    const uint32_t w4[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w4[i])));
  }
  float mx = fmaxf(__low2float(m2), __high2float(m2));
  mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));       // not negative, not NaN: ordered as integers are
  if (lane == 0) scratch[32 + warp] = mx;
  Consumers::sync();
  float a = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; w += 4) {
    const float4 f = lds_f4(scratch + 32 + w);
    a = fmaxf(fmaxf(fmaxf(a, f.x), fmaxf(f.y, f.z)), f.w);
  }
  int e = (int)((__float_as_uint(a) >> 23) & 0xffu) - 127;
  e = max(e, -100);
  if (!(a < 3.0e38f)) e = 127;
  const float qs = exp2f((float)(14 - e));
  if (tid == 0) scratch[288] = exp2f((float)(e - 14));
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const int c = tid + j * kThreads;
    if (c >= chunks) continue;
    const uint32_t w4[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
    uint32_t hw[2] = {0, 0}, lw[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int q = max(-32768, min(32767, __float2int_rn((i & 1 ? bf16hi(w4[i >> 1]) : bf16lo(w4[i >> 1])) * qs)));
      hw[i >> 2] |= (uint32_t)((q >> 8) & 0xff) << (8 * (i & 3));
      lw[i >> 2] |= (uint32_t)(q & 0xff) << (8 * (i & 3));
    }
    *reinterpret_cast<uint2*>(dst + (size_t)c * 8) = make_uint2(hw[0], hw[1]);
    *reinterpret_cast<uint2*>(dst + lstride + (size_t)c * 8) = make_uint2(lw[0] ^ 0x80808080u, lw[1] ^ 0x80808080u);       // lo - 128
  }
  Consumers::sync();
}

// ROWS: 1 (rows of up to 40 * kThreads elements), or up to 8
template <int WT, int ROWS>
__global__ void __launch_bounds__(kStreamThreads, 1) gemv_stream_kernel(const __grid_constant__ ChainParams c, const __grid_constant__ StreamFlow flow, int stages, int slots, int slot_bytes) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ StreamPart part[kMaxChain];
  __shared__ __align__(8) unsigned long long bars[2 * kStreamMaxStages + 2 * kStreamMaxSlots];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x, ncta = gridDim.x;
  const GemvParams& p0 = c.op[0];
  unsigned long long* dbg = p0.dbg == nullptr ? nullptr : p0.dbg + cta * 32;
  if (dbg != nullptr && tid == 0) dbg[0] = globaltimer_ns();
  // [staged x, its statistics | sums of units | ring]
  uint8_t* ex = smem + c.x_bytes;
  uint8_t* ring = ex + slots * slot_bytes;
  const uint32_t ring0 = smem_u32(ring), full0 = smem_u32(bars), empty0 = full0 + 8 * kStreamMaxStages;
  const uint32_t sum_full0 = empty0 + 8 * kStreamMaxStages, sum_free0 = sum_full0 + 8 * kStreamMaxSlots;
  float* scratch = reinterpret_cast<float*>(smem + c.x_bytes - 2048);
  if (tid < c.n_ops) {
    int skew = 0, slices = 1;
    for (int j = 0; j <= tid; ++j) {
      const GemvParams& p = c.op[j];
      slices = p.ws != nullptr && p.counters != nullptr ? stream_slices(p.n_tiles, p.KB, ncta) : 1;
      if (j < tid && slices == 1) skew += p.n_tiles % ncta;
    }
    part[tid] = stream_part(c.op[tid].n_tiles, c.op[tid].KB, slices, skew % ncta, cta, ncta);
  }
  if (tid == kThreads) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full0 + 8 * s, 2);
      mbar_init(empty0 + 8 * s, kWarps);
    }
    for (int s = 0; s < slots; ++s) {
      mbar_init(sum_full0 + 8 * s, kWarps);
      mbar_init(sum_free0 + 8 * s, 1);
    }
    fence_mbar_init();
  }
  __syncthreads();
  pdl_trigger();

  if (warp == kWarps || warp == kStreamCopyB) {
    // ------------------------------------------------------------ copies: weights only, which no kernel of the step writes
    if (lane == 0) {
      const int which = warp == kWarps ? 0 : 1;              // row tile of the unit
      const int flight = min(kStreamFlight, stages);
      bool ok = true;
      int s = 0, f = 0, issued = 0;                          // next stage; oldest of those under way
      uint32_t ph = 1, fph = 0;                              // a stage's first use waits for nothing
      for (int op = 0; op < c.n_ops && ok; ++op) {
        const uint8_t* const w = c.op[op].w;
        const int n_tiles = c.op[op].n_tiles, KB = c.op[op].KB;
        const StreamPart q = part[op];
        const int units = stream_units(q);
        for (int u = 0; u < units && ok; ++u) {
          const StreamUnit x = stream_unit(q, n_tiles, KB, ncta, u);
          const bool copy = which == 0 || x.two;
          const uint8_t* src = w + ((size_t)(x.tile + which) * KB + x.kt0) * 512;
          const uint32_t step = (uint32_t)x.per * 512u;
          for (uint32_t left = (uint32_t)(x.kt1 - x.kt0) * 512u; left > 0;) {
            const uint32_t bytes = min(step, left), bar = full0 + 8 * s;
            // The ring is full once.  From here on the copies wait for the consumers, who start when the kernel before has ended: its
            // time is none of this launch's, whose limit is 2 s (between ranks it may itself wait that long for a peer).
            if (issued == stages) pdl_wait();
            ok = stream_wait(empty0 + 8 * s, ph, p0.status);
            if (ok && issued >= flight) {
              ok = stream_wait(full0 + 8 * f, fph, p0.status);
              if (++f == stages) {
                f = 0;
                fph ^= 1u;
              }
            }
            if (!ok) break;
            if (copy) {
              mbar_expect_tx(bar, bytes);
              bulk_g2s(ring0 + s * kStreamStage + which * (kStreamStage / 2), src, bytes, bar);
            } else {
              mbar_arrive(bar);
            }
            src += bytes;
            left -= bytes;
            ++issued;
            if (++s == stages) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
        if (dbg != nullptr && op == 0 && which == 0) dbg[1] = globaltimer_ns();
      }
      // every copy has landed before the CTA leaves, also after a wait that ran out
      for (int i = max(0, issued - stages); i < issued; ++i) mbar_wait(full0 + 8 * (i % stages), (uint32_t)((i / stages) & 1), ok ? kStreamWaitNs : kStreamDrainNs, p0.status);
    }
    __syncwarp();
  } else if (warp < kWarps) {
    // ------------------------------------------------------------ consumers
    const int g = lane >> 2, t = lane & 3;
    int8_t* xh = reinterpret_cast<int8_t*>(smem);
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(smem);
    bool alive = true;
    int s = 0, slot = 0;
    uint32_t ph = 0, sph = 1, tag = 0;
    for (int op = 0; op < c.n_ops; ++op) {
      const GemvParams& p = c.op[op];
      const StreamPart q = part[op];
      if (dbg != nullptr && tid == 0) dbg[8 + 4 * op] = globaltimer_ns();
      RowChunks row;
      if (ROWS == 1) row.load_norm(p);
      if (op == 0) pdl_wait();
      else if (ROWS == 1 && flow.x[op]) Consumers::sync();   // all warps are done with the row before
      else sync_with_epilogue();                             // the epilogue warp has passed the grid barrier
      if (ROWS == 1 && op == 0) {
        jitter();
        tag = stream_tag(p0);
      }
      if (dbg != nullptr && tid == 0) dbg[9 + 4 * op] = globaltimer_ns();
      const int lstride = limb_stride(p.K);
      if (ROWS == 1) stage_row<WT>(p, row, flow.x[op] ? stream_packets(p0, op - 1) : nullptr, tag, smem, lstride, scratch);
      else if (WT == W_INT8) stage_limbs<Consumers>(p, 0, p.K, xh, smem + (size_t)p.M * lstride, lstride, scratch);
      else stage_bf16<Consumers>(p, xs, p.K + 8, scratch);
      if (dbg != nullptr && tid == 0) dbg[10 + 4 * op] = globaltimer_ns();
      // MMA columns: activation rows, or, of one int8 row, its high limbs, its low ones less 128 (signed, so that one MMA takes both)
      // and ones, whose sum makes up for the 128; columns without a row are zero
      const bool mine = g < (WT == W_INT8 && ROWS == 1 ? 2 : p.M);
      const uint32_t xa = WT == W_INT8 ? smem_u32(smem) + (uint32_t)(g * lstride + t * 16) : smem_u32(xs) + (uint32_t)(g * (p.K + 8) + t * 8) * 2u;
      const uint32_t xb = xa + (uint32_t)(p.M * lstride);    // int8: the low limbs
      const int M = ROWS == 1 ? 1 : p.M, units = stream_units(q);
      for (int u = 0; u < units; ++u) {
        const StreamUnit x = stream_unit(q, p.n_tiles, p.KB, ncta, u);
        int ah[4] = {0, 0, 0, 0}, al[4] = {0, 0, 0, 0};
        float af[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        for (int kt = x.kt0 + warp, end = x.kt0; end < x.kt1; kt += x.per) {
          end = min(kt - warp + x.per, x.kt1);               // k tiles of this stage: kt - warp .. end
          if (alive) alive = stream_wait(full0 + 8 * s, ph, p0.status);
          if (kt < end) {
            const uint32_t w = ring0 + s * kStreamStage + warp * 512 + lane * 16;
            const uint4 w0 = lds128(w), w1 = lds128(w + kStreamStage / 2);
            uint4 h = make_uint4(0, 0, 0, 0), l = h;
            if (WT == W_INT8 && ROWS == 1 && g == 2) h = make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
            if (mine) {
              h = lds128(xa + kt * 64);
              if (WT == W_INT8 && ROWS > 1) l = lds128(xb + kt * 64);
            }
            if (WT == W_INT8 && ROWS == 1) {
              imma_s8s8(ah, w0.x, w1.x, w0.y, w1.y, h.x, h.y);
              imma_s8s8(al, w0.z, w1.z, w0.w, w1.w, h.z, h.w);
            } else if (WT == W_INT8) {
              imma_s8s8(ah, w0.x, w1.x, w0.y, w1.y, h.x, h.y);
              imma_s8u8(al, w0.x, w1.x, w0.y, w1.y, l.x, l.y);
              imma_s8s8(ah, w0.z, w1.z, w0.w, w1.w, h.z, h.w);
              imma_s8u8(al, w0.z, w1.z, w0.w, w1.w, l.z, l.w);
            } else {
              mma_bf16_16816(af[0], w0.x, w1.x, w0.y, w1.y, h.x, h.y);
              mma_bf16_16816(af[1], w0.z, w1.z, w0.w, w1.w, h.z, h.w);
            }
          }
          __syncwarp();                                      // every lane has read the stage
          if (lane == 0) mbar_arrive(empty0 + 8 * s);
          if (++s == stages) {
            s = 0;
            ph ^= 1u;
          }
        }
        // ---- this warp's sums: [warp][activation row][16 weight rows]
        if (alive) alive = stream_wait(sum_free0 + 8 * slot, sph, p0.status);
        if (WT == W_INT8 && ROWS == 1) {
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            const int hi = ah[j] + al[j], lo = ah[j + 1] + al[j + 1], ones = __shfl_down_sync(0xffffffffu, hi, 1);      // column 2: lane t = 1
            ah[j] = hi;
            al[j] = lo + 128 * ones;
          }
        }
        uint8_t* e = ex + slot * slot_bytes + (size_t)warp * M * 16 * (WT == W_INT8 ? 8 : 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {                        // (row g + 8 (j >> 1), column 2 t + (j & 1))
          const int m = 2 * t + (j & 1), at = m * 16 + g + 8 * (j >> 1);
          if (m >= M) continue;
          if (WT == W_INT8) reinterpret_cast<int2*>(e)[at] = make_int2(ah[j], al[j]);
          else reinterpret_cast<float*>(e)[at] = af[0][j] + af[1][j];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(sum_full0 + 8 * slot);
        if (++slot == slots) {
          slot = 0;
          sph ^= 1u;
        }
      }
      if (dbg != nullptr && tid == 0) dbg[11 + 4 * op] = globaltimer_ns();
    }
    __syncwarp();
    tell_epilogue();                                         // nothing of the launch's state is read any more
  } else {
    // ------------------------------------------------------------ epilogue: lane -> weight row (lane & 15), half of the warps' sums
    typedef StreamSum<WT> Sum;
    const int row = lane & 15, half = lane >> 4;
    bool alive = true;
    int slot = 0, barriers = 0;
    uint32_t ph = 0;
    float am_v[ROWS];
    int am_i[ROWS];
#pragma unroll
    for (int m = 0; m < ROWS; ++m) {
      am_v[m] = -INFINITY;
      am_i[m] = 0x7fffffff;
    }
    pdl_wait();
    const uint32_t tag = ROWS == 1 ? stream_tag(p0) : 0;
    for (int op = 0; op < c.n_ops; ++op) {
      const GemvParams& p = c.op[op];
      const StreamPart q = part[op];
      const bool emit = ROWS == 1 && flow.emit[op];
      uint2* const packets = stream_packets(p0, op);
      const int M = ROWS == 1 ? 1 : p.M, units = stream_units(q);
      // a unit's row scale and residual values, requested a unit ahead: they come from HBM, and beside streaming weights a load
      // takes as long as a unit
      const uint2* const resid_from = ROWS == 1 && p.epi == EPI_ROWPAR && flow.resid[op] >= 0 ? stream_packets(p0, flow.resid[op]) : nullptr;
      struct Ahead {
        float scale;
        uint2 r[ROWS];             // residual: a bf16 value, or a packet
      };
      auto request = [&](int u) {
        Ahead h;
        h.scale = 1.f;
#pragma unroll
        for (int m = 0; m < ROWS; ++m) h.r[m] = make_uint2(0, 0);
        if (u >= units) return h;
        const StreamUnit x = stream_unit(q, p.n_tiles, p.KB, ncta, u);
        const int n = x.tile * 8 + row;
        if (n >= p.N || !(x.two || row < 8)) return h;
        if (WT == W_INT8) h.scale = bf16_to_f(p.scale[n]);
        if (resid_from != nullptr) {
          if (TI_CHECK(n >> 1, kStreamPacketBytes / 8, p0.status)) h.r[0] = packet_load(resid_from + (n >> 1));
        } else if (p.epi == EPI_ROWPAR) {
#pragma unroll
          for (int m = 0; m < ROWS; ++m)
            if (ROWS == 1 || m < M) h.r[m].x = (uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(p.resid) + (size_t)m * p.N + n) << 16;
        }
        return h;
      };
      Ahead next = request(0);
      for (int u = 0; u < units; ++u) {
        const StreamUnit x = stream_unit(q, p.n_tiles, p.KB, ncta, u);
        const int n = x.tile * 8 + row;
        const bool live = n < p.N && (x.two || row < 8);
        Ahead cur = next;
        next = request(u + 1);
        if (alive) alive = stream_wait(sum_full0 + 8 * slot, ph, p0.status);
        alive = __all_sync(0xffffffffu, alive);
        const uint8_t* e = ex + slot * slot_bytes;
        // a slice's sums: [pair][slice][activation row][16 weight rows], 8 bytes each
        int2* part_of = reinterpret_cast<int2*>(p.ws) + ((long long)q.pair * q.slices * M) * 16 + row;
        bool finish = true;
        Sum sum[ROWS];
#pragma unroll
        for (int m = 0; m < ROWS; ++m) {
          if (ROWS > 1 && m >= M) continue;
          sum[m].clear();
#pragma unroll
          for (int w = 0; w < kWarps / 2; ++w) sum[m].add(reinterpret_cast<const typename Sum::T*>(e)[((half * (kWarps / 2) + w) * M + m) * 16 + row]);
          sum[m].add_other_half();
          if (x.split && half == 0 && TI_CHECK((((long long)q.pair * q.slices + q.slice) * M + m) * 16 + row, kStreamPackets / 8, p0.status)) __stcg(part_of + ((size_t)q.slice * M + m) * 16, sum[m].bits());
        }
        __syncwarp();                                        // the slot has been read
        if (lane == 0) mbar_arrive(sum_free0 + 8 * slot);
        if (++slot == slots) {
          slot = 0;
          ph ^= 1u;
        }
        if (x.split) {
          jitter();
          __threadfence();
          __syncwarp();
          int last = 0;
          if (lane == 0) {
            last = atomicAdd(p.counters + q.pair, 1u) + 1 == (unsigned)q.slices;
            if (last) p.counters[q.pair] = 0;                // ready for the next product
            __threadfence();
          }
          finish = __shfl_sync(0xffffffffu, last, 0) != 0;
          __syncwarp();                                      // the other lanes read behind lane 0's fence (a shuffle orders no memory)
          if (finish)
#pragma unroll
            for (int m = 0; m < ROWS; ++m) {
              if (ROWS > 1 && m >= M) continue;
              sum[m].clear();
              for (int z = 0; z < q.slices; ++z) sum[m].add_bits(__ldcg(part_of + ((size_t)z * M + m) * 16));
            }
        }
        if (!finish) continue;
#pragma unroll
        for (int m = 0; m < ROWS; ++m) {
          if (ROWS > 1 && m >= M) continue;
          const float v = sum[m].value(WT == W_INT8 ? scratch[288 + m] : 1.f) * cur.scale;
          if (p.epi == EPI_F32) {
            if (live && half == 0) static_cast<float*>(p.out)[(size_t)m * p.ldo + n] = v;
          } else if (p.epi != EPI_ARGMAX) {
            float o = v;
            if (p.epi == EPI_SWIGLU) {                       // rows come interleaved (gate, up), each rounded to bf16 first
              const float a = round_bf16(v), b = __shfl_xor_sync(0xffffffffu, a, 1);
              o = silu_f(a) * b;
            } else if (p.epi == EPI_ROWPAR) {
              float r = __uint_as_float(cur.r[m].x);
              if (ROWS == 1 && resid_from != nullptr) {
                PollLimit limit;
                while (live && cur.r[0].y != tag && limit.more(p0.status)) cur.r[0] = packet_load(resid_from + (n >> 1));
                r = n & 1 ? bf16hi(cur.r[0].x) : bf16lo(cur.r[0].x);
                __syncwarp();
              }
              o = r + v;
            }
            const int sh = p.epi == EPI_SWIGLU ? 1 : 0;      // a result for each, or every other, weight row
            if (emit) {
              const float o2 = __shfl_xor_sync(0xffffffffu, o, 1 << sh);
              jitter();
              if (live && half == 0 && (row & ((2 << sh) - 1)) == 0 && TI_CHECK(n >> (sh + 1), kStreamPacketBytes / 8, p0.status)) packet_store(packets + (n >> (sh + 1)), pack_bf16(o, o2), tag);
            }
            if (live && half == 0 && (row & sh) == 0) static_cast<__nv_bfloat16*>(p.out)[(size_t)m * (p.epi == EPI_ROWPAR ? p.N : p.ldo) + (n >> sh)] = __float2bfloat16_rn(o);
          } else if (live && (v > am_v[m] || (v == am_v[m] && n < am_i[m]))) {
            am_v[m] = v;
            am_i[m] = n;
          }
        }
      }
      if (op + 1 < c.n_ops && !(ROWS == 1 && flow.x[op + 1])) {
        // ---- grid barrier: all results of this product are in L2
        if (dbg != nullptr && lane == 0) dbg[2 + op] = globaltimer_ns();
        jitter();
        __threadfence();
        __syncwarp();
        if (lane == 0) {
          atomicAdd(p0.sched + 2, 1);
          const int target = ++barriers * ncta;
          PollLimit limit;
          int v;
          do {
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p0.sched + 2) : "memory");
          } while (v < target && limit.more(p0.status));
          __threadfence();
        }
        __syncwarp();
        sync_with_epilogue();
      }
    }
    const GemvParams& pl = c.op[c.n_ops - 1];
    if (pl.epi == EPI_ARGMAX) {                              // one candidate per activation row of this CTA
#pragma unroll
      for (int m = 0; m < ROWS; ++m) {
        if (ROWS > 1 && m >= pl.M) continue;
#pragma unroll
        for (int o = 1; o <= 8; o <<= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, am_v[m], o);
          const int oi = __shfl_xor_sync(0xffffffffu, am_i[m], o);
          if (ov > am_v[m] || (ov == am_v[m] && oi < am_i[m])) {
            am_v[m] = ov;
            am_i[m] = oi;
          }
        }
        if (lane == 0) {
          static_cast<float*>(pl.out)[(size_t)m * pl.ldo + cta] = am_v[m];
          pl.out_idx[(size_t)m * pl.ldo + cta] = am_i[m] == 0x7fffffff ? -1 : am_i[m];
        }
      }
    }
    // The last CTA of the launch sets the counters back for the next one, and the tag on.  The consumers read the tag: a CTA without a
    // row tile in any product has nothing else in which its epilogue warp would wait for them.
    __syncwarp();
    sync_with_epilogue();
    if (lane == 0) {
      __threadfence();
      if (atomicAdd(p0.sched + 1, 1) + 1 == ncta) {
        p0.sched[1] = 0;
        p0.sched[2] = 0;
        p0.sched[3] += 1;                                    // the next launch's packets have another tag
        __threadfence();
      }
      if (dbg != nullptr) dbg[5] = globaltimer_ns();
    }
    __syncwarp();
  }
}

struct StreamPlan { int x_bytes, stages, slots, slot_bytes, rows; };
// Whether a product of several rows, or of one row longer than registers hold, takes this form: where gemv_body reads bf16 rows from
// global memory anew for every tile (us, gemv_body / here: 16480 x 5120 at 6 / 8 rows 94.7 / 40.1, 93.7 / 47.1, 5120 x 6144 at 4 / 8 32.0 / 19.6, 31.6 /
// 27.8, 8192 x 32768 at one 178 / 82), and for one row (8192 x 32768 int8 60.7 / 52.4, 3552 x 20544 22.8 / 22.2, a chain with K = 21504 107.8 / 99.5).
// Other products of several rows do not: a stage of weights costs more here with every row (int8 16480 x 5120 at 2 / 4 / 8 rows 23.0 / 27.9, 25.1 /
// 37.1, 31.1 / 56.7; bf16 32768 x 2048 at 4 / 8 29.5 / 31.3, 30.6 / 41.6).  Nor do those with few tiles per CTA, whose k the teams of gemv_body cut
// in 16 (one int8 row 256 x 32768 16.8 / 20.2, 2048 x 32768 22.9 / 25.1, 2368 x 32768 24.8 / 23.4; 256 x 8192 eight bf16 rows 10.3 / 12.7).  A decode step of several rows takes the tensor-core
// products.  Small products of several rows would gain (2048 x 2048 at 2 rows 10.1 / 7.9), but a chain would then not have the bits of its products
// launched one by one.
static bool stream_rows(const GemvParams& p, int wt, int ncta) {
  if (wt == W_BF16 && !rows_staged(p.xmode, p.M, p.K)) return p.n_tiles > ncta;
  return p.M == 1 && p.n_tiles >= 2 * ncta;
}
// Whether a launch takes this form: one GPU's products of up to 8 rows, whose staged rows leave room for 4 stages, if it is the faster one.
static bool stream_plan(const ChainParams& c, int wt, int ncta, StreamPlan& q) {
  q.x_bytes = q.slot_bytes = 0;
  int m = 0;
  for (int i = 0; i < c.n_ops; ++i) {
    const GemvParams& p = c.op[i];
    if (p.tp > 1 || p.xll || p.M > kStreamMaxRows || (wt == W_INT8 && p.K > kMaxIntK)) return false;
    const size_t x = wt == W_INT8 ? (size_t)2 * p.M * limb_stride(p.K) : (size_t)p.M * (p.K + 8) * 2;
    q.x_bytes = std::max(q.x_bytes, (int)((x + 2048 + 127) / 128 * 128));
    q.slot_bytes = std::max(q.slot_bytes, stream_slot_bytes(wt, p.M));
    m = std::max(m, p.K <= 40 * kThreads ? p.M : kStreamMaxRows);
  }
  q.rows = m;
  for (int i = 0; m > 1 && i < c.n_ops; ++i)
    if (!stream_rows(c.op[i], wt, ncta)) return false;
  q.slots = m <= 2 ? kStreamMaxSlots : 2;
  const int room = 227 * 1024 - 1024 - q.x_bytes - q.slots * q.slot_bytes;       // (1 KB static: barriers, parts)
  q.stages = std::min(kStreamMaxStages, room / kStreamStage);
  return q.stages >= kStreamMinStages;
}

// Which products of a launch hand their row on as packets.  Only where a row is exactly the results of the product before; and
// nowhere if a product reads or overwrites what an earlier one of the launch writes in any other way, which needs the barrier's order.
// What an earlier product READS from memory may be overwritten without a barrier (hidden rows go back and forth between two buffers: the
// third product of a layer's chain writes the first one's residual): no CTA has a result of product j before it holds the whole row of
// product j - 1, and so on back to i, and a result of product i is sent only after all that it is made of has been read; what a CTA
// without a part in product i reads later goes into no result.
static StreamFlow stream_flow(const ChainParams& c, int rows) {
  StreamFlow f = {};
  auto width = [&](int i) { return c.op[i].epi == EPI_SWIGLU ? c.op[i].N / 2 : c.op[i].N; };
  auto touches = [&](const void* a, size_t an, const void* b, size_t bn) { return a != nullptr && b != nullptr && (uintptr_t)a < (uintptr_t)b + bn && (uintptr_t)b < (uintptr_t)a + an; };
  auto bytes = [&](int i) { return (size_t)width(i) * (c.op[i].epi == EPI_F32 ? 4 : 2); };
  bool ok = rows == 1;
  for (int i = 0; i < c.n_ops; ++i) {
    const GemvParams& p = c.op[i];
    f.emit[i] = i + 1 < c.n_ops && p.ws != nullptr && (p.epi == EPI_STORE || p.epi == EPI_SWIGLU || p.epi == EPI_ROWPAR) && p.N % 4 == 0 && (size_t)width(i) * 4 <= kStreamPacketBytes;
    f.x[i] = i > 0 && f.emit[i - 1] && (const void*)p.x == c.op[i - 1].out && p.K == width(i - 1);
    f.resid[i] = -1;
    for (int j = 0; j < i; ++j) {
      const GemvParams& w = c.op[j];
      if (p.epi == EPI_ROWPAR && touches(p.resid, bytes(i), w.out, bytes(j))) {
        f.resid[i] = (int8_t)j;
        ok = ok && (const void*)p.resid == w.out && f.emit[j] && width(i) <= width(j);
      }
      ok = ok && !touches(p.out, bytes(i), w.out, bytes(j)) && p.ws == w.ws;
      if (!(f.x[i] && j == i - 1)) ok = ok && !touches(p.x, (size_t)p.K * 2, w.out, bytes(j));
    }
  }
  if (!ok)
    for (int i = 0; i < kMaxChain; ++i) {
      f.emit[i] = f.x[i] = 0;
      f.resid[i] = -1;
    }
  return f;
}

template <int WT, int ROWS> static int launch_stream(const ChainParams& c, const StreamPlan& q, int ncta, cudaStream_t st) {
  static bool configured = false;
  auto k = gemv_stream_kernel<WT, ROWS>;
  if (!configured) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024);
    configured = true;
  }
  const cudaError_t e = launch_kernel(k, dim3(ncta), dim3(kStreamThreads), (size_t)q.x_bytes + q.slots * q.slot_bytes + q.stages * kStreamStage, st, true, c, stream_flow(c, q.rows), q.stages, q.slots, q.slot_bytes);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace ti
