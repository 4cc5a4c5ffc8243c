// Persistent GEMM on SM pairs (tcgen05 cta_group::2):  out[token, feature] = X[token, :] . W[feature, :]
//
// Two CTAs of a cluster share one 256-token x bn-feature output tile.  Each SM keeps its own 128 token rows of A and HALF of the
// weight rows of B in shared memory and accumulates 128 x bn in its own TMEM; the even CTA's elected thread issues the MMAs for
// both.  What bounds the one-SM form of these products is operand traffic from L2, not the tensor pipe: a 128 x 256 tile reads 48 KB
// per 64-wide k-block and SM, the pair's halves read 32 KB for the same arithmetic, and the ring becomes seven stages deep.
//
// The issuing threads were the other half of it.  Behind lane == 0 an MMA took 90 cycles to issue, and a 64-bit division for the ring
// stage 400: 64-column tiles cost as much as 256-column ones.  With elect.sync and a carried stage a k-block is bound by its 512
// tensor cycles (256 columns).  Measured, single-SM kernels that issue behind lane == 0 -> this kernel (graph replays, weights from
// memory): 2048 x 4096 -> 2 x 12288 gated 348 -> 270 us (1528 TFLOP/s, the power limit's rate), 7500 tokens 1263 -> 987; 1616 x 12288 ->
// 4096 174 -> 126; 230 x 4096 -> 6144 33 -> 19.
//
// Tokens lie on the TMEM lanes, so a thread of the epilogue gets 16 features of one token row at a time.  Eight epilogue warps (two
// per lane quarter) drain one accumulator while the next tile fills the other.  bf16 results turn in shared memory (32 rows x 64
// features a warp, columns XORed with the row against bank conflicts) and leave, with the residual, as whole 128-byte lines: lanes
// that store 16 bytes each into 32 rows cost 32 requests to L2 per instruction, and short products were bound by them (6272 x 1152 -> 3456
// with bias: 61 us by lane, 51 turned, in one run; in the run of the figures above 66 on single SMs and 44 here, 1152 -> 1152 with
// residual 42 and 29).
//
// The TMA loads carry cta_group::2 only so that both CTAs' copies may report to the even CTA's barrier; every copy goes to its own CTA.
// MMA completion is reported to the even CTA, whose producer and epilogue pass it on to the odd one.
#pragma once

#include "common.cuh"

constexpr int PAIR_THREADS = 320;           // producer warp, MMA warp, eight epilogue warps
constexpr int PAIR_EPI_WARPS = 8;
constexpr int PAIR_TURN_BYTES = PAIR_EPI_WARPS * 4096;
constexpr int PAIR_GROUP = 8;               // token tiles (of 256) walked before the next feature tile

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// The same without ordering this thread's own accesses (a release at cluster scope took 1300 cycles behind TMA copies under way): for
// passing on that a stage has been read.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void pair_tmem_alloc(uint32_t* smem_slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(cols) : "memory");
}
__device__ __forceinline__ void pair_tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// Arrives on this CTA's barrier once every MMA of the pair issued so far is done.
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// mbar_wait for a barrier on which the other CTA arrives.
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity, int tag) {
  auto done = [&] {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
  };
  if (done()) return true;
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 128; ++i)
      if (done()) return true;
    if (clock64() - t0 > PRISM_WAIT_CYCLES) break;
  }
  prism_report(PRISM_ERR_MBAR_TIMEOUT, tag);
  return false;
}
__device__ __forceinline__ void pair_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// A copy into this CTA's shared memory that reports its bytes to a barrier of either CTA of the pair.
__device__ __forceinline__ void pair_tma_load_2d(void* smem_dst, const CUtensorMap* m, uint32_t cluster_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(cluster_bar), "r"(x), "r"(y)
      : "memory");
}

struct PairArgs {
  int T;         // tokens
  int N;         // columns of a full sweep: features, or gate + up rows of a gated unit (2 x outputs)
  int kb_total;  // ceil(K / 64)
  int splits, kb_per_split;  // split s multiplies k-blocks [s, s + 1) * kb_per_split into slab s of a 32-bit output
  long long split_stride;
  int bn;        // columns of a tile: a multiple of 32 (64 for a gated unit), at most 256
  int stages;
  int m_tiles, n_tiles;
  int dual;      // gated unit: the even CTA's B half holds gate rows, the odd CTA's the matching up rows
  int up_row;    // first up row of the weight matrix
  int act;
  float glu_limit;
  int out_f32;
  long long ldo, ldr;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  void* out;
  PrismSections sec;
};

__device__ __forceinline__ void add_bf16x8(float* v, const uint4& x) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __bfloat1622float2(p[e]);
    v[2 * e] += f.x;
    v[2 * e + 1] += f.y;
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const PairArgs a) {
  constexpr int A_BYTES = 128 * 64 * 2;
  constexpr int BUF_COLS = 256, TMEM_COLS = 512;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stages = a.stages;
  const int b_bytes = a.bn * 64;                       // bn / 2 rows of 128 bytes
  const int stage_bytes = A_BYTES + b_bytes;           // a multiple of 2 KB
  uint8_t* const turns = smem + (size_t)stages * stage_bytes;                          // [8] 32 rows of 128 bytes
  uint64_t* full = reinterpret_cast<uint64_t*>(turns + PAIR_TURN_BYTES);               // the even CTA's are the ones in use
  uint64_t* empty = full + stages;
  uint64_t* acc_full = empty + stages;                 // [2] MMA -> epilogue
  uint64_t* acc_empty = acc_full + 2;                  // [2] both epilogues -> MMA; the even CTA's are the ones in use
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int num_tiles = a.m_tiles * a.n_tiles * a.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * PAIR_EPI_WARPS);
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    pair_tmem_alloc(tmem_slot, TMEM_COLS);
    pair_tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  // Within a group of token tiles the token tile varies fastest: the pairs at work share a few weight tiles and the group's
  // activations, and a weight tile leaves DRAM once per group.
  auto tile_at = [&](int tile, int& m0, int& n0, int& kb0, int& kb1) {
    const int split = a.splits == 1 ? 0 : tile / (a.m_tiles * a.n_tiles);
    tile -= split * a.m_tiles * a.n_tiles;
    kb0 = split * a.kb_per_split;
    kb1 = min(a.kb_total, kb0 + a.kb_per_split);
    const int per_group = PAIR_GROUP * a.n_tiles, g = tile / per_group, first = g * PAIR_GROUP;
    const int rows = min(PAIR_GROUP, a.m_tiles - first), r = tile - g * per_group;
    m0 = (first + r % rows) * 256;
    n0 = (r / rows) * a.bn;
  };

  if (warp == 0) {
    if (elect_one()) {
      int s = 0, early = 0;        // ring stage; k-blocks whose weight tile is already under way
      uint32_t parity = 1;         // of the empty barrier: a fresh one counts as free
      bool ok = true, reused = false;  // reused: the ring has gone round, its stages are free when the MMAs say so
      int m0, n0, kb0, kb1;
      tile_at(pair, m0, n0, kb0, kb1);
      // the first ring of weight tiles depends on no earlier kernel
      const int pre = min(stages, kb1 - kb0);
      auto load_w = [&](int s, int kb, int n0) {
        if (rank == 0) mbar_expect_tx(&full[s], 2 * stage_bytes);
        const int row = a.dual ? n0 / 2 + (rank ? a.up_row : 0) : n0 + (int)rank * (a.bn / 2);
        pair_tma_load_2d(smem + (size_t)s * stage_bytes + A_BYTES, &tmW, cluster_addr(&full[s], 0), kb * 64, row);
      };
      for (int i = 0; i < pre; ++i) load_w(i, kb0 + i, n0);
      pdl_wait();  // activations come from the previous kernel
      for (int tile = pair; tile < num_tiles && ok; tile += pairs) {
        tile_at(tile, m0, n0, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = pair_wait(&empty[s], parity, 1);
          if (!ok) break;
          if (rank == 0 && reused) mbar_arrive_cluster_relaxed(cluster_addr(&empty[s], 1));
          if (early < pre) ++early;
          else load_w(s, kb, n0);
          pair_tma_load_2d(smem + (size_t)s * stage_bytes, &tmX, cluster_addr(&full[s], 0), kb * 64, m0 + (int)rank * 128);
          if (++s == stages) s = 0, parity ^= 1, reused = true;
        }
      }
      if (!ok && rank == 0) {
        // unwinding after a timed-out wait: let copies already in flight land before shared memory is released
        for (int j = 0; j < stages; ++j) {
          if (--s < 0) s = stages - 1, parity ^= 1;
          (void)mbar_wait(&full[s], parity ^ 1, 4);
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(256, a.bn);
      int s = 0, local = 0;
      uint32_t parity = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += pairs, ++local) {
        const int buf = local & 1;
        if (local >= 2) {
          ok = pair_wait(&acc_empty[buf], ((uint32_t)(local >> 1) - 1) & 1, 5);
          if (!ok) break;
          tc_fence_after();
        }
        const uint32_t acc = tmem_base + buf * BUF_COLS;
        int m0, n0, kb0, kb1;
        tile_at(tile, m0, n0, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = mbar_wait(&full[s], parity, 2);
          if (!ok) break;
          tc_fence_after();
          const uint32_t st = smem_u32(smem + (size_t)s * stage_bytes);
          const uint64_t da = umma_desc_sw128(st), db = umma_desc_sw128(st + A_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k) pair_mma(acc, da + 2 * k, db + 2 * k, idesc, kb != kb0 || k != 0);
          pair_commit(&empty[s]);
          if (++s == stages) s = 0, parity ^= 1;
        }
        if (ok) pair_commit(&acc_full[buf]);
      }
    }
  } else {
    // ------------------------------ epilogue warps 2..9 ------------------------------
    const int q = warp & 3, half = (warp - 2) >> 2;  // TMEM lane quarter this warp may read; which half of the columns
    uint4* const turn = reinterpret_cast<uint4*>(turns + (warp - 2) * 4096);
    pdl_wait();
    int local = 0;
    for (int tile = pair; tile < num_tiles; tile += pairs, ++local) {
      const int buf = local & 1;
      int m0, n0, kb0, kb1;
      tile_at(tile, m0, n0, kb0, kb1);
      // outputs of this tile: f0 + [0, width); the two warps of a lane quarter take half of the columns each, up to 64 at a time
      const int f0 = a.dual ? n0 / 2 : n0, full_width = a.dual ? a.bn / 2 : a.bn, width = min(full_width, (a.dual ? a.N / 2 : a.N) - f0);
      const int u_end = min(width, (half + 1) * (full_width / 2));
      const int row0 = m0 + (int)rank * 128 + q * 32;  // first token of this warp
      if (!pair_wait(&acc_full[buf], (uint32_t)(local >> 1) & 1, 3)) break;
      tc_fence_after();
      if (rank == 0 && warp == 2) {
        tc_fence_before();
        if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_full[buf], 1));
      }
      const uint32_t t_lane = tmem_base + buf * BUF_COLS + ((uint32_t)(q * 32) << 16);
      for (int u0 = half * (full_width / 2); u0 < u_end; u0 += 64) {
        // the unit's residual, in the order in which it will be stored
        uint4 res[8];
        const int u1 = min(u0 + 64, u_end), cu = u0 + (lane & 7) * 8;  // cu: first of the eight columns that this lane stores
        if (a.residual != nullptr) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int m = row0 + i * 4 + (lane >> 3);
            res[i] = m < a.T && cu < u1 ? *reinterpret_cast<const uint4*>(a.residual + (size_t)m * a.ldr + f0 + cu) : make_uint4(0, 0, 0, 0);
          }
        }
        for (int c0 = u0; c0 < u1; c0 += 16) {
          uint32_t r[16];
          float v[16];
          tmem_ld16(t_lane + c0, r);
          if (a.dual) {
            uint32_t ru[16];
            tmem_ld16(t_lane + a.bn / 2 + c0, ru);
            tmem_ld_wait();
            // Rows past the last token are zeros, for which the unit's division takes its slow path (257 tokens, 1024 -> 2 x 6144: 33 us,
            // 512 tokens 22): they get another gate.  A branch around the row made the plain products' epilogue slower (6272 x 1152 -> 4304
            // with GELU 57.1 -> 58.1), one around each element full gated tiles (3 to 10 %).
            const bool live = row0 + lane < a.T;
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = glu(live ? __uint_as_float(r[j]) : 1.0f, __uint_as_float(ru[j]), a.act, a.glu_limit);
          } else {
            const int f = f0 + c0;
            int act = a.act;
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
            if (a.sec.n > 0) {
              float alpha;
              prism_section_of(a.sec, f, alpha, act);
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] *= alpha;
            }
            if (a.bias != nullptr) {
              const uint4* b = reinterpret_cast<const uint4*>(a.bias + f);
              add_bf16x8(&v[0], b[0]);
              add_bf16x8(&v[8], b[1]);
            }
            if (act == PRISM_ACT_GELU_TANH) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = gelu_tanh(v[j]);
            } else if (act == PRISM_ACT_GELU_ERF) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = gelu_erf(v[j]);
            } else if (act == PRISM_ACT_SIGMOID) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = sigmoid_fast(v[j]);
            } else if (act == PRISM_ACT_DECAY) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = decay_of(v[j]);
            }
          }
          if (a.out_f32) {
            if (row0 + lane < a.T) {
              float* slab = reinterpret_cast<float*>(a.out) + (a.splits == 1 ? 0 : (kb0 / a.kb_per_split) * a.split_stride);
              float4* dst = reinterpret_cast<float4*>(slab + (size_t)(row0 + lane) * a.ldo + f0 + c0);
#pragma unroll
              for (int e = 0; e < 4; ++e) dst[e] = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
            }
            continue;
          }
          uint4 o[2];
          __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
          for (int e = 0; e < 8; ++e) op[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
          const int c = (c0 - u0) / 8;
          turn[lane * 8 + (c ^ (lane & 7))] = o[0];
          turn[lane * 8 + ((c + 1) ^ (lane & 7))] = o[1];
        }
        if (a.out_f32) continue;
        __syncwarp();
        if (cu < u1) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = i * 4 + (lane >> 3), m = row0 + r;
            uint4 o = turn[r * 8 + ((lane ^ r) & 7)];
            if (a.residual != nullptr) {
              float v[8];
              const __nv_bfloat162* op = reinterpret_cast<const __nv_bfloat162*>(&o);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 x = __bfloat1622float2(op[e]);
                v[2 * e] = x.x;
                v[2 * e + 1] = x.y;
              }
              add_bf16x8(v, res[i]);
              __nv_bfloat162* wp = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
              for (int e = 0; e < 4; ++e) wp[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
            }
            if (m < a.T) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)m * a.ldo + f0 + cu) = o;
          }
        }
        __syncwarp();
      }
      // this warp's reads of the accumulator are complete: hand the buffer back
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[buf], 0));
    }
  }
  // Neither CTA leaves while the other may still read its operands or report to its barriers.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem_base, TMEM_COLS);
  }
}
