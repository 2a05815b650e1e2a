// Table GEMM on the tensor cores: the abstract product of amsim_kernels.cuh,
//     Out[p, q] = sum_k AM(V[p, k], U[k, q]),
// for tables that factor exactly over 4-bit floats.
//
// A product is  +-2^(ev + eu - 254) * T[iv][iu]  with T the table (values 1..4 in steps of
// 2^-m).  When the table is opened the library looks for a factorisation
//     T[i][j] = unit * sum_s F[i][s] * G[j][s],   s < S slots, all F and G in {0, .5, 1, 1.5, 2, 3, 4, 6, -...}
// (factor_table in amsim.cu; every shipped table has one with S = its number of distinct rows:
// row s + 1 minus row s is a handful of small integers).  A reduction step of the GEMM is then S
// steps of a block-scaled 4-bit matrix product (tcgen05.mma kind::mxf4): an operand element
// contributes a row of S codes looked up by its mantissa index (signs by flipping the codes' sign
// bits), and its EXPONENT FIELD is the block's E8M0 scale byte as it stands.  The tensor core
// forms sum_s F * G exactly (small integers times one power of two), so the product of every
// element pair is the table's, and adds it to an FP32 accumulator in tensor memory.
//
// The accumulator add truncates (measured: one round toward zero per instruction, with at least 34 fraction bits kept
// before it), where an FP32 add rounds to nearest; a 128-slot product is two instructions.  So after a chunk of the
// reduction the tile is added (round to nearest) to an FP32 partial tile in scratch and tensor memory starts from zero;
// tiles of 128 and 64 columns spread a chunk over two and three accumulators.  A chunk is as long as leaves the error
// against 64 bits no larger than the table kernels' (code_steps in amsim.cu): with ordinary activations, weights and
// gradients 3e-9 (64 steps) to 1e-7 (10^5 steps) on either path.  Operands whose exponents spread widely lose more here:
// normal variates times 2^-10 .. 2^10 give 2e-6 (128 slots: 3.4e-6) where the table kernels give 1e-7 to 5e-7.
//
// Two CTAs (one pair of multiprocessors) share a tile of 256 rows and up to 256 columns (tcgen05 cta_group::2): each
// encodes 128 rows of V and half the columns of U, the tensor cores read both halves, and the CTA of rank 0 issues.
// Every CTA needs the scale bytes of all columns; the other half's arrive by st.async on its own barrier.
//
// Rates: 64 code steps of a 256 x 256 tile take a pair 128 clocks, so 64-slot tables run at most 256 products per clock
// and multiprocessor, 8 times the 32 table lookups per clock that bound the shared-memory kernels.  What bounds this
// kernel is making the operands: per reduction step and operand row S / 2 bytes of codes are looked up in a table,
// sign-flipped and stored.  The codes of V go to tensor memory (the product takes its first operand from there), the
// codes of U to shared memory.  With one CTA per tile of 128 x 256 every multiprocessor encoded 384 rows a step, with
// pairs 256.  The tensor pipe is active 40 % of the time with 256 columns and 15 % with 64;
// the operand warps' chains of lookups, stores and barrier operations are the rest.
//
// 32 rows or columns belong to two warps, which make the stages of a 16-step block's halves: a warp fetches the raw FP32
// elements of its rows with its own cp.async double buffer, encodes them, and signals the stage; one more warp issues
// the matrix products (rank 0) or forwards the signals (rank 1).  No barrier spans the CTA inside the loop.  Work is
// dealt out in equal runs of (tile, 16-step block) pairs as in gather_gemm's balanced mode.
//
// Measured (B200, table kernels / one CTA per tile / pairs): 3x3 256 -> 256 on 64 x 14 x 14 with MBM_7, forward
// 1255 / 318 / 272 us, filter gradient 1250 / 349 / 283 us; 8192 x 512 x 2048 with MIT_7 929 / - / 581 us.  (With 128-step
// chunks throughout and signals of the scope of a CTA; forward, both gradients and bias together 883 us then, about 915 now.)
#pragma once
#include "amsim_kernels.cuh"
#include "amsim_wide.cuh"

namespace amsim {

constexpr int CT_KB = 16;        // reduction steps per block; a warp fetches and encodes one half of each
constexpr int CT_HALF = CT_KB / 2;
constexpr int CT_RAW = 32 * CT_HALF * 4;  // one cp.async buffer of a warp
constexpr int CT_ROWS = 256;     // rows of a CTA pair's tile
constexpr int CT_MAXSPIN = 1 << 20;  // bound on every wait (see Waiter)

// How an operand's elements sit in memory.
constexpr int CT_KVEC = 0;   // 16-byte groups of four consecutive reduction steps of one row
constexpr int CT_RVEC = 1;   // 16-byte groups of four consecutive rows of one reduction step
constexpr int CT_KSCL = 2;   // element by element, lanes along the reduction
constexpr int CT_RSCL = 3;   // element by element, lanes along the rows

struct CodeParams {
  Params prm;
  const uint4* tab_v;        // code rows of the lane operand's table indices (last row: zeros)
  const uint4* tab_u;
  int rows_v, rows_u;        // indices per table (the zero row is number rows_*)
  int sh_v, sh_u;            // bits >> sh & (rows - 1) is the table index
  float unit;                // out = acc * unit (a power of two)
  int v_mode, u_mode;        // CT_* of the operands
  int step_v, step_u;        // blocks never straddle a tap and offsets fit 32 bits: step through them
  int fgrad;                 // V is gathered along p with the reduction over grid positions
  int chunk;                 // blocks summed in tensor memory before they go to the FP32 partial tile
  int no_tries;              // every wait gives up at once (for the test of the report)
  unsigned* stuck;           // (host memory) set when a bounded wait ran out
};

template <int S>
struct CodeCfg {
  static constexpr int KS = 256 / S;              // reduction steps per stage (a row of a stage is 128 bytes of codes)
  static constexpr int CH = S / 32;               // 16-byte chunks per code row
  static constexpr int W = S == 128 ? 1 : 2;      // scale words per row and stage
  static constexpr int REP = S == 128 ? 4 : 8;    // copies of a code table: lanes of a quarter warp read different banks
  static constexpr int STAGES_PER_KB = CT_KB / KS;
};

template <int S, int BN>
struct CodeSmem {
  using C = CodeCfg<S>;
  static constexpr int GU = BN / 64;              // 32-column groups of U per CTA (half of the pair's columns)
  static constexpr int NW = 2 * (4 + GU);         // two warps per group of 32 rows or columns
  static constexpr int NT = 32 * (NW + 1);
  static constexpr int NBH = (BN + 127) / 128;    // 512-byte scale chunks of U per word (both halves: every CTA needs all)
  static constexpr int NST = BN == 64 ? 8 : 6;    // stages in flight: tensor memory and shared memory hold no more
  // accumulators that a chunk's stages take in turn, added when the chunk is taken out: each has a NACC-th of the steps
  static constexpr int NACC = BN == 64 ? 3 : BN == 128 ? 2 : 1;
  static constexpr int CODE_BYTES = BN / 2 * 128; // the codes of V go to tensor memory
  static constexpr int SF_BYTES = (1 + NBH) * C::W * 512;
  static constexpr int OFF_SF = NST * CODE_BYTES;
  static constexpr int OFF_RAW = OFF_SF + NST * SF_BYTES;
  // tensor memory columns: accumulators, NST stages of V codes, two sets of scales
  static constexpr int T_CODES = NACC * BN;
  static constexpr int T_SF = T_CODES + NST * 32;
  static constexpr int SF_COLS = (1 + NBH) * C::W * 4;
  static_assert(T_SF + 2 * SF_COLS <= 512, "tensor memory");
  static constexpr int OFF_ROW = OFF_RAW + NW * 2 * CT_RAW;
  static constexpr int OFF_TAB = OFF_ROW + 8 * 512;
  static size_t bytes(int rows_v, int rows_u) {
    return 1024 + OFF_TAB + (size_t)(rows_v + 1 + rows_u + 1) * C::CH * C::REP * 16;
  }
};

// ---- tensor-core plumbing ---------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// Address in the cluster's shared memory of this CTA's `addr` in the CTA of that rank.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Stores a word in the other CTA's shared memory and counts its four bytes there (both addresses the cluster's).  The
// count is a release in the scope of the cluster.  It also serves as the signal to the other CTA, with a word nobody reads:
// an arrive that releases to the cluster waits for the thread's earlier accesses to reach it, and that made 3x3 64 -> 64 on
// 32 x 55 x 55 take 1501 us instead of 1055 (forward and backward); an arrive without a scope releases to its own CTA only.
__device__ __forceinline__ void st_async_remote(uint32_t addr, uint32_t v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// (every barrier here gets arrivals or counts from the other CTA too)
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{.reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {  // (does not wait)
  uint32_t ok;
  asm volatile("{.reg .pred p; mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Shared-memory matrix descriptor: layout 2 = rows of 128 bytes, 128-byte swizzle, 8-row groups 1024
// bytes apart; layout 0 = 8 x 16-byte core matrices, 128 bytes apart (scale chunks).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, int layout) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46) |
         ((uint64_t)layout << 61);
}
// kind::mxf4: E2M1 codes, E8M0 scales, FP32 accumulator; M = 256 over the two CTAs
__host__ __device__ constexpr uint32_t code_idesc(int n) {
  return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (1u << 28);
}
__device__ __forceinline__ void mma_codes(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                          uint32_t accumulate) {
  asm volatile(
      "{.reg .pred p; setp.ne.b32 p, %6, 0;\n"
      "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], [%5], p;}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void scales_to_tmem(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
// Arrives at this barrier of both CTAs when the products issued so far are done.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
        "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ bool elect_lane() {
  uint32_t e;
  asm volatile("{.reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p;}" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// (the clobbers keep reads of what other lanes have copied in behind the wait and the warp barrier)
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void tmem_store32(uint32_t taddr, const uint4 (&q)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
      "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(q[0].x), "r"(q[0].y), "r"(q[0].z), "r"(q[0].w), "r"(q[1].x), "r"(q[1].y), "r"(q[1].z), "r"(q[1].w), "r"(q[2].x),
      "r"(q[2].y), "r"(q[2].z), "r"(q[2].w), "r"(q[3].x), "r"(q[3].y), "r"(q[3].z), "r"(q[3].w), "r"(q[4].x), "r"(q[4].y),
      "r"(q[4].z), "r"(q[4].w), "r"(q[5].x), "r"(q[5].y), "r"(q[5].z), "r"(q[5].w), "r"(q[6].x), "r"(q[6].y), "r"(q[6].z),
      "r"(q[6].w), "r"(q[7].x), "r"(q[7].y), "r"(q[7].z), "r"(q[7].w)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void cp_async16n(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Waits for a phase of an mbarrier, at most CT_MAXSPIN tries.  A thread whose wait has run out is dead: it waits no more, signals
// nobody and issues nothing, so the warps that depend on it run out too, and only walks its work to the end (the tile
// counters stay in step, the results are wrong).  The host reads the mark at the next call.
struct Waiter {
  unsigned* stuck;
  bool dead;
  __device__ __forceinline__ void wait(uint32_t bar, uint32_t parity) {
    if (dead) return;
    for (int i = 0; i < CT_MAXSPIN; ++i)  // (a bound from the parameters: 3x3 64 -> 64 975 -> 1077 us)
      if (mbar_try(bar, parity)) return;
    dead = true;
    *(volatile unsigned*)stuck = 1u;
  }
  __device__ __forceinline__ void wait_warp(uint32_t bar, uint32_t parity) {
    wait(bar, parity);
    __syncwarp();
  }
};

// Copies a code table to shared memory as [chunk][index][copy].
template <int CH, int REP>
__device__ __forceinline__ void copy_code_table(uint4* dst, const uint4* __restrict__ src, int rows, int tid, int nthreads) {
  for (int i = tid; i < rows * CH * REP; i += nthreads) {
    const int rest = i / REP, c = rest / rows, row = rest - c * rows;
    dst[i] = __ldg(src + row * CH + c);
  }
}

// Fetches the 32 rows x 8 reduction steps (one half of a block) a warp encodes, raw FP32, into its 1 KB buffer:
// CT_K*: row r at 32 r, its two 16-byte groups at (group ^ (r >> 2 & 1)); CT_R*: step k at 128 k.
struct RowFetch {
  int k_at;              // first step of this warp's half within a block
  int e_kh, e_kw, e_ch;  // filter tap of this lane's row (group) of a filter gradient
  bool e_ok;
  // Stepping (cp.step): where a block of 16 steps never straddles a filter tap, the two 16-byte groups a
  // lane copies per block sit at offsets that advance by a constant until the tap ends.  (Decoding the tap and
  // the rows anew for every block took as many instructions as encoding a stage.)
  int off[2];            // element offsets of the next block's groups
  int left;              // blocks left in the tap
  uint32_t okm;          // bit i: group i exists

  // r: first row of the warp inside the tile; for a new tile at (p0, q0)
  __device__ __forceinline__ void new_tile(const CodeParams& cp, bool is_v, int first, int4* rowinfo, int lane) {
    left = 0;
    if (!is_v) return;
    const Params& prm = cp.prm;
    const Gather& g = prm.g;
    if (cp.fgrad) {
      const uint32_t pg = (uint32_t)(first + (cp.v_mode == CT_RVEC ? 4 * (lane & 7) : lane));
      const uint32_t tap = fdiv(pg, g.d_sc);
      e_ch = (int)(pg - tap * (uint32_t)g.SC);
      e_kh = (int)fdiv(tap, g.d_kw);
      e_kw = (int)tap - e_kh * g.KW;
      e_ok = pg < (uint32_t)prm.P;
      return;
    }
    const uint32_t pg = (uint32_t)(first + lane);
    const uint32_t n = fdiv(pg, g.d_img);
    const uint32_t rem = pg - n * (uint32_t)(g.PH * g.PW);
    const uint32_t a = fdiv(rem, g.d_pw);
    const uint32_t b = rem - a * (uint32_t)g.PW;
    const long long nb = (long long)n * ((long long)g.SH * g.SW * g.SC);
    int4 ri;
    ri.x = pg < (uint32_t)prm.P ? (int)a * g.ps_h - g.off_t : INT32_MIN / 2;  // a row past the end is never in range
    ri.y = (int)b * g.ps_w - g.off_l;
    ri.z = (int)(uint32_t)nb;
    ri.w = (int)(nb >> 32);
    __syncwarp();
    rowinfo[lane] = ri;
    __syncwarp();
  }

  __device__ __forceinline__ void issue(const Params& prm, int which, const float* __restrict__ base, int step, uint32_t dst,
                                         uint32_t dst_step) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      bool ok = (okm >> i) & 1u;
      const float* src = base + (ok ? off[i] : 0);
      ok = ok && AMSIM_IN(prm, which, src, float4);
      cp_async16n(dst + i * dst_step, src, ok ? 16 : 0);
      off[i] += step;
    }
    --left;
  }
  // CT_KVEC patch rows: group i of a lane = row 16 i + lane / 2, steps 4 (lane % 2)...
  __device__ __forceinline__ void step_v(const CodeParams& cp, const float* __restrict__ Vg, int kb, const int4* rowinfo,
                                         uint32_t dst, int lane) {
    const Params& prm = cp.prm;
    const Gather& g = prm.g;
    if (left == 0) {
      const int k = kb * CT_KB + k_at;
      const int tap = (int)fdiv((uint32_t)k, g.d_sc), ch = k - tap * g.SC;
      const int kh = (int)fdiv((uint32_t)tap, g.d_kw), kw = tap - kh * g.KW;
      left = (g.SC - ch + k_at) / CT_KB;
      okm = 0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int4 ri = rowinfo[i * 16 + (lane >> 1)];
        const int u = ri.x + kh, v = ri.y + kw;
        if ((unsigned)u < (unsigned)g.lim_h && (unsigned)v < (unsigned)g.lim_w) okm |= 1u << i;
        off[i] = ri.z + (u * g.SW + v) * g.SC + ch + 4 * (lane & 1);
      }
    }
    const int r = lane >> 1;
    issue(prm, BUF_V, Vg, CT_KB, dst + r * 32 + (((lane & 1) ^ ((r >> 2) & 1)) << 4), 16 * 32);
  }
  // CT_RVEC: group i of a lane = step 4 i + lane / 8, rows 4 (lane % 8)...; CT_KVEC: as above
  __device__ __forceinline__ void step_u(const CodeParams& cp, const float* __restrict__ Ug, int first, int kb, uint32_t dst,
                                         int lane) {
    const Params& prm = cp.prm;
    const bool rvec = cp.u_mode == CT_RVEC;
    if (left == 0) {
      const int k = kb * CT_KB + k_at;
      if (cp.fgrad) {
        left = INT32_MAX;
      } else {
        const int tap = (int)fdiv((uint32_t)k, prm.g.d_sc);
        left = (prm.g.SC - (k - tap * prm.g.SC) + k_at) / CT_KB;
      }
      const int base = (int)u_offset(cp, k);
      okm = 0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int q = first + (rvec ? 4 * (lane & 7) : i * 16 + (lane >> 1));
        if (q < prm.Q) okm |= 1u << i;
        off[i] = base + (rvec ? (4 * i + (lane >> 3)) * prm.u_sk + q : q * prm.u_sq + 4 * (lane & 1));
      }
    }
    if (rvec) {
      issue(prm, BUF_U, Ug, CT_KB * prm.u_sk, dst + lane * 16, 512);
    } else {
      const int r = lane >> 1;
      issue(prm, BUF_U, Ug, CT_KB, dst + r * 32 + (((lane & 1) ^ ((r >> 2) & 1)) << 4), 16 * 32);
    }
  }

  __device__ __forceinline__ void fetch_v(const CodeParams& cp, const float* __restrict__ Vg, int first, int kb,
                                          const int4* rowinfo, uint32_t dst, int lane) const {
    const Params& prm = cp.prm;
    const Gather& g = prm.g;
    if (cp.fgrad) {
      if (cp.v_mode == CT_RVEC) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int kl = i * 4 + (lane >> 3), pix = kb * CT_KB + k_at + kl;
          const uint32_t n = fdiv((uint32_t)pix, g.d_img);
          const uint32_t rem = (uint32_t)pix - n * (uint32_t)(g.PH * g.PW);
          const uint32_t a = fdiv(rem, g.d_pw);
          const uint32_t b = rem - a * (uint32_t)g.PW;
          const int u = (int)a * g.ps_h - g.off_t + e_kh, v = (int)b * g.ps_w - g.off_l + e_kw;
          bool ok = e_ok && pix < prm.K && (unsigned)u < (unsigned)g.lim_h && (unsigned)v < (unsigned)g.lim_w;
          const float* src = ok ? Vg + ((long long)n * ((long long)g.SH * g.SW * g.SC) + ((long long)(u * g.SW + v) * g.SC + e_ch)) : Vg;
          ok = ok && AMSIM_IN(prm, BUF_V, src, float4);
          cp_async16n(dst + kl * 128 + (lane & 7) * 16, src, ok ? 16 : 0);
        }
      } else {
#pragma unroll 4
        for (int kl = 0; kl < CT_HALF; ++kl) {
          const int pix = kb * CT_KB + k_at + kl;
          const uint32_t n = fdiv((uint32_t)pix, g.d_img);
          const uint32_t rem = (uint32_t)pix - n * (uint32_t)(g.PH * g.PW);
          const uint32_t a = fdiv(rem, g.d_pw);
          const uint32_t b = rem - a * (uint32_t)g.PW;
          const int u = (int)a * g.ps_h - g.off_t + e_kh, v = (int)b * g.ps_w - g.off_l + e_kw;
          bool ok = e_ok && pix < prm.K && (unsigned)u < (unsigned)g.lim_h && (unsigned)v < (unsigned)g.lim_w;
          const float* src = ok ? Vg + ((long long)n * ((long long)g.SH * g.SW * g.SC) + ((long long)(u * g.SW + v) * g.SC + e_ch)) : Vg;
          ok = ok && AMSIM_IN(prm, BUF_V, src, float);
          cp_async4(dst + kl * 128 + lane * 4, src, ok);
        }
      }
      return;
    }
    if (prm.v_trans) {  // V[p, k] at V[k * v_ld + p]
      if (cp.v_mode == CT_RVEC) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int kl = i * 4 + (lane >> 3), k = kb * CT_KB + k_at + kl, p = first + 4 * (lane & 7);
          bool ok = k < prm.K && p < prm.P;
          const float* src = ok ? Vg + (long long)k * prm.v_ld + p : Vg;
          ok = ok && AMSIM_IN(prm, BUF_V, src, float4);
          cp_async16n(dst + kl * 128 + (lane & 7) * 16, src, ok ? 16 : 0);
        }
      } else {
#pragma unroll 4
        for (int kl = 0; kl < CT_HALF; ++kl) {
          const int k = kb * CT_KB + k_at + kl, p = first + lane;
          bool ok = k < prm.K && p < prm.P;
          const float* src = ok ? Vg + (long long)k * prm.v_ld + p : Vg;
          ok = ok && AMSIM_IN(prm, BUF_V, src, float);
          cp_async4(dst + kl * 128 + lane * 4, src, ok);
        }
      }
      return;
    }
    const bool vec = cp.v_mode == CT_KVEC;
    const int kl = vec ? 4 * (lane & 1) : (lane & 7), k = kb * CT_KB + k_at + kl;
    const uint32_t tap = fdiv((uint32_t)k, g.d_sc);
    const int ch = k - (int)tap * g.SC;
    const int kh = (int)fdiv(tap, g.d_kw);
    const int kw = (int)tap - kh * g.KW;
    const bool k_ok = k < prm.K;
    if (vec) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = i * 16 + (lane >> 1);
        const int4 ri = rowinfo[r];
        const int u = ri.x + kh, v = ri.y + kw;
        bool ok = k_ok && (unsigned)u < (unsigned)g.lim_h && (unsigned)v < (unsigned)g.lim_w;
        const long long nb = ((long long)ri.w << 32) | (uint32_t)ri.z;
        const float* src = ok ? Vg + nb + ((long long)(u * g.SW + v) * g.SC + ch) : Vg;
        ok = ok && AMSIM_IN(prm, BUF_V, src, float4);
        cp_async16n(dst + r * 32 + (((lane & 1) ^ ((r >> 2) & 1)) << 4), src, ok ? 16 : 0);
      }
    } else {
#pragma unroll 4
      for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + (lane >> 3);
        const int4 ri = rowinfo[r];
        const int u = ri.x + kh, v = ri.y + kw;
        bool ok = k_ok && (unsigned)u < (unsigned)g.lim_h && (unsigned)v < (unsigned)g.lim_w;
        const long long nb = ((long long)ri.w << 32) | (uint32_t)ri.z;
        const float* src = ok ? Vg + nb + ((long long)(u * g.SW + v) * g.SC + ch) : Vg;
        ok = ok && AMSIM_IN(prm, BUF_V, src, float);
        cp_async4(dst + r * 32 + (((kl >> 2) ^ ((r >> 2) & 1)) << 4) + (kl & 3) * 4, src, ok);
      }
    }
  }

  // Element offset of U[k, q = 0] (see Params).
  __device__ __forceinline__ static long long u_offset(const CodeParams& cp, int k) {
    const Params& prm = cp.prm;
    if (cp.fgrad) return (long long)k * prm.u_sk;
    const Gather& g = prm.g;
    const uint32_t tap = fdiv((uint32_t)k, g.d_sc);
    const int kk = k - (int)tap * g.SC;
    const int tj = (int)fdiv(tap, g.d_kw);
    const int tp = prm.u_t0 + tj * prm.u_tj + ((int)tap - tj * g.KW) * prm.u_ti;
    return (long long)tp * prm.u_tap + (long long)kk * prm.u_sk;
  }

  __device__ __forceinline__ void fetch_u(const CodeParams& cp, const float* __restrict__ Ug, int first, int kb, uint32_t dst,
                                          int lane) const {
    const Params& prm = cp.prm;
    if (cp.u_mode == CT_RVEC) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int kl = i * 4 + (lane >> 3), k = kb * CT_KB + k_at + kl, q = first + 4 * (lane & 7);
        bool ok = k < prm.K && q < prm.Q;
        const float* src = ok ? Ug + u_offset(cp, k) + q : Ug;
        ok = ok && AMSIM_IN(prm, BUF_U, src, float4);
        cp_async16n(dst + kl * 128 + (lane & 7) * 16, src, ok ? 16 : 0);
      }
    } else if (cp.u_mode == CT_KVEC) {
      const int k = kb * CT_KB + k_at + 4 * (lane & 1);
      const float* col = Ug + u_offset(cp, k);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = i * 16 + (lane >> 1), q = first + r;
        bool ok = k < prm.K && q < prm.Q;
        const float* src = ok ? col + (long long)q * prm.u_sq : Ug;
        ok = ok && AMSIM_IN(prm, BUF_U, src, float4);
        cp_async16n(dst + r * 32 + (((lane & 1) ^ ((r >> 2) & 1)) << 4), src, ok ? 16 : 0);
      }
    } else if (cp.u_mode == CT_KSCL) {
      const int kl = lane & 7, k = kb * CT_KB + k_at + kl;
      const float* col = Ug + u_offset(cp, k);
#pragma unroll 4
      for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + (lane >> 3), q = first + r;
        bool ok = k < prm.K && q < prm.Q;
        const float* src = ok ? col + (long long)q * prm.u_sq : Ug;
        ok = ok && AMSIM_IN(prm, BUF_U, src, float);
        cp_async4(dst + r * 32 + (((kl >> 2) ^ ((r >> 2) & 1)) << 4) + (kl & 3) * 4, src, ok);
      }
    } else {
#pragma unroll 4
      for (int kl = 0; kl < CT_HALF; ++kl) {
        const int k = kb * CT_KB + k_at + kl, q = first + lane;
        bool ok = k < prm.K && q < prm.Q;
        const float* src = ok ? Ug + u_offset(cp, k) + (long long)q * prm.u_sq : Ug;
        ok = ok && AMSIM_IN(prm, BUF_U, src, float);
        cp_async4(dst + kl * 128 + lane * 4, src, ok);
      }
    }
  }
};

// The epilogue of one output of column q (see store_out_tile).
__device__ __forceinline__ float finish_out(const Params& prm, float o, int q) {
  if (prm.has_alpha) o = __fmul_rn(o, prm.alpha);
  if (prm.scale != nullptr) o = __fmul_rn(o, __ldg(prm.scale + q));
  if (prm.bias != nullptr) o = __fadd_rn(o, __ldg(prm.bias + q));
  return prm.relu && o < 0.f ? 0.f : o;
}

// Writes 4 consecutive columns of one output row through the epilogue.
__device__ __forceinline__ void store_out4(const Params& prm, float* __restrict__ orow, int qg, float (&o)[4], bool vec_out) {
  if (prm.bias != nullptr || prm.relu || prm.scale != nullptr || prm.has_alpha) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (qg + r < prm.Q) o[r] = finish_out(prm, o[r], qg + r);
  }
  if (vec_out && qg + 3 < prm.Q) {
    if (AMSIM_IN(prm, BUF_O, orow + qg, float4)) *reinterpret_cast<float4*>(orow + qg) = make_float4(o[0], o[1], o[2], o[3]);
  } else {
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (qg + r < prm.Q && AMSIM_IN(prm, BUF_O, orow + (long long)(qg + r) * prm.o_sq, float)) orow[(long long)(qg + r) * prm.o_sq] = o[r];
  }
}

// First element of output row pg of batch z.
__device__ __forceinline__ float* out_row(const Params& prm, int z, int pg) {
  const Gather& g = prm.g;
  long long row = pg;
  if (prm.o_strided) {
    const uint32_t n = fdiv((uint32_t)pg, g.d_img);
    const uint32_t rem = (uint32_t)pg - n * (uint32_t)(g.PH * g.PW);
    const uint32_t yy = fdiv(rem, g.d_pw);
    const uint32_t xx = rem - yy * (uint32_t)g.PW;
    row = ((long long)n * prm.o_h + (long long)yy * prm.o_sh + prm.o_a) * prm.o_w + (long long)xx * prm.o_sw + prm.o_b;
  }
  return prm.O + (long long)z * prm.o_bs + row * prm.o_sp;
}

// Recomputes those of 16 outputs (row pg of batch z, columns q0..) that a tile has left as NaN, as the table kernels'
// chain over the whole reduction.  An accumulator holds out / unit (1 / unit is up to 64), so sums from 2^122 on are
// infinite there, and nothing makes them finite again; FP32 holds them up to 2^128.  Operands with exponent field 255
// give NaN for every output they take part in.  A chain that has become NaN ends.
static __device__ __noinline__ void repair_outputs(const CodeParams& cp, int z, int pg, int q0) {
  const Params& prm = cp.prm;
  const Gather& g = prm.g;
  const float* const Vg = prm.V + (long long)z * prm.v_bs;
  const float* const Ug = prm.U + (long long)z * prm.u_bs;
  float* const orow = out_row(prm, z, pg);
  float s[16];
  uint32_t todo = 0;
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    const float* const at = orow + (long long)(q0 + c) * prm.o_sq;
    const float was = q0 + c < prm.Q && AMSIM_IN(prm, BUF_O, at, float) ? *at : 0.f;
    s[c] = 0.f;
    if (was != was) todo |= 1u << c;
  }
  const uint32_t redo = todo;
  for (int k = 0; k < prm.K && todo; ++k) {
    const float* src = Vg;
    bool ok = true;
    if (!cp.fgrad && prm.v_trans) {
      src += (long long)k * prm.v_ld + pg;
    } else {  // (filter gradient: pg is a filter element and k a grid position; otherwise the other way round)
      const uint32_t pix = (uint32_t)(cp.fgrad ? k : pg), el = (uint32_t)(cp.fgrad ? pg : k);
      const uint32_t n = fdiv(pix, g.d_img);
      const uint32_t rem = pix - n * (uint32_t)(g.PH * g.PW);
      const uint32_t a = fdiv(rem, g.d_pw);
      const uint32_t b = rem - a * (uint32_t)g.PW;
      const uint32_t tap = fdiv(el, g.d_sc);
      const int ch = (int)(el - tap * (uint32_t)g.SC);
      const int kh = (int)fdiv(tap, g.d_kw), kw = (int)tap - kh * g.KW;
      const int u = (int)a * g.ps_h - g.off_t + kh, v = (int)b * g.ps_w - g.off_l + kw;
      ok = (unsigned)u < (unsigned)g.lim_h && (unsigned)v < (unsigned)g.lim_w;
      if (ok) src += (long long)n * ((long long)g.SH * g.SW * g.SC) + ((long long)(u * g.SW + v) * g.SC + ch);
    }
    ok = ok && AMSIM_IN(prm, BUF_V, src, float);
    const uint32_t vb = ok ? __float_as_uint(__ldg(src)) : 0u;
    const uint32_t iv = (vb >> (23 - prm.m)) & prm.cmask;
    const long long u_at = RowFetch::u_offset(cp, k);
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      if (!((todo >> c) & 1u)) continue;
      const float* const us = Ug + u_at + (long long)(q0 + c) * prm.u_sq;
      const uint32_t ub = AMSIM_IN(prm, BUF_U, us, float) ? __float_as_uint(__ldg(us)) : 0u;
      if ((vb & 0x7F800000u) == 0x7F800000u || (ub & 0x7F800000u) == 0x7F800000u) {
        s[c] = __uint_as_float(0x7FFFFFFFu);
      } else if (vb & 0x7F800000u) {  // as in mac_step
        const uint32_t e = (uint32_t)__ldg(prm.lut + ((((ub >> (23 - prm.m)) & prm.cmask) << prm.m) | iv)) * prm.mult;
        s[c] = __fmaf_rn(__uint_as_float(ub & 0xFF800000u), __uint_as_float(e + (vb & 0xFF800000u)), s[c]);
      }
      if (s[c] != s[c]) todo &= ~(1u << c);
    }
  }
#pragma unroll
  for (int c = 0; c < 16; ++c)
    if ((redo >> c) & 1u) orow[(long long)(q0 + c) * prm.o_sq] = finish_out(prm, s[c], q0 + c);
}

// Share of a thread in draining and writing a tile: 16-column units u = g, g + NG, ... of the tile (g = warp / 4), of
// the CTA's tile row 32 * (warp % 4) + lane.
template <int S, int BN>
struct CodeAcc {
  static constexpr int NG = CodeSmem<S, BN>::NW / 4;
  static constexpr int UNITS = BN / 16;
  static constexpr int UPT = (UNITS + NG - 1) / NG;
  static constexpr int NTE = NG * 128;                 // threads that drain
  static constexpr int SLOT_FLOATS = UPT * 16 * NTE;   // one parked tile of a CTA
};

template <int S, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(CodeSmem<S, BN>::NT, 1) code_gemm(const __grid_constant__ CodeParams cp) {
  using C = CodeCfg<S>;
  using L = CodeSmem<S, BN>;
  using A = CodeAcc<S, BN>;
  constexpr int NW = L::NW, GU = L::GU, KS = C::KS, W = C::W, CH = C::CH, REP = C::REP, NST = L::NST;
  constexpr int NG = A::NG, UPT = A::UPT;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ uint64_t bars[3 * NST + 3];
  __shared__ uint32_t tmem_holder;
  __shared__ int flag_s;
  __shared__ uint32_t signal_s;  // where the other CTA's signals store their word
  __shared__ int odd_s;    // outputs that are not finite have been written (repair_outputs)
  __shared__ int wrote_s;  // this CTA has written its rows of the run's first (1) or last (2) tile, shared with other runs
  const Params& prm = cp.prm;
  const Gather& g = prm.g;
  const uint32_t smem0 = (smem_addr(smem_raw) + 1023u) & ~1023u;
  uint8_t* const smem = smem_raw + (smem0 - smem_addr(smem_raw));
  const int t = threadIdx.x, lane = t & 31;
  const int w = __shfl_sync(0xffffffffu, t >> 5, 0);
  const uint32_t rank = blockIdx.x & 1u;  // in the pair; the CTA of rank 0 issues the products of both
  const int pair = blockIdx.x >> 1;
  const uint32_t bar0 = smem_addr(bars);
  const uint32_t bar_full = bar0, bar_empty = bar0 + 8 * NST, bar_peer = bar0 + 16 * NST, bar_done = bar0 + 24 * NST,
                 bar_free = bar_done + 8, bar_exit = bar_done + 16;

  if (t == 0) {
    for (int i = 0; i < NST; ++i) {
      mbar_init(bar_full + 8 * i, NW / 2);  // half of the warps make a stage; the other CTA adds its scale bytes
      mbar_init(bar_peer + 8 * i, 1);       // (rank 0) the other CTA's stage is full: its signal, and the issue warp expecting it
      mbar_init(bar_empty + 8 * i, 1);
    }
    mbar_init(bar_done, 1);
    mbar_init(bar_exit, 1);
    mbar_init(bar_free, 4 * NG);            // (rank 0) this CTA's draining warps, and the other's signals
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    odd_s = wrote_s = 0;
  }
  if (w == NW) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_holder)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  uint4* const tab_v = reinterpret_cast<uint4*>(smem + L::OFF_TAB);
  uint4* const tab_u = tab_v + (cp.rows_v + 1) * CH * REP;
  copy_code_table<CH, REP>(tab_v, cp.tab_v, cp.rows_v + 1, t, L::NT);
  copy_code_table<CH, REP>(tab_u, cp.tab_u, cp.rows_u + 1, t, L::NT);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_holder, 0);

  const int nkb_all = (prm.K + CT_KB - 1) / CT_KB;
  int run_at = (int)balanced_begin(pair, prm.sk_iters, prm.sk_grid);  // (the launch has fewer than 2^31 blocks)
  const int run_end = (int)balanced_begin((long long)pair + 1, prm.sk_iters, prm.sk_grid);
  auto decode_tile = [&](int at, int& tp, int& tq, int& tz, int& kb0, int& kb1) {
    const uint32_t tile = (uint32_t)at / (uint32_t)nkb_all;
    kb0 = at - (int)tile * nkb_all;
    kb1 = kb0 + min(nkb_all - kb0, run_end - at);
    const uint32_t rest = tile / (uint32_t)prm.sk_qtiles;
    tq = (int)(tile - rest * (uint32_t)prm.sk_qtiles);
    tz = (int)(rest / (uint32_t)prm.sk_ptiles);
    tp = (int)rest - tz * prm.sk_ptiles;
  };
  // columns of U in the products of tile column tq; each CTA encodes one half of them
  auto tile_columns = [&](int tq) { return min(BN, (prm.Q - tq * BN + 63) / 64 * 64); };
  Waiter wt{cp.stuck, cp.no_tries != 0};
  if (cp.no_tries && t == 0) *(volatile unsigned*)cp.stuck = 1u;

  if (w == NW && rank != 0) {
    // ---- forwards "stage full" of this CTA to the issuing one: one warp fences for all, and the operand warps signal
    // inside their CTA only.  The order: an operand warp's stores, its arrive (release in the CTA), this warp's wait, the
    // fence to the proxy that the products read through, the signal (release in the cluster), the issue warp's wait.
    const uint32_t lead = cluster_addr(bar_peer, 0), signal = cluster_addr(smem_addr(&signal_s), 0);
    uint32_t b = 0, phase = 0;
    const long long stages = (long long)(run_end - run_at) * C::STAGES_PER_KB;
    for (long long i = 0; i < stages; ++i) {
      wt.wait_warp(bar_full + 8 * b, phase);
      asm volatile("tcgen05.fence::after_thread_sync;\nfence.proxy.async.shared::cta;\ntcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0 && !wt.dead) st_async_remote(signal, 0, lead + 8 * b);
      if (++b == NST) {
        b = 0;
        phase ^= 1;
      }
    }
  } else if (w == NW) {
    // ---- issue warp: moves the scales to tensor memory and issues the products --------------------
    // The whole warp walks the loop on warp-uniform values and one elected lane issues, so descriptors
    // and addresses stay in uniform registers (with a single-lane loop the moves into uniform registers
    // took 1200 clocks per stage, more than twice its products).
    const bool elected = elect_lane();
    uint32_t b = 0, phase = 0, sfset = 0, chunk = 0;
    const uint64_t desc_codes = smem_desc(smem0, 16, 1024, 2), desc_sf = smem_desc(smem0 + L::OFF_SF, 128, 128, 0);
    while (run_at < run_end) {
      int tp, tq, tz, kb0, kb1;
      decode_tile(run_at, tp, tq, tz, kb0, kb1);
      run_at += kb1 - kb0;
      const uint32_t idesc = code_idesc(tile_columns(tq));
      for (int kb = kb0; kb < kb1; kb += cp.chunk, ++chunk) {
        const int stages = (min(kb1, kb + cp.chunk) - kb) * C::STAGES_PER_KB;
        wt.wait_warp(bar_free, (chunk & 1) ^ 1);
        uint32_t acc = 0;  // first column of the stage's accumulator
#pragma unroll 1
        for (int i = 0; i < stages; ++i) {
          if (lane == 0 && !wt.dead) mbar_arrive_expect(bar_peer + 8 * b, 4);
          wt.wait(bar_full + 8 * b, phase);
          wt.wait_warp(bar_peer + 8 * b, phase);
          asm volatile("tcgen05.fence::after_thread_sync;\nfence.proxy.async.shared::cta;" ::: "memory");
          const uint64_t bd = desc_codes + b * (L::CODE_BYTES >> 4), sfd = desc_sf + b * (L::SF_BYTES >> 4);
          const uint32_t at = tmem + L::T_CODES + b * 32;
          const uint32_t sf_t = tmem + L::T_SF + sfset * L::SF_COLS;  // scale columns: V [word], U [word][128 columns]
          const uint32_t sfu_t = sf_t + W * 4;
          if (elected && !wt.dead) {
#pragma unroll
            for (int j = 0; j < W; ++j) scales_to_tmem(sf_t + 4 * j, sfd + 32 * j);
#pragma unroll
            for (int j = 0; j < W; ++j)
#pragma unroll
              for (int h = 0; h < L::NBH; ++h) scales_to_tmem(sfu_t + (j * L::NBH + h) * 4, sfd + 32 * (W + h * W + j));
#pragma unroll
            for (int s = 0; s < 4; ++s) {  // 64 code steps each; their two scale bytes sit in half (id 0 / 2) of a word
              const int word = S == 128 ? 0 : s >> 1, id = S == 128 ? (s >> 1) * 2 : (s & 1) * 2;
              mma_codes(tmem + acc, at + 8 * s, bd + 2 * s, idesc | ((uint32_t)id << 4) | ((uint32_t)id << 29), sf_t + word * 4,
                        sfu_t + word * L::NBH * 4, s > 0 || i >= L::NACC);
            }
            tc_commit(bar_empty + 8 * b);
            if (i + 1 == stages) tc_commit(bar_done);
          }
          __syncwarp();
          sfset ^= 1;
          acc = acc + BN == L::NACC * BN ? 0 : acc + BN;
          if (++b == NST) {
            b = 0;
            phase ^= 1;
          }
        }
      }
    }
    wt.wait_warp(bar_free, (chunk & 1) ^ 1);  // no signal is on its way to this CTA when it ends
  } else {
    // ---- operand warps: 32 rows of V (w < 8) or columns of U each, one half of every block ----------
    const bool is_v = w < 8;
    const int group = is_v ? w & 3 : (w - 8) % GU;
    const int half = is_v ? w >> 2 : (w - 8) / GU;
    const uint32_t raw_s = smem0 + L::OFF_RAW + w * 2 * CT_RAW;
    int4* const rowinfo = reinterpret_cast<int4*>(smem + L::OFF_ROW) + (is_v ? 32 * w : 0);
    // first row of V or column of U of this warp in a tile; -1: beyond the operand
    auto first_row = [&](int tp, int tq) {
      if (is_v) {
        const long long r = (long long)tp * CT_ROWS + (int)rank * 128 + 32 * group;
        return r < prm.P ? (int)r : -1;
      }
      const int own = tile_columns(tq) / 2, q = tq * BN + (int)rank * own + 32 * group;
      return 32 * group < own && q < prm.Q ? q : -1;
    };
    const bool kmode = is_v ? (cp.v_mode == CT_KVEC || cp.v_mode == CT_KSCL) : (cp.u_mode == CT_KVEC || cp.u_mode == CT_KSCL);
    const int rows = is_v ? cp.rows_v : cp.rows_u, sh = is_v ? cp.sh_v : cp.sh_u;
    const uint32_t row_mask = (uint32_t)rows - 1u;
    const uint32_t tab = smem0 + L::OFF_TAB + (is_v ? 0 : (cp.rows_v + 1) * CH * REP * 16) + (lane & (REP - 1)) * 16;
    const int tab_chunk = (rows + 1) * REP * 16;
    // this lane's row of V codes in tensor memory, its place among the scale words (U: set for each tile)
    const uint32_t code_t = tmem + L::T_CODES + ((uint32_t)(w & 3) << 21);
    uint32_t sf_off = L::OFF_SF + lane * 16 + group * 4;
    const uint32_t peer_smem = cluster_addr(smem0, rank ^ 1u), peer_full = cluster_addr(bar_full, rank ^ 1u);
    const uint32_t lead_free = cluster_addr(bar_free, 0), lead_signal = cluster_addr(smem_addr(&signal_s), 0);

    RowFetch rf;
    rf.k_at = half * CT_HALF;
    int ld_at = run_at;
    int ld_p = 0, ld_q = 0, ld_z = 0, ld_kb = 0, ld_kb1 = 0, ld_buf = 0, ld_first = -1;
    auto fetch_next = [&]() {
      if (ld_kb == ld_kb1 && ld_at < run_end) {
        decode_tile(ld_at, ld_p, ld_q, ld_z, ld_kb, ld_kb1);
        ld_at += ld_kb1 - ld_kb;
        ld_first = first_row(ld_p, ld_q);
        rf.new_tile(cp, is_v, ld_first < 0 ? prm.P : ld_first, rowinfo, lane);
      }
      if (ld_kb < ld_kb1) {
        const uint32_t dst = raw_s + ld_buf * CT_RAW;
        if (ld_first < 0) {
        } else if (is_v) {
          if (cp.step_v) rf.step_v(cp, prm.V + (long long)ld_z * prm.v_bs, ld_kb, rowinfo, dst, lane);
          else rf.fetch_v(cp, prm.V + (long long)ld_z * prm.v_bs, ld_first, ld_kb, rowinfo, dst, lane);
        } else {
          if (cp.step_u) rf.step_u(cp, prm.U + (long long)ld_z * prm.u_bs, ld_first, ld_kb, dst, lane);
          else rf.fetch_u(cp, prm.U + (long long)ld_z * prm.u_bs, ld_first, ld_kb, dst, lane);
        }
        ++ld_kb;
        ld_buf ^= 1;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };

    constexpr int SPH = C::STAGES_PER_KB / 2;   // stages this warp makes of a block, then the other warp of its rows as many
    // Skipping the other warp's stages, a warp may find a barrier SPH + 1 stages behind: this has to be less than one turn
    // of the ring, or the parity it waits for is that of the turn before.
    static_assert(SPH < NST, "ring");
    uint32_t b = 0, phase = 1, chunk = 0;       // stage buffer, parity of its 'empty' barrier
    auto advance = [&](int n) {
      b += n;
      if (b >= NST) {
        b -= NST;
        phase ^= 1;
      }
    };
    if (half) advance(SPH);
    // this lane's row of a stage of U codes, 16-byte place i at (i ^ row & 7) (128-byte swizzle)
    const uint32_t code_base = smem0 + (32 * group + lane) * 128 + ((uint32_t)(lane & 7) << 4);
    const int grp = w >> 2;
    float* slot = nullptr;  // this thread's place among the parked tiles
    auto read_slot = [&](int i, float (&v)[16]) {
#pragma unroll
      for (int c = 0; c < 16; ++c) v[c] = AMSIM_IN(prm, BUF_WS, slot + (i * 16 + c) * A::NTE, float) ? __ldcg(slot + (i * 16 + c) * A::NTE) : 0.f;
    };
    auto park_unit = [&](int i, const float (&v)[16]) {
#pragma unroll
      for (int c = 0; c < 16; ++c)
        if (AMSIM_IN(prm, BUF_WS, slot + (i * 16 + c) * A::NTE, float)) __stcg(slot + (i * 16 + c) * A::NTE, v[c]);
    };
    // Takes this thread's units of a finished chunk out of tensor memory, adds what earlier chunks of the segment
    // left in the slot (first: nothing) and hands them on; the next chunk's products may begin once all are out.
    // The tensor core idles meanwhile, so the slot is read a unit ahead, from before the chunk is done.
    auto take_chunk = [&](bool first, int stages, auto&& use) {
      const int units = (A::UNITS - grp + NG - 1) / NG;
      float s[16];
      if (!first) read_slot(0, s);
      wt.wait_warp(bar_done, chunk & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int i = 0; i < units; ++i) {
        float v[16];
        const uint32_t at = tmem + ((uint32_t)(w & 3) << 21) + (grp + i * NG) * 16;
        tmem_load16(at, v);
#pragma unroll
        for (int a = 1; a < L::NACC; ++a) {
          if (a >= stages) break;  // (a chunk of fewer stages than accumulators)
          float more[16];
          tmem_load16(at + a * BN, more);
#pragma unroll
          for (int c = 0; c < 16; ++c) v[c] = __fadd_rn(v[c], more[c]);
        }
        if (i + 1 == units) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0 && !wt.dead) {
            if (rank != 0) st_async_remote(lead_signal, 0, lead_free);
            else if (w == 0) mbar_arrive_expect(bar_free, 4 * 4 * NG);
            else mbar_arrive(bar_free);
          }
        }
        if (!first) {
#pragma unroll
          for (int c = 0; c < 16; ++c) v[c] = __fadd_rn(s[c], v[c]);
          if (i + 1 < units) read_slot(i + 1, s);
        }
        use(i, v);
      }
    };
    // Moves a finished chunk of the segment to the slot.
    auto drain = [&](bool first) {
      if (grp < NG) take_chunk(first, cp.chunk * C::STAGES_PER_KB, park_unit);
      ++chunk;
    };

    int buf = 0;
    fetch_next();
    while (run_at < run_end) {
      int cp_, cq, cz, kb0, kb1;
      decode_tile(run_at, cp_, cq, cz, kb0, kb1);
      run_at += kb1 - kb0;
      const bool active = first_row(cp_, cq) >= 0;
      const int own = tile_columns(cq) / 2;
      const bool sends = !is_v && 32 * group < own;  // (also for columns beyond Q: the other CTA counts on own * 4 * W bytes)
      if (!is_v) {
        const int place = (int)rank * (own / 32) + group;  // of the pair's 32-column groups
        sf_off = L::OFF_SF + (1 + (place >> 2)) * W * 512 + lane * 16 + (place & 3) * 4;
      }
      slot = prm.ws + (((long long)pair * 2 + (kb0 == 0 ? 1 : 0)) * 2 + rank) * A::SLOT_FLOATS + t;
      bool pending = false, fresh = true;
      int kc = kb0;  // first block of the chunk
      for (int kb = kb0; kb < kb1; ++kb) {
        fetch_next();
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const uint32_t rb = raw_s + buf * CT_RAW;
        buf ^= 1;
        // the next chunk's first stages are made while the last one finishes, as many as the ring holds and at most one
        // chunk: a finished chunk is taken out at once (until then the tensor core idles)
        if (pending && ((kb - kc) * C::STAGES_PER_KB + half * SPH + SPH > NST || kb - kc == cp.chunk - 1 ||
                        __all_sync(0xffffffffu, mbar_test(bar_done, chunk & 1)))) {
          drain(fresh);
          fresh = pending = false;
        }
#pragma unroll
        for (int j = 0; j < SPH; ++j) {
          uint32_t x[KS];
          uint4 q[8];
          if (!active) {
#pragma unroll
            for (int e = 0; e < KS; ++e) x[e] = 0;
          } else {
            if (kmode) {
              const uint32_t row = rb + lane * 32;
              const int flip = (lane >> 2) & 1;
              if (KS == 2) {
                const uint2 v = lds64(row + (((j >> 1) ^ flip) << 4) + (j & 1) * 8);
                x[0] = v.x; x[1] = v.y;
              } else {
#pragma unroll
                for (int i = 0; i < KS / 4; ++i) {
                  const uint4 v = lds128(row + (((j * (KS / 4) + i) ^ flip) << 4));
                  x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[(4 * i + 3) % KS] = v.w;
                }
              }
            } else {
#pragma unroll
              for (int i = 0; i < KS; ++i) x[i] = lds32(rb + (j * KS + i) * 128 + lane * 4);
            }
            // all eight 16-byte pieces are read before the first is stored (the compiler cannot tell that the
            // stage and the table do not overlap), and before the wait for the stage
#pragma unroll
            for (int e = 0; e < KS; ++e) {
              // zero and denormal elements take the table's zero row: their products are exactly 0
              const uint32_t idx = (x[e] & 0x7F800000u) ? ((x[e] >> sh) & row_mask) : (uint32_t)rows;
              const uint32_t src = tab + idx * (REP * 16);
#pragma unroll
              for (int c = 0; c < CH; ++c) q[e * CH + c] = lds128(src + c * tab_chunk);
            }
          }
          wt.wait_warp(bar_empty + 8 * b, phase);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (active) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const uint32_t sign = (uint32_t)((int)x[i / CH] >> 31) & 0x88888888u;
              q[i].x ^= sign; q[i].y ^= sign; q[i].z ^= sign; q[i].w ^= sign;
            }
            if (is_v) {
              tmem_store32(code_t + b * 32, q);
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) sts128((code_base + b * L::CODE_BYTES) ^ ((uint32_t)i << 4), q[i]);
            }
          }
          // scale bytes = exponent fields; one 32-bit word covers two matrix instructions
          if (active || sends) {
            uint32_t sf[W];
            if (S == 64) {
              sf[0] = __byte_perm(x[0] << 1, x[1] << 1, 0x7733);
              sf[W - 1] = __byte_perm(x[2 % KS] << 1, x[3 % KS] << 1, 0x7733);
            } else if (S == 128) {
              sf[0] = __byte_perm(x[0] << 1, x[1] << 1, 0x7733);
            } else {
#pragma unroll
              for (int i = 0; i < W; ++i) {
                const uint32_t lo = __byte_perm(x[(4 * i) % KS] << 1, x[(4 * i + 1) % KS] << 1, 0x0073);
                const uint32_t hi = __byte_perm(x[(4 * i + 2) % KS] << 1, x[(4 * i + 3) % KS] << 1, 0x0073);
                sf[i] = __byte_perm(lo, hi, 0x5410);
              }
            }
            const uint32_t sf_at = sf_off + b * L::SF_BYTES;
#pragma unroll
            for (int i = 0; i < W; ++i) {
              sts32(smem0 + sf_at + 512 * i, sf[i]);
              if (sends && !wt.dead) st_async_remote(peer_smem + sf_at + 512 * i, sf[i], peer_full + 8 * b);  // both CTAs need every column's scales
            }
          }
          __syncwarp();
          if (lane == 0 && !wt.dead) {
            if (is_v && group == 0) mbar_arrive_expect(bar_full + 8 * b, own * 4 * W);
            else mbar_arrive(bar_full + 8 * b);
          }
          advance(1);
        }
        advance(SPH);
        if (kb - kc == cp.chunk - 1) {
          kc = kb + 1;
          pending = kc < kb1;
        }
      }
      if (pending) {
        drain(fresh);
        fresh = false;
      }

      // ---- epilogue: the last chunk and the slot make the segment's sums ---------------------------
      if (grp < NG) {
        const long long tile = ((long long)cz * prm.sk_ptiles + cp_) * prm.sk_qtiles + cq;
        const bool shared_tile = kb0 != 0 || kb1 != nkb_all;
        const bool vec_out = prm.o_sq == 1 && (prm.o_sp & 3) == 0 && (prm.o_bs & 3) == 0 && ((reinterpret_cast<uintptr_t>(prm.O) & 15) == 0);
        auto write_unit = [&](int i, const float (&v)[16]) {
          const int u = grp + i * NG;
          const int pg = cp_ * CT_ROWS + (int)rank * 128 + (w & 3) * 32 + lane, q0 = cq * BN + u * 16;
          if (pg >= prm.P || q0 >= prm.Q) return;
          float* const orow = out_row(prm, cz, pg);
          bool finite = true;
#pragma unroll
          for (int c4 = 0; c4 < 4; ++c4) {
            float o[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              o[r] = __fmul_rn(v[4 * c4 + r], cp.unit);
              const bool odd = (__float_as_uint(o[r]) & 0x7F800000u) == 0x7F800000u;
              if (odd) o[r] = __uint_as_float(0x7FFFFFFFu);  // (stays NaN through the epilogue)
              finite = finite && !odd;
            }
            store_out4(prm, orow, q0 + 4 * c4, o, vec_out);
          }
          if (!finite) odd_s = 1;
        };
        take_chunk(fresh, ((kb1 - kb0 - 1) % cp.chunk + 1) * C::STAGES_PER_KB, [&](int i, const float (&v)[16]) {
          if (shared_tile) park_unit(i, v);
          else write_unit(i, v);
        });
        if (shared_tile) {
          // a tile shared between runs: count in; the last sharer adds the parked tiles in the order of the runs
          // (each CTA of the pair its own rows, counted apart)
          __threadfence();
          asm volatile("bar.sync 1, %0;" ::"r"(A::NTE) : "memory");
          const long long first = tile * nkb_all, last = first + nkb_all;
          int c0 = (int)(first * prm.sk_grid / prm.sk_iters);
          while (c0 > 0 && balanced_begin(c0, prm.sk_iters, prm.sk_grid) > first) --c0;
          while (balanced_begin(c0 + 1, prm.sk_iters, prm.sk_grid) <= first) ++c0;
          int c1 = (int)((last - 1) * prm.sk_grid / prm.sk_iters);
          while (c1 > 0 && balanced_begin(c1, prm.sk_iters, prm.sk_grid) > last - 1) --c1;
          while (balanced_begin(c1 + 1, prm.sk_iters, prm.sk_grid) <= last - 1) ++c1;
          if (t == 0) {
            int* const count = prm.sk_count + 2 * tile + rank;
            const int arrived = AMSIM_IN(prm, BUF_WS, count, int) ? atomicAdd(count, 1) : 0;
            flag_s = arrived == c1 - c0;
            if (arrived == c1 - c0 && AMSIM_IN(prm, BUF_WS, count, int)) *count = 0;
          }
          asm volatile("bar.sync 1, %0;" ::"r"(A::NTE) : "memory");
          const bool completes = flag_s != 0;
          if (completes && t == 0) wrote_s |= kb0 == 0 ? 2 : 1;
          asm volatile("bar.sync 1, %0;" ::"r"(A::NTE) : "memory");
          if (completes) {
            __threadfence();
#pragma unroll 1
            for (int i = 0; i < UPT; ++i) {
              if (grp + i * NG >= A::UNITS) break;
              float v[16];
#pragma unroll
              for (int c = 0; c < 16; ++c) v[c] = 0.f;
              // The sharers' tiles four at a time: 16 loads in flight (one tile after the other took a round trip to L2 each).
              // Four are summed before they are added: 74 tiles added one by one rounded the whole sum 74 times (filter
              // gradient of 64 x 256 over 96800 pixels: 1.58e-7 from the exact sum, fours 9.7e-8, the table kernels 9.8e-8).
              for (int run = c0; run <= c1; run += 4) {
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                  float part[4][4];
#pragma unroll
                  for (int r = 0; r < 4; ++r) {
                    const bool first_run = balanced_begin(run + r, prm.sk_iters, prm.sk_grid) <= first;
                    const float* src = prm.ws + (((long long)(run + r) * 2 + (first_run ? 1 : 0)) * 2 + rank) * A::SLOT_FLOATS + t;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                      const float* at = src + (i * 16 + h * 4 + c) * A::NTE;
                      part[r][c] = run + r <= c1 && AMSIM_IN(prm, BUF_WS, at, float) ? __ldcg(at) : 0.f;
                    }
                  }
                  // (in this order: sums of pairs took 150 bytes more of spills and 10 % more of 3x3 256 -> 256's time)
#pragma unroll
                  for (int r = 2; r >= 0; --r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) part[r][c] = __fadd_rn(part[r][c], part[r + 1][c]);
#pragma unroll
                  for (int c = 0; c < 4; ++c) v[h * 4 + c] = __fadd_rn(v[h * 4 + c], part[0][c]);
                }
              }
              write_unit(i, v);
            }
          }
        }
      }
      ++chunk;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  if (w == NW) {
    // Products that a dead warp left in flight have to end before the tensor memory goes.  (Otherwise this passes at once.)
    if (rank == 0 && elect_lane()) tc_commit(bar_exit);
    Waiter last{cp.stuck, false};
    last.wait_warp(bar_exit, 0);
    if (wt.dead) __nanosleep(100000);  // signals of other warps to this CTA
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (odd_s && w < 4 * NG) {  // each thread looks its own outputs over
    run_at = (int)balanced_begin(pair, prm.sk_iters, prm.sk_grid);
    while (run_at < run_end) {
      int tp, tq, tz, kb0, kb1;
      decode_tile(run_at, tp, tq, tz, kb0, kb1);
      run_at += kb1 - kb0;
      const int pg = tp * CT_ROWS + (int)rank * 128 + (w & 3) * 32 + lane;
      const bool wrote = (kb0 == 0 && kb1 == nkb_all) || (wrote_s & (kb0 == 0 ? 2 : 1));
      if (!wrote || pg >= prm.P) continue;
      for (int u = w >> 2; u < A::UNITS && tq * BN + u * 16 < prm.Q; u += NG) repair_outputs(cp, tz, pg, tq * BN + u * 16);
    }
  }
  cluster_barrier();  // neither CTA leaves while the other may still reach its shared or tensor memory
  if (w == NW) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

}  // namespace amsim
