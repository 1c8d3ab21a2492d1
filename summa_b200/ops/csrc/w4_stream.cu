// 4-bit projection of a decode step, y[M,N] = x[M,K] @ dequant(W) for few rows (weights in the k8-repacked form of
// quant.cu), as a weight stream through per-warp rings of asynchronous copies feeding warp-level mma.
//
// What bounds it: the weight bytes, if the code words can be consumed in few instructions and enough of them are in
// flight. Measured on a B200: a kernel that only loads the words of a 4096 x 28672 weight takes 14.0 us (6.3 TB/s plus
// 4.6 us of launch and ramp) with 16 warps x 4 KB in flight per SM, and 20 us with 8 warps.
//   * every product is exact whatever the range of x, the sums are fp32. Three to eight rows: a code word becomes the eight
//     bf16 values q - 8 (three shifts, four LOP3, four subtractions), and two mma.m16n8k16 take 16 columns x 32 k against all
//     8 rows of x. One or two rows: x becomes whole numbers instead, per scale group four signed digits of base 256 over a
//     power-of-two step, so that a word needs one shift and two LOP3 to be the s8 operands 16 (q - 8), and
//     ONE mma.m16n8k32 (s32 accumulation) takes 16 columns x 32 k against the 4 M digits. That holds every bf16 within a factor
//     2^21 of the group's largest exactly; a group with a smaller element that it cannot hold, an infinity or a NaN keeps its
//     bf16 values in the place of the digits and takes the bf16 products.
//   * one CTA per SM walks 16-column tiles over the whole K range; its 16 warps take the scale groups
//     round robin, each through a ring of its own in shared memory that asynchronous copies fill D groups (D KB) ahead,
//     across tiles; no barrier, no producer. (A ring in registers is held up by whatever touches a loaded register
//     early: a scale that was combined on arrival cost 27 us instead of 21.6, spilled ring registers 28 us, N 28672.)
//   * per tile every warp leaves its partial sums in one of four shared-memory buffers and streams on; the warp whose
//     turn it is adds them and runs the epilogue two tiles later (mbarriers both ways). With one block barrier and an
//     immediate epilogue per tile its latency was paid per tile. No cluster, no atomics.
//   * weights that nothing in flight writes (`static_w`) are requested before `griddepcontrol.wait`.
// Measured against the CUDA-core cluster kernel it replaces (weights from HBM, graph of launches, one row): K 4096 N 6144
// 12.0 -> 7.3 us, N 4096 7.4 -> 5.6, N 28672 28.9 -> 18.7 (gated with norm 32.9 -> 20.9), N 32000 30.3 -> 20.9, K 14336 N 4096
// 20.0 -> 12.3; four rows: 20.0 -> 9.6, 14.6 -> 7.8, 61.0 -> 26.0, 66.9 -> 28.6, 41.8 -> 19.0. Error of the sums against 64 bits
// 2.5e-6 of the result (2.7e-6), and no more with outliers of 4096 whose weights are zero (3.6e-3: that kernel multiplied
// 128 + q and took 136 times the sum of x away). The first form of the digits (three, elements below 2^-21 of the largest lost)
// took 7.3, 5.7, 20.1, 22.4 and 12.4 us; bf16 products for one row 26.0 us at N 28672. Issue slots matter: with a division and
// 64-bit products in the cursors the digits took 255 instructions a unit (16 columns x 128 k), 63 % of the slots, 21.6 us.
#include "host_util.h"
#include "sm100.cuh"
#include "w4_stream.h"

#include <type_traits>

namespace sb {

constexpr int W4S_WARPS = 16, W4S_THREADS = 512, W4S_TILE = 16, W4S_NB = 4;
constexpr int W4S_SMEM = 220 * 1024;

__device__ __forceinline__ void w4s_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void w4s_copy8(uint32_t dst_smem, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(src)) : "memory");
}
// codes of k 2 i, 2 i + 1 of a word as the bf16 pair q - 8 (0x4300 | q is 128 + q; both steps exact)
__device__ __forceinline__ uint32_t w4s_pair(uint32_t w, int i) {
  const uint32_t u = ((w >> (4 * i)) & 0x000F000Fu) | 0x43004300u;
  const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&u), __float2bfloat162_rn(136.f));
  return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ void w4s_mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                           uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// codes of k 0,4,1,5 / 2,6,3,7 of a word as s8 bytes 16 (q - 8)
__device__ __forceinline__ uint32_t w4s_lo(uint32_t w) { return ((w << 4) & 0xF0F0F0F0u) ^ 0x80808080u; }
__device__ __forceinline__ uint32_t w4s_hi(uint32_t w) { return (w & 0xF0F0F0F0u) ^ 0x80808080u; }
constexpr int W4S_MAGIC = 0x4B400000;        // float bits of 1.5 * 2^23: adding a small integer to the bits adds it to the value
constexpr float W4S_MAGICF = 12582912.f;

constexpr int W4S_SLOT = 1024 + 32;           // a group of a tile: 16 k8 rows x 64 bytes (chunks swizzled), 16 scales
struct W4SLayout {                           // shared memory, in bytes; x comes first
  int pitch, ring, sx, flags, red, psum, gsq, total;      // pitch: row of x or of digits (64 or 32 mod 128: conflict-free B loads)
};
__host__ __device__ inline W4SLayout w4s_layout(bool digits, int depth, int M, int pass_groups, int groups, bool norm, int psum_tiles) {
  W4SLayout l;
  l.pitch = digits ? pass_groups * 128 + 32 : pass_groups * 256 + 64;
  l.ring = (digits ? 4 : 1) * M * l.pitch;                                    // [warps][depth] slots
  l.sx = l.ring + W4S_WARPS * depth * W4S_SLOT;                               // digits: [pass_groups][8] fp32 steps
  l.flags = l.sx + (digits ? pass_groups * 32 : 0);                           // digits: [pass_groups][2] bytes, 1 = bf16 in their place
  l.red = l.flags + (digits ? (pass_groups * 2 + 15) & ~15 : 0);              // [buffers][warps][rows][16] fp32
  l.psum = l.red + W4S_NB * W4S_WARPS * (digits ? 8 : (M + 1) & ~1) * W4S_TILE * 4;   // [psum_tiles][M][16] fp32 (more than one K pass)
  l.gsq = l.psum + psum_tiles * M * W4S_TILE * 4;                             // [M] rstd, [M][groups] sums of squares
  l.total = l.gsq + (norm ? (M + M * groups) * 4 : 0);
  return l;
}

template <bool DIGITS, int D, int MODE>      // D: scale groups in flight per warp
__global__ void __launch_bounds__(W4S_THREADS, 1)
w4_stream_kernel(const W4StreamArgs p, const int tile_base, const int tiles, const int pass_groups, const int psum_tiles,
                 unsigned int* err) {
  extern __shared__ __align__(128) unsigned char w4s_smem[];
  __shared__ uint64_t full[W4S_NB], empty[W4S_NB];
  __shared__ int abort_flag;
  // Weights that the preceding kernel may have written are only visible behind the wait; and a following launch, which may
  // take them for settled, only starts once every CTA here has passed it.
  if (!p.static_w) asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  const int M = p.M, N = p.N, K = p.K, RP = DIGITS ? 8 : (p.M + 1) & ~1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const int groups = K >> 7;
  const W4SLayout L = w4s_layout(DIGITS, D, M, pass_groups, groups, p.gamma != nullptr, psum_tiles);
  float* sx = reinterpret_cast<float*>(w4s_smem + L.sx);
  float* red = reinterpret_cast<float*>(w4s_smem + L.red);
  float* psum = reinterpret_cast<float*>(w4s_smem + L.psum);
  float* rstd = reinterpret_cast<float*>(w4s_smem + L.gsq);
  float* gsq = rstd + M;
  // Tiles are dealt out in turn, so that the CTAs read neighbouring pieces of the same weight rows at the same time (DRAM
  // pages): N 28672 20.2 us, 21.1 with contiguous runs.
  const int t_lo = tile_base + blockIdx.x, t_hi = tile_base + tiles, t_step = gridDim.x;
  const int ntiles = (tiles - (int)blockIdx.x + t_step - 1) / t_step;
  const int I = N >> 1;                       // gated: columns of the gate half
  const int passes = (groups + pass_groups - 1) / pass_groups;
  constexpr int TILE_COLS = MODE == W4S_GATED ? 8 : W4S_TILE;       // columns (gated: gate columns) of a tile
  const int cols = MODE == W4S_GATED ? I : N;

  if (threadIdx.x == 0) {
    for (int b = 0; b < W4S_NB; ++b) { mbar_init(&full[b], W4S_WARPS); mbar_init(&empty[b], (W4S_TILE * M + 31) / 32); }
    abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();

  // Epilogue of this CTA's q-th tile (counted over the passes): 32 outputs o = m * 16 + c at a time; chunk k of the i-th
  // tile belongs to warp (i + k) % 16, which runs it two tiles later, when the other warps have long handed theirs over.
  const int chunks = (W4S_TILE * M + 31) / 32;
  int ep_q = 0, ep_pass = 0, ep_local = 0;    // the next one, its pass and its tile
  auto epilogue = [&] {
    const int q = ep_q++, pass = ep_pass, local = ep_local;
    if (++ep_local == ntiles) {
      ep_local = 0;
      ++ep_pass;
    }
    const int chunk = (warp - local) & (W4S_WARPS - 1);
    if (chunk >= chunks) return;
    const int ct = t_lo + local * t_step;
    const bool last = pass + 1 == passes;
    const float* rb = red + (q & (W4S_NB - 1)) * W4S_WARPS * RP * W4S_TILE;
    const int o = chunk * 32 + lane, m = o >> 4, c = o & 15;
    const bool row = m < M;
    const int mm = row ? m : 0;
    const int n = MODE == W4S_GATED ? ct * 8 + (c >> 1) : ct * W4S_TILE + c;
    float rv = 0.f;
    if (MODE == W4S_PLAIN && last && p.residual != nullptr && row && n < N)
      rv = bf16_lo(__ldcg(reinterpret_cast<const unsigned short*>(p.residual) + (long)m * N + n));
    if (!mbar_wait(&full[q & (W4S_NB - 1)], (q / W4S_NB) & 1, &abort_flag, err)) return;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < W4S_WARPS; ++w) {
      const float* r = rb + (w * RP + (DIGITS ? 4 * mm : mm)) * W4S_TILE + c;
      v += DIGITS ? (r[0] + r[W4S_TILE]) + (r[2 * W4S_TILE] + r[3 * W4S_TILE]) : r[0];
    }
    if (passes > 1) {
      float* ps = psum + (local * M + mm) * W4S_TILE + c;
      if (pass > 0 && row) v += *ps;
      if (!last && row) *ps = v;
    }
    if (!last) {
    } else if (MODE == W4S_GATED) {
      // the unfused path stores gate and value as bf16 before the activation
      v = __bfloat162float(__float2bfloat16(v));
      const float val = __shfl_xor_sync(0xffffffffu, v, 1);
      if (row && !(c & 1) && n < I) p.y[(long)m * I + n] = __float2bfloat16(v / (1.f + __expf(-v)) * val);
    } else if (MODE == W4S_ROPE) {
      // pairs of adjacent columns (interleaved rotary convention); the projection's output is bf16 before the rotation
      const RopeAppend& rp = p.rope;
      v = __bfloat162float(__float2bfloat16(v));
      const float u = __shfl_xor_sync(0xffffffffu, v, 1);
      if (row && !(c & 1) && n < N) {
        const int pos = min(*reinterpret_cast<const volatile int*>(rp.pos_ptr), rp.cap - 1);
        const int h = n / rp.D, dcol = n - h * rp.D;
        float a = v, b = u;
        if (h < rp.Hq + rp.Hkv) {
          const long at = (long)pos * (rp.D >> 1) + (dcol >> 1);
          const float cs = rp.cos_t[at], sn = rp.sin_t[at];
          a = v * cs - u * sn;
          b = v * sn + u * cs;
        }
        __nv_bfloat16* dst;
        if (h < rp.Hq) {
          dst = p.y + (long)m * N + n;
        } else {
          const bool is_k = h < rp.Hq + rp.Hkv;
          const int hk = is_k ? h - rp.Hq : h - rp.Hq - rp.Hkv;
          dst = (is_k ? rp.kc : rp.vc) + (long)m * rp.c_sb + (long)pos * rp.c_ss + (long)hk * rp.c_sh + dcol;
        }
        *reinterpret_cast<uint32_t*>(dst) = pack_bf16(a, b);
      }
    } else if (row && n < N) {
      p.y[(long)m * N + n] = __float2bfloat16(v + rv);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[q & (W4S_NB - 1)]);
  };
  int handed = 0;                             // tiles handed over so far

  // ---- the warp's ring. Copy: lane moves chunks (row lane / 4, chunk lane % 4) and (row + 8, same chunk); read: lane
  // (g, t) takes its two columns of k8 rows 4 j + t. Chunk c of row r lies at c ^ (r & 2), which makes both conflict-free.
  const uint32_t ring = smem_u32(w4s_smem + L.ring) + warp * (D * W4S_SLOT);
  const int cr = lane >> 2, cc = lane & 3;
  const int ccol = MODE == W4S_GATED ? (cc < 2 ? 4 * cc : I + 4 * (cc - 2)) : 4 * cc;        // first column of the chunk
  const uint32_t cdst = cr * 64 + ((cc ^ (cr & 2)) << 4);
  const uint32_t rsrc = MODE == W4S_GATED ? tq * 64 + (((gq >> 2) ^ (tq & 2)) << 4) + (gq & 3) * 4
                                          : tq * 64 + (((gq >> 1) ^ (tq & 2)) << 4) + (gq & 1) * 8;
  int lt = 0, li = 0, lmine = 0, lgpw = 1;     // load cursor: tile, unit of this warp; valid units, units per tile
  const uint32_t* lw = p.wk8;
  const __nv_bfloat16* ls = p.scales;
  long lw_next = 0, ls_next = 0;              // from past the last unit of a tile to the first one of the next
  bool live = false;                                 // the lane's columns exist (columns come in fours)
  auto tile_live = [&] { return lt < t_hi && lt * TILE_COLS + (MODE == W4S_GATED ? 4 * (cc & 1) : 4 * cc) < cols; };
  const long n8 = 8L * N, lw_step = (long)(16 * W4S_WARPS) * N, ls_step = (long)W4S_WARPS * N;
  auto load = [&](uint32_t off) {             // the next unit into the ring's slot at byte `off`; columns that do not exist keep
    if (live && li < lmine) {                 // what is there: their results go nowhere
      cp_async16_zfill(ring + off + cdst, lw, 16);
      cp_async16_zfill(ring + off + cdst + 512, lw + n8, 16);
      if (cr == 0) w4s_copy8(ring + off + 1024 + 8 * cc, ls);
    }
    cp_async_commit();
    lw += lw_step;
    ls += ls_step;
    if (++li == lgpw) {
      li = 0;
      lt += t_step;
      live = tile_live();
      lw += lw_next;
      ls += ls_next;
    }
  };

  for (int pass = 0; pass < passes; ++pass) {
    const int g0 = pass * pass_groups, g1 = min(groups, g0 + pass_groups), ng = g1 - g0;
    const int gpw = (ng + W4S_WARPS - 1) / W4S_WARPS;
    const int mine = (ng - warp + W4S_WARPS - 1) / W4S_WARPS;
    lt = t_lo; li = 0; lmine = mine; lgpw = gpw;
    lw = p.wk8 + (long)(16 * (g0 + warp) + cr) * N + (long)lt * TILE_COLS + ccol;
    ls = p.scales + (long)(g0 + warp) * N + (long)lt * TILE_COLS + ccol;
    lw_next = (long)t_step * TILE_COLS - gpw * lw_step;
    ls_next = (long)t_step * TILE_COLS - gpw * ls_step;
    live = tile_live();
    for (int d = 0; d < D; ++d) load(d * W4S_SLOT);
    // ---- the rows of x of this pass, normed on the way, as they are or as digits; half a warp takes one (row, group)
    const int l16 = threadIdx.x & 15;
    uint4 v[4];
    // `f` on the items i, i + 32, .. of this half-warp that v holds. Bf16 rows: one after another. Digits: alone, or two at a
    // time in a loop, so that the shuffles of two overlap; all four unrolled took longer in a decode step, where every launch
    // finds its instructions cold (33.6 ms for 64 tokens of eight 7B blocks against 35.2).
    auto items = [&](int i, int count, auto f) {
      const int first = i - (lane >> 4);
      if constexpr (!DIGITS) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (first + 32 * q >= count) break;
          f(std::integral_constant<int, 1>{}, i + 32 * q, v + q);
        }
      } else if (first + 32 >= count) {
        f(std::integral_constant<int, 1>{}, i, v);
      } else {
        const bool swap = first + 64 < count;
#pragma unroll 1
        for (int r = 0; r < (swap ? 2 : 1); ++r) {
          f(std::integral_constant<int, 2>{}, i + 64 * r, v);
          if (swap) {
            const uint4 t0 = v[0], t1 = v[1];
            v[0] = v[2]; v[1] = v[3];
            v[2] = t0; v[3] = t1;
          }
        }
      }
    };
    bool kept = false;                        // v holds this half-warp's items already
    int any_lost = 0;
    if (pass == 0) {
      if (p.gamma != nullptr)                 // the gains come from HBM in a decode step; ask for them early as well
        for (int i = threadIdx.x; i < K / 32; i += 32 * W4S_WARPS)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.gamma + 32 * i));
      asm volatile("griddepcontrol.wait;" ::: "memory");
      if (p.gamma != nullptr) {
        for (int i1 = 2 * warp; i1 < M * groups; i1 += 4 * 32) {               // (the warp's two halves stay together)
          const int i0 = i1 + (lane >> 4);
          kept = passes == 1 && M * groups <= 128;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + 32 * q, m = M == 1 ? 0 : i / groups, g = i - m * groups;
            v[q] = i < M * groups ? __ldcg(reinterpret_cast<const uint4*>(p.x + (long)m * p.ldx + g * 128) + l16) : make_uint4(0u, 0u, 0u, 0u);
          }
          items(i0, M * groups, [&](auto n, int i, const uint4* at) {
            constexpr int NQ = decltype(n)::value;
            float s[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
              const float a0 = bf16_lo(at[q].x), a1 = bf16_hi(at[q].x), a2 = bf16_lo(at[q].y), a3 = bf16_hi(at[q].y);
              const float a4 = bf16_lo(at[q].z), a5 = bf16_hi(at[q].z), a6 = bf16_lo(at[q].w), a7 = bf16_hi(at[q].w);
              s[q] = a0 * a0 + a1 * a1 + a2 * a2 + a3 * a3 + a4 * a4 + a5 * a5 + a6 * a6 + a7 * a7;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
              for (int q = 0; q < NQ; ++q) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
#pragma unroll
            for (int q = 0; q < NQ; ++q)
              if (l16 == 0 && i + 32 * q < M * groups) gsq[i + 32 * q] = s[q];
          });
        }
        __syncthreads();
        for (int m = warp; m < M; m += W4S_WARPS) {
          float s = 0.f;
          for (int g = lane; g < groups; g += 32) s += gsq[m * groups + g];
          s = warp_sum(s);
          if (lane == 0) rstd[m] = rsqrtf(s / static_cast<float>(K) + p.eps);
        }
        __syncthreads();
      }
    }
    for (int i1 = 2 * warp; i1 < M * ng; i1 += 4 * 32) {
      const int i0 = i1 + (lane >> 4);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = i0 + 32 * q, m = M == 1 ? 0 : i / ng, gl = i - m * ng;
        if (!kept) v[q] = i < M * ng ? __ldcg(reinterpret_cast<const uint4*>(p.x + (long)m * p.ldx + (g0 + gl) * 128) + l16) : make_uint4(0u, 0u, 0u, 0u);
      }
      items(i0, M * ng, [&](auto n, int ifirst, const uint4* from) {
        constexpr int NQ = decltype(n)::value;
        int row[NQ], grp[NQ];
        bool there[NQ];
        uint4 u[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          const int i = ifirst + 32 * q;
          there[q] = i < M * ng;
          row[q] = M == 1 || !there[q] ? 0 : i / ng;
          grp[q] = there[q] ? i - row[q] * ng : 0;
          u[q] = from[q];
          if (p.gamma != nullptr) {
            const float r = rstd[row[q]];
            const float2* gp = reinterpret_cast<const float2*>(p.gamma + (g0 + grp[q]) * 128 + 8 * l16);
            const float2 a = __ldg(gp), b = __ldg(gp + 1), c = __ldg(gp + 2), d = __ldg(gp + 3);
            u[q].x = pack_bf16(bf16_lo(u[q].x) * r * a.x, bf16_hi(u[q].x) * r * a.y);
            u[q].y = pack_bf16(bf16_lo(u[q].y) * r * b.x, bf16_hi(u[q].y) * r * b.y);
            u[q].z = pack_bf16(bf16_lo(u[q].z) * r * c.x, bf16_hi(u[q].z) * r * c.y);
            u[q].w = pack_bf16(bf16_lo(u[q].w) * r * d.x, bf16_hi(u[q].w) * r * d.y);
          }
        }
        if constexpr (!DIGITS) {
#pragma unroll
          for (int q = 0; q < NQ; ++q)
            if (there[q]) *reinterpret_cast<uint4*>(w4s_smem + row[q] * L.pitch + grp[q] * 256 + 16 * l16) = u[q];
        } else {
          // largest magnitude of the group and smallest one that is not zero, as bf16 bits (NaN > Inf > finite as unsigned
          // numbers): max in the upper half, ~(min - 1) in the lower (zeros count as 0 in either)
          uint32_t both[NQ];
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            uint32_t mx = 0u, mn = 0u;
            const uint32_t uw[4] = {u[q].x, u[q].y, u[q].z, u[q].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              mx = __vmaxu2(mx, uw[e] & 0x7FFF7FFFu);
              mn = __vmaxu2(mn, ((uw[e] | 0x80008000u) - 0x00010001u) ^ 0x7FFF7FFFu);
            }
            both[q] = __vmaxu2(__byte_perm(mn, mx, 0x7632), __byte_perm(mn, mx, 0x5410));           // (max | ~min) of either half
          }
#pragma unroll
          for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < NQ; ++q) both[q] = __vmaxu2(both[q], __shfl_xor_sync(0xffffffffu, both[q], o));
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            const uint32_t uw[4] = {u[q].x, u[q].y, u[q].z, u[q].w};
            const int top = max((int)(both[q] >> 23), 27), low = (int)(((~both[q] & 0xFFFFu) + 1u) >> 7);     // exponents (all zero: low 512)
            // whole numbers below 2^29 in steps of 2^(top - 127 - 28): exact down to exponent top - 21
            const bool lost = top > 254 || low < top - 21 || (top < 33 && low < 512);                   // (the last: steps below 2^-126)
            const float inv = __uint_as_float((274u - (uint32_t)min(top, 254)) << 23);                  // |x inv| < 2^21
            uint32_t y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float a = e & 1 ? bf16_hi(uw[e >> 1]) : bf16_lo(uw[e >> 1]);
              const float whole = fmaf(a, inv, W4S_MAGICF), rest = fmaf(fmaf(a, inv, -(whole - W4S_MAGICF)), 256.f, W4S_MAGICF);
              // 256 whole + rest, in four signed digits of base 256
              y[e] = (__float_as_uint(whole) * 256u + __float_as_uint(rest) + (0x80808080u - 257u * (uint32_t)W4S_MAGIC)) ^ 0x80808080u;
            }
            // bytes of elements 0,4,1,5 / 2,6,3,7, digit by digit
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              lo[e] = __byte_perm(y[e], y[e + 4], 0x5140);                     // digits 0 0 1 1
              hi[e] = __byte_perm(y[e], y[e + 4], 0x7362);                     // digits 2 2 3 3
            }
            // a group that the digits cannot hold: its bf16 elements 0..3 in the first row, 4..7 in the second
            const uint2 d0 = lost ? make_uint2(uw[0], uw[1]) : make_uint2(__byte_perm(lo[0], lo[1], 0x5410), __byte_perm(lo[2], lo[3], 0x5410));
            const uint2 d1 = lost ? make_uint2(uw[2], uw[3]) : make_uint2(__byte_perm(lo[0], lo[1], 0x7632), __byte_perm(lo[2], lo[3], 0x7632));
            any_lost |= lost;
            if (there[q]) {
              unsigned char* at = w4s_smem + 4 * row[q] * L.pitch + grp[q] * 128 + 8 * l16;
              *reinterpret_cast<uint2*>(at) = d0;
              *reinterpret_cast<uint2*>(at + L.pitch) = d1;
              *reinterpret_cast<uint2*>(at + 2 * L.pitch) = make_uint2(__byte_perm(hi[0], hi[1], 0x5410), __byte_perm(hi[2], hi[3], 0x5410));
              *reinterpret_cast<uint2*>(at + 3 * L.pitch) = make_uint2(__byte_perm(hi[0], hi[1], 0x7632), __byte_perm(hi[2], hi[3], 0x7632));
              // 2^(top - 127 - 28) / 16 for the lowest digit
              if (l16 < 4) sx[grp[q] * 8 + 4 * row[q] + l16] = lost ? 0.f : __uint_as_float((uint32_t)max(top - 32 + 8 * l16, 0) << 23);
              if (l16 < 2 && (l16 == 0 || M == 1)) w4s_smem[L.flags + 2 * grp[q] + row[q] + l16] = l16 == 0 && lost ? 1 : 0;
            }
          }
        }
      });
    }
    any_lost = __syncthreads_or(any_lost);

    // ---- the stream. `exact`: no group of this pass keeps bf16 values in the place of its digits
    auto stream = [&](auto exact) {
      constexpr bool EXACT = decltype(exact)::value;
      constexpr int XG = W4S_WARPS * (DIGITS ? 128 : 256);                     // bytes of x between two units of a warp
      const int xg0 = warp * (DIGITS ? 128 : 256);
      const unsigned char* xr = w4s_smem + gq * L.pitch + (DIGITS ? 8 : 16) * tq;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};      // first column, x rows (digits: digit columns) 2 t, 2 t + 1; second column
      int ci = 0, xg = xg0;                     // consume cursor: unit of the tile
      uint32_t off = 0;                         // and its slot, which the next load refills
      // One turn per tile, and at the end one per epilogue that is left (a second copy of it would be cold).
      for (int tile = 0;; ++tile) {
        if (tile < ntiles) {
          for (ci = 0; ci < gpw; ++ci) {
            cp_async_wait_group<D - 1>();
            __syncwarp();
            if (ci < mine) {
              const unsigned char* sl = w4s_smem + L.ring + warp * (D * W4S_SLOT) + off;
              auto words = [&](int j, uint32_t& w0, uint32_t& w1) {
                if (MODE == W4S_GATED) {
                  w0 = *reinterpret_cast<const uint32_t*>(sl + rsrc + 256 * j);
                  w1 = *reinterpret_cast<const uint32_t*>(sl + (rsrc ^ 32u) + 256 * j);
                } else {
                  const uint2 w = *reinterpret_cast<const uint2*>(sl + rsrc + 256 * j);
                  w0 = w.x;
                  w1 = w.y;
                }
              };
              float s0, s1;
              if (MODE == W4S_GATED) {
                s0 = bf16_lo(*reinterpret_cast<const unsigned short*>(sl + 1024 + 2 * gq));
                s1 = bf16_lo(*reinterpret_cast<const unsigned short*>(sl + 1040 + 2 * gq));
              } else {
                const uint32_t w = *reinterpret_cast<const uint32_t*>(sl + 1024 + 4 * gq);
                s0 = bf16_lo(w);
                s1 = bf16_hi(w);
              }
              uint32_t lost = 0u;                   // rows of this group that keep bf16 values
              if (!EXACT) lost = *reinterpret_cast<const unsigned short*>(w4s_smem + L.flags + (xg >> 6));
              if (DIGITS && (EXACT || lost != (M == 1 ? 1u : 0x101u))) {
                int dd[4] = {W4S_MAGIC, W4S_MAGIC, W4S_MAGIC, W4S_MAGIC};
    #pragma unroll
                for (int j = 0; j < 4; ++j) {
                  uint32_t w0, w1;
                  words(j, w0, w1);
                  const uint2 xb = gq < 4 * M ? *reinterpret_cast<const uint2*>(xr + xg + 32 * j) : make_uint2(0u, 0u);
                  w4s_mma_s8(dd, w4s_lo(w0), w4s_lo(w1), w4s_hi(w0), w4s_hi(w1), xb.x, xb.y);
                }
                const float2 st = *reinterpret_cast<const float2*>(w4s_smem + L.sx + (xg >> 2) + 8 * tq);
                acc[0] = fmaf(__int_as_float(dd[0]) - W4S_MAGICF, s0 * st.x, acc[0]);
                acc[1] = fmaf(__int_as_float(dd[1]) - W4S_MAGICF, s0 * st.y, acc[1]);
                acc[2] = fmaf(__int_as_float(dd[2]) - W4S_MAGICF, s1 * st.x, acc[2]);
                acc[3] = fmaf(__int_as_float(dd[3]) - W4S_MAGICF, s1 * st.y, acc[3]);
              }
              if (!DIGITS || (!EXACT && lost != 0u)) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                // (digits: row gq / 4 in its first digit's column)
                const bool xrow = DIGITS ? (gq & 3) == 0 && gq < 4 * M && (lost >> (2 * gq) & 1u) != 0 : gq < M;
    #pragma unroll
                for (int j = 0; j < 4; ++j) {
                  uint32_t w0, w1;
                  words(j, w0, w1);
                  uint4 xv = make_uint4(0u, 0u, 0u, 0u);
                  if (xrow) {
                    if (DIGITS) {
                      const uint2 lo = *reinterpret_cast<const uint2*>(xr + xg + 32 * j), hi = *reinterpret_cast<const uint2*>(xr + L.pitch + xg + 32 * j);
                      xv = make_uint4(lo.x, lo.y, hi.x, hi.y);
                    } else {
                      xv = *reinterpret_cast<const uint4*>(xr + xg + 64 * j);
                    }
                  }
                  w4s_mma(d, w4s_pair(w0, 0), w4s_pair(w1, 0), w4s_pair(w0, 1), w4s_pair(w1, 1), xv.x, xv.y);
                  w4s_mma(d, w4s_pair(w0, 2), w4s_pair(w1, 2), w4s_pair(w0, 3), w4s_pair(w1, 3), xv.z, xv.w);
                }
                acc[0] = fmaf(d[0], s0, acc[0]);
                acc[1] = fmaf(d[1], s0, acc[1]);
                acc[2] = fmaf(d[2], s1, acc[2]);
                acc[3] = fmaf(d[3], s1, acc[3]);
              }
            }
            __syncwarp();                         // everyone has read the slot
            load(off);
            off = off == (D - 1) * W4S_SLOT ? 0u : off + W4S_SLOT;
            xg += XG;
          }
          // ---- tile done: hand this warp's sums over
          xg = xg0;
          const int hb = handed & (W4S_NB - 1);
          if (handed >= W4S_NB && !mbar_wait(&empty[hb], ((handed / W4S_NB) - 1) & 1, &abort_flag, err)) return false;
          if (DIGITS || 2 * tq < M) {
            float* r = red + ((hb * W4S_WARPS + warp) * RP + 2 * tq) * W4S_TILE + 2 * gq;
            *reinterpret_cast<float2*>(r) = make_float2(acc[0], acc[2]);
            *reinterpret_cast<float2*>(r + W4S_TILE) = make_float2(acc[1], acc[3]);
          }
          acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
          __syncwarp();
          if (lane == 0) mbar_arrive(&full[hb]);
          if (++handed - ep_q <= 2) continue;
        } else if (pass + 1 < passes || ep_q == handed) {
          return true;
        }
        epilogue();
      }
    };
    bool ok;
    if constexpr (DIGITS) ok = any_lost ? stream(std::false_type{}) : stream(std::true_type{});
    else ok = stream(std::true_type{});
    cp_async_wait_all();
    if (!ok) return;
    if (pass + 1 < passes) __syncthreads();   // every warp is done with x
  }
}

// How a call is cut: digits or bf16 products, ring depth, scale groups per K pass, column tiles per launch. The rows of x of a
// pass stay in shared memory while the CTA walks its tiles. Six groups in flight per warp while that leaves room for all of x,
// four otherwise; K in passes when that is not enough either: partial sums then wait in shared memory (at least
// W4S_PSUM_TILES tiles per CTA, or all of them), what does not fit goes to further launches. One or two rows take the
// digits (two: only where all of x fits; K 14336, N 4096 15.3 us against 16.1 with bf16 products), which cost twice the room.
constexpr int W4S_PSUM_TILES = 8;
struct W4SPlan { bool digits; int depth, pass_groups, tiles_per_cta; };      // tiles_per_cta: tiles of a launch per CTA, 0 = all at once
static bool w4s_plan(int M, int K, int tiles, int sms, bool norm, W4SPlan& out) {
  const int groups = K / 128;
  for (int digits = M <= 2; digits >= (M == 1 ? 1 : 0); --digits)
    for (int depth = 6; depth >= 4; depth -= 2)
      if (w4s_layout(digits, depth, M, groups, groups, norm, 0).total <= W4S_SMEM) {
        out = {digits != 0, depth, groups, 0};
        return true;
      }
  const bool digits = M == 1;
  const int all = (tiles + sms - 1) / sms, kept = all < W4S_PSUM_TILES ? all : W4S_PSUM_TILES;
  auto left = [&](int pass_groups, int psum_tiles) { return W4S_SMEM - w4s_layout(digits, 4, M, pass_groups, groups, norm, psum_tiles).total; };
  int fit = left(0, kept) / (digits ? M * 512 + 34 : M * 256);
  while (fit > 0 && left(fit, kept) < 0) --fit;                   // (the flags are padded to 16 bytes)
  if (fit < 1) return false;
  const int passes = (groups + fit - 1) / fit;
  int pass_groups = ((groups + passes - 1) / passes + W4S_WARPS - 1) / W4S_WARPS * W4S_WARPS;      // whole rounds of the warps
  if (pass_groups > fit) pass_groups = fit < W4S_WARPS ? fit : fit / W4S_WARPS * W4S_WARPS;
  const int room = left(pass_groups, 0) / (M * W4S_TILE * 4);
  out = {digits, 4, pass_groups, room < all ? room : all};
  return true;
}

template <bool DIGITS, int D, int MODE>
static int w4s_launch(const W4StreamArgs& a, const W4SPlan& plan, int tiles, cudaStream_t st) {
  const int groups = a.K / 128;
  unsigned int* err = error_word();
  if (!err) return SB_ERR_CUDA;
  auto kern = w4_stream_kernel<DIGITS, D, MODE>;
  static bool attr_set[64] = {false};
  int dev = 0;
  SB_CHECK_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev & 63]) {
    SB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, W4S_SMEM));
    attr_set[dev & 63] = true;
  }
  const int most = plan.tiles_per_cta > 0 ? plan.tiles_per_cta * num_sms() : tiles;
  for (int t0 = 0; t0 < tiles; t0 += most) {
    const int nt = tiles - t0 < most ? tiles - t0 : most;
    const int grid = nt < num_sms() ? nt : num_sms();
    const int psum_tiles = plan.tiles_per_cta > 0 ? (nt + grid - 1) / grid : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(W4S_THREADS, 1, 1);
    cfg.dynamicSmemBytes = w4s_layout(DIGITS, D, a.M, plan.pass_groups, groups, a.gamma != nullptr, psum_tiles).total;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    // programmatic dependent launch: this grid may start while its predecessor in the stream still runs; before
    // `griddepcontrol.wait` it reads weights at most (static_w), and it writes nothing
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, a, t0, nt, plan.pass_groups, psum_tiles, err));
  }
  return SB_OK;
}

bool w4_stream_preferred(int M, int K) {
  W4SPlan plan;
  return M <= 4 || (M <= W4S_MAX_ROWS && w4s_plan(M, K, 1, 1, false, plan) && plan.pass_groups == K / 128);
}

template <int MODE>
static int w4s_planned(const W4StreamArgs& a, cudaStream_t st) {
  const int tiles = MODE == W4S_GATED ? (a.N / 2 + 7) / 8 : (a.N + W4S_TILE - 1) / W4S_TILE;
  W4SPlan plan;
  SB_CHECK_ARG(w4s_plan(a.M, a.K, tiles, num_sms(), a.gamma != nullptr, plan));
  if (plan.digits)
    return plan.depth == 6 ? w4s_launch<true, 6, MODE>(a, plan, tiles, st) : w4s_launch<true, 4, MODE>(a, plan, tiles, st);
  return plan.depth == 6 ? w4s_launch<false, 6, MODE>(a, plan, tiles, st) : w4s_launch<false, 4, MODE>(a, plan, tiles, st);
}

int launch_w4_stream(const W4StreamArgs& a, W4StreamMode mode, cudaStream_t st) {
  SB_CHECK_ARG(a.M >= 1 && a.M <= (mode == W4S_PLAIN ? W4S_MAX_ROWS : 4) && a.K > 0 && a.K % 128 == 0 && a.N > 0 && a.N % 4 == 0 && a.ldx % 8 == 0);
  SB_CHECK_ARG(((reinterpret_cast<uintptr_t>(a.wk8) | reinterpret_cast<uintptr_t>(a.x)) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.scales) & 7) == 0);
  if (mode == W4S_GATED) {
    SB_CHECK_ARG(a.N % 8 == 0);
    return w4s_planned<W4S_GATED>(a, st);
  }
  return mode == W4S_ROPE ? w4s_planned<W4S_ROPE>(a, st) : w4s_planned<W4S_PLAIN>(a, st);
}

}  // namespace sb

extern "C" int sb_w4_stream_preferred(int M, int K) { return sb::w4_stream_preferred(M, K) ? 1 : 0; }

// Host check of the cut of a call on a GPU of `sms` SMs: dynamic shared memory of its largest launch in bytes, -1 when the call
// would be refused. passes (may be null) receives the number of K passes.
extern "C" int sb_w4_stream_smem(int M, int N, int K, int norm, int sms, int* passes) {
  using namespace sb;
  const int groups = K / 128, tiles = (N + W4S_TILE - 1) / W4S_TILE;
  W4SPlan plan;
  if (!w4s_plan(M, K, tiles, sms, norm != 0, plan)) return -1;
  if (passes) *passes = (groups + plan.pass_groups - 1) / plan.pass_groups;
  const int bytes = w4s_layout(plan.digits, plan.depth, M, plan.pass_groups, groups, norm != 0, plan.tiles_per_cta).total;
  return bytes <= W4S_SMEM && plan.tiles_per_cta >= (plan.pass_groups < groups ? 1 : 0) ? bytes : -1;
}
