// y[M,N] = x[M,K] @ W[K,N] (+ bias, + residual) for few rows, W bf16 row-major: a weight stream through per-warp rings of
// asynchronous copies, feeding warp-level mma (the bf16 sibling of w4_stream.cu).
//
// What bounds it: the weight bytes. The tcgen05 GEMM pads x to 128 rows and has N / 128 tiles to hand out, so at decode
// sizes it leaves most SMs idle (K 4096 N 4096: 32 CTAs). Here one CTA per SM walks tiles of 16 or 32 columns over the
// whole K range; its 16 warps take blocks of 64 or 32 k round robin, each through its own ring (three blocks of 2 KB in
// flight per warp, 96 KB per SM). A block is stored `[k][columns]` as it comes; ldmatrix.trans turns it into A fragments
// (rows = columns of W) and ldmatrix takes x as B fragments (columns = rows of x), so a 2 KB block costs about 45
// instructions. Per tile every warp leaves its partial sums in one of the shared-memory buffers and streams on; the warp
// whose turn it is adds them and runs the epilogue two tiles later. Measured against the tcgen05 GEMM, 6 rows, weights from
// HBM: K 4096 N 4096 23.7 -> 8.8 us, N 6144 24.4 -> 13.7, N 28672 50.0 -> 43.7, K 14336 N 4096 72.4 -> 28.4, K 3072 N 1536
// 18.5 -> 5.3; N 32000 53.4 -> 54.3 (1 row 52.9 -> 51.1).
#include "bf16_stream.h"
#include "host_util.h"
#include "sm100.cuh"

namespace sb {

constexpr int BFS_WARPS = 16, BFS_THREADS = 512, BFS_D = 3, BFS_SLOT = 2048;
// TC columns per tile (16 or 32), blocks of BFS_UK k, BFS_NB hand-over buffers
template <int TC> constexpr int BFS_UK = 1024 / TC;
template <int TC> constexpr int BFS_NB = TC == 16 ? 4 : 3;
constexpr int BFS_SMEM = 220 * 1024;

__device__ __forceinline__ void bfs_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void bfs_ldsm(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void bfs_ldsm_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

struct BfsLayout {                           // shared memory, in bytes
  int pitch, x, red, psum, total;            // pitch: row of x (16 mod 128: conflict-free ldmatrix)
};
template <int TC>
__host__ __device__ inline BfsLayout bfs_layout(int rows, int M, int pass_blocks, int psum_tiles) {
  BfsLayout l;
  l.pitch = pass_blocks * BFS_UK<TC> * 2 + 16;
  l.x = BFS_WARPS * BFS_D * BFS_SLOT;
  l.red = (l.x + M * l.pitch + 15) & ~15;                           // [buffers][warps][rows][TC] fp32
  l.psum = l.red + BFS_NB<TC> * BFS_WARPS * rows * TC * 4;          // [psum_tiles][M][TC] fp32 (more than one K pass)
  l.total = l.psum + psum_tiles * M * TC * 4;
  return l;
}

template <int TC>
__global__ void __launch_bounds__(BFS_THREADS, 1)
bf16_stream_kernel(const Bf16StreamArgs p, const int static_w, const int tile_base, const int tiles, const int pass_blocks,
                   const int psum_tiles, unsigned int* err) {
  constexpr int ROWS = 8, D = BFS_D, UK = BFS_UK<TC>, NB = BFS_NB<TC>, CH = TC / 16, CPR = TC / 8;
  extern __shared__ __align__(128) unsigned char bfs_smem[];
  __shared__ uint64_t full[NB], empty[NB];
  __shared__ int abort_flag;
  asm volatile("griddepcontrol.launch_dependents;");
  const int M = p.M, N = p.N, K = p.K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const BfsLayout L = bfs_layout<TC>(ROWS, M, pass_blocks, psum_tiles);
  float* red = reinterpret_cast<float*>(bfs_smem + L.red);
  float* psum = reinterpret_cast<float*>(bfs_smem + L.psum);
  // Tiles are dealt out in turn, so that the CTAs read neighbouring pieces of the same weight rows at the same time (DRAM
  // pages): K 4096 N 28672 41 us, 55 with contiguous runs.
  const int t_lo = tile_base + blockIdx.x, t_hi = tile_base + tiles, t_step = gridDim.x;
  const int ntiles = (tiles - (int)blockIdx.x + t_step - 1) / t_step;
  const int blocks = (K + UK - 1) / UK;
  const int passes = (blocks + pass_blocks - 1) / pass_blocks;
  const int chunks = (TC * M + 31) / 32;
  if (threadIdx.x == 0) {
    for (int b = 0; b < NB; ++b) { mbar_init(&full[b], BFS_WARPS); mbar_init(&empty[b], chunks); }
    abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();

  // Epilogue of this CTA's q-th tile (counted over the passes): 32 outputs o = m * TC + c at a time; chunk k of the i-th tile
  // belongs to warp (i + k) % 16.
  auto epilogue = [&](int q) {
    const int pass = q / ntiles, local = q - pass * ntiles, ct = t_lo + local * t_step;
    const int chunk = (warp - local) & (BFS_WARPS - 1);
    if (chunk >= chunks) return;
    const bool last = pass + 1 == passes;
    const float* rb = red + (q % NB) * BFS_WARPS * ROWS * TC;
    const int o = chunk * 32 + lane, m = o / TC, c = o % TC, n = ct * TC + c;
    const bool row = m < M, out = row && n < N && last;
    const int mm = row ? m : 0;
    float rv = 0.f, bv = 0.f;
    if (out && p.residual != nullptr) rv = bf16_lo(__ldcg(reinterpret_cast<const unsigned short*>(p.residual) + (long)m * N + n));
    if (out && p.bias != nullptr)
      bv = p.bias_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[n]) : static_cast<const float*>(p.bias)[n];
    if (!mbar_wait(&full[q % NB], (q / NB) & 1, &abort_flag, err)) return;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < BFS_WARPS; ++w) v += rb[(w * ROWS + mm) * TC + c];
    if (passes > 1) {
      float* ps = psum + (local * M + mm) * TC + c;
      if (pass > 0 && row) v += *ps;
      if (!last && row) *ps = v;
    }
    if (out) {
      v += bv;
      // the projection's own output is bf16; the sum is rounded once more, as the separate addition does
      if (p.residual != nullptr) v = __bfloat162float(__float2bfloat16(v)) + rv;
      p.y[(long)m * p.ldy + n] = __float2bfloat16(v);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[q % NB]);
  };
  int handed = 0;                             // tiles handed over so far

  // ---- the warp's ring: UK rows of TC columns, 16-byte chunk c of row k at c ^ swz(k); a lane copies rows cr + UK / 4 i
  auto swz = [](int k) { return TC == 16 ? (k >> 2) & 1 : (k >> 1) & 3; };
  const uint32_t ring = smem_u32(bfs_smem) + warp * (D * BFS_SLOT);
  const int cr = lane / CPR, cc = lane % CPR;
  const uint32_t cdst = cr * (TC * 2) + ((cc ^ swz(cr)) << 4);
  int lt, li, lmine, lbpw, lb0;               // load cursor: tile, block of this warp; valid blocks, blocks per tile
  uint32_t lslot = 0;
  auto load = [&] {
    if (lt < t_hi && li < lmine) {
      const int k0 = (lb0 + warp + BFS_WARPS * li) * UK + cr, n0 = lt * TC + 8 * cc;
      const __nv_bfloat16* src = p.w + (long)k0 * p.ldw + n0;
      const int bytes = min(16, max(0, 2 * (N - n0)));
      const uint32_t dst = ring + lslot * BFS_SLOT + cdst;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int nb = k0 + UK / 4 * i < K ? bytes : 0;
        cp_async16_zfill(dst + 512 * i, nb > 0 ? src + (long)(UK / 4 * i) * p.ldw : p.w, nb);
      }
    }
    cp_async_commit();
    lslot = lslot + 1 == D ? 0 : lslot + 1;
    if (++li == lbpw) {
      li = 0;
      lt += t_step;
    }
  };

  if (!static_w) asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int pass = 0; pass < passes; ++pass) {
    const int b0 = pass * pass_blocks, nb = min(blocks, b0 + pass_blocks) - b0;
    const int bpw = (nb + BFS_WARPS - 1) / BFS_WARPS;
    const int mine = (nb - warp + BFS_WARPS - 1) / BFS_WARPS;
    const int total = ntiles * bpw;
    lt = t_lo; li = 0; lmine = mine; lbpw = bpw; lb0 = b0; lslot = 0;
    for (int d = 0; d < D; ++d) load();
    if (pass == 0 && static_w) {
      if (p.gamma != nullptr)                 // the gains come from HBM in a decode step; ask for them early as well
        for (int i = threadIdx.x; i < K / 32; i += BFS_THREADS) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.gamma + 32 * i));
      asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    // ---- the rows of x of this pass (zero beyond K), normed in place
    const uint32_t xs = smem_u32(bfs_smem + L.x);
    const int cpr = nb * (UK / 8);        // 16-byte chunks per row
    for (int i = threadIdx.x; i < M * cpr; i += BFS_THREADS) {
      const int m = i / cpr, c = i - m * cpr, k = b0 * UK + 8 * c;
      cp_async16_zfill(xs + m * L.pitch + 16 * c, k < K ? p.x + (long)m * p.ldx + k : p.x, k < K ? 16 : 0);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if (p.gamma != nullptr) {                 // (one pass)
      const int wpr = M <= 1 ? 16 : (M <= 2 ? 8 : (M <= 4 ? 4 : (M <= 8 ? 2 : 1)));       // warps per row
      const int m = warp / wpr, sub = warp % wpr;
      float* ssq = red;                       // [16], before any tile is handed over
      if (m < M) {
        const uint4* row = reinterpret_cast<const uint4*>(bfs_smem + L.x + m * L.pitch);
        float s = 0.f;
        for (int c = sub * 32 + lane; c < cpr; c += wpr * 32) {
          const uint4 v = row[c];
          const float a0 = bf16_lo(v.x), a1 = bf16_hi(v.x), a2 = bf16_lo(v.y), a3 = bf16_hi(v.y);
          const float a4 = bf16_lo(v.z), a5 = bf16_hi(v.z), a6 = bf16_lo(v.w), a7 = bf16_hi(v.w);
          s += a0 * a0 + a1 * a1 + a2 * a2 + a3 * a3 + a4 * a4 + a5 * a5 + a6 * a6 + a7 * a7;
        }
        s = warp_sum(s);
        if (lane == 0) ssq[warp] = s;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < M * (K / 8); i += BFS_THREADS) {
        const int mm = i / (K / 8), c = i - mm * (K / 8);
        float sq = 0.f;
        for (int w = 0; w < wpr; ++w) sq += ssq[mm * wpr + w];
        const float r = rsqrtf(sq / static_cast<float>(K) + p.eps);
        const float4 g0 = __ldg(reinterpret_cast<const float4*>(p.gamma) + 2 * c), g1 = __ldg(reinterpret_cast<const float4*>(p.gamma) + 2 * c + 1);
        uint4* at = reinterpret_cast<uint4*>(bfs_smem + L.x + mm * L.pitch) + c;
        uint4 v = *at;
        v.x = pack_bf16(bf16_lo(v.x) * r * g0.x, bf16_hi(v.x) * r * g0.y);
        v.y = pack_bf16(bf16_lo(v.y) * r * g0.z, bf16_hi(v.y) * r * g0.w);
        v.z = pack_bf16(bf16_lo(v.z) * r * g1.x, bf16_hi(v.z) * r * g1.y);
        v.w = pack_bf16(bf16_lo(v.w) * r * g1.z, bf16_hi(v.w) * r * g1.w);
        *at = v;
      }
      __syncthreads();
    }

    // ---- the stream
    float acc[CH][4];
#pragma unroll
    for (int h = 0; h < CH; ++h)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[h][c] = 0.f;
    // ldmatrix rows: A matrix i = lane / 8 holds k 8 (i / 2) .. + 8, columns 8 (i % 2) .. + 8; B matrix i holds k 8 i .. + 8
    const int mi = lane >> 3, mr = lane & 7, ak = 8 * (mi >> 1) + mr;
    const uint32_t a_off = ak * (TC * 2) + (((mi & 1) ^ swz(ak)) << 4);       // (swz(ak + 16) = swz(ak); columns + 16: chunk ^ 2)
    const uint32_t x_off = xs + min(mr, M - 1) * L.pitch + 16 * mi;              // (rows beyond M: results unused)
    int ci = 0;                               // consume cursor: block of the tile
    uint32_t slot = 0;
    for (int it = 0; it < total; ++it) {
      cp_async_wait_group<D - 1>();
      __syncwarp();
      if (ci < mine) {
        const uint32_t sl = ring + slot * BFS_SLOT + a_off;
        const uint32_t kb = (warp + BFS_WARPS * ci) * (UK * 2);
#pragma unroll
        for (int s = 0; s < UK / 32; ++s) {
          uint32_t b[4];
          bfs_ldsm(b, x_off + kb + 64 * s);
#pragma unroll
          for (int h = 0; h < CH; ++h) {
            uint32_t a0[4], a1[4];
            bfs_ldsm_t(a0, (sl ^ (32 * h)) + s * (64 * TC));
            bfs_ldsm_t(a1, (sl ^ (32 * h)) + s * (64 * TC) + 32 * TC);
            bfs_mma(acc[h], a0, b[0], b[1]);
            bfs_mma(acc[h], a1, b[2], b[3]);
          }
        }
      }
      __syncwarp();                           // everyone has read the slot
      load();
      slot = slot + 1 == D ? 0 : slot + 1;
      if (++ci < bpw) continue;
      // ---- tile done: hand this warp's sums over
      ci = 0;
      const int hb = handed % NB;
      if (handed >= NB && !mbar_wait(&empty[hb], ((handed / NB) - 1) & 1, &abort_flag, err)) {
        cp_async_wait_all();                  // (no copy may land in shared memory that is someone else's by then)
        return;
      }
#pragma unroll
      for (int h = 0; h < CH; ++h) {
        float* r = red + ((hb * BFS_WARPS + warp) * ROWS + 2 * tq) * TC + 16 * h + gq;
        r[0] = acc[h][0];                     // column g, rows 2 t, 2 t + 1
        r[TC] = acc[h][1];
        r[8] = acc[h][2];                     // column g + 8
        r[TC + 8] = acc[h][3];
        acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.f;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[hb]);
      if (++handed > 2) epilogue(handed - 3);
    }
    cp_async_wait_all();
    if (pass + 1 < passes) __syncthreads();   // every warp is done with x
  }
  for (int q = max(handed - 2, 0); q < handed; ++q) epilogue(q);
}

// blocks of k whose x rows fit next to rings and buffers
template <int TC>
static int bfs_fit(int M) {
  return (BFS_SMEM - bfs_layout<TC>(8, 0, 0, 0).total - 4096 - 16 * M) / (M * BFS_UK<TC> * 2);     // 4 KB: partial sums
}

template <int TC>
static int bfs_launch(const Bf16StreamArgs& a, bool static_w, cudaStream_t st) {
  constexpr int ROWS = 8;
  const int blocks = (a.K + BFS_UK<TC> - 1) / BFS_UK<TC>;
  const int tiles = (a.N + TC - 1) / TC;
  const int fit = bfs_fit<TC>(a.M);
  const int passes = (blocks + fit - 1) / fit;
  int pass_blocks = (blocks + passes - 1) / passes;
  if (passes > 1) {             // whole rounds of the warps
    pass_blocks = (pass_blocks + BFS_WARPS - 1) / BFS_WARPS * BFS_WARPS;
    if (pass_blocks > fit) pass_blocks = fit < BFS_WARPS ? fit : fit / BFS_WARPS * BFS_WARPS;
  }
  const int base_smem = bfs_layout<TC>(ROWS, a.M, pass_blocks, 0).total;
  int most = tiles;
  if (pass_blocks < blocks)     // partial sums wait in shared memory: as many tiles per CTA as fit, the rest in further launches
    most = (BFS_SMEM - base_smem) / (a.M * TC * 4) * num_sms();
  SB_CHECK_ARG(base_smem <= BFS_SMEM && most > 0 && (a.gamma == nullptr || pass_blocks == blocks));
  unsigned int* err = error_word();
  if (!err) return SB_ERR_CUDA;
  auto kern = bf16_stream_kernel<TC>;
  static bool attr_set[64] = {false};
  int dev = 0;
  SB_CHECK_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev & 63]) {
    SB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BFS_SMEM));
    attr_set[dev & 63] = true;
  }
  for (int t0 = 0; t0 < tiles; t0 += most) {
    const int nt = tiles - t0 < most ? tiles - t0 : most;
    const int grid = nt < num_sms() ? nt : num_sms();
    const int psum_tiles = pass_blocks < blocks ? (nt + grid - 1) / grid : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(BFS_THREADS, 1, 1);
    cfg.dynamicSmemBytes = bfs_layout<TC>(ROWS, a.M, pass_blocks, psum_tiles).total;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    // programmatic dependent launch: before `griddepcontrol.wait` the grid reads weights at most, and writes nothing
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, a, static_w ? 1 : 0, t0, nt, pass_blocks, psum_tiles, err));
  }
  return SB_OK;
}

bool bf16_stream_one_pass(int M, int K) { return (K + BFS_UK<32> - 1) / BFS_UK<32> <= bfs_fit<32>(M) && (K + BFS_UK<16> - 1) / BFS_UK<16> <= bfs_fit<16>(M); }

bool bf16_stream_takes(const Bf16StreamArgs& a) {
  return a.M >= 1 && a.M <= BFS_MAX_ROWS && a.N > 0 && a.K > 0 && a.K % 8 == 0 && a.ldx % 8 == 0 && a.ldw % 8 == 0 &&
         ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w)) & 15) == 0;
}

int launch_bf16_stream(const Bf16StreamArgs& a, bool static_w, cudaStream_t st) {
  SB_CHECK_ARG(bf16_stream_takes(a));
  // 32 columns a tile read 64 contiguous bytes of a row (16: 32 bytes, K 14336 N 4096 40.4 us against 21.0); 16 columns as
  // long as those give every tile an SM of its own (K 3072 N 352: 2.9 us against 4.2, N 1536 level)
  return (a.N + 15) / 16 <= num_sms() ? bfs_launch<16>(a, static_w, st) : bfs_launch<32>(a, static_w, st);
}

}  // namespace sb

// y[M, N] = (rmsnorm(x) or x)[M, K] @ W[K, N] (+ bias) (+ residual [M, N]) for M <= 8 rows of a decode step; W bf16
// row-major with row stride ldw. static_w != 0: W is not being written by anything in flight on the stream.
extern "C" int sb_decode_linear(const void* x, const void* w, const void* bias, int bias_is_bf16, const void* residual, void* y,
                                int M, int N, int K, long ldx, long ldw, const float* gamma, float eps, int static_w,
                                cudaStream_t st) {
  using namespace sb;
  const Bf16StreamArgs a = {(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, bias, bias_is_bf16, (const __nv_bfloat16*)residual,
                            (__nv_bfloat16*)y, M, N, K, ldx, ldw, (long)N, gamma, eps};
  return launch_bf16_stream(a, static_w != 0, st);
}

// 1 when sb_decode_linear takes M rows of K with a fused norm
extern "C" int sb_decode_linear_one_pass(int M, int K) { return M >= 1 && M <= sb::BFS_MAX_ROWS && sb::bf16_stream_one_pass(M, K) ? 1 : 0; }
