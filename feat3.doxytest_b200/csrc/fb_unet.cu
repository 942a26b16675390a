// Learned warm start: a small convolutional U-Net on vertex grids (G = 2^k + 1 points per side)
// that maps (f, log kappa) to an approximation of u, trained on solutions of the FP64 multigrid.
// No counterpart in the reference (its solve path has no learned component).
//
// Network (channels 16/32/64/64, 3x3 "same" convolutions, zero padding):
//   L1 conv 2->16 @G1, ReLU = e1;  S = injection (every other vertex)
//   L2 conv 16->32 @G2 on S(e1), ReLU = e2
//   L3 conv 32->64 @G3 on S(e2), ReLU = e3
//   L4 conv 64->64 @G4 on S(e3), then two more 64->64 convolutions @G4 with dilation 2 and 4
//      (ReLU after each) = e4: the bottleneck sees 15 x 15 of its 17 x 17 points (for G1 = 129), so
//      the prediction can couple the whole domain as the solution operator does
//   L5 conv 128->64 @G3 on [U(e4), e3], ReLU = d3;  U = bilinear vertex upsampling (the Q1
//      prolongation stencil: coincident vertex 1, edge midpoints 1/2 + 1/2, cell centres 4 x 1/4)
//   L6 conv 96->32 @G2 on [U(d3), e2], ReLU = d2
//   L7 conv 48->16 @G1 on [U(d2), e1], ReLU = d1
//   L8 conv 16->1 @G1 on d1 (no activation) = output
// Activations are stored as BF16 in NHWC layout (channels padded to multiples of 8); the
// convolutions are implicit GEMMs on the tensor cores (mma.sync m16n8k16, BF16 operands, FP32
// accumulation); bias, ReLU and the upsampling averages are computed in FP32 and rounded to BF16
// once.  Parameters are FP32 masters (Adam), converted to BF16 GEMM layouts after every update.
//
// Parameter layout (the flat FP32 vector of fb_unet_get_params): per layer, W[co][tap][ci] with
// tap = (dy+1)*3 + (dx+1) (dy along the grid's slow axis), then bias[co].
#include "fb_common.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

namespace fb
{
namespace un
{
  typedef uint16_t bf;

  __device__ __forceinline__ float bf2f(bf v) { return __uint_as_float(uint32_t(v) << 16); }
  __device__ __forceinline__ bf f2bf(float f) { return __bfloat16_as_ushort(__float2bfloat16_rn(f)); }
  // all ones in each half of a BF16 pair that is greater than zero
  __device__ __forceinline__ uint32_t mask2(uint32_t q)
  {
    return (bf2f(bf(q)) > 0.f ? 0xFFFFu : 0u) | (bf2f(bf(q >> 16)) > 0.f ? 0xFFFF0000u : 0u);
  }

  constexpr int NLAYER = 10;
  struct LayerDef { int cin, cout, level; };
  // real channel counts; level = resolution index (0 = finest grid)
  constexpr LayerDef LAYERS[NLAYER] = {{2, 16, 0}, {16, 32, 1}, {32, 64, 2}, {64, 64, 3}, {64, 64, 3}, {64, 64, 3},
                                       {128, 64, 2}, {96, 32, 1}, {48, 16, 0}, {16, 1, 0}};

  __host__ __device__ inline int pad8(int c) { return (c + 7) & ~7; }

  // ------------------------------------------------------------------ tensor-core helpers
  __device__ __forceinline__ uint32_t smem_addr(const void* p)
  {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
  }
  // 16-byte async copy global -> shared; src_bytes 0 fills zeros (halo / padding)
  __device__ __forceinline__ void cp16(void* dst, const void* src, int src_bytes)
  {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(smem_addr(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
  }
  __device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
  template<int N>
  __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

  // ldmatrix from a shared-memory address: each lane points at one 16-byte row
  __device__ __forceinline__ void ldm_x4a(uint32_t (&r)[4], uint32_t p)
  {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(p));
  }
  __device__ __forceinline__ void ldm_x4a_t(uint32_t (&r)[4], uint32_t p)
  {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(p));
  }
  __device__ __forceinline__ void ldm_x2a_t(uint32_t (&r)[2], uint32_t p)
  {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1]) : "r"(p));
  }
  __device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
  {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }

  // ------------------------------------------------------------------ tiles
  // Every convolution kernel works on T x T pixel tiles of one image (T <= 11, so that a tile's
  // 121 pixels fill the 128 rows of an MMA tile and 33, 65 and 129 points per side divide into
  // whole tiles with 1-5% overhang) and stages the tile's input with its halo of `dil` pixels in
  // shared memory once.  The nine taps then read that one copy at shifted addresses: each ldmatrix
  // lane points at its own pixel's 16-byte chunk, so no im2col copy of the input is ever made (a
  // gather per tap reads the input nine times and spends its issue slots on address arithmetic).
  // Pixel stride: PXC 16-byte chunks, odd, so that the eight rows of an ldmatrix fall into
  // different banks.
  constexpr int TMAX = 11;
  __host__ __device__ constexpr int px_chunks(int c) { return (c / 8) | 1; }
  __host__ __device__ constexpr int halo_dim(int dil) { return TMAX + 2 * dil; }
  __host__ __device__ constexpr int halo_bytes(int c, int dil)
  {
    return halo_dim(dil) * halo_dim(dil) * px_chunks(c) * 16;
  }

  struct Tiling
  {
    int G, T, nt;        // points per side, tile side, tiles per side
  };

  // where a convolution's input comes from
  enum InMode
  {
    IN_PLAIN,            // BF16 [B][G][G][C]
    IN_SUB,              // injection: every other vertex of BF16 [B][2G-1][2G-1][C]
    IN_CAT,              // [U(coarse), skip]: the first cu channels are the bilinear vertex
                         // upsampling of BF16 [B][(G+1)/2][(G+1)/2][cu] (FP32 average rounded
                         // once), the others BF16 [B][G][G][C - cu]
    IN_PAIR,             // BF16 pairs [B][G][G][2]: channels 0, 1 of 8 (the others zero)
    IN_SCALAR            // FP32 [B][G][G]: channel 0 of 8, rounded to BF16
  };

  struct Input
  {
    const void* x;       // IN_CAT: the coarse tensor
    const bf* skip;      // IN_CAT
    int cu;              // IN_CAT: upsampled channels
    int ct;              // channels of the tensor (IN_PLAIN, IN_SUB) or of the concatenation
    int c0;              // first channel of this kernel's range
  };

  __device__ __forceinline__ uint32_t pack2(float lo, float hi)
  {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }

  // The halo tile of the channels [c0, c0 + C) of [U(coarse), skip].  One work item of the upsampled
  // channels is a coarse cell: its four corners' 16-byte chunks give the cell's four fine pixels (the
  // vertex, two edge midpoints, the centre; FP32 averages rounded once), so a corner is loaded and
  // converted once for them.  The averages bound this loader, not the copies: one item per fine pixel
  // (four loads and four-point averages each) spent three quarters of the kernel's issue slots here
  // (batch 32 at 129 points: the 48 -> 16 convolution 107 -> 81 us, its weight gradient 87 -> 65).
  template<int C, int DIL, int NT>
  __device__ __forceinline__ void load_cat(const Input& in, const Tiling& t, int b, int y0, int x0, bf* sh)
  {
    constexpr int HD = halo_dim(DIL), CH = C / 8, PXC = px_chunks(C);
    const int hd = t.T + 2 * DIL, G = t.G, Gc = (G + 1) / 2;
    const unsigned nu = unsigned(max(0, min(CH, (in.cu - in.c0) / 8))), ns = CH - nu;
    for(unsigned e = threadIdx.x; e < HD * HD * ns; e += NT)
    {
      const unsigned p = e / ns, ch = nu + e - p * ns;
      const int hy = int(p) / HD, hx = int(p) - hy * HD;
      if(hy >= hd || hx >= hd)
        continue;
      const int y = y0 + hy - DIL, x = x0 + hx - DIL;
      const bool ok = y >= 0 && y < G && x >= 0 && x < G;
      cp16(sh + (p * PXC + ch) * 8,
        ok ? in.skip + ((size_t(b) * G + y) * G + x) * (in.ct - in.cu) + (in.c0 + int(ch) * 8 - in.cu) : in.skip,
        ok ? 16 : 0);
    }
    const int cy0 = (y0 - DIL) >> 1, cx0 = (x0 - DIL) >> 1;
    const unsigned ncx = unsigned(((x0 + t.T + DIL - 1) >> 1) - cx0 + 1), ncy = unsigned(((y0 + t.T + DIL - 1) >> 1) - cy0 + 1);
    const bf* cb = static_cast<const bf*>(in.x) + size_t(b) * Gc * Gc * in.cu + in.c0;
    #pragma unroll 1
    for(unsigned e = threadIdx.x; e < ncy * ncx * nu; e += NT)
    {
      const unsigned q = e / nu, ch = e - q * nu, iy = q / ncx;
      const int cy = cy0 + int(iy), cx = cx0 + int(q - iy * ncx);
      // corners outside the coarse grid belong to pixels outside the fine one
      const int ya = min(max(cy, 0), Gc - 1), yb = min(max(cy + 1, 0), Gc - 1);
      const int xa = min(max(cx, 0), Gc - 1), xb = min(max(cx + 1, 0), Gc - 1);
      uint32_t v[4][4];
      const bf* cc = cb + ch * 8;
      *reinterpret_cast<uint4*>(v[0]) = __ldg(reinterpret_cast<const uint4*>(cc + (size_t(ya) * Gc + xa) * in.cu));
      *reinterpret_cast<uint4*>(v[1]) = __ldg(reinterpret_cast<const uint4*>(cc + (size_t(ya) * Gc + xb) * in.cu));
      *reinterpret_cast<uint4*>(v[2]) = __ldg(reinterpret_cast<const uint4*>(cc + (size_t(yb) * Gc + xa) * in.cu));
      *reinterpret_cast<uint4*>(v[3]) = __ldg(reinterpret_cast<const uint4*>(cc + (size_t(yb) * Gc + xb) * in.cu));
      uint32_t o[4][4];
      #pragma unroll
      for(int k = 0; k < 4; ++k)
      {
        float f[4][2];
        #pragma unroll
        for(int u = 0; u < 4; ++u)
        {
          f[u][0] = __uint_as_float(v[u][k] << 16);
          f[u][1] = __uint_as_float(v[u][k] & 0xffff0000u);
        }
        o[0][k] = v[0][k];
        o[1][k] = pack2((f[0][0] + f[1][0]) * 0.5f, (f[0][1] + f[1][1]) * 0.5f);
        o[2][k] = pack2((f[0][0] + f[2][0]) * 0.5f, (f[0][1] + f[2][1]) * 0.5f);
        o[3][k] = pack2(((f[0][0] + f[1][0]) + (f[2][0] + f[3][0])) * 0.25f,
          ((f[0][1] + f[1][1]) + (f[2][1] + f[3][1])) * 0.25f);
      }
      #pragma unroll
      for(int u = 0; u < 4; ++u)
      {
        const int y = 2 * cy + (u >> 1), x = 2 * cx + (u & 1), hy = y - y0 + DIL, hx = x - x0 + DIL;
        if(hy < 0 || hy >= hd || hx < 0 || hx >= hd)
          continue;
        const bool ok = y >= 0 && y < G && x >= 0 && x < G;
        *reinterpret_cast<uint4*>(sh + ((hy * HD + hx) * PXC + ch) * 8) =
          ok ? make_uint4(o[u][0], o[u][1], o[u][2], o[u][3]) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }

  // The halo tile of channels [c0, c0 + C) around the tile at (y0, x0) of image b into shared
  // memory, zeros outside the grid.  Asynchronous copies where the data is already BF16.
  template<int C, int DIL, int IN, int NT>
  __device__ __forceinline__ void load_halo(const Input& in, const Tiling& t, int b, int y0, int x0, bf* sh)
  {
    if constexpr(IN == IN_CAT)
    {
      load_cat<C, DIL, NT>(in, t, b, y0, x0, sh);
      return;
    }
    constexpr int HD = halo_dim(DIL), CH = C / 8, PXC = px_chunks(C);
    const int hd = t.T + 2 * DIL;
    const int G = t.G;
    for(int e = threadIdx.x; e < HD * HD * CH; e += NT)
    {
      const int ch = e % CH, p = e / CH;
      const int hy = p / HD, hx = p - hy * HD;
      if(hy >= hd || hx >= hd)
        continue;
      const int y = y0 + hy - DIL, x = x0 + hx - DIL;
      const bool ok = y >= 0 && y < G && x >= 0 && x < G;
      bf* dst = sh + (p * PXC + ch) * 8;
      if constexpr(IN == IN_PLAIN)
      {
        const bf* src = static_cast<const bf*>(in.x);
        cp16(dst, ok ? src + ((size_t(b) * G + y) * G + x) * in.ct + in.c0 + ch * 8 : src, ok ? 16 : 0);
      }
      else if constexpr(IN == IN_SUB)
      {
        const bf* src = static_cast<const bf*>(in.x);
        const int Gf = 2 * G - 1;
        cp16(dst, ok ? src + ((size_t(b) * Gf + 2 * y) * Gf + 2 * x) * in.ct + in.c0 + ch * 8 : src, ok ? 16 : 0);
      }
      else
      {
        uint32_t w = 0u;
        if(ok)
        {
          const size_t q = (size_t(b) * G + y) * G + x;
          w = IN == IN_PAIR ? __ldg(static_cast<const uint32_t*>(in.x) + q)
                            : uint32_t(f2bf(__ldg(static_cast<const float*>(in.x) + q)));
        }
        *reinterpret_cast<uint4*>(dst) = make_uint4(w, 0u, 0u, 0u);
      }
    }
  }

  // ------------------------------------------------------------------ convolution
  // y[p, n] = bias[n] + sum_{tap, c} x[p + off(tap), c] * w[tap*C + c][n] for the BN columns from
  // n0 = blockIdx.y * BN (zero outside the grid); w: BF16 rows of n_ld.  One block of four warps per
  // tile, persistent over tiles; warp w takes MMA rows 32 w .. 32 w + 31 and all BN columns.  The
  // same kernel is the data gradient (x = the output gradient, w = flipped transposed weights).
  // Weights stay in shared memory for all of a block's tiles where the nine taps fit (NST = 9),
  // otherwise they are streamed tap by tap through two buffers (NST = 2).  Bound by shared-memory
  // reads: per 16-deep step a warp issues 2 + BN/16 ldmatrix.x4 for BN/4 MMAs.
  enum OutMode
  {
    OUT_RELU,            // BF16 [P][n], max(v + bias, 0)
    OUT_FIRST,           // FP32 [P]: v + bias of column 0 only
    OUT_F32,             // FP32, columns < nsplit to y [P][nsplit], the others to y2 [P][n - nsplit]
    OUT_MASK             // BF16 [P][n]: v where post > 0, else 0
  };

  struct ConvArgs
  {
    Input in;
    Tiling t;
    const bf* w;
    const float* bias;   // n entries (OUT_RELU), 1 (OUT_FIRST)
    void* y;
    float* y2;
    const bf* post;
    int n, n_ld, nsplit;
    int ntiles;
  };

  constexpr int CNT = 128;

  template<int C, int BN, int NST>
  __host__ __device__ constexpr int conv_wbytes()
  {
    return (C == 8 ? 80 : NST * C) * (BN + 8) * 2;
  }
  template<int C, int BN, int DIL, int NST>
  __host__ __device__ constexpr int conv_smem()
  {
    return conv_wbytes<C, BN, NST>() + halo_bytes(C, DIL);
  }

  // Resident blocks per SM: by shared memory, and with registers for the accumulators (BN columns) and
  // the fragments in flight.  The kernels are compiled for it: left alone the unrolled taps take 120 to
  // 170 registers, so that three or four blocks were resident of a grid of eight per SM (the 48 -> 16 layer, batch 32 at 129 points: 81 -> 68 us).
  template<int C, int BN, int DIL, int IN, int NST>
  __host__ __device__ constexpr int conv_blocks()
  {
    constexpr int by_smem = 227 * 1024 / (conv_smem<C, BN, DIL, NST>() + 1024);
    constexpr int by_regs = BN > 32 ? 4 : BN > 16 || IN == IN_CAT ? 5 : 6;
    return by_smem < by_regs ? by_smem : by_regs;
  }

  template<int C, int BN, int DIL, int IN, int OUT, int NST>
  __global__ void __launch_bounds__(CNT, conv_blocks<C, BN, DIL, IN, NST>()) k_conv(const ConvArgs a)
  {
    constexpr int HD = halo_dim(DIL), PXC = px_chunks(C), NT8 = BN / 8, BST = BN + 8;
    constexpr int WROWS = C == 8 ? 80 : C;         // weight rows of one stage
    extern __shared__ __align__(16) unsigned char smem[];
    bf* sw = reinterpret_cast<bf*>(smem);
    bf* sx = reinterpret_cast<bf*>(smem + conv_wbytes<C, BN, NST>());
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = a.t.T, G = a.t.G, nt = a.t.nt, TT = T * T;
    const int n0 = blockIdx.y * BN;

    auto load_w = [&](int stage, int buf)
    {
      constexpr int CHB = BN / 8;
      for(int q = tid; q < WROWS * CHB; q += CNT)
      {
        const int r = q / CHB, c = q % CHB;
        cp16(sw + (buf * WROWS + r) * BST + c * 8, a.w + size_t(stage * WROWS + r) * a.n_ld + n0 + c * 8, 16);
      }
    };
    // shared-memory addresses of this lane's two A rows (pixels outside the tile read pixel 0)
    uint32_t arow[2];
    #pragma unroll
    for(int mt = 0; mt < 2; ++mt)
    {
      int m = warp * 32 + mt * 16 + (lane & 15);
      if(m >= TT)
        m = 0;
      arow[mt] = smem_addr(sx) + uint32_t((m / T * HD + m % T) * PXC * 16);
    }
    const uint32_t brow = smem_addr(sw) + uint32_t((lane & 15) * BST + (lane >> 4) * 8) * 2;
    const int half = lane >> 4;
    // what the missing tenth tap of eight channels reads: zeros, since its zero weights would turn an
    // infinite pixel into NaN
    __shared__ __align__(16) uint4 zeros;
    if(C == 8 && tid == 0)
      zeros = make_uint4(0u, 0u, 0u, 0u);

    // the weights that stay are fetched before the wait for the kernel ahead: no kernel that is followed
    // by a convolution directly writes them, and none lets its dependents start before its own wait is over
    // (dependents start when every block has exited), so the kernels before it have ended
    if constexpr(C == 8)
      load_w(0, 0);
    else if constexpr(NST == 9)
      for(int s = 0; s < 9; ++s)
        load_w(s, s);
    pdl_wait();
    bool first = true;
    for(int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x)
    {
      const int b = tile / (nt * nt), r = tile - b * (nt * nt);
      const int y0 = r / nt * T, x0 = (r - r / nt * nt) * T;
      if(!first)
        __syncthreads();                            // the previous tile's reads are done
      load_halo<C, DIL, IN, CNT>(a.in, a.t, b, y0, x0, sx);
      if constexpr(C != 8 && NST != 9)
        load_w(0, 0);
      cp_commit();
      float acc[2][NT8][4];
      #pragma unroll
      for(int i = 0; i < 2; ++i)
        #pragma unroll
        for(int j = 0; j < NT8; ++j)
          #pragma unroll
          for(int e = 0; e < 4; ++e)
            acc[i][j][e] = 0.f;
      // one 16-deep step: A chunks at aoff (bytes), B rows at boff (bytes); zero: this lane's are zeros
      auto step = [&](uint32_t aoff, uint32_t boff, bool zero = false)
      {
        uint32_t af[2][4];
        #pragma unroll
        for(int mt = 0; mt < 2; ++mt)
          ldm_x4a(af[mt], zero ? smem_addr(&zeros) : arow[mt] + aoff);
        #pragma unroll
        for(int j = 0; j < NT8; j += 2)
        {
          if(j + 1 < NT8)
          {
            uint32_t bfr[4];
            ldm_x4a_t(bfr, brow + boff + j * 16);
            #pragma unroll
            for(int mt = 0; mt < 2; ++mt)
            {
              mma16816(acc[mt][j], af[mt], bfr[0], bfr[1]);
              mma16816(acc[mt][j + 1], af[mt], bfr[2], bfr[3]);
            }
          }
          else
          {
            uint32_t bfr[2];
            ldm_x2a_t(bfr, brow - half * 16 + boff + j * 16);
            #pragma unroll
            for(int mt = 0; mt < 2; ++mt)
              mma16816(acc[mt][j], af[mt], bfr[0], bfr[1]);
          }
        }
      };
      if constexpr(C == 8)
      {
        cp_wait<0>();
        __syncthreads();
        // a 16-deep step holds two taps; the tenth chunk's weight rows are zero
        #pragma unroll
        for(int s = 0; s < 5; ++s)
        {
          const int q0 = 2 * s, q1 = 2 * s + 1 < 9 ? 2 * s + 1 : 0;
          const int o0 = (q0 / 3 * HD + q0 % 3) * DIL * PXC * 16, o1 = (q1 / 3 * HD + q1 % 3) * DIL * PXC * 16;
          step(uint32_t(half ? o1 : o0), uint32_t(s * 16 * BST * 2), s == 4 && half);
        }
      }
      else if constexpr(NST == 9)
      {
        cp_wait<0>();
        __syncthreads();
        #pragma unroll
        for(int tap = 0; tap < 9; ++tap)
          #pragma unroll
          for(int c = 0; c < C / 16; ++c)
            step(uint32_t(((tap / 3 * HD + tap % 3) * DIL * PXC + 2 * c + half) * 16),
              uint32_t((tap * C + c * 16) * BST * 2));
      }
      else
      {
        for(int tap = 0; tap < 9; ++tap)
        {
          if(tap + 1 < 9)
            load_w(tap + 1, (tap + 1) & 1);
          cp_commit();
          cp_wait<1>();
          __syncthreads();
          const uint32_t ao = uint32_t(((tap / 3 * HD + tap % 3) * DIL * PXC + half) * 16);
          const uint32_t bo = uint32_t((tap & 1) * C * BST * 2);
          #pragma unroll
          for(int c = 0; c < C / 16; ++c)
            step(ao + c * 32, bo + c * 16 * BST * 2);
          __syncthreads();
        }
      }
      first = false;
      // epilogue: fragment rows g and g + 8 of each 16-row tile, columns 8 j + 2 tg, + 1
      const int g = lane >> 2, tg = lane & 3;
      #pragma unroll
      for(int mt = 0; mt < 2; ++mt)
        #pragma unroll
        for(int h = 0; h < 2; ++h)
        {
          const int m = warp * 32 + mt * 16 + g + h * 8;
          const int ty = m / T, y = y0 + ty, x = x0 + m - ty * T;
          const bool ok = m < TT && y < G && x < G;
          const size_t p = (size_t(b) * G + y) * G + x;
          if constexpr(OUT == OUT_FIRST)
          {
            if(ok && tg == 0)
              static_cast<float*>(a.y)[p] = acc[mt][0][h * 2] + __ldg(a.bias);
          }
          else if constexpr(OUT == OUT_F32)
          {
            if(ok)
              #pragma unroll
              for(int j = 0; j < NT8; ++j)
              {
                const int col = n0 + j * 8 + tg * 2;
                float* q = col < a.nsplit ? static_cast<float*>(a.y) + p * a.nsplit + col
                                          : a.y2 + p * (a.n - a.nsplit) + (col - a.nsplit);
                *reinterpret_cast<float2*>(q) = make_float2(acc[mt][j][h * 2], acc[mt][j][h * 2 + 1]);
              }
          }
          else
          {
            // two 8-column groups at a time: the four lanes of a row exchange so that each stores
            // 8 consecutive bytes of the row's 32 (whole sectors)
            #pragma unroll
            for(int j = 0; j < NT8; j += 2)
            {
              uint32_t pk[2];
              #pragma unroll
              for(int u = 0; u < 2; ++u)
              {
                float v0 = acc[mt][j + u][h * 2], v1 = acc[mt][j + u][h * 2 + 1];
                if constexpr(OUT == OUT_RELU)
                {
                  const int col = n0 + (j + u) * 8 + tg * 2;
                  v0 = fmaxf(v0 + __ldg(a.bias + col), 0.f);
                  v1 = fmaxf(v1 + __ldg(a.bias + col + 1), 0.f);
                }
                pk[u] = uint32_t(f2bf(v0)) | (uint32_t(f2bf(v1)) << 16);
              }
              const int s0 = (lane & ~3) | ((tg & 1) * 2);
              const uint32_t a0 = __shfl_sync(0xffffffffu, pk[0], s0), a1 = __shfl_sync(0xffffffffu, pk[0], s0 + 1);
              const uint32_t b0 = __shfl_sync(0xffffffffu, pk[1], s0), b1 = __shfl_sync(0xffffffffu, pk[1], s0 + 1);
              uint2 v = tg < 2 ? make_uint2(a0, a1) : make_uint2(b0, b1);
              if(ok)
              {
                const size_t o = p * a.n + n0 + j * 8 + tg * 4;
                if constexpr(OUT == OUT_MASK)
                {
                  const uint2 q = __ldg(reinterpret_cast<const uint2*>(a.post + o));
                  v.x &= mask2(q.x);
                  v.y &= mask2(q.y);
                }
                *reinterpret_cast<uint2*>(static_cast<bf*>(a.y) + o) = v;
              }
            }
          }
        }
    }
  }

  // ------------------------------------------------------------------ weight gradient
  // part[block][co][tap*ct + c0 + c] = sum over the block's tiles of dy[p, co] * x[p + off(tap), c],
  // part_b[block][co] = sum of dy[p, co]: M = output channels, N = 9 C columns, K = the 128 pixel
  // slots of each tile (slots outside the tile or the grid hold zeros in dy).  Both operands are
  // read transposed by ldmatrix.trans from the staged tiles; warp w takes GPW groups of 16 columns
  // and all M rows, so a warp issues MT + GPW ldmatrix.x4 for 2 MT GPW MMAs.  Blocks are
  // persistent over tiles and write one partial each (FP32), which k_grad_reduce sums in block order.
  // A slot outside the tile or the grid reads zeros for x too: its zero in dy would turn an infinite
  // activation into NaN.
  struct WgradArgs
  {
    Input in;
    Tiling t;
    const void* dy;      // BF16 [P][M] or FP32 [P] (SCALAR: M = 16 rows of which row 0 is real)
    float* part;         // [blocks][m_real * 9 ct]
    float* part_b;       // [blocks][m_real]
    int m_real;
    int ntiles;
  };

  template<int C, int M, int DIL>
  __host__ __device__ constexpr int wgrad_stage()
  {
    return halo_bytes(C, DIL) + 128 * px_chunks(M) * 16;
  }
  template<int C, int M, int DIL>
  __host__ __device__ constexpr int wgrad_smem() { return 2 * wgrad_stage<C, M, DIL>(); }

  // Resident blocks per SM by the accumulators' registers: layers of few weights take three or four
  // (batch 32 at 129 points: 48 -> 16 62 -> 57 us, 2 -> 16 31 -> 19, 16 -> 1 32 -> 26); 96 -> 32 takes one of
  // 18 warps, three column groups each, where nine warps with six held 14% of the SM's warps (58 -> 47 us)
  template<int C, int M>
  __host__ __device__ constexpr int wgrad_resident() { return C * M <= 256 ? 4 : C * M <= 768 ? 3 : 1; }

  template<int C, int M, int DIL, int IN, bool SCALAR, int NW>
  __global__ void __launch_bounds__(NW * 32, wgrad_resident<C, M>()) k_wgrad(const WgradArgs a)
  {
    constexpr int NT = NW * 32, HD = halo_dim(DIL), PXC = px_chunks(C), PXD = px_chunks(M);
    constexpr int MT = M / 16, CH = C / 8;
    constexpr int NCH = 9 * CH;                     // 8-column chunks
    constexpr int GPW = ((NCH + 1) / 2 + NW - 1) / NW;
    extern __shared__ __align__(16) unsigned char smem[];
    bf* sx = reinterpret_cast<bf*>(smem);
    bf* sd = reinterpret_cast<bf*>(smem + halo_bytes(C, DIL));
    constexpr int STAGE = wgrad_stage<C, M, DIL>();
    __shared__ int pxo[2][128];                     // halo offset (bytes) of each pixel slot, -1: none
    __shared__ __align__(16) uint4 zeros;
    Input in = a.in;
    in.c0 += int(blockIdx.y) * C;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = a.t.T, G = a.t.G, nt = a.t.nt, TT = T * T;
    if(tid == 0)
      zeros = make_uint4(0u, 0u, 0u, 0u);
    // byte offset of this lane's chunk of each column group (chunks past the end read chunk 0)
    uint32_t goff[GPW];
    #pragma unroll
    for(int k = 0; k < GPW; ++k)
    {
      int q = 2 * (warp * GPW + k) + (lane >> 4);
      if(q >= NCH)
        q = 0;
      const int tap = q / CH, c = q - tap * CH;
      goff[k] = smem_addr(sx) + uint32_t(((tap / 3 * HD + tap % 3) * DIL * PXC + c) * 16);
    }
    const int lj = lane >> 3, li = lane & 7;
    const uint32_t drow = smem_addr(sd) + uint32_t(((lj >> 1) * 8 + li) * PXD * 16 + (lj & 1) * 16);
    float acc[MT][GPW][2][4], accb[MT][4];
    #pragma unroll
    for(int i = 0; i < MT; ++i)
    {
      #pragma unroll
      for(int j = 0; j < GPW; ++j)
        #pragma unroll
        for(int e = 0; e < 4; ++e)
          acc[i][j][0][e] = acc[i][j][1][e] = 0.f;
      #pragma unroll
      for(int e = 0; e < 4; ++e)
        accb[i][e] = 0.f;
    }
    // a tile's input and output gradient into buffer `buf`
    auto load = [&](int tile, int buf)
    {
      const int b = tile / (nt * nt), r = tile - b * (nt * nt);
      const int y0 = r / nt * T, x0 = (r - r / nt * nt) * T;
      load_halo<C, DIL, IN, NT>(in, a.t, b, y0, x0, sx + buf * (STAGE / 2));
      for(int m = tid; m < 128; m += NT)
      {
        const int ty = m / T, tx = m - ty * T;
        pxo[buf][m] = m < TT && y0 + ty < G && x0 + tx < G ? (ty * HD + tx) * PXC * 16 + buf * STAGE : -1;
      }
      for(int e = tid; e < 128 * (M / 8); e += NT)
      {
        const int ch = e % (M / 8), m = e / (M / 8);
        const int ty = m / T, y = y0 + ty, x = x0 + m - ty * T;
        const bool ok = m < TT && y < G && x < G;
        const size_t p = (size_t(b) * G + y) * G + x;
        bf* dst = sd + buf * (STAGE / 2) + (m * PXD + ch) * 8;
        if constexpr(SCALAR)
        {
          const uint32_t w = ok && ch == 0 ? uint32_t(f2bf(__ldg(static_cast<const float*>(a.dy) + p))) : 0u;
          *reinterpret_cast<uint4*>(dst) = make_uint4(w, 0u, 0u, 0u);
        }
        else
        {
          const bf* src = static_cast<const bf*>(a.dy);
          cp16(dst, ok ? src + p * M + ch * 8 : src, ok ? 16 : 0);
        }
      }
      cp_commit();
    };
    int buf = 0;
    pdl_wait();
    if(int(blockIdx.x) < a.ntiles)
      load(int(blockIdx.x), 0);
    for(int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, buf ^= 1)
    {
      // the next tile's copies run under this tile's products (its buffer's reads ended with the last
      // round's barrier)
      if(tile + int(gridDim.x) < a.ntiles)
      {
        load(tile + int(gridDim.x), buf ^ 1);
        cp_wait<1>();
      }
      else
        cp_wait<0>();
      __syncthreads();
      const uint32_t so = uint32_t(buf * STAGE);
      #pragma unroll 2
      for(int k = 0; k < 8; ++k)
      {
        const int px = pxo[buf][k * 16 + (lane & 15)];
        uint32_t bfr[GPW][4];
        #pragma unroll
        for(int j = 0; j < GPW; ++j)
          ldm_x4a_t(bfr[j], px < 0 ? smem_addr(&zeros) : goff[j] + uint32_t(px));
        #pragma unroll
        for(int mt = 0; mt < MT; ++mt)
        {
          uint32_t af[4];
          ldm_x4a_t(af, drow + so + uint32_t(k * 16 * PXD * 16 + mt * 32));
          #pragma unroll
          for(int j = 0; j < GPW; ++j)
          {
            mma16816(acc[mt][j][0], af, bfr[j][0], bfr[j][1]);
            mma16816(acc[mt][j][1], af, bfr[j][2], bfr[j][3]);
          }
          if(warp == NW - 1)
            mma16816(accb[mt], af, 0x3F803F80u, 0x3F803F80u);   // times ones: the bias gradient
        }
      }
      __syncthreads();                              // this buffer's reads are done
    }
    const int g = lane >> 2, tg = lane & 3;
    const int n9 = 9 * in.ct;
    float* out = a.part + size_t(blockIdx.x) * a.m_real * n9;
    #pragma unroll
    for(int mt = 0; mt < MT; ++mt)
      #pragma unroll
      for(int h = 0; h < 2; ++h)
      {
        const int m = mt * 16 + g + h * 8;
        if(m >= a.m_real)
          continue;
        #pragma unroll
        for(int j = 0; j < GPW; ++j)
          #pragma unroll
          for(int u = 0; u < 2; ++u)
          {
            const int q = 2 * (warp * GPW + j) + u;
            if(q < NCH)
              *reinterpret_cast<float2*>(out + size_t(m) * n9 + q / CH * in.ct + in.c0 + q % CH * 8 + tg * 2) =
                make_float2(acc[mt][j][u][h * 2], acc[mt][j][u][h * 2 + 1]);
          }
        if(warp == NW - 1 && tg == 0 && blockIdx.y == 0)
          a.part_b[size_t(blockIdx.x) * a.m_real + m] = accb[mt][h * 2];
      }
  }

  // ------------------------------------------------------------------ parameters
  // Where each layer's parameters, BF16 GEMM copies and gradient partials lie.
  struct LayerMap
  {
    int woff, boff, cin, cout, cin_pad, cout_pad;
    bf *wf, *wd;
    const float *part, *part_b;
    int blocks;
  };
  struct NetMap
  {
    LayerMap l[NLAYER];
    int n;
  };

  __device__ __forceinline__ int layer_of(const NetMap& net, int e)
  {
    int l = 0;
    #pragma unroll
    for(int k = 1; k < NLAYER; ++k)
      l += e >= net.l[k].woff ? 1 : 0;
    return l;
  }

  // Every parameter's gradient: its partials summed in four groups (group g takes partials g, g + 4,
  // ...), then the groups in order.  64 parameters per block: a group's loads are whole 128-byte
  // lines, and four groups keep four times as many of them in flight as one thread per parameter.
  constexpr int GR_E = 64, GR_G = 4;
  __global__ void __launch_bounds__(GR_E * GR_G) k_grad_reduce(const __grid_constant__ NetMap net,
    float* __restrict__ grad, int accumulate)
  {
    pdl_wait();
    __shared__ float sh[GR_G][GR_E];
    const int x = threadIdx.x % GR_E, grp = threadIdx.x / GR_E;
    const int e = blockIdx.x * GR_E + x;
    float s = 0.f;
    if(e < net.n)
    {
      const LayerMap& L = net.l[layer_of(net, e)];
      const float* p;
      int stride;
      if(e >= L.boff)
      {
        p = L.part_b + (e - L.boff);
        stride = L.cout;
      }
      else
      {
        const int w = e - L.woff, ci = w % L.cin, t = w / L.cin;
        p = L.part + t * L.cin_pad + ci;            // t = co * 9 + tap
        stride = L.cout * 9 * L.cin_pad;
      }
      const int blocks = L.blocks;
      #pragma unroll 8
      for(int k = grp; k < blocks; k += GR_G)
        s += __ldg(p + size_t(k) * stride);
    }
    sh[grp][x] = s;
    __syncthreads();
    if(grp == 0 && e < net.n)
    {
      const float t = ((s + sh[1][x]) + sh[2][x]) + sh[3][x];
      grad[e] = accumulate ? grad[e] + t : t;
    }
  }

  // FP32 master -> BF16 GEMM layouts: forward wf[tap*cin_pad + ci][co] (rows of cout_pad) and data
  // gradient wd[t*cout_pad + co][ci] = W[co][8-t][ci] (rows of cin_pad); padding entries stay zero
  __device__ __forceinline__ void store_weight(const LayerMap& L, int w, float v)
  {
    const int ci = w % L.cin, t = w / L.cin, tap = t % 9, co = t / 9;
    const bf h = f2bf(v);
    L.wf[(tap * L.cin_pad + ci) * L.cout_pad + co] = h;
    if(L.wd)
      L.wd[((8 - tap) * L.cout_pad + co) * L.cin_pad + ci] = h;
  }
  __global__ void __launch_bounds__(256) k_prep_weights(const __grid_constant__ NetMap net, const float* __restrict__ p)
  {
    pdl_wait();
    const int e = blockIdx.x * 256 + threadIdx.x;
    if(e >= net.n)
      return;
    const LayerMap& L = net.l[layer_of(net, e)];
    if(e < L.boff)
      store_weight(L, e - L.woff, p[e]);
  }

  // Adam (Kingma & Ba 2015, Algorithm 1) on the FP32 masters, and the BF16 copies of the new weights
  __global__ void __launch_bounds__(256) k_adam(const __grid_constant__ NetMap net, float* __restrict__ p,
    const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2, float eps,
    float c1, float c2)
  {
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if(i >= net.n)
      return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    const LayerMap& L = net.l[layer_of(net, i)];
    if(i < L.boff)
      store_weight(L, i - L.woff, pi);
  }

  // ------------------------------------------------------------------ packing and masked gradients
  // NCHW FP32 input (2 channels) -> BF16 pairs per pixel (kept for the first layer's weight gradient)
  __global__ void k_pack_input(const float* __restrict__ in, int B, int G, uint32_t* __restrict__ x)
  {
    pdl_wait();
    const size_t n = size_t(G) * G;
    for(size_t p = blockIdx.x * size_t(blockDim.x) + threadIdx.x; p < n * B; p += size_t(gridDim.x) * blockDim.x)
    {
      const size_t b = p / n, r = p - b * n;
      x[p] = uint32_t(f2bf(in[b * 2 * n + r])) | (uint32_t(f2bf(in[(b * 2 + 1) * n + r])) << 16);
    }
  }

  __device__ __forceinline__ void store8(bf* dst, const float (&s)[8], const uint4& post)
  {
    const uint32_t q[4] = {post.x, post.y, post.z, post.w};
    uint32_t o[4];
    #pragma unroll
    for(int k = 0; k < 4; ++k)
      o[k] = (uint32_t(f2bf(s[2 * k])) | (uint32_t(f2bf(s[2 * k + 1])) << 16)) & mask2(q[k]);
    *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  __device__ __forceinline__ void load8(const float* p, float (&v)[8])
  {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p + 4));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }

  // adjoint of U for a fine FP32 gradient [B][Gf][Gf][C]: gc(i, j) = sum_{dy,dx in -1..1} w(dy) w(dx)
  // gf(2i+dy, 2j+dx) (in-grid points), w(0) = 1, w(+-1) = 1/2; the four corner products of a cell
  // centre carry 1/4 each.  Then dpre = mask(post) * gc as BF16.  Eight channels per thread.
  __global__ void __launch_bounds__(256) k_upsample_bwd_mask(const float* __restrict__ gf, int C, int B, int Gf,
    const bf* __restrict__ post, bf* __restrict__ dpre)
  {
    pdl_wait();
    const int Gc = (Gf + 1) / 2, C8 = C / 8;
    const size_t n = size_t(B) * Gc * Gc * C8;
    for(size_t e = blockIdx.x * size_t(256) + threadIdx.x; e < n; e += size_t(gridDim.x) * 256)
    {
      const int ch = int(e % C8);
      const size_t p = e / C8;
      const int x = int(p % Gc), y = int((p / Gc) % Gc);
      const size_t b = p / (size_t(Gc) * Gc);
      float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      #pragma unroll
      for(int dy = -1; dy <= 1; ++dy)
        #pragma unroll
        for(int dx = -1; dx <= 1; ++dx)
        {
          const int yf = 2 * y + dy, xf = 2 * x + dx;
          if(yf < 0 || yf >= Gf || xf < 0 || xf >= Gf)
            continue;
          const float w = (dy == 0 ? 1.f : 0.5f) * (dx == 0 ? 1.f : 0.5f);
          float v[8];
          load8(gf + ((b * Gf + yf) * Gf + xf) * C + ch * 8, v);
          #pragma unroll
          for(int k = 0; k < 8; ++k)
            s[k] += w * v[k];
        }
      store8(dpre + e * 8, s, __ldg(reinterpret_cast<const uint4*>(post + e * 8)));
    }
  }

  // dpre = mask(post) * (g1 + (even-even pixel ? g2 of the coarse vertex : 0)): the gradient through
  // the skip connection and through the injection.  Eight channels per thread.
  __global__ void __launch_bounds__(256) k_grad_mask(const bf* __restrict__ post, int C, int B, int G,
    const float* __restrict__ g1, const float* __restrict__ g2, bf* __restrict__ dpre)
  {
    pdl_wait();
    const int Gc = (G + 1) / 2, C8 = C / 8;
    const size_t n = size_t(B) * G * G * C8;
    for(size_t e = blockIdx.x * size_t(256) + threadIdx.x; e < n; e += size_t(gridDim.x) * 256)
    {
      const int ch = int(e % C8);
      const size_t p = e / C8;
      const int x = int(p % G), y = int((p / G) % G);
      float s[8];
      load8(g1 + e * 8, s);
      if(!(x & 1) && !(y & 1))
      {
        const size_t b = p / (size_t(G) * G);
        float v[8];
        load8(g2 + ((b * Gc + y / 2) * Gc + x / 2) * C + ch * 8, v);
        #pragma unroll
        for(int k = 0; k < 8; ++k)
          s[k] += v[k];
      }
      store8(dpre + e * 8, s, __ldg(reinterpret_cast<const uint4*>(post + e * 8)));
    }
  }

  // loss = sum (y - t)^2 / n over [n]; grad = 2 (y - t) / n (per-block partials, summed in block
  // order by the last block)
  constexpr int MSE_NT = 256;
  __global__ void __launch_bounds__(MSE_NT) k_mse(const float* __restrict__ y, const float* __restrict__ t, size_t n,
    float* __restrict__ grad, RedSlot slot, double* __restrict__ loss)
  {
    pdl_wait();
    __shared__ double sh[32];
    double s = 0.0;
    const float inv = 1.f / float(n);
    for(size_t i = blockIdx.x * size_t(MSE_NT) + threadIdx.x; i < n; i += size_t(gridDim.x) * MSE_NT)
    {
      const float d = y[i] - t[i];
      if(grad)
        grad[i] = 2.f * d * inv;
      s += double(d) * double(d);
    }
    double total;
    if(grid_sum_last<MSE_NT>(s, slot, sh, total))
      *loss = total / double(n);
  }
} // namespace un
} // namespace fb

using namespace fb;
using namespace fb::un;

struct fb_unet
{
  int G[4] = {0, 0, 0, 0};
  int max_batch = 0;
  size_t nparam = 0;
  size_t woff[NLAYER], boff[NLAYER];
  int cin_pad[NLAYER], cout_pad[NLAYER], kpad[NLAYER], kpad_d[NLAYER];
  void* arena = nullptr;       // every device buffer of the network
  float *param = nullptr, *grad = nullptr, *adam_m = nullptr, *adam_v = nullptr;
  bf* wf[NLAYER] = {};
  bf* wd[NLAYER] = {};
  // activations (BF16 NHWC): xp (input pairs), e1..e4, the two further bottleneck outputs, d3, d2, d1
  uint32_t* xp = nullptr;
  bf *e[4] = {}, *d[3] = {};
  bf* b4[2] = {};              // bottleneck: outputs of the dilation-2 and dilation-4 convolutions
  // backward scratch: BF16 pre-activation gradients (two, used in turn); FP32 data gradients of the
  // concatenated inputs, upsampled channels du and skip channels dk, and of the subsampled ones (gs)
  bf* dpre[2] = {};
  float *du[3] = {}, *dk[3] = {}, *gs = nullptr;
  float* part[NLAYER] = {};    // weight- and bias-gradient partials, one per block
  float* part_b[NLAYER] = {};
  int blocks_max[NLAYER] = {};
  double* mse_part = nullptr;
  unsigned int* mse_counter = nullptr;
  bool weights_ready = false;
};

namespace
{
  constexpr int SMS = 148;

#define UN_TRY(x)                      \
  do {                                 \
    fb_status t_ = (x);                \
    if(t_ != FB_OK) return t_;         \
  } while(0)

  unsigned grid_for(size_t n, int nt = 256)
  {
    return unsigned(std::min<size_t>(std::max<size_t>((n + nt - 1) / nt, 1), SMS * 16));
  }

  // tiles of at most TMAX x TMAX points, as even as they come
  Tiling tiling(int G)
  {
    Tiling t;
    t.G = G;
    t.nt = (G + TMAX - 1) / TMAX;
    t.T = (G + t.nt - 1) / t.nt;
    return t;
  }
  int tiles(const Tiling& t, int B) { return B * t.nt * t.nt; }

  // The blocks of a layer's weight-gradient kernel: a tile each up to what the SMs hold.  Two tiles per
  // block of the 64 x 64 and larger layers halve what the reduction reads, but their FP32 sums are twice as
  // long (relative error of the 64 x 64 layers' gradients at 129 points and batch 1 9e-8, against 4e-8) and
  // the step is no faster (240 us, against 221; batch 32 755, against 749).
  int wgrad_blocks(const fb_unet* u, int l, int B)
  {
    const int nt = tiles(tiling(u->G[LAYERS[l].level]), B);
    const int w = u->cin_pad[l] * pad8(LAYERS[l].cout);
    const int cap = l == 6 ? SMS / 2 : w <= 256 ? 4 * SMS : w <= 768 ? 3 * SMS : SMS;
    return std::max(1, std::min(nt, cap));
  }

  NetMap net_map(const fb_unet* u, int B)
  {
    NetMap m;
    m.n = int(u->nparam);
    for(int l = 0; l < NLAYER; ++l)
    {
      LayerMap& L = m.l[l];
      L.woff = int(u->woff[l]);
      L.boff = int(u->boff[l]);
      L.cin = LAYERS[l].cin;
      L.cout = LAYERS[l].cout;
      L.cin_pad = u->cin_pad[l];
      L.cout_pad = u->cout_pad[l];
      L.wf = u->wf[l];
      L.wd = u->wd[l];
      L.part = u->part[l];
      L.part_b = u->part_b[l];
      L.blocks = B > 0 ? wgrad_blocks(u, l, B) : 0;
    }
    return m;
  }

  // A launch with programmatic stream serialisation: scheduled while the kernel ahead finishes, every
  // kernel waits for it in pdl_wait.  Ten layers forward and forty kernels of a training step spent 2 us
  // each between one's end and the next one's first load (a prediction of batch 1: 83 -> 52 us).
  template<typename... KA, typename... A>
  cudaError_t launch(void (*k)(KA...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, A&&... args)
  {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = grid;
    lc.blockDim = dim3(block);
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = &at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k, KA(args)...);
  }

  template<int C, int BN, int DIL, int IN, int OUT, int NST>
  fb_status launch_conv(const ConvArgs& a, cudaStream_t st)
  {
    constexpr int smem = conv_smem<C, BN, DIL, NST>();
    if(smem > 48 * 1024)
      FB_CUDA(cudaFuncSetAttribute(k_conv<C, BN, DIL, IN, OUT, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    constexpr int occ = conv_blocks<C, BN, DIL, IN, NST>();
    const int ny = a.n / BN;
    dim3 grid(unsigned(std::min(a.ntiles, std::max(1, SMS * occ / ny))), unsigned(ny));
    FB_CUDA(launch(k_conv<C, BN, DIL, IN, OUT, NST>, dim3(grid), CNT, smem, st, a));
    FB_LAUNCHED(1);
    return FB_OK;
  }

  Input plain(const bf* x, int c) { return Input{x, nullptr, 0, c, 0}; }
  Input concat(const bf* coarse, int cu, const bf* skip, int cs) { return Input{coarse, skip, cu, cu + cs, 0}; }

  // layer l's convolution of `in` at its grid; y BF16 with ReLU, or FP32 [P] for the last layer.
  // NARROW: 16 output columns per block instead of all, for grids of few tiles: the blocks of one
  // tile share its pixels, so a batch of one (4 to 36 tiles on the coarse grids) spreads over four
  // times as many SMs, and each streams a quarter of the weights.
  template<int C, int BN, int DIL, int IN, int OUT, int NST, int NARROW_NST = 9>
  fb_status conv_fwd(fb_unet* u, int l, const Input& in, int B, void* y, cudaStream_t st)
  {
    ConvArgs a{};
    a.in = in;
    a.t = tiling(u->G[LAYERS[l].level]);
    a.w = u->wf[l];
    a.bias = u->param + u->boff[l];
    a.y = y;
    a.n = a.n_ld = u->cout_pad[l];
    a.ntiles = tiles(a.t, B);
    if constexpr(BN > 16)
      if(a.ntiles * (a.n / BN) < SMS)
        return launch_conv<C, 16, DIL, IN, OUT, NARROW_NST>(a, st);
    return launch_conv<C, BN, DIL, IN, OUT, NST>(a, st);
  }

  // data gradient of layer l: from dpre (`in`, cout_pad channels) to its input's cin_pad channels
  template<int C, int BN, int DIL, int IN, int OUT, int NST>
  fb_status conv_bwd(fb_unet* u, int l, const Input& in, int B, void* y, float* y2, int nsplit, const bf* post,
    cudaStream_t st)
  {
    ConvArgs a{};
    a.in = in;
    a.t = tiling(u->G[LAYERS[l].level]);
    a.w = u->wd[l];
    a.y = y;
    a.y2 = y2;
    a.post = post;
    a.n = a.n_ld = u->cin_pad[l];
    a.nsplit = nsplit;
    a.ntiles = tiles(a.t, B);
    return launch_conv<C, BN, DIL, IN, OUT, NST>(a, st);
  }

  // weight- and bias-gradient partials of layer l (cin_pad = C * ny channels, ny halves)
  template<int C, int M, int DIL, int IN, bool SCALAR, int NW>
  fb_status wgrad(fb_unet* u, int l, const void* dy, const Input& in, int B, cudaStream_t st)
  {
    constexpr int smem = wgrad_smem<C, M, DIL>();
    if(smem > 48 * 1024 - 2048)
      FB_CUDA(cudaFuncSetAttribute(k_wgrad<C, M, DIL, IN, SCALAR, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    WgradArgs a{};
    a.in = in;
    a.t = tiling(u->G[LAYERS[l].level]);
    a.dy = dy;
    a.part = u->part[l];
    a.part_b = u->part_b[l];
    a.m_real = LAYERS[l].cout;
    a.ntiles = tiles(a.t, B);
    const dim3 grid(unsigned(wgrad_blocks(u, l, B)), unsigned(u->cin_pad[l] / C));
    FB_CUDA(launch(k_wgrad<C, M, DIL, IN, SCALAR, NW>, dim3(grid), NW * 32, smem, st, a));
    FB_LAUNCHED(1);
    return FB_OK;
  }

  fb_status prep_weights(fb_unet* u, cudaStream_t st)
  {
    FB_CUDA(launch(k_prep_weights, dim3(unsigned((u->nparam + 255) / 256)), 256, 0, st, net_map(u, 0), u->param));
    FB_LAUNCHED(1);
    u->weights_ready = true;
    return FB_OK;
  }
} // namespace

extern "C" {

fb_status fb_unet_create(fb_unet** out, int grid, int max_batch)
{
  if(!out || max_batch < 1 || grid < 9 || ((grid - 1) & 7) != 0 || ((grid - 1) & (grid - 2)) != 0)
  {
    set_error("unet_create: grid must be 2^k + 1 (k >= 3), max_batch >= 1");
    return FB_ERR_ARG;
  }
  std::unique_ptr<fb_unet> u(new fb_unet());
  u->max_batch = max_batch;
  u->G[0] = grid;
  for(int i = 1; i < 4; ++i)
    u->G[i] = (u->G[i - 1] + 1) / 2;
  size_t off = 0;
  for(int l = 0; l < NLAYER; ++l)
  {
    const LayerDef& L = LAYERS[l];
    u->woff[l] = off;
    off += size_t(L.cout) * 9 * L.cin;
    u->boff[l] = off;
    off += size_t(L.cout);
    u->cin_pad[l] = pad8(L.cin);
    u->cout_pad[l] = pad8(L.cout);
    // GEMM depth rounded up to whole 32-deep steps (the rows past 9 channels stay zero)
    u->kpad[l] = (9 * u->cin_pad[l] + 31) / 32 * 32;
    u->kpad_d[l] = (9 * u->cout_pad[l] + 31) / 32 * 32;
  }
  u->nparam = off;
  fb_unet* p = u.get();
  // one allocation for all buffers (an allocation each takes the driver longer than their use in a
  // short training step); the zeroed ones first
  std::vector<std::pair<void**, size_t>> want;
  size_t total = 0;
  auto take = [&](auto*& ptr, size_t bytes)
  {
    want.emplace_back(reinterpret_cast<void**>(&ptr), total);
    total += (std::max<size_t>(bytes, 256) + 255) & ~size_t(255);
  };
  take(p->param, sizeof(float) * off);
  take(p->grad, sizeof(float) * off);
  take(p->adam_m, sizeof(float) * off);
  take(p->adam_v, sizeof(float) * off);
  for(int l = 0; l < NLAYER; ++l)
  {
    take(p->wf[l], sizeof(bf) * p->kpad[l] * p->cout_pad[l]);
    if(l > 0)
      take(p->wd[l], sizeof(bf) * p->kpad_d[l] * p->cin_pad[l]);
  }
  take(p->mse_counter, sizeof(unsigned int));
  const size_t zeroed = total;
  for(int l = 0; l < NLAYER; ++l)
  {
    const size_t nb = size_t(wgrad_blocks(p, l, max_batch));
    take(p->part[l], sizeof(float) * nb * LAYERS[l].cout * 9 * p->cin_pad[l]);
    take(p->part_b[l], sizeof(float) * nb * LAYERS[l].cout);
  }
  const size_t B = size_t(max_batch);
  auto pix = [&](int lv) { return B * size_t(p->G[lv]) * p->G[lv]; };
  take(p->xp, sizeof(uint32_t) * pix(0));
  const int ech[4] = {16, 32, 64, 64};
  for(int i = 0; i < 4; ++i)
    take(p->e[i], sizeof(bf) * pix(i) * ech[i]);
  for(int i = 0; i < 2; ++i)
    take(p->b4[i], sizeof(bf) * pix(3) * 64);
  // d[0] = d1 @G1 (16), d[1] = d2 @G2 (32), d[2] = d3 @G3 (64)
  for(int i = 0; i < 3; ++i)
    take(p->d[i], sizeof(bf) * pix(i) * ech[i]);
  // largest pre-activation gradient: G1 x 16, G2 x 32, G3 x 64 or G4 x 64 channels
  const size_t dmax = std::max(std::max(pix(0) * 16, pix(1) * 32), std::max(pix(2) * 64, pix(3) * 64));
  for(int i = 0; i < 2; ++i)
    take(p->dpre[i], sizeof(bf) * dmax);
  // data gradients of [U(d2), e1] @G1, [U(d3), e2] @G2, [U(e4), e3] @G3
  const int uch[3] = {32, 64, 64};
  for(int i = 0; i < 3; ++i)
  {
    take(p->du[i], sizeof(float) * pix(i) * uch[i]);
    take(p->dk[i], sizeof(float) * pix(i) * ech[i]);
  }
  take(p->gs, sizeof(float) * std::max(pix(3) * 64, std::max(pix(2) * 32, pix(1) * 16)));
  take(p->mse_part, sizeof(double) * 1024);
  FB_CUDA(cudaMalloc(&p->arena, total));
  const cudaError_t z = cudaMemset(p->arena, 0, zeroed);
  if(z != cudaSuccess)
  {
    cudaFree(p->arena);
    return cuda_fail(z, "cudaMemset");
  }
  for(const auto& w : want)
    *w.first = static_cast<unsigned char*>(p->arena) + w.second;
  *out = u.release();
  return FB_OK;
}

void fb_unet_destroy(fb_unet* u)
{
  if(!u)
    return;
  cudaFree(u->arena);
  delete u;
}

fb_status fb_unet_num_params(const fb_unet* u, uint64_t* n)
{
  if(!u || !n)
  {
    set_error("unet_num_params: bad arguments");
    return FB_ERR_ARG;
  }
  *n = u->nparam;
  return FB_OK;
}

fb_status fb_unet_set_params(fb_unet* u, const float* host)
{
  if(!u || !host)
  {
    set_error("unet_set_params: bad arguments");
    return FB_ERR_ARG;
  }
  FB_CUDA(cudaMemcpy(u->param, host, sizeof(float) * u->nparam, cudaMemcpyHostToDevice));
  FB_CUDA(cudaMemset(u->adam_m, 0, sizeof(float) * u->nparam));
  FB_CUDA(cudaMemset(u->adam_v, 0, sizeof(float) * u->nparam));
  UN_TRY(prep_weights(u, 0));
  FB_CUDA(cudaDeviceSynchronize());
  return FB_OK;
}

fb_status fb_unet_get_params(const fb_unet* u, float* host)
{
  if(!u || !host)
  {
    set_error("unet_get_params: bad arguments");
    return FB_ERR_ARG;
  }
  FB_CUDA(cudaDeviceSynchronize());
  FB_CUDA(cudaMemcpy(host, u->param, sizeof(float) * u->nparam, cudaMemcpyDeviceToHost));
  return FB_OK;
}

fb_status fb_unet_get_grads(const fb_unet* u, float* host)
{
  if(!u || !host)
  {
    set_error("unet_get_grads: bad arguments");
    return FB_ERR_ARG;
  }
  FB_CUDA(cudaDeviceSynchronize());
  FB_CUDA(cudaMemcpy(host, u->grad, sizeof(float) * u->nparam, cudaMemcpyDeviceToHost));
  return FB_OK;
}

// in: DEVICE [batch][2][G][G] FP32 (f, log kappa, already scaled); out: DEVICE [batch][G][G] FP32
fb_status fb_unet_forward(fb_unet* u, const float* in, float* out, int batch, void* stream)
{
  if(!u || !in || !out || batch < 1 || batch > u->max_batch || !u->weights_ready)
  {
    set_error("unet_forward: bad arguments (or parameters not set)");
    return FB_ERR_ARG;
  }
  cudaStream_t st = as_stream(stream);
  const int B = batch;
  FB_CUDA(launch(k_pack_input, dim3(grid_for(size_t(B) * u->G[0] * u->G[0])), 256, 0, st, in, B, u->G[0], u->xp));
  FB_LAUNCHED(1);
  UN_TRY((conv_fwd<8, 16, 1, IN_PAIR, OUT_RELU, 9>(u, 0, Input{u->xp, nullptr, 0, 8, 0}, B, u->e[0], st)));
  UN_TRY((conv_fwd<16, 32, 1, IN_SUB, OUT_RELU, 9>(u, 1, plain(u->e[0], 16), B, u->e[1], st)));
  UN_TRY((conv_fwd<32, 64, 1, IN_SUB, OUT_RELU, 9>(u, 2, plain(u->e[1], 32), B, u->e[2], st)));
  UN_TRY((conv_fwd<64, 64, 1, IN_SUB, OUT_RELU, 2>(u, 3, plain(u->e[2], 64), B, u->e[3], st)));
  // bottleneck: dilation 2 and 4
  UN_TRY((conv_fwd<64, 64, 2, IN_PLAIN, OUT_RELU, 2>(u, 4, plain(u->e[3], 64), B, u->b4[0], st)));
  UN_TRY((conv_fwd<64, 64, 4, IN_PLAIN, OUT_RELU, 2>(u, 5, plain(u->b4[0], 64), B, u->b4[1], st)));
  // decoder
  UN_TRY((conv_fwd<128, 64, 1, IN_CAT, OUT_RELU, 2>(u, 6, concat(u->b4[1], 64, u->e[2], 64), B, u->d[2], st)));
  UN_TRY((conv_fwd<96, 32, 1, IN_CAT, OUT_RELU, 2>(u, 7, concat(u->d[2], 64, u->e[1], 32), B, u->d[1], st)));
  UN_TRY((conv_fwd<48, 16, 1, IN_CAT, OUT_RELU, 9>(u, 8, concat(u->d[1], 32, u->e[0], 16), B, u->d[0], st)));
  UN_TRY((conv_fwd<16, 8, 1, IN_PLAIN, OUT_FIRST, 9>(u, 9, plain(u->d[0], 16), B, out, st)));
  return FB_OK;
}

// Gradients of the parameters for d loss / d out = dout (DEVICE [batch][G][G] FP32) at the
// activations of the last fb_unet_forward (same batch).  accumulate != 0 adds to the stored gradients.
fb_status fb_unet_backward(fb_unet* u, const float* dout, int batch, int accumulate, void* stream)
{
  if(!u || !dout || batch < 1 || batch > u->max_batch)
  {
    set_error("unet_backward: bad arguments");
    return FB_ERR_ARG;
  }
  cudaStream_t st = as_stream(stream);
  const int B = batch;
  const int* G = u->G;
  bf *p0 = u->dpre[0], *p1 = u->dpre[1];
  auto n8 = [&](int lv, int C) { return size_t(B) * G[lv] * G[lv] * (C / 8); };
  // dpre = mask(post) * U^T(du) at level lv + 1 (C channels)
  auto up_bwd = [&](int lv, int C, const bf* post, bf* dpre)
  {
    FB_CUDA(launch(k_upsample_bwd_mask, dim3(grid_for(n8(lv + 1, C))), 256, 0, st, u->du[lv], C, B, G[lv], post, dpre));
    FB_LAUNCHED(1);
    return fb_status(FB_OK);
  };
  // dpre = mask(e[lv]) * (skip gradient + S^T(gs))
  auto skip_bwd = [&](int lv, int C, bf* dpre)
  {
    FB_CUDA(launch(k_grad_mask, dim3(grid_for(n8(lv, C))), 256, 0, st, u->e[lv], C, B, G[lv], u->dk[lv], u->gs, dpre));
    FB_LAUNCHED(1);
    return fb_status(FB_OK);
  };
  // L8 (input d1)
  const Input dy8{dout, nullptr, 0, 8, 0};
  UN_TRY((wgrad<16, 16, 1, IN_PLAIN, true, 9>(u, 9, dout, plain(u->d[0], 16), B, st)));
  UN_TRY((conv_bwd<8, 16, 1, IN_SCALAR, OUT_MASK, 9>(u, 9, dy8, B, p0, nullptr, 0, u->d[0], st)));
  // L7 (input [U(d2), e1])
  UN_TRY((wgrad<48, 16, 1, IN_CAT, false, 9>(u, 8, p0, concat(u->d[1], 32, u->e[0], 16), B, st)));
  UN_TRY((conv_bwd<16, 48, 1, IN_PLAIN, OUT_F32, 9>(u, 8, plain(p0, 16), B, u->du[0], u->dk[0], 32, nullptr, st)));
  UN_TRY(up_bwd(0, 32, u->d[1], p1));
  // L6 (input [U(d3), e2])
  UN_TRY((wgrad<96, 32, 1, IN_CAT, false, 18>(u, 7, p1, concat(u->d[2], 64, u->e[1], 32), B, st)));
  UN_TRY((conv_bwd<32, 48, 1, IN_PLAIN, OUT_F32, 9>(u, 7, plain(p1, 32), B, u->du[1], u->dk[1], 64, nullptr, st)));
  UN_TRY(up_bwd(1, 64, u->d[2], p0));
  // L5 (input [U(e4), e3])
  UN_TRY((wgrad<64, 64, 1, IN_CAT, false, 12>(u, 6, p0, concat(u->b4[1], 64, u->e[2], 64), B, st)));
  UN_TRY((conv_bwd<64, 64, 1, IN_PLAIN, OUT_F32, 2>(u, 6, plain(p0, 64), B, u->du[2], u->dk[2], 64, nullptr, st)));
  UN_TRY(up_bwd(2, 64, u->b4[1], p1));
  // bottleneck: dilation 4 (input b4[0]), dilation 2 (input e4 = e[3]), L4 (input S(e3))
  UN_TRY((wgrad<64, 64, 4, IN_PLAIN, false, 12>(u, 5, p1, plain(u->b4[0], 64), B, st)));
  UN_TRY((conv_bwd<64, 64, 4, IN_PLAIN, OUT_MASK, 2>(u, 5, plain(p1, 64), B, p0, nullptr, 0, u->b4[0], st)));
  UN_TRY((wgrad<64, 64, 2, IN_PLAIN, false, 12>(u, 4, p0, plain(u->e[3], 64), B, st)));
  UN_TRY((conv_bwd<64, 64, 2, IN_PLAIN, OUT_MASK, 2>(u, 4, plain(p0, 64), B, p1, nullptr, 0, u->e[3], st)));
  UN_TRY((wgrad<64, 64, 1, IN_SUB, false, 12>(u, 3, p1, plain(u->e[2], 64), B, st)));
  UN_TRY((conv_bwd<64, 64, 1, IN_PLAIN, OUT_F32, 2>(u, 3, plain(p1, 64), B, u->gs, nullptr, 64, nullptr, st)));
  // L3 (input S(e2))
  UN_TRY(skip_bwd(2, 64, p0));
  UN_TRY((wgrad<32, 64, 1, IN_SUB, false, 9>(u, 2, p0, plain(u->e[1], 32), B, st)));
  UN_TRY((conv_bwd<64, 32, 1, IN_PLAIN, OUT_F32, 2>(u, 2, plain(p0, 64), B, u->gs, nullptr, 32, nullptr, st)));
  // L2 (input S(e1))
  UN_TRY(skip_bwd(1, 32, p1));
  UN_TRY((wgrad<16, 32, 1, IN_SUB, false, 9>(u, 1, p1, plain(u->e[0], 16), B, st)));
  UN_TRY((conv_bwd<32, 16, 1, IN_PLAIN, OUT_F32, 9>(u, 1, plain(p1, 32), B, u->gs, nullptr, 16, nullptr, st)));
  // L1 (input f, log kappa)
  UN_TRY(skip_bwd(0, 16, p0));
  UN_TRY((wgrad<8, 16, 1, IN_PAIR, false, 5>(u, 0, p0, Input{u->xp, nullptr, 0, 8, 0}, B, st)));
  FB_CUDA(launch(k_grad_reduce, dim3(unsigned((u->nparam + GR_E - 1) / GR_E)), GR_E * GR_G, 0, st, net_map(u, B), u->grad, accumulate ? 1 : 0));
  FB_LAUNCHED(1);
  return FB_OK;
}

// Adam step on the FP32 masters with the stored gradients (step t >= 1 for the bias corrections),
// then the BF16 GEMM copies.
fb_status fb_unet_adam(fb_unet* u, float lr, float beta1, float beta2, float eps, int t, void* stream)
{
  if(!u || t < 1)
  {
    set_error("unet_adam: bad arguments");
    return FB_ERR_ARG;
  }
  cudaStream_t st = as_stream(stream);
  const float c1 = 1.f - std::pow(beta1, float(t)), c2 = 1.f - std::pow(beta2, float(t));
  FB_CUDA(launch(k_adam, dim3(unsigned((u->nparam + 255) / 256)), 256, 0, st, net_map(u, 0), u->param, u->grad, u->adam_m, u->adam_v, lr,
    beta1, beta2, eps, c1, c2));
  FB_LAUNCHED(1);
  u->weights_ready = true;
  return FB_OK;
}

// Mean squared error over n entries (DEVICE arrays): *loss (DEVICE double) = sum (y - t)^2 / n;
// grad (DEVICE, may be NULL) = 2 (y - t) / n.
fb_status fb_unet_mse(fb_unet* u, const float* y, const float* t, uint64_t n, float* grad, double* loss, void* stream)
{
  if(!u || !y || !t || !loss || n == 0)
  {
    set_error("unet_mse: bad arguments");
    return FB_ERR_ARG;
  }
  cudaStream_t st = as_stream(stream);
  const int nb = int(std::min<uint64_t>(1024, (n + MSE_NT - 1) / MSE_NT));
  FB_CUDA(launch(k_mse, dim3(nb), MSE_NT, 0, st, y, t, size_t(n), grad, RedSlot{u->mse_part, u->mse_counter}, loss));
  FB_LAUNCHED(1);
  return FB_OK;
}

} // extern "C"
