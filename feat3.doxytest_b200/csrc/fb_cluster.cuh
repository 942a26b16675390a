// The bottom of a V-cycle, and whole PCG solves of small systems, in one thread-block cluster.
//
// A level of a few thousand rows costs a launched pass 3-7 us whatever it computes: launch, cold
// instruction fetch, matrix values from L2 and a grid-wide reduction by arrival counter.  Here one
// cluster of CL_CS blocks (one per SM) keeps every level that fits in shared memory: the matrices'
// values and columns, the inverse diagonals, the masks and the vectors.  The rows of a level are
// dealt out in contiguous ranges to the blocks 0 .. CL_CS - 2; levels of at most CL_SMALL rows
// belong to the last block alone, which runs them with block barriers only.  A pass reads the vector
// entries of other blocks through distributed shared memory, and passes are separated by a barrier
// in the blocks' shared memory (ClBar).  What is left is latency: a pass is one or two rows' chain of
// shared or distributed loads per thread and a barrier, 0.5 us to 2 us; a whole solve of 2D FP64 level
// 5 (1,089 rows, 5 iterations) takes 205 us with host work, 370 us as launched passes, and level 7
// (16,641 rows, 6 iterations) 390 us against 556 us.  One short loop runs a list of passes written by the host: the code
// of a pass is fetched once per launch and reused, where the single-block tail's straight-line
// sequence waits for instruction fetch.
//
// Every row is computed in its stored entry order with separately rounded products and sums, the
// arithmetic of fb_rows.cuh, so a V-cycle is bitwise the grid kernels'.  Norms and dot products are
// per-warp partial sums that every block adds in the same order (deterministic, and the same value
// in every thread of the cluster, so all blocks take the same branches).
//
// Matrix data (the image) is staged by bulk copies before the programmatic-dependent-launch wait: no
// kernel of a solve writes it.
#pragma once

#include "fb_common.cuh"
#include "fb_rows.cuh"

namespace fb
{
  constexpr int CL_CS = 16;               // blocks of the cluster (non-portable size)
  // 12 warps: every barrier and every word of a pass costs issue slots per warp, and a level-7 FP64
  // block's 1,110 rows keep 384 threads busy three times (512 threads: 6% slower V-cycles)
  constexpr int CL_NT = 384;
  constexpr int CL_NW = CL_NT / 32;
  constexpr uint32_t CL_SMALL = 300;      // rows of a level one block runs alone
  constexpr uint32_t CL_ROWS = 4096;      // rows of a level per block at most (12-bit local index)
  constexpr int CL_PASSES = 73;           // twelve levels of V(2,2)
  constexpr uint32_t CL_NONE = 0xffffffffu;
  constexpr uint32_t CL_SMEM_MAX = 227 * 1024;
  constexpr uint32_t CL_COPY = 32768;     // bytes of one bulk copy

  enum : uint32_t
  {
    CLF_SMALL = 1,       // the last block's pass
    CLF_W = 2,           // the value is D .* u, otherwise u
    CLF_SKIP = 4,        // the smoother's skip test (latest norm) applies to the value
    CLF_SKIP_ZERO = 8,   // skipped rows store 0, otherwise a2 + 0
    CLF_NORM = 16,       // ||u|| is the latest norm
    CLF_COARSE = 32,     // the exact coarse solve
    CLF_SKIP_EXT = 64,   // the skip flag comes from the kernel before
    CLF_B = 128, CLF_A1 = 256, CLF_A2 = 512, CLF_OUT2 = 1024,   // the vector is there
    CLF_U9 = 2048,       // staged, a multiple of nine entries per row
    CLF_U4 = 4096,       // staged, a multiple of four entries per row
    CLF_LOCAL = 8192,    // every entry gathered lies in the block itself
    CLF_CLUSTER = 16384  // a cluster barrier ends the pass, otherwise the last block's own
  };

  // One pass over a level's rows: s = (M g)[i], u = F(b - s) or F(s + 0), w = F(D u),
  // v = u or w, v = a1 + v, skip test, out = a2 + v (or v), out2 = 0 + w.  Two 16-byte words, the
  // second read only by warps with rows: each costs the 12 warps of a block 48 cycles of shared-memory
  // issue.  Offsets in units of 16 bytes; those of absent vectors point at `out`.
  struct __align__(16) ClPass
  {
    uint16_t flags, k, n, rpc;            // entries per row; rows; rows per block
    uint16_t ns, dinv, dm, g;             // row stride of M's arrays; image offsets; gathered vector
    uint16_t val, code, b, a1;            // M's values and columns (image); vectors (shared memory)
    uint16_t a2, out, out2, pad;
  };

  struct __align__(16) ClParams
  {
    int npass, cs;
    int small_end;                        // the last block's last pass (it hands over to the others)
    uint32_t vec_base_img;                // shared-memory offset of the image (blocks 0 .. cs - 2)
    uint32_t vec_base_img_small;          // the same in the last block
    uint32_t staged, staged_small;        // image bytes staged in shared memory
    uint32_t img_stride;                  // image bytes per block in global memory
    const unsigned char* img;
    const uint32_t* free_dofs;            // coarse solve
    const double* inv;
    uint32_t m;
    // the top level of the cluster: rows, distribution, vectors b, x1 and the final iterate
    uint32_t n, rpc, vb, vx, vout;
    int top_small;
    uint32_t dinv, dm;
    // whole solves: the FP64 system matrix (image offsets), PCG vectors p, q, r (shared memory; in
    // FP64 r is the V-cycle's b and q its defect vector)
    uint32_t a64, acode, ans, ak, vp, vq, vr;
    ClPass pass[CL_PASSES];
  };

  // What the phases share through memory: the PCG's scalars, and what few instructions need.  In
  // registers they would be live across the V-cycle and leave its passes too few: a row's loads no longer
  // all in flight (twice the time per pass), or spills, whose stores every barrier's release then waits
  // for (1,000 cycles more per barrier; level 7 FP64, one solve: 470 -> 416 us without).
  struct ClState
  {
    double d0, dc, scale, gamma, gamma_prev, alpha, beta;
    const unsigned char* gimg;            // this block's image in global memory
    int* err;
    uint32_t staged, img;                 // bytes of it staged in shared memory, and where
    double* x;                            // whole solves: the iterate
    const Scalars* sc;
    int it, status;
  };

  // shared-memory map: parameters, PCG scalars, two arrays of partial sums, norm flags (two words of
  // this block's, two sets of one word per block), barriers, vectors and image from CL_VEC0 on
  constexpr uint32_t CL_STATE = (uint32_t(sizeof(ClParams)) + 15u) & ~15u;
  constexpr uint32_t CL_PART = (CL_STATE + uint32_t(sizeof(ClState)) + 15u) & ~15u;
  constexpr uint32_t CL_PARTS = CL_CS * CL_NW * 8u;
  constexpr uint32_t CL_FLAGS = CL_PART + 2u * CL_PARTS;
  constexpr uint32_t CL_FSET = CL_FLAGS + 16u;
  constexpr uint32_t CL_BAR = CL_FSET + 2u * CL_CS * 4u;   // staging barrier, two cluster barriers
  constexpr uint32_t CL_OK = CL_BAR + 24u;
  constexpr uint32_t CL_HUGE = CL_BAR + 28u;
  constexpr uint32_t CL_VEC0 = (CL_BAR + 32u + 127u) & ~127u;
  constexpr uint32_t CL_SPIN = 1u << 22;

  __device__ __forceinline__ void cl_sync()
  {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  __device__ __forceinline__ uint32_t cl_rank()
  {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
  }
  __device__ __forceinline__ uint32_t cl_smem(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

  // bounded wait for a phase of a shared-memory barrier, acquiring what was released to it in the cluster
  __device__ __forceinline__ bool cl_wait(uint32_t bar, uint32_t parity)
  {
    uint32_t done = 0;
    for(uint32_t k = 0; k < CL_SPIN && !done; ++k)
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                   "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
  }

  // The barrier between passes: each block arrives once at a shared-memory barrier of every block and
  // waits at its own.  (The hardware's cluster barrier takes an arrival from every thread: 800 to 900
  // cycles after the last block.)  Two barriers in turn: a block ahead can arrive at the next one, but
  // not at the one after, before all have left this one.  NORM: the block's flag word travels along
  // and all blocks' are returned.
  struct ClBar
  {
    // barriers passed; the top bit: a wait expired, no further ones (the error word is set)
    uint32_t n = 0;
    template<bool NORM>
    __device__ __forceinline__ uint32_t sync(unsigned char* sm, uint32_t me, uint32_t cs, uint32_t f, uint32_t turn)
    {
      volatile uint32_t* word = reinterpret_cast<volatile uint32_t*>(sm + CL_FLAGS + turn * 4u);
      if(NORM)
      {
        if(threadIdx.x == 0)
          *reinterpret_cast<volatile uint32_t*>(sm + CL_FLAGS + (turn ^ 1u) * 4u) = 0u;
        if(f & ~*word)
          atomicOr(const_cast<uint32_t*>(word), f);
      }
      __syncthreads();
      const uint32_t base = uint32_t(__cvta_generic_to_shared(sm));
      const uint32_t bar = base + CL_BAR + 8u + (n & 1u) * 8u, set = CL_FSET + (n & 1u) * (CL_CS * 4u);
      if(threadIdx.x < cs)
      {
        if(NORM)
          asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\tst.shared::cluster.u32 [r], %2;\n\t}"
                       :: "r"(base + set + me * 4u), "r"(threadIdx.x), "r"(*word) : "memory");
        asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\t"
                     "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [r];\n\t}"
                     :: "r"(bar), "r"(threadIdx.x) : "memory");
      }
      if(!(n >> 31) && !cl_wait(bar, (n >> 1) & 1u))
      {
        n |= 1u << 31;
        *reinterpret_cast<ClState*>(sm + CL_STATE)->err = 1;
      }
      ++n;
      if(!NORM)
        return 0u;
      const uint32_t lane = threadIdx.x & 31u;
      __syncwarp();
      return __reduce_or_sync(0xffffffffu, lane < cs ? *reinterpret_cast<volatile uint32_t*>(sm + set + lane * 4u) : 0u);
    }
  };

  // Entry `addr` (this block's shared address of it) in block `cta`.  One load whichever block that
  // is: a predicated pair (own block / other) serialises on the shared destination register and
  // measured 16% slower per V-cycle.
  __device__ __forceinline__ double cl_get(uint32_t addr, uint32_t cta, double)
  {
    double v;
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %1, %2;\n\tld.shared::cluster.f64 %0, [r];\n\t}"
                 : "=d"(v) : "r"(addr), "r"(cta));
    return v;
  }
  __device__ __forceinline__ float cl_get(uint32_t addr, uint32_t cta, float)
  {
    float v;
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %1, %2;\n\tld.shared::cluster.f32 %0, [r];\n\t}"
                 : "=f"(v) : "r"(addr), "r"(cta));
    return v;
  }

  __device__ __forceinline__ double cl_warp_sum(double v)
  {
    #pragma unroll
    for(int o = 16; o > 0; o >>= 1)
      v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;   // the same value in every lane: each step adds the two halves' sums
  }
  // this warp's sum to its slot of the partial sums in every block (cs <= 32)
  __device__ __forceinline__ void cl_put(uint32_t part, double v, uint32_t me, uint32_t cs)
  {
    v = cl_warp_sum(v);
    const uint32_t lane = threadIdx.x & 31u;
    if(lane < cs)
      asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\tst.shared::cluster.f64 [r], %2;\n\t}"
                   :: "r"(part + (me * CL_NW + (threadIdx.x >> 5)) * 8u), "r"(lane), "d"(v) : "memory");
    __syncwarp();
  }
  // sum of the partial sums [lo, lo + cnt), the same in every thread of every block
  __device__ __forceinline__ double cl_total(const volatile double* part, uint32_t lo, uint32_t cnt)
  {
    double s = 0.0;
    for(uint32_t j = threadIdx.x & 31u; j < cnt; j += 32u)
      s += part[lo + j];
    return cl_warp_sum(s);
  }

  // (M g)[i] in stored entry order: column code = block << 12 | local index
  template<typename V, typename X>
  __device__ __forceinline__ X cl_row(const V* __restrict__ val, const uint16_t* __restrict__ code, uint32_t ns,
    uint32_t K, uint32_t g)
  {
    constexpr uint32_t U = 9;
    X sum = X(0);
    for(uint32_t k0 = 0; k0 < K; k0 += U)
    {
      X v[U], x[U];
      uint32_t c[U];
      #pragma unroll
      for(uint32_t u = 0; u < U; ++u)
        if(k0 + u < K)
        {
          c[u] = code[(k0 + u) * ns];
          v[u] = X(to_acc(val[(k0 + u) * ns]));
        }
      #pragma unroll
      for(uint32_t u = 0; u < U; ++u)
        if(k0 + u < K)
          x[u] = cl_get(g + (c[u] & 0xfffu) * uint32_t(sizeof(X)), c[u] >> 12, X(0));
      #pragma unroll
      for(uint32_t u = 0; u < U; ++u)
        if(k0 + u < K)
          sum = add(sum, mul(v[u], x[u]));
    }
    return sum;
  }
  // U entries at a time, K a multiple of U; LOCAL: all in this block (`gv` the vector itself,
  // `mine` the block's code bits)
  template<typename V, typename X, int U, bool LOCAL>
  __device__ __forceinline__ X cl_rowu(const V* __restrict__ val, const uint16_t* __restrict__ code, uint32_t ns,
    uint32_t K, uint32_t g, const X* gv, uint32_t mine)
  {
    X sum = X(0);
    #pragma unroll 1
    for(uint32_t k = 0; k < K; k += U, val += U * ns, code += U * ns)
    {
      X v[U], x[U];
      uint32_t c[U];
      #pragma unroll
      for(int u = 0; u < U; ++u)
      {
        c[u] = code[uint32_t(u) * ns];
        v[u] = X(to_acc(val[uint32_t(u) * ns]));
      }
      // a warp whose rows' entries all lie in this block reads them as its own (three of four warps on
      // a level-7 band); a cluster load of an own entry takes the slower path all the same
      bool own = LOCAL;
      if(!LOCAL)
      {
        uint32_t far = 0;
        #pragma unroll
        for(int u = 0; u < U; ++u)
          far |= c[u] ^ mine;
        own = !__any_sync(__activemask(), far >> 12);
      }
      if(own)
      {
        #pragma unroll
        for(int u = 0; u < U; ++u)
          x[u] = gv[c[u] & 0xfffu];
      }
      else
      {
        #pragma unroll
        for(int u = 0; u < U; ++u)
          x[u] = cl_get(g + (c[u] & 0xfffu) * uint32_t(sizeof(X)), c[u] >> 12, X(0));
      }
      #pragma unroll
      for(int u = 0; u < U; ++u)
        sum = add(sum, mul(v[u], x[u]));
    }
    return sum;
  }

  // bounds of a defect entry that decide the skip test without the norm: one entry above CL_BIG
  // makes ||u|| > eps^2, and no entry above CL_HUGE keeps the sum of squares finite
  template<typename S> __device__ __forceinline__ S cl_big() { return S(2) * eps_sq<S>(); }
  __device__ __forceinline__ bool cl_huge(double u) { return !(fabs(u) <= 1e150); }
  __device__ __forceinline__ bool cl_huge(float u) { return !isfinite(u); }

  // The rows of one pass.  U: entries taken at a time from staged arrays (0: any row length, staged
  // or not).  Returns the norm flags of this thread's rows: 1 an entry above CL_BIG, 2 one above
  // CL_HUGE.
  template<typename V, typename S, int U, bool LOCAL>
  __device__ __forceinline__ uint32_t cl_rows(const uint4& d0, const uint4& d1, unsigned char* sm, uint32_t img,
    uint32_t nl, uint32_t me, bool skip)
  {
    const uint32_t fl = d0.x & 0xffffu, K = d0.x >> 16, ns = d0.z & 0xffffu;
    const S* dinv = reinterpret_cast<const S*>(sm + img + (d0.z >> 16) * 16u);
    const uint8_t* dm = sm + img + (d0.w & 0xffffu) * 16u;
    const uint32_t go = (d0.w >> 16) * 16u, vo_ = (d1.x & 0xffffu) * 16u, co_ = (d1.x >> 16) * 16u;
    const S* vb = reinterpret_cast<const S*>(sm + (d1.y & 0xffffu) * 16u);
    const S* v1 = reinterpret_cast<const S*>(sm + (d1.y >> 16) * 16u);
    const S* v2 = reinterpret_cast<const S*>(sm + (d1.z & 0xffffu) * 16u);
    S* vo = reinterpret_cast<S*>(sm + (d1.z >> 16) * 16u);
    S* vo2 = reinterpret_cast<S*>(sm + (d1.w & 0xffffu) * 16u);
    const uint32_t ga = cl_smem(sm) + go;
    const S* gv = reinterpret_cast<const S*>(sm + go);
    uint32_t f = 0;
    for(uint32_t i = threadIdx.x; i < nl; i += CL_NT)
    {
      // (the row's own entries: ahead of the sum in FP32, behind it in FP64, whose sum takes the registers)
      bool d;
      S di, bi, c1, c2;
      auto own_entries = [&]()
      {
        d = dm[i] != 0;
        di = dinv[i];
        bi = vb[i];
        c1 = v1[i];
        c2 = v2[i];
      };
      if(sizeof(S) == 4)
        own_entries();
      S s;
      if constexpr(U == 0)
      {
        const ClState& st = *reinterpret_cast<const ClState*>(sm + CL_STATE);
        s = cl_row<V, S>(reinterpret_cast<const V*>((vo_ < st.staged ? sm + img : st.gimg) + vo_) + i,
                         reinterpret_cast<const uint16_t*>((co_ < st.staged ? sm + img : st.gimg) + co_) + i, ns, K, ga);
      }
      else
        s = cl_rowu<V, S, U, LOCAL>(reinterpret_cast<const V*>(sm + img + vo_) + i,
                                    reinterpret_cast<const uint16_t*>(sm + img + co_) + i, ns, K, ga, gv, me << 12);
      if(sizeof(S) == 8)
        own_entries();
      const S u = d ? S(0) : ((fl & CLF_B) ? sub(bi, s) : add(s, S(0)));
      const S w = d ? S(0) : mul(di, u);
      S v = (fl & CLF_W) ? w : u;
      v = (fl & CLF_A1) ? add(c1, v) : v;
      v = skip ? S(0) : v;
      if((fl & CLF_A2) && !(skip && (fl & CLF_SKIP_ZERO)))
        v = add(c2, v);
      vo[i] = v;
      if(fl & CLF_OUT2)
        vo2[i] = add(S(0), w);
      f |= (fabs(u) > cl_big<S>() ? 1u : 0u) | (cl_huge(u) ? 2u : 0u);
    }
    return f;
  }

  // the last block's own passes run in its first CL_SW warps (CL_SMALL rows at most)
  constexpr int CL_SW = 10;
  static_assert(CL_SW * 32 >= int(CL_SMALL), "one row per thread");
  __device__ __forceinline__ void cl_small_sync() { asm volatile("bar.sync 1, 320;" ::: "memory"); }
  __device__ __forceinline__ bool cl_small_or(bool p)
  {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, 320, p;\n\t"
                 "selp.u32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"(uint32_t(p)) : "memory");
    return r != 0u;
  }

  // The passes of one V-cycle.  `ext`: the top level's skip flag.  Not inlined: inside the solve kernel
  // its loop would share registers with the calls around it and spill.
  template<typename V, typename S>
  __device__ __noinline__ ClBar cl_vcycle(bool ext, ClBar bar)
  {
    extern __shared__ __align__(128) unsigned char cl_sm[];
    unsigned char* const sm = cl_sm;
    const ClParams& cp = *reinterpret_cast<const ClParams*>(cl_sm);
    const uint32_t cs = uint32_t(cp.cs), me = cl_rank(), img = reinterpret_cast<const ClState*>(sm + CL_STATE)->img;
    const bool last = me == cs - 1u;
    double* part = reinterpret_cast<double*>(sm + CL_PART);
    const uint32_t base = cl_smem(sm);
    const int np = cp.npass;
    const uint32_t lane = threadIdx.x & 31u, w0 = threadIdx.x & ~31u;
    const bool small_warp = last && w0 < CL_SW * 32u;
    bool skip = false;          // the latest norm's skip flag
    uint32_t turn = 0;          // the flag word of the next norm
    if(threadIdx.x < 2u)
      *reinterpret_cast<volatile uint32_t*>(sm + CL_FLAGS + threadIdx.x * 4u) = 0u;
    const uint4* dp = reinterpret_cast<const uint4*>(cp.pass);
    uint4 d0 = dp[0];
    for(int pc = 0; pc < np; ++pc)
    {
      const uint4 d = d0;
      const uint32_t fl = d.x & 0xffffu, n = d.y & 0xffffu, rpc = d.y >> 16;
      const bool small = (fl & CLF_SMALL) != 0;
      if(small && !small_warp)
      {
        // the last block's passes: wait for its hand-over
        pc = cp.small_end;
        if(pc + 1 < np)
          d0 = dp[2 * (pc + 1)];
        bar.sync<false>(sm, me, cs, 0u, 0u);
        continue;
      }
      const uint32_t r0 = small ? 0u : me * rpc;
      const uint32_t nl = (small || !last) && r0 < n ? min(rpc, n - r0) : 0u;
      uint32_t f = 0, vout = 0;
      if(fl & CLF_COARSE)
      {
        // exact solve on the free DOFs (FP64 arithmetic whatever S is)
        const uint4 d1 = dp[2 * pc + 1];
        const S* b = reinterpret_cast<const S*>(sm + (d1.y & 0xffffu) * 16u);
        S* x = reinterpret_cast<S*>(sm + (d1.z >> 16) * 16u);
        if(threadIdx.x < n)
          x[threadIdx.x] = S(0);
        cl_small_sync();
        if(threadIdx.x < cp.m)
        {
          double s = 0.0;
          for(uint32_t j = 0; j < cp.m; ++j)
            s = add(s, mul(__ldg(cp.inv + size_t(threadIdx.x) * cp.m + j), double(b[__ldg(cp.free_dofs + j)])));
          x[__ldg(cp.free_dofs + threadIdx.x)] = S(s);
        }
      }
      else if(w0 < nl)
      {
        const uint4 d1 = dp[2 * pc + 1];
        vout = (d1.z >> 16) * 16u;
        const bool sk = (fl & CLF_SKIP_EXT) ? ext : ((fl & CLF_SKIP) ? skip : false);
        if(fl & CLF_U9)
          f = (fl & CLF_LOCAL) ? cl_rows<V, S, 9, true>(d, d1, sm, img, nl, me, sk)
                               : cl_rows<V, S, 9, false>(d, d1, sm, img, nl, me, sk);
        else if(fl & CLF_U4)
          f = (fl & CLF_LOCAL) ? cl_rows<V, S, 4, true>(d, d1, sm, img, nl, me, sk)
                               : cl_rows<V, S, 4, false>(d, d1, sm, img, nl, me, sk);
        else
          f = cl_rows<V, S, 0, false>(d, d1, sm, img, nl, me, sk);
      }
      // the next pass's word: its latency runs beside the barrier's
      if(pc + 1 < np)
        d0 = dp[2 * (pc + 1)];
      if(!(fl & CLF_NORM))
      {
        if(small && !(fl & CLF_CLUSTER))
          cl_small_sync();
        else
          bar.sync<false>(sm, me, cs, 0u, 0u);
      }
      else if(!small)
      {
        const uint32_t all = bar.sync<true>(sm, me, cs, f, turn);
        turn ^= 1u;
        const bool big = (all & 1u) != 0u, huge = (all & 2u) != 0u;
        skip = false;
        if(!big || huge)
        {
          // undecided (the same in every block): the norm itself
          vout = (dp[2 * pc + 1].z >> 16) * 16u;
          double sq = 0.0;
          const S* u = reinterpret_cast<const S*>(sm + vout);
          for(uint32_t i = threadIdx.x; i < nl; i += CL_NT)
            sq += double(u[i]) * double(u[i]);
          cl_put(base + CL_PART, sq, me, cs);
          bar.sync<false>(sm, me, cs, 0u, 0u);
          skip = skip_from_norm<S>(sqrt(cl_total(part, 0u, cs * CL_NW))) != 0;
          bar.sync<false>(sm, me, cs, 0u, 0u);
        }
      }
      else
      {
        if(f & 2u)
          *reinterpret_cast<volatile int*>(sm + CL_HUGE) = 1;
        const bool big = cl_small_or((f & 1u) != 0u);
        skip = false;
        if(!big || *reinterpret_cast<volatile int*>(sm + CL_HUGE))
        {
          vout = (dp[2 * pc + 1].z >> 16) * 16u;
          const S* u = reinterpret_cast<const S*>(sm + vout);
          const double sq = cl_warp_sum(threadIdx.x < n ? double(u[threadIdx.x]) * double(u[threadIdx.x]) : 0.0);
          if(lane == 0u)
            part[threadIdx.x >> 5] = sq;
          cl_small_sync();
          skip = skip_from_norm<S>(sqrt(cl_total(part, 0u, CL_SW))) != 0;
          if(threadIdx.x == 0)
            *reinterpret_cast<volatile int*>(sm + CL_HUGE) = 0;
          cl_small_sync();
        }
        if(fl & CLF_CLUSTER)
          bar.sync<false>(sm, me, cs, 0u, 0u);
      }
    }
    return bar;
  }

  // stages the image, copies the parameters; false when a staging wait expired anywhere in the
  // cluster (the error word is set and every block returns)
  template<class F>
  __device__ __forceinline__ bool cl_start(const ClParams* __restrict__ gp, unsigned char* sm, uint32_t me, uint32_t cs,
    uint32_t img_off, uint32_t staged, const unsigned char* gimg, int* err, F after_wait)
  {
    const uint32_t bar = cl_smem(sm) + CL_BAR;
    if(threadIdx.x == 0)
    {
      asm volatile("mbarrier.init.shared.b64 [%0], 1;" :: "r"(bar) : "memory");
      asm volatile("mbarrier.init.shared.b64 [%0], %1;" :: "r"(bar + 8u), "r"(cs) : "memory");
      asm volatile("mbarrier.init.shared.b64 [%0], %1;" :: "r"(bar + 16u), "r"(cs) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.shared.b64 t, [%0], %1;\n\t}"
                   :: "r"(bar), "r"(staged) : "memory");
      for(uint32_t o = 0; o < staged; o += CL_COPY)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     :: "r"(cl_smem(sm) + img_off + o), "l"(gimg + o), "r"(min(CL_COPY, staged - o)), "r"(bar)
                     : "memory");
    }
    {
      const uint32_t nw = uint32_t(offsetof(ClParams, pass) / 4) + uint32_t(gp->npass) * uint32_t(sizeof(ClPass) / 4);
      for(uint32_t k = threadIdx.x; k < nw; k += CL_NT)
        reinterpret_cast<uint32_t*>(sm)[k] = __ldg(reinterpret_cast<const uint32_t*>(gp) + k);
    }
    if(threadIdx.x == 0)
    {
      *reinterpret_cast<volatile int*>(sm + CL_HUGE) = 0;
      ClState& st = *reinterpret_cast<ClState*>(sm + CL_STATE);
      st.gimg = gimg;
      st.staged = staged;
      st.img = img_off;
      st.err = err;
    }
    __syncthreads();
    pdl_wait();
    if(!after_wait())
    {
      // the gate is closed (the same answer in every block): drain the copies and leave
      if(threadIdx.x == 0)
        for(int k = 0; k < 1 << 20; ++k)
        {
          uint32_t done;
          asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared.b64 p, [%1], 0;\n\t"
                       "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar) : "memory");
          if(done)
            break;
        }
      __syncthreads();
      return false;
    }
    uint32_t done = 0;
    for(int k = 0; k < 1 << 20 && !done; ++k)
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared.b64 p, [%1], 0;\n\t"
                   "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar) : "memory");
    const int ok = __syncthreads_and(done != 0);
    if(threadIdx.x == 0)
      *reinterpret_cast<volatile int*>(sm + CL_OK) = ok;
    cl_sync();
    int all = 1;
    for(uint32_t c = 0; c < cs; ++c)
    {
      int v;
      asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %1, %2;\n\tld.shared::cluster.s32 %0, [r];\n\t}"
                   : "=r"(v) : "r"(cl_smem(sm) + CL_OK), "r"(c));
      all &= v;
    }
    cl_sync();
    if(!all && threadIdx.x == 0 && me == 0)
      *err = 1;
    return all != 0;
  }

  // ---------------------------------------------------------------- the image
  // How a level's rows are dealt out: `last` = the block that holds them all, or CL_NONE
  struct ClMap
  {
    uint32_t n, rpc, last;
    __device__ __forceinline__ uint32_t owner(uint32_t i) const { return last == CL_NONE ? i / rpc : last; }
    __device__ __forceinline__ uint32_t local(uint32_t i) const { return last == CL_NONE ? i % rpc : i; }
  };
  // A matrix as the launched passes store it and where its rows go in the image: K entries per row at
  // stride ns, values at offset `val`, column codes at `code` (CL_NONE: values only)
  template<typename V>
  struct ClMat
  {
    DCsr<V> M;
    const uint32_t* mask;    // diagonal storage of more than K diagonals: each row's own ones, as bits
    ClMap rows, cols;
    uint32_t K, ns, val, code;
    unsigned char* img;
    uint32_t stride;
  };

  // entry k of row i, in stored order; slots past a row's entries hold 0 at the row's own column where there is
  // one, so that they do not make a warp's loads leave the block (at the level's first column: 2D level 7
  // FP64, one solve 416 us, against 390)
  template<typename V>
  __device__ __forceinline__ void cl_copy_entry(const ClMat<V>& m, uint32_t i, uint32_t k)
  {
    const uint32_t sl = i >> 5;
    unsigned char* base = m.img + size_t(m.rows.owner(i)) * m.stride;
    const size_t o = size_t(k) * m.ns + m.rows.local(i);
    const uint32_t b0 = m.M.kw ? sl * 32u * m.M.kw : m.M.soff[sl], w = m.M.kw ? m.M.kw : (m.M.soff[sl + 1] - b0) >> 5;
    const uint32_t u = m.mask ? __fns(m.mask[i], 0u, int(k) + 1) : k;
    V val{};
    uint32_t col = m.cols.n;
    if(u < w)
    {
      const uint32_t e = b0 + (i & 31u) + u * 32u;
      val = m.M.val[e];
      if(m.code != CL_NONE)
        col = m.M.doff ? uint32_t(int32_t(i) + m.M.doff[u])
                       : (m.M.dcol ? uint32_t(int32_t(i) + int32_t(m.M.dcol[e])) : m.M.col[e]);
    }
    reinterpret_cast<V*>(base + m.val)[o] = val;
    if(m.code == CL_NONE)
      return;
    if(col >= m.cols.n)
      col = i < m.cols.n ? i : 0u;
    reinterpret_cast<uint16_t*>(base + m.code)[o] = uint16_t(m.cols.owner(col) << 12 | m.cols.local(col));
  }

  // A matrix's rows into the image, and (dinv given) the level's inverse diagonal and mask; blockIdx.y = the
  // entry within the row
  template<typename V, typename S>
  __global__ void __launch_bounds__(256) k_cl_image(const ClMat<V> m, const S* __restrict__ dinv,
    const uint8_t* __restrict__ dm, uint32_t odinv, uint32_t odm)
  {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if(i >= m.rows.n)
      return;
    cl_copy_entry(m, i, blockIdx.y);
    if(!dinv || blockIdx.y)
      return;
    unsigned char* base = m.img + size_t(m.rows.owner(i)) * m.stride;
    reinterpret_cast<S*>(base + odinv)[m.rows.local(i)] = dinv[i];
    base[odm + m.rows.local(i)] = dm[i];
  }

  // The V-cycle below the launched levels: b and sol1 of the cluster's top level come from the
  // restriction before, its iterate goes back to global memory.
  template<typename V, typename S>
  __global__ void __launch_bounds__(CL_NT, 1) k_cl_bottom(const ClParams* __restrict__ gp, const S* __restrict__ gb,
    const S* __restrict__ gx, S* __restrict__ gout, const int* __restrict__ skip_pre, const Scalars* __restrict__ sc,
    int* err)
  {
    extern __shared__ __align__(128) unsigned char cl_sm[];
    const uint32_t me = cl_rank();
    const uint32_t cs = uint32_t(gp->cs);
    const bool last = me == cs - 1u;
    const uint32_t img_off = last ? gp->vec_base_img_small : gp->vec_base_img;
    const uint32_t staged = last ? gp->staged_small : gp->staged;
    const unsigned char* gimg = gp->img + size_t(me) * gp->img_stride;
    const ClParams& cp = *reinterpret_cast<const ClParams*>(cl_sm);
    bool ext = false;
    uint32_t r0 = 0, nl = 0;
    if(!cl_start(gp, cl_sm, me, cs, img_off, staged, gimg, err, [&]
       {
         if(gate_closed(sc))
           return false;
         ext = *(volatile const int*)skip_pre != 0;
         if(cp.top_small ? last : !last)
         {
           r0 = cp.top_small ? 0u : me * cp.rpc;
           nl = r0 < cp.n ? min(cp.rpc, cp.n - r0) : 0u;
           S* b = reinterpret_cast<S*>(cl_sm + cp.vb);
           S* x = reinterpret_cast<S*>(cl_sm + cp.vx);
           for(uint32_t i = threadIdx.x; i < nl; i += CL_NT)
           {
             b[i] = gb[r0 + i];
             x[i] = gx[r0 + i];
           }
         }
         return true;
       }))
      return;
    cl_vcycle<V, S>(ext, ClBar());
    const S* o = reinterpret_cast<const S*>(cl_sm + cp.vout);
    for(uint32_t i = threadIdx.x; i < nl; i += CL_NT)
      gout[r0 + i] = o[i];
    cl_sync();   // no block leaves while another may still read its vectors or arrive at its barriers
  }

  // What the PCG's phases work on, from the shared parameters
  template<typename V, typename S>
  struct ClPcg
  {
    static constexpr bool F64 = sizeof(S) == 8;
    unsigned char* sm;
    const ClParams& cp;
    volatile ClState& st;
    uint32_t me, cs, img, plo, pcnt, r0, nl, base;
    bool mine;
    S *vb, *vx1;
    const S* vz;
    double *vp, *vq, *vr;                 // in FP64 r is the V-cycle's input vb
    const S* dinv;
    const uint8_t* dm;
    const double *a64, *part;
    const uint16_t* acode;

    __device__ __forceinline__ explicit ClPcg(unsigned char* s)
      : sm(s), cp(*reinterpret_cast<const ClParams*>(s)), st(*reinterpret_cast<volatile ClState*>(s + CL_STATE)), me(cl_rank()),
        cs(uint32_t(cp.cs)), img(st.img)
    {
      const bool last = me == cs - 1u;
      plo = cp.top_small ? (cs - 1u) * CL_NW : 0u;
      pcnt = cp.top_small ? uint32_t(CL_NW) : (cs - 1u) * CL_NW;
      mine = cp.top_small ? last : !last;
      r0 = cp.top_small ? 0u : me * cp.rpc;
      nl = mine && r0 < cp.n ? min(cp.rpc, cp.n - r0) : 0u;
      base = cl_smem(s);
      vb = reinterpret_cast<S*>(s + cp.vb);
      vx1 = reinterpret_cast<S*>(s + cp.vx);
      vz = reinterpret_cast<const S*>(s + cp.vout);
      vp = reinterpret_cast<double*>(s + cp.vp);
      vq = reinterpret_cast<double*>(s + cp.vq);
      vr = reinterpret_cast<double*>(s + cp.vr);
      dinv = reinterpret_cast<const S*>(s + img + cp.dinv);
      dm = s + img + cp.dm;
      a64 = reinterpret_cast<const double*>((cp.a64 < st.staged ? s + img : st.gimg) + cp.a64);
      acode = reinterpret_cast<const uint16_t*>(s + img + cp.acode);
      part = reinterpret_cast<const double*>(s + CL_PART);
    }
    // (A p)[i]
    __device__ __forceinline__ double product(uint32_t i) const
    {
      if(F64 && cp.ak % 9u == 0u)
        return cl_rowu<double, double, 9, false>(reinterpret_cast<const double*>(sm + img + cp.a64) + i, acode + i, cp.ans,
                                                 cp.ak, base + cp.vp, vp, me << 12);
      return cl_row<double, double>(a64 + i, acode + i, cp.ans, cp.ak, base + cp.vp);
    }
    // the next V-cycle's input from the defect rv: b = S(rv scale), sol1 = F(D .* b)
    __device__ __forceinline__ void input(uint32_t i, double rv, double scale) const
    {
      const S b = F64 ? S(rv) : S(mul(rv, scale));
      vb[i] = b;
      const S c = dm[i] ? S(0) : mul(dinv[i], b);
      vx1[i] = add(S(0), c);
      if(!F64)
        vr[i] = rv;
    }
  };

  // r = F(rhs - A x), ||r||, the first V-cycle's input (iterative.hpp:748-771)
  template<typename V, typename S>
  __device__ __noinline__ ClBar cl_pcg_init(const double* rhs, ClBar bar)
  {
    extern __shared__ __align__(128) unsigned char cl_sm[];
    const ClPcg<V, S> w(cl_sm);
    const uint32_t me = w.me;
    const double* gx = w.st.x;
    for(uint32_t i = threadIdx.x; i < w.nl; i += CL_NT)
      w.vp[i] = gx[w.r0 + i];
    bar.sync<false>(cl_sm, me, w.cs, 0u, 0u);
    double sq = 0.0;
    for(uint32_t i = threadIdx.x; i < w.nl; i += CL_NT)
    {
      const double b = rhs[w.r0 + i];
      const double s = w.product(i);
      const double rv = w.dm[i] ? 0.0 : sub(b, s);
      sq += mul(rv, rv);
      if(w.F64)
        w.input(i, rv, 1.0);
      else
        w.vr[i] = rv;
    }
    if(w.mine)
      cl_put(w.base + CL_PART, sq, me, w.cs);
    bar.sync<false>(cl_sm, me, w.cs, 0u, 0u);
    const double d0 = sqrt(cl_total(w.part, w.plo, w.pcnt));
    int status = FB_SOLVER_PROGRESS;
    if(!isfinite(d0))
      status = FB_SOLVER_ABORTED;
    else if(d0 <= EPS64 * EPS64)
      status = FB_SOLVER_SUCCESS;
    double scale = 1.0;
    if(!w.F64 && status == FB_SOLVER_PROGRESS)
    {
      scale = pow2_near_inverse(d0);
      for(uint32_t i = threadIdx.x; i < w.nl; i += CL_NT)
        w.input(i, w.vr[i], scale);
    }
    if(threadIdx.x == 0)
    {
      w.st.d0 = d0;
      w.st.dc = d0;
      w.st.scale = scale;
      w.st.gamma = 0.0;
      w.st.gamma_prev = 0.0;
      w.st.alpha = 0.0;
      w.st.beta = 0.0;
      w.st.it = 0;
      w.st.status = status;
    }
    // every block has read the partial sums and p before the next pass writes them
    bar.sync<false>(cl_sm, me, w.cs, 0u, 0u);
    return bar;
  }

  // The PCG iteration after the V-cycle, up to the next V-cycle's input
  template<typename V, typename S>
  __device__ __noinline__ ClBar cl_pcg_step(ClBar bar)
  {
    extern __shared__ __align__(128) unsigned char cl_sm[];
    const ClPcg<V, S> w(cl_sm);
    const uint32_t me = w.me;
    double* gx = w.st.x;
    // z = x_top / scale (FP64), r.z -> beta; p = z + beta p
    const int it = w.st.it;
    const double dc0 = w.st.dc, gamma_prev = w.st.gamma, inv_scale = 1.0 / w.st.scale;
    double rz = 0.0;
    for(uint32_t i = threadIdx.x; i < w.nl; i += CL_NT)
      rz += mul(w.vr[i], mul(double(w.vz[i]), inv_scale));
    if(w.mine)
      cl_put(w.base + CL_PART, rz, me, w.cs);
    bar.sync<false>(cl_sm, me, w.cs, 0u, 0u);
    const double gamma = cl_total(w.part, w.plo, w.pcnt);
    const double beta = gamma / gamma_prev;
    for(uint32_t i = threadIdx.x; i < w.nl; i += CL_NT)
    {
      const double z = mul(double(w.vz[i]), inv_scale);
      w.vp[i] = it == 0 ? z : add(mul(w.vp[i], beta), z);
    }
    bar.sync<false>(cl_sm, me, w.cs, 0u, 0u);
    // q = F(A p), q.p -> alpha
    double qp = 0.0;
    for(uint32_t i = threadIdx.x; i < w.nl; i += CL_NT)
    {
      const double s = w.product(i);
      const double qv = w.dm[i] ? 0.0 : add(s, 0.0);
      w.vq[i] = qv;
      qp += mul(qv, w.vp[i]);
    }
    if(w.mine)
      cl_put(w.base + CL_PART + CL_PARTS, qp, me, w.cs);
    bar.sync<false>(cl_sm, me, w.cs, 0u, 0u);
    const double alpha = gamma / cl_total(w.part + CL_PARTS / 8u, w.plo, w.pcnt);
    // x += alpha p; r -= alpha q; ||r||; the next V-cycle's input
    const double nscale = w.F64 ? 1.0 : pow2_near_inverse(dc0);
    double rr = 0.0;
    for(uint32_t i = threadIdx.x; i < w.nl; i += CL_NT)
    {
      const double xo = gx[w.r0 + i];
      const double rn = add(w.vr[i], mul(-alpha, w.vq[i]));
      w.input(i, rn, nscale);
      rr += mul(rn, rn);
      gx[w.r0 + i] = add(xo, mul(alpha, w.vp[i]));
    }
    if(w.mine)
      cl_put(w.base + CL_PART, rr, me, w.cs);   // (every block has read r.z: barriers lie between)
    bar.sync<false>(cl_sm, me, w.cs, 0u, 0u);
    const double dc = sqrt(cl_total(w.part, w.plo, w.pcnt));
    if(threadIdx.x == 0)
    {
      const double d0 = w.st.d0;
      const Scalars* sc = w.st.sc;
      int status = FB_SOLVER_PROGRESS;
      if(!isfinite(dc))
        status = FB_SOLVER_ABORTED;
      else if(dc > sc->div_abs || dc > sc->div_rel * d0)
        status = FB_SOLVER_DIVERGED;
      else if(it + 1 < sc->min_iter)
        status = FB_SOLVER_PROGRESS;
      else if(dc <= sc->tol_abs && (dc <= sc->tol_rel * d0 || dc <= 0.0))
        status = FB_SOLVER_SUCCESS;
      else if(it + 1 >= sc->max_iter)
        status = FB_SOLVER_MAX_ITER;
      w.st.dc = dc;
      w.st.scale = nscale;
      w.st.gamma = gamma;
      w.st.gamma_prev = gamma_prev;
      w.st.alpha = alpha;
      w.st.beta = beta;
      w.st.it = it + 1;
      w.st.status = status;
    }
    __syncthreads();
    return bar;
  }

  // A whole PCG solve (kernel/solver/pcg.hpp:159-286): x is the initial guess and the result; the
  // scalars go to *sc as the launched passes leave them.
  template<typename V, typename S>
  __global__ void __launch_bounds__(CL_NT, 1) k_cl_solve(const ClParams* __restrict__ gp, double* gx,
    const double* rhs, Scalars* sc, int* err)
  {
    extern __shared__ __align__(128) unsigned char cl_sm[];
    const uint32_t me = cl_rank();
    const uint32_t cs = uint32_t(gp->cs);
    const bool last = me == cs - 1u;
    const uint32_t img = last ? gp->vec_base_img_small : gp->vec_base_img;
    const uint32_t staged = last ? gp->staged_small : gp->staged;
    const unsigned char* gimg = gp->img + size_t(me) * gp->img_stride;
    if(!cl_start(gp, cl_sm, me, cs, img, staged, gimg, err, [] { return true; }))
      return;
    volatile ClState& st = *reinterpret_cast<volatile ClState*>(cl_sm + CL_STATE);
    if(threadIdx.x == 0)
    {
      st.x = gx;
      st.sc = sc;
    }
    __syncthreads();
    ClBar bar = cl_pcg_init<V, S>(rhs, ClBar());
    while(st.status == FB_SOLVER_PROGRESS)
    {
      bar = cl_vcycle<V, S>(skip_from_norm<S>(st.dc * st.scale) != 0, bar);
      bar = cl_pcg_step<V, S>(bar);
    }
    cl_sync();   // no block leaves while another may still arrive at its barriers; all have read *sc
    if(threadIdx.x == 0 && me == 0u)
    {
      sc->gamma = st.gamma;
      sc->gamma_prev = st.gamma_prev;
      sc->alpha = st.alpha;
      sc->beta = st.beta;
      sc->def_init = st.d0;
      sc->def_cur = st.dc;
      sc->mg_scale = st.scale;
      sc->mg_inv_scale = 1.0 / st.scale;
      sc->iter = st.it;
      sc->status = st.status;
    }
  }
} // namespace fb
