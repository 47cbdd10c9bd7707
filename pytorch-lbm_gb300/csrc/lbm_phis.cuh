// The phi pass of a state in source form, and the populations back from it.
//
// With tau_f == 1 (the reference's default tau_h) the post-collision phase-field
// populations of a node are a function of seven of its values: phi, u and the
// source vector S (FEval, lbm_kernels.cu).  Storing S instead of the 19
// populations takes 64 bytes per node (float; 26 in half storage) off the
// update kernel's stores and 48 (10) off the next phi pass's loads, and the
// populations are evaluated where they are summed.
//
// A block walks cx planes of x over a ty x tz tile of the (y, z) plane, two
// planes at a time, one thread per node of the tile and its one-node halo
// (periodic).  Per pair of planes (x, x + 1) each thread loads its two nodes'
// seven values (the next pair's loads are in flight meanwhile), evaluates the
// 19 populations of both as packed float pairs and puts the 16 that stream off
// the node's column into shared memory; after the barrier the threads of the
// tile's inner nodes complete the planes x - 1 and x: the e_x = +1 populations
// come from the pair before, the e_x = -1 ones from this pair, the e_x = 0 ones
// half from each (the second half is kept in registers).  Packed arithmetic
// (fma.rn.f32x2 and the like) halves the instructions, which bound the pass: one
// plane and scalar arithmetic per iteration ran at 71 us on the 150x150x107
// case against 51 us.
// The values and the order of their sum are those of the pass over stored
// populations (half storage: each value is rounded to the stored deviation on
// the way, as a store and a load would), so the two give the same bits.
// Included by lbm_kernels.cu.
#pragma once

namespace lbm {

// rows of float pairs in shared memory: the 4 e_x = +1 velocities of two pairs
// of planes, the 8 e_x = 0 and the 4 e_x = -1 ones of one (the column's own 0,
// 1, 2 stay in registers)
constexpr int kPhisRows = 4 * 2 + 8 + 4;
constexpr size_t kPhisShared = (size_t)kPhisRows * kPhisNT * sizeof(float2);

// Lets the phi pass's kernel use its shared memory, once per kernel and device
// (the attribute call costs about as much as a launch).
template <typename Kern>
static cudaError_t phis_shared(Kern fn) {
  static std::atomic<unsigned long long> done{0ull};  // one bit per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPhisShared);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

// Index of population q (3..18) among those of its e_x that go through shared memory.
__host__ __device__ constexpr int phis_row(int q) {
  int r = 0;
  for (int p = 3; p < q; ++p) r += ex(p) == ex(q) ? 1 : 0;
  return r;
}

// Packed pairs.  ptxas fuses a packed multiplication into a packed addition
// that takes its result (seen on the results of __fmul2_rn and __fadd2_rn, and
// of the .rn instructions themselves); a product that is added is therefore
// formed by two scalar multiplications (p2_prod), which it leaves alone.
__device__ __forceinline__ float2 p2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 p2_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 p2_sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 p2_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 p2_prod(float2 a, float b) { return make_float2(mul_rn(a.x, b), mul_rn(a.y, b)); }
__device__ __forceinline__ float2 p2_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// e_q.(a0, a1, a2) of the first velocity q of an opposite pair (edot)
__device__ __forceinline__ float2 p2_edot(int q, float2 a0, float2 a1, float2 a2) {
  const float2 v[3] = {a0, a1, a2};
  const int e[3] = {ex(q), ey(q), ez(q)};
  int i = e[0] != 0 ? 0 : (e[1] != 0 ? 1 : 2);       // first component, +1 or -1
  int j = i < 2 && e[2] != 0 ? 2 : (i < 1 && e[1] != 0 ? 1 : -1);  // second one, always +1
  if (j < 0) return v[i];
  return e[i] > 0 ? p2_add(v[i], v[j]) : p2_sub(v[j], v[i]);
}

// What is stored and read back of population v of velocity q (the identity
// unless the storage type is half).
template <typename S>
__device__ __forceinline__ float stored_f(const Consts<float>& k, int q, float v, float ref) {
  using IO = PopIO<float, S>;
  return IO::ld_f(IO::st_f(v, q, ref, k), q, ref, k);
}

// The populations of a node from phi, u and S, as the update kernel evaluates them.
template <typename S>
__device__ __forceinline__ void feval_all(const Consts<float>& k, float phi, const float (&u)[3], const float (&src)[3],
                                          float (&f)[Q]) {
  const float usq = fma_(u[2], u[2], fma_(u[1], u[1], mul_rn(u[0], u[0])));
  constexpr float it = Lat<float>::inv_two_cs2(), ic = Lat<float>::inv_cs2();
  const float ob = PopIO<float, S>::kDev ? fma_(-usq, it, 1.0f) : sub_rn(1.0f, mul_rn(usq, it));
  const float ux = mul_rn(u[0], ic), uy = mul_rn(u[1], ic), uz = mul_rn(u[2], ic);
  const FEval<float> fe(k, phi, ux, uy, uz, ob, src[0], src[1], src[2]);
  f[0] = fe.f0;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int q = pair_first(i);
    fe.pair(q, edot(q, ux, uy, uz), f[q], f[opp(q)]);
  }
}

// fetch_f of a fluid node of a state in source form (s.fin holds S): the value of
// each slot that node n reads, evaluated at the slot's node.  Linear layout.
template <typename S>
__device__ __forceinline__ void fetch_f_source(float (&v)[Q], const Consts<float>& k, const State<float, S>& s, int n,
                                               const Nbr& nb, uint8_t c, float eps) {
  constexpr bool DEV = PopIO<float, S>::kDev;
  const float* src = reinterpret_cast<const float*>(s.fin);
  const unsigned Np = (unsigned)k.Np;
  const float corr = s.cbuf[s.c_prev];
  // population q of node m, stored with the deviation reference ref and read back
  auto slot = [&](int q, unsigned m, float ref) {
    const float u[3] = {s.u[m], s.u[Np + m], s.u[2 * Np + m]}, sv[3] = {src[m], src[Np + m], src[2 * Np + m]};
    float f[Q];
    feval_all<S>(k, s.phi_in[m], u, sv, f);
    return DEV ? stored_f<S>(k, q, f[q], ref) : f[q];
  };
  const float ref_self = DEV ? s.phi_in[n] : 0.0f, one_m = sub_rn(1.0f, eps);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const unsigned m = (unsigned)nb.at(n, -ex(q), -ey(q), -ez(q));
    v[q] = slot(q, m, ref_self);
    // blended with the node's own opposite slot, whose reader is x - e_q
    if (c & kPartial) v[q] = fma_(one_m, v[q], mul_rn(eps, slot(opp(q), (unsigned)n, DEV ? s.phi_in[m] : 0.0f)));
    v[q] = mul_rn(v[q], corr);
  }
  relax_f<float, S, false>(v, k, s, n, c, corr);
}

template <typename S>
__device__ __forceinline__ void phis_block(const Consts<float>& k, const State<float, S>& s, const PhiTile& t, int b,
                                           int nblk, float2* sm) {
  constexpr bool DEV = PopIO<float, S>::kDev;
  const Pol pol = Pol::make();
  const int bt = b / t.ntz, bz = b - bt * t.ntz, bx = bt / t.nty, by = bt - bx * t.nty;
  const int x0 = bx * t.cx, x1 = min(x0 + t.cx, k.nx);
  const int y0 = by * t.ty, z0 = bz * t.tz;
  const int ey_ = min(t.ty, k.ny - y0), ez_ = min(t.tz, k.nz - z0), EZ = ez_ + 2;
  const int tid = threadIdx.x, ly = tid / EZ, lz = tid - ly * EZ;
  const bool act = ly < ey_ + 2;
  const bool inner = ly >= 1 && ly <= ey_ && lz >= 1 && lz <= ez_;
  int y = y0 - 1 + ly, z = z0 - 1 + lz;
  y = act ? (y < 0 ? y + k.ny : (y >= k.ny ? y - k.ny : y)) : 0;
  z = z < 0 ? z + k.nz : (z >= k.nz ? z - k.nz : z);
  const unsigned m = (unsigned)(y * k.nz + z), P = (unsigned)(k.ny * k.nz), Np = (unsigned)k.Np;
  const float* src = reinterpret_cast<const float*>(s.fin);
  const float corr = s.cbuf[s.c_prev];

  struct Nodes {  // of two planes
    float2 phi, u[3], s[3];
    uint8_t c0, c1;
  };
  auto wrap = [&](int x) { return (unsigned)(x < 0 ? x + k.nx : (x >= k.nx ? x - k.nx : x)); };
  auto load = [&](int x) {
    Nodes v;
    const unsigned n0 = wrap(x) * P + m, n1 = wrap(x + 1 > x1 ? x1 : x + 1) * P + m;
    v.phi = make_float2(ld_pol(s.phi_in + n0, pol.keep), ld_pol(s.phi_in + n1, pol.keep));
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      v.u[d] = make_float2(ld_pol(s.u + (d * Np + n0), pol.keep), ld_pol(s.u + (d * Np + n1), pol.keep));
      v.s[d] = make_float2(ld_pol(src + (d * Np + n0), pol.once), ld_pol(src + (d * Np + n1), pol.once));
    }
    v.c0 = s.cls[n0];
    v.c1 = s.cls[n1];
    return v;
  };
  float2* const sa = sm + tid;                  // e_x = +1: two rings of 4 rows
  float2* const sb = sm + 8 * kPhisNT + tid;    // e_x = 0: 8 rows
  float2* const sc = sm + 16 * kPhisNT + tid;   // e_x = -1: 4 rows

  TileSum<float> part;
  // carried from the pair before: f_0 of its second plane, f_1 of both, the
  // gathered e_x = 0 populations, phi and class of its second plane
  float f0_last = 0.0f, phi_last = 0.0f, b_last[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float2 f1_last = p2(0.0f);
  uint8_t c_last = 0;

  // plane x of this thread's column from its 19 streamed populations times corr
  // (already in w), their sum in velocity order
  auto finish = [&](int x, uint8_t c, float phi_prev, float sum, auto population) {
    float phi = 0.0f;
    const unsigned n = (unsigned)x * P + m;
    if (!(c & kSolid)) {
      phi = clamp01(sum);
      // a top-surface node is rescaled only where its corrected phi lies in the relaxation's range
      const float pb = clamp01(mul_rn(phi_prev, corr));
      const bool relaxed = k.relax_on && (c & kTop) && pb > 0.15f && pb < 0.85f;
      if (relaxed || (c & kPartial)) {
        // rare: blended with the node's own populations, or rescaled
        float w[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) w[q] = population(q);
        if (c & kPartial) {
          const float eps = s.eps[n], one_m = sub_rn(1.0f, eps);
          const float u[3] = {s.u[n], s.u[Np + n], s.u[2 * Np + n]}, sv[3] = {src[n], src[Np + n], src[2 * Np + n]};
          float o[Q];
          feval_all<S>(k, phi_prev, u, sv, o);
          if (DEV) {
            // each with the deviation reference of its reader x + e_q
            const Nbr nb = make_nbr_xyz(x, y, z, k.nx, k.ny, k.nz);
#pragma unroll
            for (int q = 0; q < Q; ++q)
              o[q] = stored_f<S>(k, q, o[q], ld_state(s.phi_in + nb.at((int)n, ex(q), ey(q), ez(q))));
          }
#pragma unroll
          for (int q = 0; q < Q; ++q) w[q] = fma_(one_m, w[q], mul_rn(eps, o[opp(q)]));
        }
        phi = phi_of<float, S, false>(k, s, (int)n, c, w, corr, phi_prev);
      }
    }
    st_pol(s.phi_out + n, phi, pol.keep);  // read back (stencil) by the update kernel
    part.add(phi);
  };

  Nodes nxt = load(x0 - 1);
  for (int x = x0 - 1, j = 0; x <= x1; x += 2, j ^= 1) {
    const Nodes v = nxt;
    if (x + 2 <= x1) nxt = load(x + 2);
    // the 19 populations of both nodes (FEval)
    float2 f0, f1, f2;
    {
      const float2 usq = p2_fma(v.u[2], v.u[2], p2_fma(v.u[1], v.u[1], p2_mul(v.u[0], v.u[0])));
      constexpr float it = Lat<float>::inv_two_cs2(), ic = Lat<float>::inv_cs2();
      const float2 ob = DEV ? p2_fma(usq, p2(-it), p2(1.0f)) : p2_sub(p2(1.0f), p2_prod(usq, it));
      const float2 ux = p2_prod(v.u[0], ic), uy = p2_prod(v.u[1], ic), uz = p2_prod(v.u[2], ic);
      const float2 wa_p = p2_mul(v.phi, p2(Lat<float>::w(1))), wd_p = p2_mul(v.phi, p2(Lat<float>::w(7)));
      const float2 wa_A = p2_mul(wa_p, ob), wd_A = p2_mul(wd_p, ob);
      const float2 wa_H = p2_mul(p2(0.5f), wa_p), wd_H = p2_mul(p2(0.5f), wd_p);
      const float2 ca = p2(k.wac3[1]), cd = p2(k.wac3[7]);
      f0 = p2_mul(p2_mul(v.phi, p2(Lat<float>::w(0))), ob);
      __syncthreads();  // the pair before has been read
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const int q = pair_first(i);
        const bool ax = i < 3;
        const float2 ec = p2_edot(q, ux, uy, uz), es = p2_edot(q, v.s[0], v.s[1], v.s[2]);
        const float2 e = p2_fma(p2_mul(ax ? wa_H : wd_H, ec), ec, ax ? wa_A : wd_A);
        const float2 o = p2_fma(ax ? wa_p : wd_p, ec, p2_mul(ax ? ca : cd, es));
        const float2 fq = p2_add(e, o), fp = p2_sub(e, o);
        auto put = [&](int r, float2 w) {
          if (r == 1) f1 = w;
          else if (r == 2) f2 = w;
          else if (ex(r) > 0) sa[(j * 4 + phis_row(r)) * kPhisNT] = w;
          else if (ex(r) == 0) sb[phis_row(r) * kPhisNT] = w;
          else sc[phis_row(r) * kPhisNT] = w;
        };
        put(q, fq);
        put(opp(q), fp);
      }
    }
    __syncthreads();
    if (inner) {
      // planes x - 1 and x, populations in velocity order
      const float2 ref = make_float2(phi_last, v.phi.x);
      float b_now[8];
      auto at = [&](int q) {
        const int off = -ey(q) * EZ - ez(q);
        if (q == 0) return make_float2(f0_last, f0.x);
        if (q == 1) return f1_last;
        if (q == 2) return f2;
        if (ex(q) > 0) return sa[((j ^ 1) * 4 + phis_row(q)) * kPhisNT + off];
        if (ex(q) < 0) return sc[phis_row(q) * kPhisNT + off];
        const float2 g = sb[phis_row(q) * kPhisNT + off];
        b_now[phis_row(q)] = g.y;
        return make_float2(b_last[phis_row(q)], g.x);
      };
      auto val = [&](int q) {
        const float2 w = at(q);
        return DEV ? make_float2(stored_f<S>(k, q, w.x, ref.x), stored_f<S>(k, q, w.y, ref.y)) : w;
      };
      float2 sum = p2_prod(val(0), corr);
#pragma unroll
      for (int q = 1; q < Q; ++q) sum = p2_add(sum, p2_prod(val(q), corr));
      if (x > x0) finish(x - 1, c_last, phi_last, sum.x, [&](int q) { return val(q).x; });
      if (x >= x0 && x < x1) finish(x, v.c0, v.phi.x, sum.y, [&](int q) { return val(q).y; });
#pragma unroll
      for (int i = 0; i < 8; ++i) b_last[i] = b_now[i];
    }
    f0_last = f0.y;
    f1_last = f1;
    phi_last = v.phi.y;
    c_last = v.c1;
  }
  phi_finish(s, part, b, nblk);
}

template <typename T, typename S>
__global__ void __launch_bounds__(kPhisNT, kPhisPerSm) k_phis_one(const __grid_constant__ CaseDesc<T, S> d) {
  extern __shared__ __align__(16) float2 phis_sm[];
  pdl_trigger();
  pdl_wait();  // S and u of the previous update kernel
  if (other_form(d.s)) return;
  phis_block<S>(d.k, d.s, d.tile, blockIdx.x, gridDim.x, phis_sm);
}

template <typename T, typename S>
__global__ void __launch_bounds__(kPhisNT, kPhisPerSm) k_phis_batch(const CaseDesc<T, S>* __restrict__ cases,
                                                           const unsigned short* __restrict__ blk2case) {
  extern __shared__ __align__(16) float2 phis_sm[];
  __shared__ CaseDesc<T, S> d;
  load_desc(d, cases + blk2case[blockIdx.x]);
  pdl_trigger();
  pdl_wait();
  phis_block<S>(d.k, d.s, d.tile, blockIdx.x - d.phs_blk0, d.tile.blocks(), phis_sm);
}

// Whether node n of class c does more than pull its f: solid and partial nodes, and
// top-surface ones whose corrected phi lies in the boundary-phi relaxation's range.
template <typename T, typename S>
__device__ __forceinline__ bool special_reader(const Consts<T>& k, const State<T, S>& s, unsigned n, uint8_t c, T corr) {
  if (c & (kSolid | kPartial)) return true;
  if (!(k.relax_on && (c & kTop))) return false;
  const T pb = clamp01(mul_rn(s.phi_in[n], corr));
  return pb > T(0.15) && pb < T(0.85);
}

// f of solid node n of a state in source form: its own opposite slots, whose readers
// are its neighbours.
template <typename T, typename S>
__device__ __forceinline__ void solid_f_source(T (&v)[Q], const Consts<T>& k, const State<T, S>& s, int n, const Nbr& nb,
                                               T corr) {
  const unsigned Np = (unsigned)k.Np;
  const T* src = reinterpret_cast<const T*>(s.fin);
  const T u[3] = {s.u[n], s.u[Np + n], s.u[2 * Np + n]}, sv[3] = {src[n], src[Np + n], src[2 * Np + n]};
  T f[Q];
  feval_all<S>(k, s.phi_in[n], u, sv, f);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (PopIO<T, S>::kDev) f[q] = stored_f<S>(k, q, f[q], s.phi_in[nb.at(n, ex(q), ey(q), ez(q))]);
    v[opp(q)] = mul_rn(f[q], corr);
  }
}

// f and g (may be null) of a state in source form as the reference holds them
// between steps, without writing anything of the state.  Below kReadSmall nodes
// every node evaluates the 19 values that it reads (k_read_small).  Above, a thread
// evaluates its node's f once and writes each value, corrected, to the slot of the
// node that pulls it, and pulls its g (k_read_source); f of the special readers follows
// from k_read_special, over what the first kernel wrote there: its blocks collect those of
// kSpecialRun nodes each (a wall puts one or two into most warps; a lookup of 18
// classes per node instead costs 35 us at 128x128x96) and do all but their stores
// before the first kernel has ended.
// us for f and g, float (half): 128x128x96 84 (86), by k_read_small 112 (130),
// k_expand and reading what it wrote 94; read-outs of stored populations take 78 (76),
// but the next step then reads them.  A step and a read-out of f and g there: 227 (230)
// against 261 (279) on stored populations; by k_read_small / the two kernels 24^3 20.4 /
// 22.7 (20.4 / 26.5), 48^3 26.7 / 28.7 (28.7 / 30.8), 60^3 39.1 / 37.7 (41.4 / 41.1).
constexpr int kSpecialRun = 8 * kBlock;
constexpr int kReadSmall = 200000;

template <typename T, typename S>
__global__ void __launch_bounds__(kBlock) k_read_special(Consts<T> k, State<T, S> s, T* f_o) {
  if (other_form(s)) {
    pdl_wait();
    return;
  }
  const int n0 = blockIdx.x * kSpecialRun;
  __shared__ unsigned short list[kSpecialRun];
  __shared__ int count;
  const T corr = s.cbuf[s.c_prev];
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  // eight classes per thread in one load (the array is padded with zeros to a multiple of 32)
  const int i0 = 8 * threadIdx.x;
  if (n0 + i0 < k.N) {
    const uint2 w = *reinterpret_cast<const uint2*>(s.cls + n0 + i0);
    for (int i = 0; i < 8; ++i) {
      const uint8_t c = (uint8_t)((i < 4 ? w.x : w.y) >> (8 * (i & 3)));
      if (n0 + i0 + i < k.N && special_reader(k, s, (unsigned)(n0 + i0 + i), c, corr))
        list[atomicAdd(&count, 1)] = (unsigned short)(i0 + i);
    }
  }
  __syncthreads();
  const unsigned N = (unsigned)k.N;
  for (int i = threadIdx.x; i < count || i < kBlock; i += kBlock) {
    T v[Q];
    int n = 0;
    if (i < count) {
      n = n0 + list[i];
      const uint8_t c = s.cls[n];
      int ix, iy, iz;
      decode(k.dz, k.dy, n, k.nz, k.ny, ix, iy, iz);
      const Nbr nb = make_nbr_xyz(ix, iy, iz, k.nx, k.ny, k.nz);
      if (c & kSolid) {
        solid_f_source(v, k, s, n, nb, corr);
      } else {
        fetch_f_source<S>(v, k, s, n, nb, c, (c & kPartial) ? s.eps[n] : T(0));
      }
    }
    if (i < kBlock) pdl_wait();  // all threads of the block, once
    if (i < count) {
#pragma unroll
      for (int q = 0; q < Q; ++q) f_o[q * N + n] = v[q];
    }
  }
}

template <typename T, typename S>
__global__ void __launch_bounds__(kBlock, 4) k_read_source(Consts<T> k, State<T, S> s, T* f_o, T* g_o) {
  pdl_trigger();
  if (other_form(s)) return;
  const int n = blockIdx.x * kBlock + threadIdx.x;
  if (n >= k.N) return;
  const unsigned N = (unsigned)k.N, Np = (unsigned)k.Np;
  int ix, iy, iz;
  decode(k.dz, k.dy, n, k.nz, k.ny, ix, iy, iz);
  const Nbr nb = make_nbr_xyz(ix, iy, iz, k.nx, k.ny, k.nz);
  {
    const T* src = reinterpret_cast<const T*>(s.fin);
    const T corr = s.cbuf[s.c_prev];
    const T u[3] = {s.u[n], s.u[Np + n], s.u[2 * Np + n]}, sv[3] = {src[n], src[Np + n], src[2 * Np + n]};
    T f[Q];
    feval_all<S>(k, s.phi_in[n], u, sv, f);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const unsigned m = (unsigned)nb.at(n, ex(q), ey(q), ez(q));
      const T v = PopIO<T, S>::kDev ? stored_f<S>(k, q, f[q], s.phi_in[m]) : f[q];
      f_o[q * N + m] = mul_rn(v, corr);
    }
  }
  if (g_o) {
    const uint8_t c = s.cls[n];
    T v[Q];
    fetch_pop<T, S, false, false, false>(v, k, s.gin, s.phi_in, n, (size_t)N, nb, c, (c & kPartial) ? s.eps[n] : T(0), T(1));
#pragma unroll
    for (int q = 0; q < Q; ++q) g_o[q * N + n] = v[q];
  }
}

template <typename T, typename S>
__global__ void __launch_bounds__(kBlock) k_read_small(Consts<T> k, State<T, S> s, T* f_o, T* g_o) {
  const int n = blockIdx.x * kBlock + threadIdx.x;
  if (n >= k.N || other_form(s)) return;
  const unsigned N = (unsigned)k.N;
  const uint8_t c = s.cls[n];
  int ix, iy, iz;
  decode(k.dz, k.dy, n, k.nz, k.ny, ix, iy, iz);
  const Nbr nb = make_nbr_xyz(ix, iy, iz, k.nx, k.ny, k.nz);
  const T eps = (c & kPartial) ? s.eps[n] : T(0);
  T v[Q];
  if (c & kSolid) solid_f_source(v, k, s, n, nb, s.cbuf[s.c_prev]);
  else fetch_f_source<S>(v, k, s, n, nb, c, eps);
#pragma unroll
  for (int q = 0; q < Q; ++q) f_o[q * N + n] = v[q];
  if (g_o) {
    fetch_pop<T, S, false, false, false>(v, k, s.gin, s.phi_in, n, (size_t)N, nb, c, eps, T(1));
#pragma unroll
    for (int q = 0; q < Q; ++q) g_o[q * N + n] = v[q];
  }
}

// The populations of a state in source form: s.fin holds S, s.phi_in the phi
// and s.u the velocity it belongs to; written to s.fout.
template <typename T, typename S>
__global__ void __launch_bounds__(kBlock) k_expand(Consts<T> k, State<T, S> s) {
  const int n = blockIdx.x * kBlock + threadIdx.x;
  if (n >= k.N || other_form(s)) return;
  using IO = PopIO<T, S>;
  const size_t Np = (size_t)k.Np;
  const T* src = reinterpret_cast<const T*>(s.fin);
  int ix, iy, iz;
  decode(k.dz, k.dy, n, k.nz, k.ny, ix, iy, iz);
  const Nbr nb = make_nbr_xyz(ix, iy, iz, k.nx, k.ny, k.nz);
  const T u[3] = {s.u[n], s.u[Np + n], s.u[2 * Np + n]}, sv[3] = {src[n], src[Np + n], src[2 * Np + n]};
  T f[Q];
  feval_all<S>(k, s.phi_in[n], u, sv, f);
#pragma unroll
  for (int q = 0; q < Q; ++q)
    s.fout[q * Np + n] = IO::st_f(f[q], q, IO::kDev ? s.phi_in[nb.at(n, ex(q), ey(q), ez(q))] : T(0), k);
}

}  // namespace lbm
