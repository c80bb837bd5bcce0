// field_engine.cuh -- swap trials of fcc/bcc chains whose sites' fields fit in
// shared memory.
//
// Field.  For every site i and species s the fixed-point energy that an atom
// of species s would have there,
//   h(i, s) = sum over i's entries (dx, dy, dz, shell) of F(s, shell, species
//             at i + (dx, dy, dz)),
// kept relative to species 1 (g(i, s) = h(i, s) - h(i, 1), s = 2..ns).  The
// energy change of swapping sites a and b of species sa and sb is then
//   g(a, sb) - g(a, sa) + g(b, sa) - g(b, sb)
// plus, when the two are neighbours, a constant of their displacement and
// species: four loads instead of the 2z neighbours' species and tables.  An
// accepted swap updates the g of the 2z sites that have a or b as a
// neighbour.  Most evaluated trials are rejected, so the loads saved far
// outnumber the updates.  The sums are the fast tier's own integers (each term
// once, added in another order), so every decision is the one the gathered sum
// gives.
#pragma once

#include "halo_engine.cuh"
#include "kernels.cuh"

namespace brawl {

// A position's static record (the trial that would start there):
//   A  index of site 1, of site 2; byte address of the neighbours' constants
//      of its displacement class; the caller's, from the acceptance word
//   B  coordinates of site 1, of site 2 (x | y << 10 | z << 20); the caller's,
//      from the acceptance word; whether a site may have both as neighbours
// Four warps make them, a window each of a part of four; two parts are held.
constexpr int kFieldMakers = 4;
constexpr int kFieldPart = kFieldMakers * kWin, kFieldRing = 2 * kFieldPart;
// Words generated before the first part, and ahead of the stream at most (the
// stream in a part, the next one made, the words of one more).
constexpr int kFieldAhead = 5 * kWin;
using FieldWords = StreamRing<kFieldAhead + 2 * kFieldPart>;

// Shared memory of a chain with fields: the stream's rings, the records, then
// V, the update table U, the neighbours' constants C, W and F, the entries,
// the axis tables, the displacement classes, the exact tier's codes, the
// fields and the compact lattice.
struct FieldLayout {
  static constexpr uint32_t kA = FieldWords::kWords * 4;
  static constexpr uint32_t kB = kA + kFieldRing * 16;
  static constexpr uint32_t kV = kB + kFieldRing * 16;
  uint32_t U, C, W, F, ents, tabs[3], sstart, dtab, codes, g, lat, total;
};
static_assert(FieldLayout::kA % 16 == 0 && FieldLayout::kV % 16 == 0, "16-byte records, tables of doubles");

// Fields a site keeps: ns - 1, three padded to four so that a site's are read
// and written as one vector.
__host__ __device__ __forceinline__ int field_stride(int ns) { return ns == 4 ? 4 : ns - 1; }

// The kernel's variant: one, two or four fields a site as a vector, or 0.
__host__ __device__ __forceinline__ int field_variant(int ns) {
  const int r = field_stride(ns);
  return r == 1 || r == 2 || r == 4 ? r : 0;
}

__host__ __device__ inline FieldLayout field_layout(const Geom& g, const FieldGeom& f) {
  FieldLayout L;
  const uint32_t ns = (uint32_t)g.ns, r = (uint32_t)field_stride(g.ns), nsh = (uint32_t)g.nsh;
  L.U = align_up(FieldLayout::kV + ns * ns * nsh * 8, 16);
  L.C = L.U + ns * ns * nsh * r * 4;
  L.W = L.C + (uint32_t)f.n_class * ns * ns * 4;
  L.F = L.W + nsh * ns * r * 4;
  L.ents = L.F + (ns + 1) * nsh * (ns + 1) * 4;
  L.tabs[0] = L.ents + (uint32_t)g.z * 4;
  L.tabs[1] = L.tabs[0] + (2 * (uint32_t)g.n1 + 2 * kHalo) * 4;
  L.tabs[2] = L.tabs[1] + (2 * (uint32_t)g.n2 + 2 * kHalo) * 4;
  L.sstart = L.tabs[2] + (2 * (uint32_t)g.n3 + 2 * kHalo) * 4;
  L.dtab = L.sstart + (nsh + 1) * 2;
  L.codes = L.dtab + (uint32_t)(f.side[0] * f.side[1] * f.side[2]);
  L.g = align_up(L.codes + 2u * (uint32_t)g.z, 16);
  L.lat = align_up(L.g + (uint32_t)g.n_sites * r * 4, 16);
  L.total = align_up(L.lat + (uint32_t)g.n_sites, 16);
  return L;
}

// Tables, lattice (4 (species - 1) a site: a byte offset into rows by species)
// and fields from the job, by all the block's threads.  Ends with a
// __syncthreads.
__device__ inline void field_stage(const ChainJob& J, const Geom& g, const FieldLayout& L, unsigned char* smem, int tid,
                                   int nt) {
  const int ns = g.ns, nsp = ns + 1, r = field_stride(ns), nsh = g.nsh;
  double* V = reinterpret_cast<double*>(smem + FieldLayout::kV);
  int32_t* U = reinterpret_cast<int32_t*>(smem + L.U);
  int32_t* C = reinterpret_cast<int32_t*>(smem + L.C);
  int32_t* W = reinterpret_cast<int32_t*>(smem + L.W);
  int32_t* F = reinterpret_cast<int32_t*>(smem + L.F);
  uint32_t* ents = reinterpret_cast<uint32_t*>(smem + L.ents);
  int16_t* sstart = reinterpret_cast<int16_t*>(smem + L.sstart);
  uint8_t* dtab = smem + L.dtab;
  int32_t* G = reinterpret_cast<int32_t*>(smem + L.g);
  uint8_t* lat = smem + L.lat;
  const FieldGeom& f = J.fg;
  for (int i = tid; i < ns * ns * nsh; i += nt) V[i] = J.V[i];
  for (int i = tid; i < nsp * nsh * nsp; i += nt) F[i] = J.F[i];
  for (int i = tid; i < g.z; i += nt) ents[i] = J.entries[i];
  for (int i = tid; i <= nsh; i += nt) sstart[i] = J.shell_start[i];
  const int cells = f.side[0] * f.side[1] * f.side[2];
  for (int i = tid; i < cells; i += nt) dtab[i] = f.dtab[i];
  for (int a = 0; a < 3; ++a) {
    // wrapping axis tables: coordinate t - kHalo to its part of the compact index
    int32_t* tab = reinterpret_cast<int32_t*>(smem + L.tabs[a]);
    const int Wp = a == 0 ? 2 * g.n1 : a == 1 ? 2 * g.n2 : 2 * g.n3;
    for (int i = tid; i < Wp + 2 * kHalo; i += nt) {
      int w = (i - kHalo) % Wp;
      w += w < 0 ? Wp : 0;
      tab[i] = a == 0 ? w >> g.xs : a == 1 ? (w >> g.ys) * g.sy : w * g.sz;
    }
  }
  {
    // 4 (species - 1) a site, four sites at a time
    const int n4 = g.n_sites >> 2;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(J.lat);
    uint32_t* dst = reinterpret_cast<uint32_t*>(smem + L.lat);
    for (int i = tid; i < n4; i += nt) dst[i] = (src[i] - 0x01010101u) << 2;
    for (int i = (n4 << 2) + tid; i < g.n_sites; i += nt) lat[i] = (uint8_t)((J.lat[i] - 1) << 2);
  }
  __syncthreads();
  auto Fv = [&](int a, int sh, int b) { return F[(a * nsh + sh) * nsp + b]; };
  // W[sh][s - 1][s2 - 2]: a neighbour of species s in shell sh, to g(., s2)
  for (int i = tid; i < nsh * ns * r; i += nt) {
    const int s2 = i % r + 2, s = (i / r) % ns + 1, sh = i / (r * ns);
    W[i] = s2 <= ns ? Fv(s2, sh, s) - Fv(1, sh, s) : 0;
  }
  // U[old - 1][new - 1][sh][s2 - 2]: a neighbour changing from old to new
  for (int i = tid; i < ns * ns * nsh * r; i += nt) {
    const int s2 = i % r + 2, sh = (i / r) % nsh, sn = (i / (r * nsh)) % ns + 1, so = i / (r * nsh * ns) + 1;
    U[i] = s2 <= ns ? (Fv(s2, sh, sn) - Fv(1, sh, sn)) - (Fv(s2, sh, so) - Fv(1, sh, so)) : 0;
  }
  // C[class][sa - 1][sb - 1]: an entry that meets the other site finds our old
  // species there after the swap, not the other site's own
  for (int i = tid; i < f.n_class * ns * ns; i += nt) {
    const int sb = i % ns + 1, sa = (i / ns) % ns + 1, c = i / (ns * ns);
    int v = 0;
    for (int sh = 0; sh < nsh; ++sh) {
      const int na = f.sig[(c * nsh + sh) * 2], nb = f.sig[(c * nsh + sh) * 2 + 1];
      if (na) v += na * (Fv(sb, sh, sa) - Fv(sb, sh, sb));
      if (nb) v += nb * (Fv(sa, sh, sb) - Fv(sa, sh, sa));
    }
    C[i] = v;
  }
  __syncthreads();
  // The fields: per shell the neighbours are counted by species (six bits each,
  // a shell has at most 48; five species at a time), then weighted.
  const unsigned char* tx = smem + L.tabs[0] + kHalo * 4;
  const unsigned char* ty = smem + L.tabs[1] + kHalo * 4;
  const unsigned char* tz = smem + L.tabs[2] + kHalo * 4;
  for (int i = tid; i < g.n_sites; i += nt) {
    int x, y, z;
    decode_site(g, i, x, y, z);
    const unsigned char *bx = tx + 4 * x, *by = ty + 4 * y, *bz = tz + 4 * z;
    for (int sh = 0; sh < nsh; ++sh) {
      const int k0 = sstart[sh], k1 = sstart[sh + 1];
      for (int s0 = 0; s0 < ns; s0 += 5) {
        unsigned n5 = 0;
        auto count = [&](int k) {
          const uint32_t e = ents[k];
          const int dx = (int)(e << 24) >> 24, dy = (int)(e << 16) >> 24, dz = (int)(e << 8) >> 24;
          const int at = *reinterpret_cast<const int32_t*>(bx + 4 * dx) + *reinterpret_cast<const int32_t*>(by + 4 * dy) +
                         *reinterpret_cast<const int32_t*>(bz + 4 * dz);
          const unsigned s = (unsigned)((lat[at] >> 2) - s0);
          return s < 5u ? 1u << (6u * s) : 0u;
        };
        int k = k0;
        for (; k + 6 <= k1; k += 6) {
          unsigned c[6];
#pragma unroll
          for (int u = 0; u < 6; ++u) c[u] = count(k + u);
#pragma unroll
          for (int u = 0; u < 6; ++u) n5 += c[u];
        }
        for (; k < k1; ++k) n5 += count(k);
        for (int p = 0; p < r; ++p) {
          int v = sh == 0 && s0 == 0 ? 0 : G[i * r + p];
          const int32_t* w = W + (sh * ns + s0) * r + p;
          unsigned m = n5;
          for (int s = s0; s < min(ns, s0 + 5); ++s, m >>= 6, w += r) v += (int)(m & 63u) * *w;
          G[i * r + p] = v;
        }
      }
    }
  }
  __syncthreads();
}

// A thread's share of an update by the team: the first half of it takes the
// sites around swapped site 1, the second half around site 2; entries (tid mod
// half) + half j.  Entry e of a site leads to the swapped site when the site lies
// one entry before it.
template <int NJ>
struct FieldPlan {
  int ex[NJ], ey[NJ], ez[NJ];  // byte addresses of the axis tables at -entry
  int ush[NJ];                 // the entry's shell in a row of U, bytes
  int valid;                   // bit j: entry j exists
};

// The team that decides trials and updates fields: four of a block's warps.
constexpr int kFieldTeam = 128, kFieldHalf = kFieldTeam / 2;
__device__ __forceinline__ void team_sync() { asm volatile("bar.sync 6, 128;" ::: "memory"); }

template <int R>
struct FieldVec;
template <>
struct FieldVec<1> {
  using T = int;
  static __device__ __forceinline__ T add(T a, T b) { return a + b; }
};
template <>
struct FieldVec<2> {
  using T = int2;
  static __device__ __forceinline__ T add(T a, T b) { return make_int2(a.x + b.x, a.y + b.y); }
};
template <>
struct FieldVec<4> {
  using T = int4;
  static __device__ __forceinline__ T add(T a, T b) { return make_int4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
};

// sign = 1: the sites one entry after it instead, the same sites with the same
// shells when every entry's opposite is an entry of its shell.
template <int NJ>
__device__ __forceinline__ void field_plan(const Geom& g, const FieldLayout& L, const unsigned char* smem, int tid,
                                           FieldPlan<NJ>& P, int sign = -1) {
  const uint32_t* ents = reinterpret_cast<const uint32_t*>(smem + L.ents);
  P.valid = 0;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int k = (tid & (kFieldHalf - 1)) + kFieldHalf * j;
    int dx = 0, dy = 0, dz = 0, sh = 0;
    if (k < g.z) {
      unpack_entry(ents[k], dx, dy, dz, sh);
      P.valid |= 1 << j;
    }
    P.ex[j] = (int)L.tabs[0] + (kHalo + sign * dx) * 4;
    P.ey[j] = (int)L.tabs[1] + (kHalo + sign * dy) * 4;
    P.ez[j] = (int)L.tabs[2] + (kHalo + sign * dz) * 4;
    P.ush[j] = sh * field_stride(g.ns) * 4;
  }
}

// The plan's sites around the site at coordinates xyz (compact indices).
template <int NJ>
__device__ __forceinline__ void field_sites(const unsigned char* smem, const FieldPlan<NJ>& P, int xyz, int* at) {
  const int x = (xyz & 1023) << 2, y = (xyz >> 8) & 4092, z = (xyz >> 18) & 4092;
  auto tab = [&](int a) { return *reinterpret_cast<const int32_t*>(smem + a); };
#pragma unroll
  for (int j = 0; j < NJ; ++j) at[j] = tab(P.ex[j] + x) + tab(P.ey[j] + y) + tab(P.ez[j] + z);
}

// This thread's share of the fields' update for a swap: the plan's sites around
// its site (field_sites) and U's row of that site's change (byte address).  Plain loads, adds and
// stores: an entry's sites are distinct for one swapped site, and where a site
// may be around both, the halves go one after the other.  On lattices so small
// that several entries of a site lead to one other (distinct = 0) the adds are
// atomic.  R: fields a site keeps (1, 2 or 4 as one vector; 0: r of them).  The
// team meets once more before the fields are read.
template <int NJ, int R>
__device__ __forceinline__ void field_update(const FieldLayout& L, unsigned char* smem, const FieldPlan<NJ>& P,
                                             int distinct, int r, const int (&sites)[NJ], int row, bool both,
                                             bool second) {
  using F = FieldVec<R == 0 ? 1 : R>;
  using T = typename F::T;
  const int rs = R == 0 ? r : R;
  int at[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) at[j] = (int)L.g + 4 * rs * sites[j];
  if (!distinct) {
    for (int p = 0; p < rs; ++p)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        if ((P.valid >> j) & 1)
          atomicAdd(reinterpret_cast<int32_t*>(smem + at[j] + 4 * p),
                    *reinterpret_cast<const int32_t*>(smem + row + P.ush[j] + 4 * p));
    return;
  }
  auto add = [&]() {
    for (int p = 0; p < (R == 0 ? r : 1); ++p) {
      T d[NJ], v[NJ];
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        d[j] = *reinterpret_cast<const T*>(smem + row + P.ush[j] + 4 * p);
        v[j] = *reinterpret_cast<const T*>(smem + at[j] + 4 * p);
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        if ((P.valid >> j) & 1) *reinterpret_cast<T*>(smem + at[j] + 4 * p) = F::add(v[j], d[j]);
    }
  };
  if (both) {
    if (!second) add();
    team_sync();
    if (second) add();
  } else {
    add();
  }
}

// The reference-order FP64 pair energies before and after a swap
// (exact_pair_energies: same values, same order): the neighbours' species of
// both sites are gathered by all lanes, then lane c < 4 nsh adds, in list order
// from 0.0, the terms of shell c % nsh of evaluation c / nsh (site 1 before,
// site 2 before, site 1 after, site 2 after).
struct FieldExact {
  int z, ns, nsh;
  uint32_t ents, tx, ty, tz, sstart, codes, lat;  // addresses; the axis tables at coordinate 0
};

__device__ __forceinline__ FieldExact field_exact_setup(const Geom& g, const FieldLayout& L) {
  return {g.z, g.ns, g.nsh, L.ents, L.tabs[0] + kHalo * 4, L.tabs[1] + kHalo * 4, L.tabs[2] + kHalo * 4, L.sstart,
          L.codes, L.lat};
}

static __device__ __noinline__ double2 field_exact_pair(const FieldExact X, int xyz1, int xyz2, int i1, int i2, int s1,
                                                        int s2, int lane) {
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t* ents = reinterpret_cast<const uint32_t*>(smem + X.ents);
  const int16_t* sstart = reinterpret_cast<const int16_t*>(smem + X.sstart);
  const double* V = reinterpret_cast<const double*>(smem + FieldLayout::kV);
  uint8_t* codes = smem + X.codes;
  const int z = X.z, ns = X.ns, nsh = X.nsh;
  constexpr int kOther = 0x40;  // the neighbour is the other site
  const bool second = lane >= 16;
  const int c0 = second ? xyz2 : xyz1, other = second ? i1 : i2;
  const int32_t* tx = reinterpret_cast<const int32_t*>(smem + X.tx) + (c0 & 1023);
  const int32_t* ty = reinterpret_cast<const int32_t*>(smem + X.ty) + ((c0 >> 10) & 1023);
  const int32_t* tz = reinterpret_cast<const int32_t*>(smem + X.tz) + (c0 >> 20);
  __syncwarp();
  for (int k = lane & 15; k < z; k += 16) {
    int dx, dy, dz, sh;
    unpack_entry(ents[k], dx, dy, dz, sh);
    const int i = tx[dx] + ty[dy] + tz[dz];
    codes[(second ? z : 0) + k] = (uint8_t)((smem[X.lat + i] >> 2) + 1 + (i == other ? kOther : 0));
  }
  __syncwarp();
  const int nc = 4 * nsh;
  double part[2] = {0.0, 0.0};
#pragma unroll 1
  for (int q = 0; q < 2; ++q) {
    const int c = lane + 32 * q;
    double sum = 0.0;
    if (c < nc) {
      const int ev = c / nsh, sh = c - ev * nsh;
      const bool on2 = ev & 1, after = ev >= 2;
      const int own = on2 ? s2 : s1, oth = on2 ? s1 : s2;
      const double* Vr = V + ((after ? oth : own) - 1) + ns * ns * sh - ns;  // + ns * species
      const uint8_t* code = codes + (on2 ? z : 0);
      const int k1 = sstart[sh + 1];
#pragma unroll 4
      for (int k = sstart[sh]; k < k1; ++k) {
        const int v = code[k];
        // the other site holds our old species after the swap
        const int s = (after && (v & kOther)) ? own : (v & 63);
        sum = __dadd_rn(sum, Vr[ns * s]);
      }
    }
    part[q] = sum;
  }
  double e_un, e_sw;
  combine_pair_energies(part, nsh, lane, e_un, e_sw);
  return make_double2(e_un, e_sw);
}

// Named hardware barriers of the team's warps and the makers' (N threads
// together), per part h of the record ring: its records are made (1 + h); they
// have been used (3 + h); and of the makers alone (5).
template <int N = kFieldTeam + 32 * kFieldMakers>
__device__ __forceinline__ void made_arrive(int h) {
  asm volatile("bar.arrive %0, %1;" ::"r"(1 + h), "n"(N) : "memory");
}
template <int N = kFieldTeam + 32 * kFieldMakers>
__device__ __forceinline__ void made_wait(int h) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + h), "n"(N) : "memory");
}
template <int N = kFieldTeam + 32 * kFieldMakers>
__device__ __forceinline__ void used_arrive(int h) {
  asm volatile("bar.arrive %0, %1;" ::"r"(3 + h), "n"(N) : "memory");
}
template <int N = kFieldTeam + 32 * kFieldMakers>
__device__ __forceinline__ void used_wait(int h) {
  asm volatile("bar.sync %0, %1;" ::"r"(3 + h), "n"(N) : "memory");
}
__device__ __forceinline__ void makers_meet() { asm volatile("bar.sync 5, 128;" ::: "memory"); }

// The walk through a window of decided positions from this lane's position: like
// pairs (accepted without an energy evaluation or a draw) and certain
// rejections are passed, up to a trial that is neither or past the window.
// Bits 0-7: that position (32 and more: past the window), 8-15: trials passed,
// 16-23: rejections among them.
__device__ __forceinline__ unsigned field_walk(unsigned like, unsigned rej, int lane, int n_base, bool nbr) {
  unsigned path = 1u << lane;
#pragma unroll
  for (int i = 0; i < 5; ++i) path |= ((path & like) << n_base) | ((path & rej) << (n_base + 1));
  if (nbr) {  // eight trials can start in a window, six otherwise
    path |= ((path & like) << n_base) | ((path & rej) << (n_base + 1));
    path |= ((path & like) << n_base) | ((path & rej) << (n_base + 1));
  }
  // the positions passed, by n_base words each and one more per rejection
  const unsigned passed = __popc(path & (like | rej)), n_rej = __popc(path & rej);
  return ((unsigned)lane + passed * (unsigned)n_base + n_rej) | passed << 8 | n_rej << 16;
}

// What the team tells the makers at the end.
struct FieldEnd {
  unsigned long long words;
  int done;
};

// A making warp (`mine` of kFieldMakers): its window's static records of every
// part, two parts at most before the team has used one, and its 32 words of the
// stream one part further on.  make(w, slot): the record at place `slot` of the
// ring, of the position of words w[0], w[1], ...  N: the threads of the barriers.
template <int N = kFieldTeam + 32 * kFieldMakers, class Make>
__device__ __forceinline__ void stream_produce(uint32_t* rng, unsigned char* smem, FieldEnd* end, int mine, int lane,
                                               Make make) {
  using Ring = FieldWords;
  uint32_t* mt = reinterpret_cast<uint32_t*>(smem);
  uint32_t* tw = mt + Ring::kTwAt;
  const int pos0 = (int)rng[kMTN];
  MtRoll R = {pos0, 0, 0};
  if (mine == 0) {
    mt_roll_load<Ring>(rng, mt, pos0, lane);
    __syncwarp();
#pragma unroll 1
    for (int k = 0; k < kFieldAhead / kWin; ++k) {
      mt_roll<Ring>(mt, tw, R, lane);
      __syncwarp();
    }
  }
  // this warp's rows of the stream: the first after those, then every fourth
  R = {pos0 + kFieldAhead + mine * kWin, kFieldAhead + mine * kWin, kFieldAhead + mine * kWin};
  unsigned long long made = kFieldAhead;
  int at = mine * kWin;  // the window's place in the ring of tempered words
  bool wrapped = false;  // two parts have been made
  for (int h = 0;; h ^= 1) {
    if (wrapped) used_wait<N>(h);
    wrapped = wrapped || h == 1;
    if (*(volatile int*)&end->done) break;
    makers_meet();  // the words of the part before
    make(tw + at + lane, (kFieldMakers * h + mine) * kWin + lane);
    mt_roll<Ring>(mt, tw, R, lane, kFieldMakers - 1);
    made += kFieldPart;
    at = at + kFieldPart >= Ring::kTw ? at + kFieldPart - Ring::kTw : at + kFieldPart;
    made_arrive<N>(h);
  }
  if (mine == 0) mt_roll_store<Ring>(mt, tw, R, pos0, end->words, made, rng, lane);
}

// stream_produce for trials (records A and B).  test(w): the records' last word
// of A and third of B from the acceptance word.
template <class Test>
__device__ __forceinline__ void field_produce(const ChainJob& J, const Geom& g, const FieldLayout& L,
                                              unsigned char* smem, FieldEnd* end, int mine, int lane, Test test) {
  const FieldGeom f = J.fg;
  const uint8_t* dtab = smem + L.dtab;
  const bool bcc = g.lattice == kBcc;
  const bool nbr = J.nbr_swap != 0;
  const int W1 = 2 * g.n1, W2 = 2 * g.n2, W3 = 2 * g.n3;
  const int ns4 = 4 * g.ns, c_at = (int)L.C;
  stream_produce(J.rng, smem, end, mine, lane, [&](const uint32_t* w, int slot) {
    int ax, ay, az, Ya, Xa, bx, by, bz, Yb, Xb;
    draw_site_halo(g, bcc, w[0], w[1], w[2], ax, ay, az, Ya, Xa);
    if (nbr) {
      // draw_nbr's neighbour; its steps are -1, 0, 1
      const int8_t* v = cNbrSwap[g.lattice][umulhi32(w[3], (uint32_t)g.nbr_k)];
      bx = wrap_fast(ax + v[0], W1);
      by = wrap_fast(ay + v[1], W2);
      bz = wrap_fast(az + v[2], W3);
      Yb = by >> g.ys;
      Xb = bx >> 1;
    } else {
      draw_site_halo(g, bcc, w[3], w[4], w[5], bx, by, bz, Yb, Xb);
    }
    const int2 th = test(w[nbr ? 4 : 6]);
    const int t1 = wrap_fast(bx - ax + f.dm[0], W1), t2 = wrap_fast(by - ay + f.dm[1], W2),
              t3 = wrap_fast(bz - az + f.dm[2], W3);
    const int both = nbr || words_near(f.both_c, f.both_2c, w);  // a site may be around both
    int cls = 0;
    if (t1 < f.side[0] && t2 < f.side[1] && t3 < f.side[2]) cls = dtab[(t3 * f.side[1] + t2) * f.side[0] + t1];
    const int ia = az * g.sz + Ya * g.sy + Xa, ib = bz * g.sz + Yb * g.sy + Xb;
    *reinterpret_cast<int4*>(smem + FieldLayout::kA + slot * 16) =
        make_int4(ia, ib, c_at + cls * g.ns * ns4, th.x);
    *reinterpret_cast<int4*>(smem + FieldLayout::kB + slot * 16) =
        make_int4(ax | ay << 10 | az << 20, bx | by << 10 | bz << 20, th.y, both);
  });
}

}  // namespace brawl
