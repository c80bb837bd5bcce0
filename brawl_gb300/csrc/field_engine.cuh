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

#include "kernels.cuh"

namespace brawl {

// A position's static record (the trial that would start there):
//   at   coordinates of site 1, of site 2 (x | y << 10 | z << 20), index of
//        site 1 | index of site 2 << 16, displacement class (0: no entry)
//   th   the larger of rej_above and the band; acc_below
constexpr int kFieldRing = 4 * kWin;  // positions held: two halves of two windows

// Shared memory of a chain with fields: the stream's rings, the records, then
// V, the update table U, the neighbours' constants C, W and F, the entries,
// the axis tables, the displacement classes, the exact tier's codes, the
// fields and the compact lattice.
struct FieldLayout {
  static constexpr uint32_t kAt = kRollWords * 4;
  static constexpr uint32_t kTh = kAt + kFieldRing * 16;
  static constexpr uint32_t kV = kTh + kFieldRing * 8;
  uint32_t U, C, W, F, ents, tabs[3], sstart, dtab, codes, g, lat, total;
};
static_assert(FieldLayout::kAt % 16 == 0 && FieldLayout::kV % 16 == 0, "16-byte records, tables of doubles");

__host__ __device__ inline FieldLayout field_layout(const Geom& g, const FieldGeom& f) {
  FieldLayout L;
  const uint32_t ns = (uint32_t)g.ns, r = ns - 1, nsh = (uint32_t)g.nsh;
  L.U = FieldLayout::kV + ns * ns * nsh * 8;
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

// Tables, lattice and fields from the job, by all the block's threads.  Ends
// with a __syncthreads.
__device__ inline void field_stage(const ChainJob& J, const Geom& g, const FieldLayout& L, unsigned char* smem, int tid,
                                   int nt) {
  const int ns = g.ns, nsp = ns + 1, r = ns - 1, nsh = g.nsh;
  double* V = reinterpret_cast<double*>(smem + FieldLayout::kV);
  int32_t* U = reinterpret_cast<int32_t*>(smem + L.U);
  int32_t* C = reinterpret_cast<int32_t*>(smem + L.C);
  int32_t* W = reinterpret_cast<int32_t*>(smem + L.W);
  int32_t* F = reinterpret_cast<int32_t*>(smem + L.F);
  uint32_t* ents = reinterpret_cast<uint32_t*>(smem + L.ents);
  int16_t* sstart = reinterpret_cast<int16_t*>(smem + L.sstart);
  uint8_t* dtab = smem + L.dtab;
  int32_t* G = reinterpret_cast<int32_t*>(smem + L.g);
  int8_t* lat = reinterpret_cast<int8_t*>(smem + L.lat);
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
    const int n16 = g.n_sites >> 4;
    const uint4* src = reinterpret_cast<const uint4*>(J.lat);
    uint4* dst = reinterpret_cast<uint4*>(lat);
    for (int i = tid; i < n16; i += nt) dst[i] = src[i];
    for (int i = (n16 << 4) + tid; i < g.n_sites; i += nt) lat[i] = J.lat[i];
  }
  __syncthreads();
  auto Fv = [&](int a, int sh, int b) { return F[(a * nsh + sh) * nsp + b]; };
  // W[sh][s - 1][s2 - 2]: a neighbour of species s in shell sh, to g(., s2)
  for (int i = tid; i < nsh * ns * r; i += nt) {
    const int s2 = i % r + 2, s = (i / r) % ns + 1, sh = i / (r * ns);
    W[i] = Fv(s2, sh, s) - Fv(1, sh, s);
  }
  // U[old - 1][new - 1][sh][s2 - 2]: a neighbour changing from old to new
  for (int i = tid; i < ns * ns * nsh * r; i += nt) {
    const int s2 = i % r + 2, sh = (i / r) % nsh, sn = (i / (r * nsh)) % ns + 1, so = i / (r * nsh * ns) + 1;
    U[i] = (Fv(s2, sh, sn) - Fv(1, sh, sn)) - (Fv(s2, sh, so) - Fv(1, sh, so));
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
  // The fields: per shell the neighbours are counted by species (a byte each
  // of a 64-bit word, eight species at a time), then weighted.
  const int32_t* tx = reinterpret_cast<const int32_t*>(smem + L.tabs[0]) + kHalo;
  const int32_t* ty = reinterpret_cast<const int32_t*>(smem + L.tabs[1]) + kHalo;
  const int32_t* tz = reinterpret_cast<const int32_t*>(smem + L.tabs[2]) + kHalo;
  for (int i = tid; i < g.n_sites; i += nt) {
    int x, y, z;
    decode_site(g, i, x, y, z);
    for (int sh = 0; sh < nsh; ++sh) {
      for (int s0 = 0; s0 < ns; s0 += 8) {
        unsigned long long n8 = 0;
        const int k1 = sstart[sh + 1];
#pragma unroll 4
        for (int k = sstart[sh]; k < k1; ++k) {
          int dx, dy, dz, s_;
          unpack_entry(ents[k], dx, dy, dz, s_);
          const int s = lat[tx[x + dx] + ty[y + dy] + tz[z + dz]] - 1 - s0;
          n8 += (unsigned)s < 8u ? 1ull << (8 * s) : 0ull;
        }
        for (int p = 0; p < r; ++p) {
          int v = sh == 0 && s0 == 0 ? 0 : G[p * g.n_sites + i];
          for (int s = s0; s < min(ns, s0 + 8); ++s)
            v += (int)((n8 >> (8 * (s - s0))) & 0xffull) * W[(sh * ns + s) * r + p];
          G[p * g.n_sites + i] = v;
        }
      }
    }
  }
  __syncthreads();
}

// This lane's share of an update: lanes 0-15 the sites that have site 1 as a
// neighbour, 16-31 site 2; entry (lane & 15) + 16 j of such a site leads back
// to it, so the site lies one entry before it.
template <int NJ>
struct FieldPlan {
  int ex[NJ], ey[NJ], ez[NJ];  // byte addresses of the axis tables at -entry
  int ush[NJ];                 // the entry's shell in a row of U, bytes
  unsigned valid;
};

template <int NJ>
__device__ __forceinline__ void field_plan(const Geom& g, const FieldLayout& L, const unsigned char* smem, int lane,
                                           FieldPlan<NJ>& P) {
  const uint32_t* ents = reinterpret_cast<const uint32_t*>(smem + L.ents);
  P.valid = 0;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int k = (lane & 15) + 16 * j;
    int dx = 0, dy = 0, dz = 0, sh = 0;
    if (k < g.z) {
      unpack_entry(ents[k], dx, dy, dz, sh);
      P.valid |= 1u << j;
    }
    P.ex[j] = (int)L.tabs[0] + (kHalo - dx) * 4;
    P.ey[j] = (int)L.tabs[1] + (kHalo - dy) * 4;
    P.ez[j] = (int)L.tabs[2] + (kHalo - dz) * 4;
    P.ush[j] = sh * (g.ns - 1) * 4;
  }
}

// The swap of sites 1 and 2 (coordinates xyz1, xyz2, indices, species before):
// the lattice and the fields.  All lanes of one warp; a __syncwarp follows
// before either is read.  Sites can meet in several entries, so the adds are
// atomic.
template <int NJ>
__device__ __forceinline__ void field_swap(const Geom& g, const FieldLayout& L, unsigned char* smem,
                                           const FieldPlan<NJ>& P, int xyz1, int xyz2, int i1, int i2, int s1, int s2,
                                           int lane) {
  const bool second = lane >= 16;
  const int c = second ? xyz2 : xyz1;
  const int so = second ? s2 : s1, sn = second ? s1 : s2;
  const int x4 = (c & 1023) << 2, y4 = (c >> 8) & 4092, z4 = (c >> 18) & 4092;
  const int r = g.ns - 1;
  const int row = (int)L.U + (((so - 1) * g.ns + (sn - 1)) * g.nsh * r) * 4;
  int at[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j)
    at[j] = *reinterpret_cast<const int32_t*>(smem + P.ex[j] + x4) +
            *reinterpret_cast<const int32_t*>(smem + P.ey[j] + y4) +
            *reinterpret_cast<const int32_t*>(smem + P.ez[j] + z4);
  if (lane == 0) smem[L.lat + i1] = (unsigned char)s2;
  if (lane == 16) smem[L.lat + i2] = (unsigned char)s1;
  for (int p = 0; p < r; ++p) {
    int32_t* G = reinterpret_cast<int32_t*>(smem + L.g) + p * g.n_sites;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int u = *reinterpret_cast<const int32_t*>(smem + row + P.ush[j] + 4 * p);
      if ((P.valid >> j) & 1u) atomicAdd(G + at[j], u);
    }
  }
}

// The reference-order FP64 pair energies' difference e_swapped - e_unswapped
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

static __device__ __noinline__ double field_exact_delta(const FieldExact X, int xyz1, int xyz2, int i1, int i2, int s1,
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
    codes[(second ? z : 0) + k] = (uint8_t)(smem[X.lat + i] | (i == other ? kOther : 0));
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
  return __dsub_rn(e_sw, e_un);
}

}  // namespace brawl
