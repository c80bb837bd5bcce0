// halo_shear.cuh -- fcc/bcc lattices with a periodic halo whose neighbour
// steps are the same at every site.
//
// The compact lattice (Z, Y, X) = (z, y >> ys, x >> 1) halves coordinates, so
// the index step of a neighbour depends on the site's parity.  Here each row
// (fcc) or plane (bcc) is shifted by half its own coordinate, which undoes the
// halving's dependence:
//   fcc: index = z SZ + y SY + (x + y + z)/2    (x + y + z is even)
//   bcc: index = z SZ + (y - z)/2 SY + (x - z)/2  (x, y, z of one parity)
// Both are linear in (x, y, z), so an entry (dx, dy, dz) is one step for every
// site, and so is a period (the images an accepted swap writes).  SY and SZ
// leave the shifted rows and planes room; the layout is 2-5% larger than the
// unshifted one (1.8% for bcc 24^3 with six shells).  A neighbour's address is
// one add instead of a select and an add.
#pragma once

#include "chain_engine.cuh"

namespace brawl {

// The index of compact cell (Z, Y, X), halo cells (negative or past the
// extents) included.
__host__ __device__ __forceinline__ int shear_cell(bool bcc, const HaloGeom& H, int Z, int Y, int X) {
  const int at = H.korg + Z * H.kSZ + Y * H.kSY + X;
  return bcc ? at - (Z >> 1) * (H.kSY + 1) : at + ((Y + Z + 1) >> 1);
}

// The index step of an entry.
__host__ __device__ __forceinline__ int shear_step(bool bcc, const HaloGeom& H, int dx, int dy, int dz) {
  return bcc ? dz * H.kSZ + (dy - dz) / 2 * H.kSY + (dx - dz) / 2 : dz * H.kSZ + dy * H.kSY + (dx + dy + dz) / 2;
}

// A lane's walk over the cells (Z, Y, X) of a box, X fastest, 32 cells on at a time.
struct BoxWalk {
  int nx, ny;  // the box's rows and their length
  int dx, dy;  // 32 cells on: so many rows and cells
  int x, y, z;
};

__device__ __forceinline__ BoxWalk box_walk(int nx, int ny, int lane) {
  return {nx, ny, 32 % nx, 32 / nx, lane % nx, lane / nx % ny, lane / nx / ny};
}

__device__ __forceinline__ void box_step(BoxWalk& w) {
  w.x += w.dx;
  const int row = w.x >= w.nx;
  w.x -= row ? w.nx : 0;
  w.y += w.dy + row;
  while (w.y >= w.ny) {  // (once, unless the box is tiny)
    w.y -= w.ny;
    ++w.z;
  }
}

// Fills every cell of the layout from the compact lattice with 4 times the
// species (the byte offset of its column in the tables).  The latency of the loads
// and the index arithmetic bound it, so kAhead cells are in flight.
__device__ inline void shear_fill(const Geom& g, const HaloGeom& H, const int8_t* lat_c, uint8_t* lat, int lane) {
  const bool bcc = g.lattice == kBcc;
  const int PX = H.NX + 2 * H.hx, PY = H.NY + 2 * H.hy, total = PX * PY * (H.NZ + 2 * H.hz);
  BoxWalk w = box_walk(PX, PY, lane);
  constexpr int kAhead = 16;
  for (int t = lane; t < total; t += 32 * kAhead) {
    int at[kAhead];
    int8_t v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      int X = w.x - H.hx, Y = w.y - H.hy, Z = w.z - H.hz;
      const bool on = t + 32 * u < total;
      at[u] = on ? shear_cell(bcc, H, Z, Y, X) : -1;
      X += X < 0 ? H.NX : X >= H.NX ? -H.NX : 0;
      Y += Y < 0 ? H.NY : Y >= H.NY ? -H.NY : 0;
      Z += Z < 0 ? H.NZ : Z >= H.NZ ? -H.NZ : 0;
      v[u] = on ? lat_c[Z * g.sz + Y * g.sy + X] : (int8_t)0;
      box_step(w);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (at[u] >= 0) lat[at[u]] = (uint8_t)(v[u] << 2);
  }
}

// Copies the lattice's own cells back to the compact one.
__device__ inline void shear_store(const Geom& g, const HaloGeom& H, const uint8_t* lat, int8_t* lat_c, int lane) {
  const bool bcc = g.lattice == kBcc;
  BoxWalk w = box_walk(H.NX, H.NY, lane);
#pragma unroll 8
  for (int t = lane; t < g.n_sites; t += 32) {
    lat_c[t] = (int8_t)(lat[shear_cell(bcc, H, w.z, w.y, w.x)] >> 2);
    box_step(w);
  }
}

}  // namespace brawl
