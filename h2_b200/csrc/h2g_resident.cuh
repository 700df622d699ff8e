// h2g_resident.cuh -- the preconditioner with its vector resident on the chip, and CalcAX behind it.
//
// One cooperative launch runs the Krylov update that makes the right-hand side, the 10 colour passes
// of Preconditioner! (src/NonUniform.jl:531-559) and CalcAX! of its result with the iteration's inner
// products (NonUniform.jl:296-326): 3 launches an iteration instead of 23.
//
// What bounds it: the colour passes as separate launches read x, b and the coefficients through L1
// and L2 on every pass (155 instructions per cell, 7 us a pass at 240x240x30).  Here x and b stay in
// the shared memory of the SMs from the first pass to the last, so a pass costs the shared-memory
// reads of its stencil and one exchange with the neighbouring tiles.
//
// Split.  A block owns a tile of 32 positions x R rows x every plane (all of a column, so that the
// z-neighbours are always its own) and there are at most as many tiles as SMs.  A warp owns NP pairs
// of planes of the tile: 32 lanes along the positions, R rows each.  Marching along the rows instead of
// along z keeps a lane's coefficients in registers from row to row while the stencil class stays the
// same, which it does inside a layer; where it changes they come from the tile's own copy of its rows of
// the class table in shared memory (k_tile_classes numbers a tile's classes; from L1, beside 225 KB of x
// and b, they mostly missed).
//
// Exchange.  The rows and columns on a tile's edge go to the neighbouring tiles through global
// memory: a cell is stored with the number of the pass that made it, in one 16-byte store, and the
// reader polls the 16 bytes until the number is the one it waits for.  There is no grid barrier and
// no fence; one message is one trip through L2, about 1000 cycles.  Inside a tile a warp waits for the
// warps of the planes below and above, not for the block.  A pass updates its first and last row
// first, so that their messages travel while the rows between are updated.  One slot per cell and colour
// suffices: a cell is overwritten a sweep later, by an update that needs the reader's value of the pass in between, which
// the reader made after reading the slot.  Every wait is bounded like the grid barriers'.
//
// Results are the bits of the separate launches: the same operations per cell, the same quotient (see
// div_by) and the same order in the inner products (row sums in the shuffle order of k_ax's warps,
// then k_ax's sum over 8 rows, then reduce_finish's sum over blocks).
#pragma once
#include <type_traits>

#include "h2g_device.cuh"

namespace h2g {

constexpr int kRsRowPitch = 34;   // doubles per row in shared memory: 32 positions and one on each side
constexpr int kRsBox = 72;        // messages per tile, plane and colour: first row, last row, x edges
constexpr int kRsZero = 4 * kRsBox;  // slots before the first tile's that nobody writes (zeros)
constexpr int kRsMaxRows = 8;
constexpr int kRsMaxWarps = 15;   // 128 registers a thread: four of the warps share a scheduler's 16384

// Number of the next launch (part of every message's pass number), arrivals of the current launch or barrier.
struct RsCtl {
  unsigned long long epoch;
  unsigned int ticket;
  unsigned int go;  // passes of a grid barrier (k_resident_sor)
};

struct RsArgs {
  OpParams<double> op;
  double* xx;       // M^-1 bb
  double* v;        // bb: VM 0 read; VM 1 p, updated; VM 2 s, written
  const double* r;
  const double* q;
  double* y;        // A xx (VM 1, 2)
  const double* u;  // r0, the second factor of the inner product (VM 1)
  SolverState* st;
  ulonglong2* box;      // messages
  ulonglong2* rowsum;   // row sums of the inner products as messages: [NDOT][blocks of k_ax][8]
  double* partials;     // k_ax's block sums: [NDOT][blocks of k_ax]
  RsCtl* ctl;
  const uint16_t* lcls;  // per cell: its class in the tile's own numbering, 0: not updated
  const uint16_t* list;  // per tile (kRsMaxTab): the tile's classes
  const int* count;      // per tile: how many
  int* err;
  long long limit;
  int ntab;         // rows of the tile table in shared memory (the largest count + 1)
  int nxb, ntj;     // tiles along the positions and along the rows
};

constexpr int kRsMaxTab = 1024;
// A row of a tile's table: (cx-, cx+), (cx+, cx-), (cy-, cy+), (cz-, cz+), (dd, 1/dd).
constexpr int kRsTabRow = 10;

// Shared memory: x (an even number of planes between two planes of zeros, so that every neighbour lies at
// a constant distance), the tile's rows of the class table, the classes of every pair of planes and, if
// there is room (BS), b.
__host__ __device__ constexpr size_t rs_x_elems(int R, int NZ) {
  return (size_t)((NZ + 1) / 2 * 2 + 2) * 2 * R * kRsRowPitch;
}
__host__ __device__ constexpr size_t rs_smem(int R, int NZ, int ntab, bool bs) {
  return sizeof(double) * (rs_x_elems(R, NZ) + kRsTabRow * (size_t)ntab) +
         (size_t)((NZ + 1) / 2) * 2 * R * 32 * (sizeof(unsigned) + (bs ? 2 * sizeof(double) : 0));
}

// One message: 16 bytes, stored and loaded as one (a .b128 access is single-copy atomic).
// The pass number is 32 bits: 16 for each launch since the messages were cleared, which they are long before it
// comes round again (resident_prepare).
__device__ __forceinline__ void msg_store(ulonglong2* p, double v, unsigned seq) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"((unsigned long long)seq));
}
__device__ __forceinline__ void msg_load(const ulonglong2* p, double& v, unsigned& seq) {
  unsigned long long b, q;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(b), "=l"(q)
               : "l"(p));
  v = __longlong_as_double(b);
  seq = (unsigned)q;
}

// Shared memory by 32-bit address and constant distance (bytes).  The compiler takes these for opaque
// operations in program order; __syncwarp() separates them from other accesses.
__device__ __forceinline__ unsigned saddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
template <int D>
__device__ __forceinline__ double lds(unsigned a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1+%2];" : "=d"(v) : "r"(a), "n"(D));
  return v;
}
template <int D>
__device__ __forceinline__ unsigned ldsu(unsigned a) {
  unsigned v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(D));
  return v;
}
template <int D>
__device__ __forceinline__ void sts(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0+%1], %2;" ::"r"(a), "n"(D), "d"(v));
}

// A value that this launch overwrites: an ordinary load (a read-only one may return old values), which the
// compiler may move like a read-only one: the value is used up before its place is written.
__device__ __forceinline__ double ld_once(const double* p) {
  double v;
  asm("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// Coefficients of a cell.  cxa multiplies the x-neighbour at the cell's own position in an even row of
// the tile, cxb the other one; in an odd row they change places.
struct RsCoef {
  double cxa, cxb, cym, cyp, czm, czp, dd, y;
};
// Coefficients of a cell and of the cell of the plane above (classes packed in 16 bits each), loaded
// where the class is not that of the lane's last cell: in 39 % of the rows of a warp (240x240x30), by
// predicated loads (a branch round them cost 2000 cycles a pass more, 10 % of a solve).  oa: 0 if the
// neighbour at the first plane's cell's own position is the one at x- (e = 1 in an even row), else 16.
__device__ __forceinline__ void rs_coef(unsigned tab, unsigned cl, unsigned oa, unsigned& cur, RsCoef (&k)[2]) {
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const unsigned on = w ? (cl ^ cur) >> 16 : (cl ^ cur) & 0xffffu;
    const unsigned t = tab + 8u * kRsTabRow * (w ? cl >> 16 : cl & 0xffffu);
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %8, 0;\n\t@p ld.shared.v2.f64 {%0, %1}, [%10];\n\t"
        "@p ld.shared.v2.f64 {%2, %3}, [%9+32];\n\t@p ld.shared.v2.f64 {%4, %5}, [%9+48];\n\t"
        "@p ld.shared.v2.f64 {%6, %7}, [%9+64];\n\t}"
        : "+d"(k[w].cxa), "+d"(k[w].cxb), "+d"(k[w].cym), "+d"(k[w].cyp), "+d"(k[w].czm), "+d"(k[w].czp),
          "+d"(k[w].dd), "+d"(k[w].y)
        : "r"(on), "r"(t), "r"(t + (w ? 16u - oa : oa)));
  }
  cur = cl;
}
// e of every cell of the row changes with the colour
__device__ __forceinline__ void rs_turn(RsCoef (&k)[2]) {
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const double t = k[w].cxa;
    k[w].cxa = k[w].cxb;
    k[w].cxb = t;
  }
}

// The quotient where div_bad(a).  The row of the cells without a class, zeros with dd = 1, has y = 0: their
// quotient is 0 whatever lies in their b or beside them (zero times infinity is not 0).  A selection of the
// row's result instead cost a transient solve of 181x179x30 1.7 %.
__device__ __forceinline__ double div_fix(double a, double d, double y, double q) {
  return !div_bad(a) ? q : y != 0.0 ? __ddiv_rn(a, d) : 0.0;
}

// A warp's pair of planes: where its messages, rows and classes are.
struct RsPair {
  // messages of plane 0, colour 0 that it reads: the rows before its first (lo) and after its last (hi)
  // and, per row (lane r: row r), the cell beside its first or last position; xa: of (plane w, colour w),
  // xb: the others.  Where there is no neighbour: slots that stay zero, and a mask of zeros.
  const ulonglong2 *lo, *hi, *xa, *xb;
  unsigned mlo, mhi, mxa, mxb;
  ulonglong2* box;  // its own, of plane 0, colour 0
  unsigned x;       // shared memory: row 0 of plane 0, colour 0, the lane's element
  unsigned edge;    // lane r: row r of plane 0, colour 0, from the cell beside its first position on
  unsigned pad;     // lane r: where there the message of colour 0 belongs (0 or 33 positions on)
  unsigned cls;     // classes of row 0, colour 0, the lane's
};

// The messages of a pair of planes, in flight or arrived.
struct RsMsg {
  double vlo[2], vhi[2], vxe[2];
  unsigned slo[2], shi[2], sxe[2];
  __device__ __forceinline__ void fetch_edges(const RsPair& a, int c) {
    msg_load((c ? a.xb : a.xa) + c * kRsBox, vxe[0], sxe[0]);
    msg_load((c ? a.xa : a.xb) + (2 + c) * kRsBox, vxe[1], sxe[1]);
  }
  __device__ __forceinline__ void fetch(const RsPair& a, int c) {
    const ulonglong2 *l = a.lo + c * kRsBox, *h = a.hi + c * kRsBox;
    msg_load(l, vlo[0], slo[0]);
    msg_load(l + 2 * kRsBox, vlo[1], slo[1]);
    msg_load(h, vhi[0], shi[0]);
    msg_load(h + 2 * kRsBox, vhi[1], shi[1]);
    fetch_edges(a, c);
  }
  // zero if the x edges of the lanes with mask `lanes` carry seq
  __device__ __forceinline__ unsigned edges_missing(const RsPair& a, int c, unsigned seq, unsigned lanes) const {
    return (((sxe[0] ^ seq) & (c ? a.mxb : a.mxa)) | ((sxe[1] ^ seq) & (c ? a.mxa : a.mxb))) & lanes;
  }
  __device__ __forceinline__ unsigned rows_missing(const RsPair& a, unsigned seq) const {
    return (((slo[0] ^ seq) | (slo[1] ^ seq)) & a.mlo) | (((shi[0] ^ seq) | (shi[1] ^ seq)) & a.mhi);
  }
};

// One turn of a bounded wait that has lasted since t0: true once it ran out here or elsewhere.
__device__ __forceinline__ bool rs_give_up(long long t0, const RsArgs& A) {
  const bool late = clock64() - t0 > A.limit;
  if (!__any_sync(kFull, late || ld_relaxed_s32(A.err))) return false;
  if (late) {
    atomicExch(A.err, 1);
    if (A.st) {
      A.st->stop = 1;
      A.st->reason = kTimeout;
    }
  }
  return true;
}

// Polls until the rows' messages of colour c, and the x edges of the lanes with mask `lanes`, carry seq.
// False in every lane if the wait ran out.
__device__ __forceinline__ bool rs_wait(RsMsg& m, const RsPair& a, int c, unsigned seq, unsigned lanes,
                                        const RsArgs& A) {
  if (!__any_sync(kFull, m.rows_missing(a, seq) | m.edges_missing(a, c, seq, lanes))) return true;
  const long long t0 = clock64();
  do {
    if (rs_give_up(t0, A)) return false;
    m.fetch(a, c);
  } while (__any_sync(kFull, m.rows_missing(a, seq) | m.edges_missing(a, c, seq, lanes)));
  return true;
}
// The x edges alone: once this warp has sent its first and last row the tile beside them may go on and
// overwrite theirs.
__device__ __forceinline__ bool rs_wait_edges(RsMsg& m, const RsPair& a, int c, unsigned seq, unsigned lanes,
                                              const RsArgs& A) {
  if (!__any_sync(kFull, m.edges_missing(a, c, seq, lanes))) return true;
  const long long t0 = clock64();
  do {
    if (rs_give_up(t0, A)) return false;
    m.fetch_edges(a, c);
  } while (__any_sync(kFull, m.edges_missing(a, c, seq, lanes)));
  return true;
}

// Writes the x edges of colour c (lanes with mask `lanes`) beside their rows.
template <int R>
__device__ __forceinline__ void rs_put_edges(const RsMsg& m, const RsPair& a, int c, bool lanes) {
  constexpr int PL = 2 * R * kRsRowPitch * 8, CP = R * kRsRowPitch * 8;
  if (lanes) {
    const unsigned e = a.edge + (c ? CP : 0), o = c ? 264u - a.pad : a.pad;
    sts<0>(e + o, m.vxe[0]);
    sts<PL + 264>(e - o, m.vxe[1]);
  }
  __syncwarp();
}
// Sends the cells of colour c beside the neighbouring tiles: the first position's if e is 0, the last's if it is 1.
template <int R>
__device__ __forceinline__ void rs_send_edges(const RsPair& a, int c, unsigned seq, bool lanes) {
  constexpr int PL = 2 * R * kRsRowPitch * 8, CP = R * kRsRowPitch * 8;
  __syncwarp();
  if (lanes) {
    const unsigned e = a.edge + (c ? CP : 0), o = (c ? 264u - a.pad : a.pad) ? 8u : 256u;
    ulonglong2* box = a.box + c * kRsBox + 64;
    if (c ? a.mxa : a.mxb) msg_store(box, lds<0>(e + o), seq);
    if (c ? a.mxb : a.mxa) msg_store(box + 2 * kRsBox, lds<PL + 264>(e - o), seq);
  }
}

// Passes a warp has finished, for the warps of the planes below and above (shared memory).
__device__ __forceinline__ void rs_post(unsigned* prog, unsigned n) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0)
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(prog)), "r"(n) : "memory");
}
__device__ __forceinline__ unsigned rs_progress(const unsigned* prog) {
  unsigned v;
  asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"((unsigned)__cvta_generic_to_shared(prog)) : "memory");
  return v;
}
// Waits until the two warps have finished n passes: their planes are then up to date, and nobody reads
// what this warp's next pass overwrites.  Lanes may read different counts, so the warp votes: all of its
// lanes go on, or give up, in the same turn.
__device__ __forceinline__ bool rs_planes_ready(const unsigned* below, const unsigned* above, unsigned n) {
  return __all_sync(kFull, rs_progress(below) >= n && rs_progress(above) >= n);
}
__device__ __forceinline__ bool rs_wait_planes(const unsigned* below, const unsigned* above, unsigned n,
                                               const RsArgs& A) {
  if (rs_planes_ready(below, above, n)) return true;
  const long long t0 = clock64();
  for (unsigned turn = 1;; ++turn) {
    if (rs_planes_ready(below, above, n)) return true;
    if ((turn & 63u) == 0 && rs_give_up(t0, A)) return false;
  }
}

// Six products of a cell in the reference's order (nb_sum); the first two, whose sum does not depend on
// their order, by position: oc at the cell's own position, ot beside it.
__device__ __forceinline__ double rs_sum(const RsCoef& k, double ca, double cb, double oc, double ot, double yp,
                                         double ym, double zp, double zm) {
  double s = mul(ca, oc);
  s = add(s, mul(cb, ot));
  s = add(s, mul(k.cyp, yp));
  s = add(s, mul(k.cym, ym));
  s = add(s, mul(k.czp, zp));
  return add(s, mul(k.czm, zm));
}

// Addresses of a row of the pair's first plane (shared memory): the updated colour, the other colour, and
// the other colour beside the cell in an even and in an odd row; the second plane and the planes below and
// above the pair lie at constant distances.
struct RsAddr {
  unsigned x, o, oe, oo, cls;
};

// What a pass with relaxation and residual sums (SOR) needs beside the rest: omega, RN(1/omega), the lane that
// keeps the sum of row 0, the sums kept.
struct RsSor {
  double omega, romega, sum;
  int at;
};

// The update of a row of the pair of planes (D: distance of the row).  The two planes are each other's
// z-neighbours, which saves two of the loads, and two independent chains of dependent FP64 operations.
template <int R, int D, bool ODD, bool SOR>
__device__ __forceinline__ void rs_row(const RsAddr& a, unsigned tab, unsigned oa, unsigned cl, unsigned& cur,
                                       RsCoef (&k)[2], double om0, double oc0, double on0, double om1, double oc1,
                                       double on1, double b0, double b1, double& n0, double& n1, RsSor& sor) {
  constexpr int PL = 2 * R * kRsRowPitch * 8;
  const double ot0 = lds<D>(ODD ? a.oo : a.oe), ot1 = lds<D + PL>(ODD ? a.oe : a.oo);
  const double z0 = lds<D - PL>(a.o), z1 = lds<D + 2 * PL>(a.o);
  const double p0 = lds<D>(a.x), p1 = lds<D + PL>(a.x);
  rs_coef(tab, cl, oa, cur, k);
  const double a0 = sub(rs_sum(k[0], ODD ? k[0].cxb : k[0].cxa, ODD ? k[0].cxa : k[0].cxb, oc0, ot0, on0, om0, oc1, z0), b0);
  const double a1 = sub(rs_sum(k[1], ODD ? k[1].cxb : k[1].cxa, ODD ? k[1].cxa : k[1].cxb, oc1, ot1, on1, om1, z1, oc0), b1);
  double q0 = div_by(a0, k[0].dd, k[0].y), q1 = div_by(a1, k[1].dd, k[1].y);
  if (div_bad(a0) || div_bad(a1)) {
#pragma unroll 1
    for (int w = 0; w < 2; ++w) {  // one copy of the division
      const double q = div_fix(w ? a1 : a0, w ? k[1].dd : k[0].dd, w ? k[1].y : k[0].y, w ? q1 : q0);
      if (w) q1 = q;
      else q0 = q;
    }
  }
  if constexpr (!SOR) {
    n0 = add(p0, sub(q0, p0));
    n1 = add(p1, sub(q1, p1));
    sts<D>(a.x, n0);
    sts<D + PL>(a.x, n1);
  } else {
    // cells without a class keep what they have: a guard of an isothermal face is a neighbour like any other
    const double d0 = sub(q0, p0), d1 = sub(q1, p1);
    n0 = cl & 0xffffu ? add(p0, mul(sor.omega, d0)) : p0;
    n1 = cl >> 16 ? add(p1, mul(sor.omega, d1)) : p1;
    sts<D>(a.x, n0);
    sts<D + PL>(a.x, n1);
    // the residual of rb_pass_column; cx- is cxa in both parities of the row if oa is 0 (first plane)
    const double g0 = mul(add(k[0].dd, mul(sor.omega, add(add(oa ? k[0].cxb : k[0].cxa, k[0].cym), k[0].czm))), d0);
    const double g1 = mul(add(k[1].dd, mul(sor.omega, add(add(oa ? k[1].cxa : k[1].cxb, k[1].cym), k[1].czm))), d1);
    double r0 = div_by(g0, sor.omega, sor.romega), r1 = div_by(g1, sor.omega, sor.romega);
    if (div_bad(g0) || div_bad(g1)) {
#pragma unroll 1
      for (int w = 0; w < 2; ++w) {
        const double r = div_fix(w ? g1 : g0, sor.omega, sor.romega, w ? r1 : r0);
        if (w) r1 = r;
        else r0 = r;
      }
    }
    double v = add(cl & 0xffffu ? mul(r0, r0) : 0.0, cl >> 16 ? mul(r1, r1) : 0.0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if (((int)threadIdx.x & 31) == sor.at + D / (kRsRowPitch * 8)) sor.sum = v;
  }
}

template <int I, int N, typename F>
__device__ __forceinline__ void rs_each(F& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    rs_each<I + 1, N>(f);
  }
}

// One colour pass over the R rows of a pair of planes, in one copy of the code for both colours and
// parities: a launch starts with a cold instruction cache (with a copy for each, the first two passes took
// 8000 cycles longer).  The first and the last row come first; mid() is called between them and the rest
// (false ends the pass).
// b: from shared memory (BS: bs, row 0 of the colour, the lane's element), or from the vector itself (bv,
// pitches row and plane), loaded two rows ahead of its use; f and l are those of the first and last row.
// (What a cell without a class gets for b does not matter: see div_fix.)
template <int R, bool BS, bool SOR, typename Mid>
__device__ __forceinline__ bool rs_rows(RsAddr a, unsigned tab, unsigned oa, unsigned bs, const double* bv, int row,
                                        int plane, double (&f)[2], double (&l)[2], RsCoef (&k)[2], unsigned& cur,
                                        const RsMsg& m, ulonglong2* box, bool to_lo, bool to_hi, unsigned seq,
                                        RsSor& sor, Mid mid) {
  constexpr int P = kRsRowPitch * 8, PL = 2 * R * P, L = R - 1, BP = 2 * R * 256;
  double n0, n1, om0, om1, oc0, oc1, b0, b1, c0, c1;
  if (!BS && R > 2) {
    bv += row;
    b0 = bv[0];
    b1 = bv[plane];
  }
  om0 = lds<0>(a.o);
  om1 = lds<PL>(a.o);
  oc0 = R > 1 ? lds<(R > 1 ? P : 0)>(a.o) : m.vhi[0];
  oc1 = R > 1 ? lds<(R > 1 ? P : 0) + PL>(a.o) : m.vhi[1];
  if (BS) {
    f[0] = lds<0>(bs);
    f[1] = lds<BP>(bs);
  }
  rs_row<R, 0, false, SOR>(a, tab, oa, ldsu<0>(a.cls), cur, k, m.vlo[0], om0, oc0, m.vlo[1], om1, oc1, f[0], f[1], n0, n1,
                            sor);
  if (to_lo) {
    msg_store(box, n0, seq);
    msg_store(box + 2 * kRsBox, n1, seq);
  }
  if constexpr (R > 1) {
    if (!BS && R > 3) {
      bv += row;
      c0 = bv[0];
      c1 = bv[plane];
    }
    if (BS) {
      l[0] = lds<L * 256>(bs);
      l[1] = lds<L * 256 + BP>(bs);
    }
    rs_row<R, L * P, (L & 1) != 0, SOR>(a, tab, oa, ldsu<L * 128>(a.cls), cur, k, lds<(L - 1) * P>(a.o), lds<L * P>(a.o),
                                   m.vhi[0], lds<(L - 1) * P + PL>(a.o), lds<L * P + PL>(a.o), m.vhi[1], l[0], l[1],
                                   n0, n1, sor);
  }
  if (to_hi) {
    msg_store(box + 32, n0, seq);
    msg_store(box + 2 * kRsBox + 32, n1, seq);
  }
  if (!mid()) return false;
  if constexpr (R > 2) {
    auto next = [&](auto rc) {
      constexpr int r = decltype(rc)::value;
      const double on0 = lds<(r + 1) * P>(a.o), on1 = lds<(r + 1) * P + PL>(a.o);
      double u0, u1;
      if (BS) {
        u0 = lds<r * 256>(bs);
        u1 = lds<r * 256 + BP>(bs);
      } else {
        u0 = b0;
        u1 = b1;
        b0 = c0;
        b1 = c1;
        if (r + 2 < L) {
          bv += row;
          c0 = bv[0];
          c1 = bv[plane];
        }
      }
      rs_row<R, r * P, (r & 1) != 0, SOR>(a, tab, oa, ldsu<r * 128>(a.cls), cur, k, om0, oc0, on0, om1, oc1, on1, u0, u1, n0, n1,
                                               sor);
      om0 = oc0;
      om1 = oc1;
      oc0 = on0;
      oc1 = on1;
    };
    rs_each<1, L>(next);
  }
  return true;
}

// One step of a sum over the warp's lanes of N values a lane: lanes that differ in bit o exchange
// halves, each keeps the sums of its half (N = 1: both keep the sum).  Steps 16, 8, 4, 2, 1 add the
// lanes in the order of a shuffle-down tree.
template <int N>
__device__ __forceinline__ void rs_fold(double* v, int o, int lane) {
  if constexpr (N == 1) {
    v[0] += __shfl_xor_sync(kFull, v[0], o);
  } else {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      const double keep = up ? v[i + N / 2] : v[i], send = up ? v[i] : v[i + N / 2];
      v[i] = keep + __shfl_xor_sync(kFull, send, o);
    }
  }
}

// The tile's classes: numbers the distinct classes of a tile from 1 (0: not updated) in the order of
// their numbers in the grid's table.  count[tile] may exceed kRsMaxTab: the list is then cut off.
// One block per tile; bitmap of the grid's classes in shared memory.
static __global__ void __launch_bounds__(256) k_tile_classes(Geo g, const uint16_t* __restrict__ cls,
                                                             uint16_t* __restrict__ lcls, uint16_t* __restrict__ list,
                                                             int* __restrict__ count, int R, int nxb) {
  __shared__ unsigned bits[2048];
  __shared__ int before[256];
  const int t = threadIdx.x, xb = blockIdx.x % nxb, j0 = 1 + (blockIdx.x / nxb) * R;
  for (int q = t; q < 2048; q += 256) bits[q] = 0u;
  __syncthreads();
  const int cells = g.NZ * R * 64;
  auto offset = [&](int q) {
    const int p = xb * 32 + (q & 31), c = (q >> 5) & 1, r = (q >> 6) % R, k = 1 + (q >> 6) / R, j = j0 + r;
    return j <= g.NY && p < g.HN ? g.row(c, j, k) + p : -1;
  };
  for (int q = t; q < cells; q += 256) {
    const int o = offset(q);
    const unsigned cl = o >= 0 ? cls[o] : kNoClass;
    if (cl != kNoClass) atomicOr(bits + (cl >> 5), 1u << (cl & 31));
  }
  __syncthreads();
  int n = 0;
  for (int q = 0; q < 8; ++q) n += __popc(bits[8 * t + q]);
  before[t] = n;
  __syncthreads();
  if (t == 0) {
    int sum = 0;
    for (int q = 0; q < 256; ++q) {
      const int v = before[q];
      before[q] = sum;
      sum += v;
    }
    count[blockIdx.x] = sum;
  }
  __syncthreads();
  auto rank = [&](unsigned cl) {
    int v = before[cl >> 8];
    for (unsigned q = (cl >> 8) * 8; q < (cl >> 5); ++q) v += __popc(bits[q]);
    return v + __popc(bits[cl >> 5] & ((1u << (cl & 31)) - 1u));
  };
  for (int q = t; q < cells; q += 256) {
    const int o = offset(q);
    if (o < 0) continue;
    const unsigned cl = cls[o];
    if (cl == kNoClass) {
      lcls[o] = 0;
      continue;
    }
    const int v = rank(cl);
    lcls[o] = (uint16_t)min(v + 1, kRsMaxTab);
    if (v < kRsMaxTab) list[(size_t)blockIdx.x * kRsMaxTab + v] = (uint16_t)cl;
  }
}

// VM 0: xx = M^-1 v.  VM 1: p = r + beta (p - omega q) in v, xx = M^-1 p, y = A xx, (y, u) ->
// kStageAlpha.  VM 2: s = r - alpha q in v, xx = M^-1 s, y = A xx, (y, y) and (y, s) -> kStageOmega.
// Grid nxb * ntj blocks (cooperative), block 32 * ceil(NZ / (2 NP)) threads.
// An iteration (two of these and the update) against the separate launches: 20x20x30 47 us (63), 120x120x30 64
// (88), 180x180x30 99 (143), 240x240x30 158 (216).  16 iterations in one launch, with both stages in one kernel,
// spilled 600 to 1500 bytes a thread and took 98 us at 120x120x30.
template <int R, int NP, int VM, bool BS>
__global__ void __launch_bounds__(32 * kRsMaxWarps, 1) k_resident(const __grid_constant__ RsArgs A) {
  extern __shared__ double sh[];
  __shared__ unsigned prog[kRsMaxWarps + 2];  // passes finished by each warp, between two that always have
  __shared__ int am_last;
  __shared__ double red[16];
  const Geo& g = A.op.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int tile = blockIdx.x, xb = tile % A.nxb, tj = tile / A.nxb;
  const int NZ = g.NZ, j0 = 1 + tj * R, p = xb * 32 + lane;
  constexpr int P = kRsRowPitch, CP = R * P, PL = 2 * CP;  // colour and plane pitch of x
  constexpr int BP = 2 * R * 32;                           // plane pitch of b
  double* X = sh + PL;                                     // [planes][2][R][P], position p at p + 1
  double* T = sh + rs_x_elems(R, NZ);                      // [ntab][kRsTabRow]
  double* B = T + kRsTabRow * A.ntab;                             // BS: [even number of planes][2][R][32]
  // [pair][2][R][32]: the tile's classes of the pair's planes, 16 bits each
  unsigned* K = reinterpret_cast<unsigned*>(B + (BS ? (NZ + 1) / 2 * 2 * BP : 0));
  constexpr int KP = 2 * R * 32;
  // neighbours
  const bool n_lo = tj > 0, n_hi = tj + 1 < A.ntj, n_xm = xb > 0, n_xp = xb + 1 < A.nxb;
  const int rows = min(R, g.NY - j0 + 1);  // inside the grid
  RsCoef cf[2];
  unsigned cur = 0xffffffffu;
  const unsigned tab = saddr(T);
  const bool par0 = (1 + j0 + 1) & 1;  // e of colour 0 in row 0 of a pair's first plane
  // messages of a plane and colour; with an odd NZ a tile has a plane more, which nobody reads
  const int NZe = (NZ + 1) & ~1;
  auto box_of = [&](int t, int pl) { return A.box + (size_t)(t * NZe + pl) * (2 * kRsBox); };

  // where the messages, rows and classes of the pair of planes pl0, pl0 + 1 are
  auto pair_at = [&](int pl0) {
    RsPair a;
    const ulonglong2* zero = A.box - kRsZero;
    a.box = box_of(tile, pl0) + lane;
    a.mlo = n_lo ? ~0u : 0u;
    a.mhi = n_hi ? ~0u : 0u;
    a.lo = n_lo ? box_of(tile - A.nxb, pl0) + 32 + lane : zero;
    a.hi = n_hi ? box_of(tile + A.nxb, pl0) + lane : zero;
    // the reader's e at row `lane`, for the messages of colour 0 in the first plane (it updates colour 1)
    const bool e = (1 + 1 + j0 + lane + pl0 + 1) & 1;
    const bool xa = lane < R && (e ? n_xp : n_xm), xb = lane < R && (e ? n_xm : n_xp);
    a.mxa = xa ? ~0u : 0u;
    a.mxb = xb ? ~0u : 0u;
    a.xa = xa ? box_of(e ? tile + 1 : tile - 1, pl0) + 64 + lane : zero;
    a.xb = xb ? box_of(e ? tile - 1 : tile + 1, pl0) + 64 + lane : zero;
    a.x = saddr(X + pl0 * PL + 1 + lane);
    a.edge = saddr(X + pl0 * PL + (lane < R ? lane : 0) * P);
    a.pad = e ? 264u : 0u;
    a.cls = saddr(K + (pl0 / 2) * KP + lane);
    return a;
  };

  // ---- the tile's table, right-hand side and first pass (x = 0: colour 0 gets (0 - b)/dd) ----------------
  if (threadIdx.x < kRsTabRow) T[threadIdx.x] = threadIdx.x == 8 ? 1.0 : 0.0;  // no class: 0, dd = 1, y = 0
  {
    const int n = A.count[tile];
    const uint16_t* list = A.list + (size_t)tile * kRsMaxTab;
    const double2* src = reinterpret_cast<const double2*>(A.op.ctab);
    for (int q = threadIdx.x; q < 4 * n; q += blockDim.x) {
      const double2 v = __ldg(src + 4 * (int)__ldg(list + (q >> 2)) + (q & 3));
      double2* t = reinterpret_cast<double2*>(T) + 5 * (1 + (q >> 2));
      t[(q & 3) + ((q & 3) > 0)] = v;
      if ((q & 3) == 0) t[1] = make_double2(v.y, v.x);
    }
  }
  if (threadIdx.x == 0) prog[0] = prog[nw + 1] = 16u;
  if (lane == 0) prog[warp + 1] = 0u;
  const int NZx = (NZ + 1) / 2 * 2;
  for (int q = threadIdx.x; q < PL; q += blockDim.x) {
    X[q - PL] = 0.0;
    X[NZx * PL + q] = 0.0;
  }
  // Programmatic launch: the set-up above overlaps the tail of the kernel before (its last reduction), whose
  // writes are read from here on.  240x240x30: 63.0 -> 58.9 ms a solve, 121x117x30 13.1 -> 12.6.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if ((A.st && A.st->stop) || ld_relaxed_s32(A.err)) return;  // the same for every block
  const unsigned seq0 = (unsigned)A.ctl->epoch * 16u;
  double beta = 0.0, omg = 0.0, alpha = 0.0;
  int first = 0;
  if (VM == 1) {
    first = A.st->first;
    beta = A.st->beta;
    omg = A.st->omega;
  } else if (VM == 2) {
    alpha = A.st->alpha;
  }
  // cell (row r, colour c, plane w of the pair): inside the grid, and where
  auto inside = [&](int pl0, int r, int c, int w) {
    const int i = 2 * p + (((1 + j0 + r + pl0 + w + 1) & 1) ^ c);
    return pl0 + w < NZ && r < rows && p < g.HN && i >= 1 && i <= g.NX;
  };
  auto where = [&](int pl0, int r, int c, int w) { return g.row(c, j0 + r, pl0 + w + 1) + p; };
#pragma unroll 1
  for (int np = 0; np < NP; ++np) {
    const int pl0 = (warp * NP + np) * 2;
    // r, q, v and classes of a row, two colours and two planes, loaded a row ahead
    double lr[4], lq[4], lv[4];
    unsigned lc[4];
    auto load = [&](int r) {
#pragma unroll
      for (int cw = 0; cw < 4; ++cw) {
        lr[cw] = lq[cw] = lv[cw] = 0.0;
        lc[cw] = 0u;
        if (inside(pl0, r, cw >> 1, cw & 1)) {
          const int ci = where(pl0, r, cw >> 1, cw & 1);
          lc[cw] = __ldg(A.lcls + ci);
          if (VM != 0) lr[cw] = __ldg(A.r + ci);
          if (VM != 0) lq[cw] = VM == 1 ? ld_once(A.q + ci) : __ldg(A.q + ci);
          if (VM != 2) lv[cw] = ld_once(A.v + ci);
        }
      }
    };
    load(0);
    if (np == 0) __syncthreads();  // the table
    if (pl0 >= NZ) break;
    ulonglong2* box = box_of(tile, pl0) + lane;
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
      double bv[4];
      unsigned cl[4];
#pragma unroll
      for (int cw = 0; cw < 4; ++cw) {
        cl[cw] = lc[cw];
        if (VM == 0) bv[cw] = lv[cw];
        else if (VM == 1) bv[cw] = first ? lr[cw] : add(lr[cw], mul(beta, sub(lv[cw], mul(omg, lq[cw]))));
        else bv[cw] = add(mul(-alpha, lq[cw]), lr[cw]);
      }
      load(r + 1);
      unsigned* kr = K + (pl0 / 2) * KP + r * 32 + lane;
      kr[0] = cl[0] | (cl[1] << 16);
      kr[R * 32] = cl[2] | (cl[3] << 16);
      rs_coef(tab, cl[0] | (cl[1] << 16), par0 ? 0u : 16u, cur, cf);
#pragma unroll
      for (int cw = 0; cw < 4; ++cw) {
        if (VM != 0 && inside(pl0, r, cw >> 1, cw & 1)) A.v[where(pl0, r, cw >> 1, cw & 1)] = bv[cw];
        if (BS) B[(pl0 + (cw & 1)) * BP + ((cw >> 1) * R + r) * 32 + lane] = cl[cw] ? bv[cw] : 1.0;
      }
      double n[2];
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const double a = sub(0.0, bv[w]);
        n[w] = div_by(a, cf[w].dd, cf[w].y);
        if (div_bad(a)) n[w] = div_fix(a, cf[w].dd, cf[w].y, n[w]);
        n[w] = cl[w] ? add(0.0, sub(n[w], 0.0)) : 0.0;
        double* x = X + (pl0 + w) * PL + r * P + 1 + lane;
        x[0] = n[w];
        x[CP] = 0.0;
        if (lane == 0) x[-1] = x[CP - 1] = 0.0;
        if (lane == 31) x[1] = x[CP + 1] = 0.0;
      }
      if (r == 0 && n_lo) {
        msg_store(box, n[0], seq0);
        msg_store(box + 2 * kRsBox, n[1], seq0);
      }
      if (r == R - 1 && n_hi) {
        msg_store(box + 32, n[0], seq0);
        msg_store(box + 2 * kRsBox + 32, n[1], seq0);
      }
    }
    rs_send_edges<R>(pair_at(pl0), 0, seq0, lane < R);
  }
  rs_post(prog + warp + 1, 1u);

  // ---- passes 2 to 10 --------------------------------------------------------------------------------
  bool ok = true;
  RsMsg m;
  // x edges of the first and the last row, and of the rows between
  const bool ends = lane == 0 || lane == R - 1, rest = lane < R && !ends;
  RsPair a = pair_at(warp * NP * 2);
#pragma unroll 1
  for (unsigned n = 1; n < 2 * kSweeps && ok; ++n) {
    const int c = n & 1;
    const unsigned seq = seq0 + n;
    const bool par = par0 ^ (c != 0);
    double f[2], l[2];
    const double* bv;
    // with an odd NZ the second plane of the last pair is not there: its b is not used
    auto first_b = [&](int pl) {
      bv = A.v + g.row(c, j0, pl + 1) + p;
      const int pp = pl + 1 < NZ ? (int)g.plane : 0;
      f[0] = bv[0];
      f[1] = bv[pp];
      if (R > 1) {
        l[0] = bv[(R - 1) * 2 * g.HP];
        l[1] = bv[(R - 1) * 2 * g.HP + pp];
      }
      return pp;
    };
    int plane = 0;
    if (NP == 1) {
      m.fetch(a, c ^ 1);
      if (!BS) plane = first_b(warp * 2);
    }
    rs_turn(cf);
    ok = rs_wait_planes(prog + warp, prog + warp + 2, n, A);
#pragma unroll 1
    for (int np = 0; np < NP && ok; ++np) {
      const int pl = (warp * NP + np) * 2;
      if (pl >= NZ) break;
      if (NP > 1) {
        a = pair_at(pl);
        m.fetch(a, c ^ 1);
        if (!BS) plane = first_b(pl);
      }
      ok = rs_wait(m, a, c ^ 1, seq - 1, ends ? ~0u : 0u, A);
      if (!ok) break;
      rs_put_edges<R>(m, a, c ^ 1, ends);
      if (R > 2 && __any_sync(kFull, m.edges_missing(a, c ^ 1, seq - 1, rest ? ~0u : 0u))) m.fetch_edges(a, c ^ 1);
      auto mid = [&] {
        rs_send_edges<R>(a, c, seq, ends);
        if (R <= 2) return true;
        if (!rs_wait_edges(m, a, c ^ 1, seq - 1, rest ? ~0u : 0u, A)) return false;
        rs_put_edges<R>(m, a, c ^ 1, rest);
        return true;
      };
      RsAddr ad;
      ad.x = a.x + (c ? CP * 8 : 0);
      ad.o = a.x + (c ? 0 : CP * 8);
      ad.oe = ad.o + (par ? 8u : -8u);
      ad.oo = ad.o - (par ? 8u : -8u);
      ad.cls = a.cls + (c ? R * 128 : 0);
      RsSor none;
      ok = rs_rows<R, BS, false>(ad, tab, par ? 0u : 16u, saddr(B + pl * BP + c * (R * 32) + lane), bv, 2 * g.HP, plane, f, l,
                          cf, cur, m, a.box + c * kRsBox, n_lo, n_hi, seq, none, mid);
      if (R > 2) rs_send_edges<R>(a, c, seq, rest);
    }
    rs_post(prog + warp + 1, n + 1);
  }
  if (ok) ok = rs_wait_planes(prog + warp, prog + warp + 2, 2 * kSweeps, A);

  // ---- xx, and y = A xx with the inner products ----------------------------------------------------------
  constexpr int NDOT = VM;  // 0, 1 or 2
  const int gy = (g.NY + kBY - 1) / kBY, nb = A.nxb * gy * NZ;
  auto block_id = [&](int group, int pl) { return xb + A.nxb * (group + gy * pl); };
#pragma unroll 1
  for (int np = 0; np < NP; ++np) {
    const int pl0 = (warp * NP + np) * 2;
    if (pl0 >= NZ || !ok) break;
    // the second factor of the inner product, a row ahead
    double un[4];
    auto load_u = [&](int r) {
#pragma unroll
      for (int cw = 0; cw < 4; ++cw) {
        un[cw] = 0.0;
        if (VM == 1 && inside(pl0, r, cw >> 1, cw & 1)) un[cw] = __ldg(A.u + where(pl0, r, cw >> 1, cw & 1));
        if (VM == 2 && BS) un[cw] = B[(pl0 + (cw & 1)) * BP + ((cw >> 1) * R + r) * 32 + lane];
        if (VM == 2 && !BS && inside(pl0, r, cw >> 1, cw & 1)) un[cw] = A.v[where(pl0, r, cw >> 1, cw & 1)];
      }
    };
    double om[4] = {0.0, 0.0, 0.0, 0.0};  // [colour * 2 + plane]: the row before
    if (VM != 0) {
      // colour 0's messages of its last pass are still in the boxes; its x edges are already in X
      if (NP > 1) a = pair_at(pl0);
      m.fetch(a, 0);
      load_u(0);
      ok = rs_wait(m, a, 0, seq0 + 2 * kSweeps - 2, 0u, A);
      if (!ok) break;
      om[0] = m.vlo[0];
      om[1] = m.vlo[1];
      const double h0 = m.vhi[0], h1 = m.vhi[1];
      m.fetch(a, 1);
      ok = rs_wait(m, a, 1, seq0 + 2 * kSweeps - 1, ~0u, A);
      if (!ok) break;
      rs_put_edges<R>(m, a, 1, lane < R);
      om[2] = m.vlo[0];
      om[3] = m.vlo[1];
      m.vlo[0] = h0;  // from here on: the row after the last, colour 0
      m.vlo[1] = h1;
    }
    const double* x0 = X + pl0 * PL + 1 + lane;
    const unsigned* kp = K + (pl0 / 2) * KP + lane;
    double xc[4];  // [colour * 2 + plane]: this row
#pragma unroll
    for (int cw = 0; cw < 4; ++cw) xc[cw] = x0[(cw & 1) * PL + (cw >> 1) * CP];
    // row sums, folded to one value a lane and kept by the lanes of the row (see below)
    double mine_sum = 0.0;
    constexpr int S = VM == 1 ? 2 : 1;
    cur = 0xffffffffu;
    // one copy of the code for both parities, like the passes
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
      const bool e0 = par0 ^ (r & 1);  // e of colour 0 in the first plane
      double d[4] = {0.0, 0.0, 0.0, 0.0}, uc[4], on[4];
      const double* x = x0 + r * P;
#pragma unroll
      for (int cw = 0; cw < 4; ++cw) {
        uc[cw] = un[cw];
        on[cw] = r + 1 < R ? x[(cw & 1) * PL + (cw >> 1) * CP + P] : cw < 2 ? m.vlo[cw & 1] : m.vhi[cw & 1];
      }
      if (VM != 0) load_u(r + 1);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (VM != 0) rs_coef(tab, kp[(c * R + r) * 32], 16u, cur, cf);  // cxa: x+ (plane 0), x- (plane 1)
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const int o = c ^ 1, cw = c * 2 + w, ow = o * 2 + w;
          const bool e = e0 ^ (c ^ w);
          const bool in = inside(pl0, r, c, w);
          const int ci = where(pl0, r, c, w);
          if (in) A.xx[ci] = xc[cw];
          if (VM != 0) {
            const double ot = x[w * PL + o * CP + (e ? 1 : -1)];
            const double dn = w ? xc[o * 2] : x[o * CP - PL], up = w ? x[o * CP + 2 * PL] : xc[o * 2 + 1];
            // cxa multiplies x+ in the first plane and x- in the second
            const double pa = (e != (w != 0)) ? ot : xc[ow], pb = (e != (w != 0)) ? xc[ow] : ot;
            // a cell without a class: 0 - 1 * 0 (a selection instead costs 240x240x30 1.2 % of a solve; the zero is not one
            // beside an infinity, which ends the solve in this iteration)
            const double out =
                sub(rs_sum(cf[w], cf[w].cxa, cf[w].cxb, pa, pb, on[ow], om[ow], up, dn), mul(cf[w].dd, xc[cw]));
            if (in) {
              A.y[ci] = out;
              if (VM == 1) {
                d[w] = __fma_rn(out, uc[cw], d[w]);
              } else {
                d[w] = __fma_rn(out, out, d[w]);
                d[2 + w] = __fma_rn(out, uc[cw], d[2 + w]);
              }
            }
          }
        }
      }
#pragma unroll
      for (int cw = 0; cw < 4; ++cw) {
        om[cw] = xc[cw];
        xc[cw] = on[cw];
      }
      if (VM == 1) {
        rs_fold<2>(d, 16, lane);
        rs_fold<1>(d, 8, lane);
        rs_fold<1>(d, 4, lane);
        rs_fold<1>(d, 2, lane);
        rs_fold<1>(d, 1, lane);
      } else if (VM == 2) {
        rs_fold<4>(d, 16, lane);
        rs_fold<2>(d, 8, lane);
        rs_fold<1>(d, 4, lane);
        rs_fold<1>(d, 2, lane);
        rs_fold<1>(d, 1, lane);
      }
      if (((lane / S) & 7) == r) mine_sum = d[0];
    }
    if (VM != 0) {
      // row sums: lane (q * 2 + w) * 8 + r (VM 2) or w * 16 + 2 r (VM 1) gets product q, plane w, row r
      const int q = VM == 1 ? 0 : lane >> 4, w = VM == 1 ? lane >> 4 : (lane >> 3) & 1;
      const int r = (lane / S) & 7, pl = pl0 + w, row = tj * R + r;
      const bool mine = pl < NZ && (VM == 2 || !(lane & 1));
      if (mine && r < rows)
        msg_store(A.rowsum + ((size_t)q * nb + block_id(row >> 3, pl)) * 8 + (row & 7), mine_sum, seq0);
      // k_ax's block sums: the tile that holds a group's first row adds its 8 rows in block_sum's order
      const int group = (tj * R + 7) >> 3;
      if (group * 8 < tj * R + R && group * 8 < g.NY) {
        const ulonglong2* src = mine && group * 8 + r < g.NY
                                    ? A.rowsum + ((size_t)q * nb + block_id(group, pl)) * 8 + r
                                    : nullptr;
        double v = 0.0;
        unsigned sv = seq0;
        if (src) msg_load(src, v, sv);
        const long long t0 = clock64();
        while (!__all_sync(kFull, sv == seq0)) {
          if (sv != seq0) msg_load(src, v, sv);
          if (__all_sync(kFull, sv == seq0)) break;
          if (rs_give_up(t0, A)) {
            ok = false;
            break;
          }
        }
        v += __shfl_down_sync(kFull, v, 4 * S);
        v += __shfl_down_sync(kFull, v, 2 * S);
        v += __shfl_down_sync(kFull, v, S);
        if (mine && r == 0) A.partials[(size_t)q * nb + block_id(group, pl)] = v;
      }
    }
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (__syncthreads_or(!ok)) return;
  if (threadIdx.x == 0) {
    __threadfence();
    am_last = atomicAdd(&A.ctl->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  if (threadIdx.x == 0) {
    A.ctl->ticket = 0;
    A.ctl->epoch += 1;
  }
  if constexpr (VM != 0) {
    // reduce_finish's order over the blocks: 256 threads' strided sums, then block_sum
    for (int vw = warp; vw < 8 * NDOT; vw += nw) {
      const double* src = A.partials + (size_t)(vw >> 3) * nb;
      double acc = 0.0;
      for (int b0 = (vw & 7) * 32 + lane; b0 < nb; b0 += 256 * 8) {
        double t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) t[u] = b0 + 256 * u < nb ? __ldcg(src + b0 + 256 * u) : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) acc += t[u];
      }
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(kFull, acc, o);
      if (lane == 0) red[vw] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double s[2] = {0.0, 0.0};
      for (int q = 0; q < NDOT; ++q) {
        const double* v = red + 8 * q;
        s[q] = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
      }
      finish_stage(VM == 1 ? kStageAlpha : kStageOmega, A.st, s[0], s[1]);
    }
  }
}

// ------------------------------------------------------------------------------------------
// solveSOR!'s passes (k_sor_pass) with theta on the chip: up to `sweeps` passes over both colours in one
// cooperative launch.  The tiles, messages and row updates are k_resident's; theta comes from memory, guards
// and masked cells included, and goes back at the end.  After each pass over both colours the tiles leave the
// blocks' sums of k_sor_pass and meet; the last one to arrive adds them in its order and tests for the end.
// What bounds it: the chain of row updates and messages of the two colour passes, then the chain of row sums,
// barrier and test (about half of the time of a small grid).  A pass over both colours: 169x169x30 15.1 us
// (two launches of k_sor_pass: 22.6), 72x70x30 10.2 us (14.9).
// ------------------------------------------------------------------------------------------
template <int R, int NP, bool BS>
__global__ void __launch_bounds__(32 * kRsMaxWarps, 1)
    k_resident_sor(const __grid_constant__ RsArgs A, double omega, double romega, int sweeps,
                   cudaGraphConditionalHandle hc, int use_cond) {
  extern __shared__ double sh[];
  __shared__ unsigned prog[kRsMaxWarps + 2];
  __shared__ int am_last, ended;
  __shared__ double red[16];
  // Fail-safe loop bound: every launch first ends the loop, before any test; only the finisher of a pass
  // (which runs after block 0 has arrived) can continue it.
  if (blockIdx.x == 0 && threadIdx.x == 0) set_cond(hc, use_cond, 0);
  if (A.st->stop || ld_relaxed_s32(A.err)) return;  // the same for every block
  const Geo& g = A.op.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int tile = blockIdx.x, xb = tile % A.nxb, tj = tile / A.nxb;
  const int NZ = g.NZ, j0 = 1 + tj * R, p = xb * 32 + lane;
  constexpr int P = kRsRowPitch, CP = R * P, PL = 2 * CP, BP = 2 * R * 32, KP = 2 * R * 32;
  double* X = sh + PL;
  double* T = sh + rs_x_elems(R, NZ);
  double* B = T + kRsTabRow * A.ntab;
  unsigned* K = reinterpret_cast<unsigned*>(B + (BS ? (NZ + 1) / 2 * 2 * BP : 0));
  const unsigned long long epoch = A.ctl->epoch;
  const unsigned seq0 = (unsigned)epoch * 16u;
  unsigned gen = ld_relaxed_u32(&A.ctl->go) & ~1u;
  const bool n_lo = tj > 0, n_hi = tj + 1 < A.ntj, n_xm = xb > 0, n_xp = xb + 1 < A.nxb;
  const int rows = min(R, g.NY - j0 + 1);
  const unsigned tab = saddr(T);
  const bool par0 = (1 + j0 + 1) & 1;
  const int NZe = (NZ + 1) & ~1;
  auto box_of = [&](int t, int pl) { return A.box + (size_t)(t * NZe + pl) * (2 * kRsBox); };
  auto pair_at = [&](int pl0) {
    RsPair a;
    const ulonglong2* zero = A.box - kRsZero;
    a.box = box_of(tile, pl0) + lane;
    a.mlo = n_lo ? ~0u : 0u;
    a.mhi = n_hi ? ~0u : 0u;
    // beside the first and the last row of the grid: boxes that hold the guards' theta
    a.lo = box_of(n_lo ? tile - A.nxb : (int)gridDim.x + xb, pl0) + 32 + lane;
    a.hi = box_of(n_hi ? tile + A.nxb : (int)gridDim.x + A.nxb + xb, pl0) + lane;
    const bool e = (1 + 1 + j0 + lane + pl0 + 1) & 1;
    const bool xa = lane < R && (e ? n_xp : n_xm), xb = lane < R && (e ? n_xm : n_xp);
    a.mxa = xa ? ~0u : 0u;
    a.mxb = xb ? ~0u : 0u;
    a.xa = xa ? box_of(e ? tile + 1 : tile - 1, pl0) + 64 + lane : zero;
    a.xb = xb ? box_of(e ? tile - 1 : tile + 1, pl0) + 64 + lane : zero;
    a.x = saddr(X + pl0 * PL + 1 + lane);
    a.edge = saddr(X + pl0 * PL + (lane < R ? lane : 0) * P);
    a.pad = e ? 264u : 0u;
    a.cls = saddr(K + (pl0 / 2) * KP + lane);
    return a;
  };
  auto inside = [&](int pl0, int r, int c, int w) {
    const int i = 2 * p + (((1 + j0 + r + pl0 + w + 1) & 1) ^ c);
    return pl0 + w < NZ && r < rows && p < g.HN && i >= 1 && i <= g.NX;
  };
  auto where = [&](int pl0, int r, int c, int w) { return g.row(c, j0 + r, pl0 + w + 1) + p; };
  // theta of any cell, guards and masked cells included (0 beyond the guards)
  auto theta = [&](int c, int j, int k) {
    return p < g.HN && j <= g.NY + 1 && k <= NZ + 1 ? __ldcg(A.xx + g.row(c, j, k) + p) : 0.0;
  };

  // ---- the tile's table, theta, classes, b; theta of colour 1 to the neighbours --------------------------
  if (threadIdx.x < kRsTabRow) T[threadIdx.x] = threadIdx.x == 8 ? 1.0 : 0.0;
  {
    const int n = A.count[tile];
    const uint16_t* list = A.list + (size_t)tile * kRsMaxTab;
    const double2* src = reinterpret_cast<const double2*>(A.op.ctab);
    for (int q = threadIdx.x; q < 4 * n; q += blockDim.x) {
      const double2 v = __ldg(src + 4 * (int)__ldg(list + (q >> 2)) + (q & 3));
      double2* t = reinterpret_cast<double2*>(T) + 5 * (1 + (q >> 2));
      t[(q & 3) + ((q & 3) > 0)] = v;
      if ((q & 3) == 0) t[1] = make_double2(v.y, v.x);
    }
  }
  if (threadIdx.x == 0) {
    prog[0] = prog[nw + 1] = ~0u;
    if (tile == 0) A.st->passes += 1;
  }
  if (lane == 0) prog[warp + 1] = 0u;
  const int NZx = (NZ + 1) / 2 * 2;
  for (int rc = warp; rc < 2 * R; rc += nw) {  // the planes below the first and above the last pair
    X[-PL + rc * P + 1 + lane] = theta(rc / R, j0 + rc % R, 0);
    X[NZx * PL + rc * P + 1 + lane] = theta(rc / R, j0 + rc % R, NZx + 1);
  }
#pragma unroll 1
  for (int np = 0; np < NP; ++np) {
    const int pl0 = (warp * NP + np) * 2;
    if (pl0 >= NZ) break;
    const RsPair a = pair_at(pl0);
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
      unsigned cl[4];
#pragma unroll
      for (int cw = 0; cw < 4; ++cw) {
        const int c = cw >> 1, w = cw & 1;
        const bool in = inside(pl0, r, c, w);
        const double t = theta(c, j0 + r, pl0 + w + 1);
        cl[cw] = in ? __ldg(A.lcls + where(pl0, r, c, w)) : 0u;
        double* x = X + (pl0 + w) * PL + c * CP + r * P + 1 + lane;
        x[0] = t;
        if (lane == 0) x[-1] = 0.0;
        if (lane == 31) x[1] = 0.0;
        if (BS) B[(pl0 + w) * BP + (c * R + r) * 32 + lane] = cl[cw] ? __ldg(A.v + where(pl0, r, c, w)) : 1.0;
        if (c == 1 && r == 0 && n_lo) msg_store(a.box + kRsBox + w * 2 * kRsBox, t, seq0);
        if (c == 1 && r == R - 1 && n_hi) msg_store(a.box + kRsBox + w * 2 * kRsBox + 32, t, seq0);
      }
      unsigned* kr = K + (pl0 / 2) * KP + r * 32 + lane;
      kr[0] = cl[0] | (cl[1] << 16);
      kr[R * 32] = cl[2] | (cl[3] << 16);
    }
#pragma unroll
    for (int cw = 0; cw < 4; ++cw) {
      const int c = cw >> 1, w = cw & 1, at = c * kRsBox + w * 2 * kRsBox;
      if (!n_lo) msg_store(const_cast<ulonglong2*>(a.lo) + at, theta(c, j0 - 1, pl0 + w + 1), 0u);
      if (!n_hi) msg_store(const_cast<ulonglong2*>(a.hi) + at, theta(c, j0 + R, pl0 + w + 1), 0u);
    }
    rs_send_edges<R>(a, 1, seq0, lane < R);
  }
  __syncthreads();
  rs_post(prog + warp + 1, 1u);

  bool ok = true;
  RsMsg m;
  RsCoef cf[2];
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    cf[w].cxa = cf[w].cxb = cf[w].cym = cf[w].cyp = cf[w].czm = cf[w].czp = cf[w].y = 0.0;
    cf[w].dd = 1.0;
  }
  unsigned cur = 0xffffffffu;
  const bool ends = lane == 0 || lane == R - 1, rest = lane < R && !ends;
  RsPair a = pair_at(warp * NP * 2);
  RsSor sor;
  sor.omega = omega;
  sor.romega = romega;
  const int gy = (g.NY + kBY - 1) / kBY, nb = A.nxb * gy * ((NZ + 1) / 2);
#pragma unroll 1
  for (unsigned n = 1;; ++n) {
    const int c = (n - 1) & 1;
    const unsigned seq = seq0 + n;
    const bool par = par0 ^ (c != 0);
    double f[2], l[2];
    const double* bv;
    auto first_b = [&](int pl) {
      bv = A.v + g.row(c, j0, pl + 1) + p;
      const int pp = pl + 1 < NZ ? (int)g.plane : 0;
      f[0] = bv[0];
      f[1] = bv[pp];
      if (R > 1) {
        l[0] = bv[(R - 1) * 2 * g.HP];
        l[1] = bv[(R - 1) * 2 * g.HP + pp];
      }
      return pp;
    };
    int plane = 0;
    if (NP == 1) {
      m.fetch(a, c ^ 1);
      if (!BS) plane = first_b(warp * 2);
    }
    rs_turn(cf);
    ok = rs_wait_planes(prog + warp, prog + warp + 2, n, A);
    // a warp has at most two pairs: their sums one after the other
    double sums[NP];
#pragma unroll
    for (int np = 0; np < NP; ++np) {
      sums[np] = 0.0;
      const int pl = (warp * NP + np) * 2;
      if (pl >= NZ || !ok) continue;
      if (NP > 1) {
        a = pair_at(pl);
        m.fetch(a, c ^ 1);
        if (!BS) plane = first_b(pl);
      }
      ok = rs_wait(m, a, c ^ 1, seq - 1, ends ? ~0u : 0u, A);
      if (!ok) continue;
      rs_put_edges<R>(m, a, c ^ 1, ends);
      if (R > 2 && __any_sync(kFull, m.edges_missing(a, c ^ 1, seq - 1, rest ? ~0u : 0u))) m.fetch_edges(a, c ^ 1);
      auto mid = [&] {
        rs_send_edges<R>(a, c, seq, ends);
        if (R <= 2) return true;
        if (!rs_wait_edges(m, a, c ^ 1, seq - 1, rest ? ~0u : 0u, A)) return false;
        rs_put_edges<R>(m, a, c ^ 1, rest);
        return true;
      };
      RsAddr ad;
      ad.x = a.x + (c ? CP * 8 : 0);
      ad.o = a.x + (c ? 0 : CP * 8);
      ad.oe = ad.o + (par ? 8u : -8u);
      ad.oo = ad.o - (par ? 8u : -8u);
      ad.cls = a.cls + (c ? R * 128 : 0);
      sor.sum = 0.0;
      sor.at = 0;
      ok = rs_rows<R, BS, true>(ad, tab, par ? 0u : 16u, saddr(B + pl * BP + c * (R * 32) + lane), bv, 2 * g.HP, plane,
                                f, l, cf, cur, m, a.box + c * kRsBox, n_lo, n_hi, seq, sor, mid);
      sums[np] = sor.sum;
      if (R > 2) rs_send_edges<R>(a, c, seq, rest);
      // lane r has row r's sum
      if (lane < rows)
        msg_store(A.rowsum + ((size_t)c * nb + xb + A.nxb * (((tj * R + lane) >> 3) + gy * (pl / 2))) * 8 +
                      ((tj * R + lane) & 7),
                  sums[np], seq);
    }
    rs_post(prog + warp + 1, n + 1);
    if (ok && c == 0) continue;

    // ---- after both colours: k_sor_pass's block sums, by the tile that holds a group's first row --------
    const int group = (tj * R + 7) >> 3;
    if (group * 8 < tj * R + R && group * 8 < g.NY) {
#pragma unroll 1
      for (int np = 0; np < NP; ++np) {
        const int pl = (warp * NP + np) * 2;
        if (pl >= NZ || !ok) break;
        const size_t id = (size_t)(lane >> 3) * nb + xb + A.nxb * (group + gy * (pl / 2));  // lane: colour * 8 + row
        const unsigned want = (lane >> 3) ? seq : seq - 1;
        const ulonglong2* src = lane < 16 && group * 8 + (lane & 7) < g.NY ? A.rowsum + id * 8 + (lane & 7) : nullptr;
        double v = 0.0;
        unsigned sv = want;
        if (src) msg_load(src, v, sv);
        const long long t0 = clock64();
        while (!__all_sync(kFull, sv == want)) {
          if (sv != want) msg_load(src, v, sv);
          if (__all_sync(kFull, sv == want)) break;
          if (rs_give_up(t0, A)) {
            ok = false;
            break;
          }
        }
        v += __shfl_down_sync(kFull, v, 4);
        v += __shfl_down_sync(kFull, v, 2);
        v += __shfl_down_sync(kFull, v, 1);
        if (lane == 0 || lane == 8) A.partials[id] = v;
      }
    }
    // ---- every block meets; the last one tests for the end -------------------------------------------------
    if (__syncthreads_or(!ok)) return;
    if (threadIdx.x == 0) {
      __threadfence();
      am_last = atomicAdd(&A.ctl->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    gen += 2;  // the lowest bit: the solve has ended
    bool good = true;
    if (am_last) {
      __threadfence();
      // ordered_sum and block_sum of k_sor_pass's 256 threads
      for (int vw = warp; vw < 16; vw += nw) {
        const double* src = A.partials + (size_t)(vw >> 3) * nb;
        double acc = 0.0;
        for (int b0 = (vw & 7) * 32 + lane; b0 < nb; b0 += 256 * 8) {
          double t[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) t[u] = b0 + 256 * u < nb ? __ldcg(src + b0 + 256 * u) : 0.0;
#pragma unroll
          for (int u = 0; u < 8; ++u) acc += t[u];
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(kFull, acc, o);
        if (lane == 0) red[vw] = acc;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        auto tree8 = [&](const double* v) {
          return ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
        };
        finish_stage(kStageSorHalf, A.st, tree8(red), 0.0);
        finish_stage(kStageSorIter, A.st, tree8(red + 8), 0.0);
        const bool stop = A.st->stop;
        if (n >= 2u * (unsigned)sweeps && !stop) set_cond(hc, use_cond, A.st->passes <= A.st->maxItr + 1);
        A.ctl->ticket = 0;
        A.ctl->epoch = epoch + n / 16u + 1;
        ended = stop;
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&A.ctl->go), "r"(gen | (stop ? 1u : 0u)) : "memory");
      }
    } else if (threadIdx.x == 0) {
      const long long t0 = clock64();
      for (;;) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&A.ctl->go) : "memory");
        if ((v & ~1u) == gen) {
          ended = v & 1u;
          break;
        }
        const bool late = clock64() - t0 > A.limit;
        if (late || ld_relaxed_s32(A.err)) {
          if (late) {
            atomicExch(A.err, 1);
            A.st->stop = 1;
            A.st->reason = kTimeout;
          }
          good = false;
          break;
        }
      }
    }
    if (__syncthreads_or(!good)) return;
    if (ended || n >= 2u * (unsigned)sweeps) break;
  }

  // ---- theta back to memory ------------------------------------------------------------------------------
#pragma unroll 1
  for (int np = 0; np < NP; ++np) {
    const int pl0 = (warp * NP + np) * 2;
    if (pl0 >= NZ) break;
#pragma unroll 1
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int cw = 0; cw < 4; ++cw)
        if (inside(pl0, r, cw >> 1, cw & 1))
          A.xx[where(pl0, r, cw >> 1, cw & 1)] = X[(pl0 + (cw & 1)) * PL + (cw >> 1) * CP + r * P + 1 + lane];
  }
}

}  // namespace h2g
