/* The fast pass of classify: one warp classifies a group of up to 32 nearby
 * points, one lane per point (included by wb_classify.cu).
 *
 * A group is up to 32 points that lie close together (groupOrderKernel puts
 * the points of a super-cell in an order whose runs of 32, and within them of
 * 8, are compact), so they share their neighbourhood, and the groups are its
 * index too: the warp walks the super-cells around its group once, the groups
 * of each, and the octets (runs of 8 points) of those.  A box at each of these
 * levels is read only if some lane's own hyperboloid can reach its lowest
 * point in a direction that still matters to the lane; the points of the
 * octets that remain are tested by all lanes, each against its own point.
 *
 * What a lane keeps of the directions seen.  The point is surrounded when
 * every circular gap between its directions is below 144 degrees.  A gap
 * below that can never decide the point again (gaps only shrink), and at most
 * two gaps of 144 degrees fit a circle, so a lane keeps only those: its open
 * arcs, as pairs of unit rays.  A candidate inside the hyperboloid matters
 * only if its direction falls into an open arc; two cross products say so,
 * no direction is formed, and an arc that is split keeps the halves that are
 * still wide enough.  No open arc left: surrounded.
 *
 * Error of the arcs.  The rays are FP32 unit vectors (error below 5e-7 rad)
 * and are turned inward by kRayPad, so a direction that rounding puts on the
 * wrong side of a ray moves it by less than the pad and an arc never grows.
 * An arc narrower than 144 degrees - kArcBand is closed and one wider than
 * 144 degrees + kArcBand proves the point not surrounded; a point whose widest
 * arc ends between the two is ambiguous and re-run (with exact directions, or
 * in the precision mode with the FP32 directions of the one-point kernel).
 * kArcBand is 1.2e-5 rad.
 *
 * Lengths are in x record units, heights divided by the slope: a point is
 * inside the hyperboloid when zd > 0 and zd^2 - ex^2 - ey^2 >= por^2.
 *
 * Bound: instruction issue (80% of the slots at 24 warps per SM, DRAM idle; 50M
 * points at 100 per square metre: 30,500 warp instructions a group, of which
 * 42% test candidates and update arcs, 20% octet boxes, 11% group boxes, 10%
 * staging, 15% listing).  The classify stage takes 50.3 ms there; 104 ms before
 * with groups of one column's points by height, 8 direction bins a lane (FP32
 * arctangents) and envelope tests only.  On the way: arcs instead of bins 85,
 * the lane's own reach per column, four candidates a step and updates by the
 * lanes that need them 58, compact groups as the index with octet boxes 54,
 * packed FP32 52, candidates held against the arcs before the update 50 ms. */

constexpr float kRayPad = 1e-6f;
/* cos(144 degrees -+ kArcBand) */
constexpr float kCosOpen = -0.809009940f, kCosSure = -0.809024048f;
/* Groups a group reads before it hands its undecided points over to the
 * one-point kernel.  A point alone needs nearly as many reads as its group (at
 * 64 reads 50M points take 92 ms, at 128 60, at 256 52, at 400 and 700 50.4), so
 * the limit only bounds the longest group. */
constexpr int kGroupReads = 512;

/* Two FP32 values in one register pair: the packed instructions take one
 * issue slot for both. */
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float a, float b)
{
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void split(f32x2 v, float &a, float &b)
{
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

struct GroupShared
{
  /* the group being read: x, y, -z in record units from the origin of the
     warp's own group, -z minus infinity where there is no point to test
     in FP32; the octets' boxes (WbBoxF) and lowest z */
  alignas(16) float cx[32], cy[32], cz[32];
  float4 obox[4];
  float oz[4];
  /* a lane's second open arc, while it has one */
  float2 arc2a[32], arc2b[32];
  /* the groups and super-cells the lanes hold while the warp walks them */
  float4 nbox[32], sbox[32];
  int4 nrec[32];   /* zmin (a float from the origin), first, points, flags */
  int4 srec[32];   /* zmin (likewise), first group, groups, flags */
};

/* Monotone map of floats to signed integers, and back. */
__device__ __forceinline__ int orderedInt(float f)
{
  const int i = __float_as_int(f);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float orderedFloat(int i)
{
  return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}

/* A lane's open arcs.  nDir: 0 no direction yet, 1 one direction (or a cluster
 * of them too narrow to tell its two ends apart: b its clockwise end, a its
 * counter-clockwise end), 2 open arcs with two rays.  The first arc runs
 * counter-clockwise from side * a to side * b, side -1 for an arc wider than a
 * half turn: a direction c falls into it when
 * side * min(cross(a, c), cross(c, b)) > 0.  A second one is in shared memory
 * (two).  open false: no open arc is left, the point is surrounded. */
struct LaneArcs
{
  float ax, ay, bx, by, side;
  int nDir;
  bool two, open;
};

/* Whether the arc from ray p counter-clockwise to ray q is open, at least 144
 * degrees - kArcBand wide: cr and dt their cross and dot product.  A half
 * narrower than the pads, whose rays have crossed, has cr near 0 from below and
 * dt near 1: not open. */
__device__ __forceinline__ bool arcOpen(float cr, float dt)
{
  return (dt <= kCosOpen) | (cr < -1e-5f);
}

/* Adds direction (ux, uy), a unit vector, to a lane's arcs: splits the open
 * arc it falls into.  Arc starts are turned counter-clockwise by the pad, arc
 * ends back. */
__device__ __noinline__ LaneArcs addDirection(LaneArcs s, float ux, float uy, float2 *arc2a, float2 *arc2b)
{
  if (s.nDir == 0)
  {
    s.nDir = 1;
    s.ax = s.bx = ux;
    s.ay = s.by = uy;
    return s;
  }
  const float lx = __fmaf_rn(-kRayPad, uy, ux), ly = __fmaf_rn(kRayPad, ux, uy);   // u as the start of an arc
  const float rx = __fmaf_rn(kRayPad, uy, ux), ry = __fmaf_rn(-kRayPad, ux, uy);   // u as the end of an arc
  // the arc u splits, from p to q, and the lane's other one, from o to n
  float px = s.ax * s.side, py = s.ay * s.side, qx = s.bx * s.side, qy = s.by * s.side;
  float ox = 0.f, oy = 0.f, nx = 0.f, ny = 0.f;
  bool other = false;
  if (s.nDir == 1)
  {
    const float cr = s.ax * uy - s.ay * ux, dt = s.ax * ux + s.ay * uy;
    const bool near = fabsf(cr) <= 1e-3f && dt > 0.f;
    if (near)
    {
      // within a milliradian of the cluster: widen it
      if (cr > 0.f)
      {
        s.ax = ux;
        s.ay = uy;
      }
      else if (s.bx * uy - s.by * ux < 0.f)
      {
        s.bx = ux;
        s.by = uy;
      }
      if (!(fabsf(s.bx * s.ay - s.by * s.ax) > 5e-4f))
        return s;
    }
    // the cluster's ends as rays of one open arc from a around to b
    px = __fmaf_rn(-kRayPad, s.ay, s.ax);
    py = __fmaf_rn(kRayPad, s.ax, s.ay);
    qx = __fmaf_rn(kRayPad, s.by, s.bx);
    qy = __fmaf_rn(-kRayPad, s.bx, s.by);
    s.nDir = 2;
    if (near)
    {
      s.side = -1.f;
      s.ax = -px;
      s.ay = -py;
      s.bx = -qx;
      s.by = -qy;
      return s;
    }
  }
  else
  {
    if (s.two)
    {
      // u can fall into one of the two arcs
      const float2 p2 = *arc2a, q2 = *arc2b;
      const bool w2 = p2.x * q2.y - p2.y * q2.x < 0.f;
      const float c0 = p2.x * uy - p2.y * ux, c1 = ux * q2.y - uy * q2.x;
      other = true;
      ox = p2.x;
      oy = p2.y;
      nx = q2.x;
      ny = q2.y;
      if (w2 ? (c0 > 0.f || c1 > 0.f) : (c0 > 0.f && c1 > 0.f))
      {
        ox = px;
        oy = py;
        nx = qx;
        ny = qy;
        px = p2.x;
        py = p2.y;
        qx = q2.x;
        qy = q2.y;
      }
    }
    const float c0 = px * uy - py * ux, c1 = ux * qy - uy * qx;
    if (!(px * qy - py * qx < 0.f ? (c0 > 0.f || c1 > 0.f) : (c0 > 0.f && c1 > 0.f)))
      return s;
  }
  const bool o0 = arcOpen(px * ry - py * rx, px * rx + py * ry), o1 = arcOpen(lx * qy - ly * qx, lx * qx + ly * qy);
  s.open = o0 || o1 || other;
  s.two = o0 ? (o1 || other) : (o1 && other);
  if (s.two)
  {
    *arc2a = o0 && o1 ? make_float2(lx, ly) : make_float2(ox, oy);
    *arc2b = o0 && o1 ? make_float2(qx, qy) : make_float2(nx, ny);
  }
  const bool none = !o0 && !o1;
  const float nax = none ? ox : (o0 ? px : lx), nay = none ? oy : (o0 ? py : ly);
  const float nbx = none ? nx : (o0 ? rx : qx), nby = none ? ny : (o0 ? ry : qy);
  s.side = nax * nby - nay * nbx < 0.f ? -1.f : 1.f;
  s.ax = nax * s.side;
  s.ay = nay * s.side;
  s.bx = nbx * s.side;
  s.by = nby * s.side;
  return s;
}

/* Splits a lane's only open arc by a direction (ux, uy) inside it: the half
 * that stays open replaces the arc.  Returns the open halves; with both open
 * the second is left in (lx, ly)-(qx, qy). */
__device__ __forceinline__ int splitArc(float ux, float uy, float &ax, float &ay, float &bx, float &by, float &side,
                                        float2 &l, float2 &q)
{
  const float lx = __fmaf_rn(-kRayPad, uy, ux), ly = __fmaf_rn(kRayPad, ux, uy);
  const float rx = __fmaf_rn(kRayPad, uy, ux), ry = __fmaf_rn(-kRayPad, ux, uy);
  const float cr0 = side * __fmaf_rn(ax, ry, -(ay * rx)), d0 = side * __fmaf_rn(ax, rx, ay * ry);
  const float cr1 = side * __fmaf_rn(lx, by, -(ly * bx)), d1 = side * __fmaf_rn(lx, bx, ly * by);
  const bool o0 = arcOpen(cr0, d0), o1 = arcOpen(cr1, d1);
  l = make_float2(lx, ly);
  q = make_float2(bx * side, by * side);
  const float ns = (o0 ? cr0 : cr1) < 0.f ? -1.f : 1.f, t = ns * side;
  ax = o0 ? ax * t : lx * ns;
  ay = o0 ? ay * t : ly * ns;
  bx = o0 ? rx * ns : bx * t;
  by = o0 ? ry * ns : by * t;
  side = ns;
  return (int)o0 + (int)o1;
}

/* The block of a point outside the root cube, from the origin (X, Y, Z) in record
 * units: x and y range, top and bottom of its cube. */
struct BlockBounds
{
  float x0, x1, y0, y1, top, bottom;
};
__device__ __noinline__ BlockBounds blockBounds(const ClsArgs &a, uint32_t j, int X, int Y, int Z)
{
  const uint32_t l = a.leafId[j];
  double cx, cy, cz, side;
  wb_leaf_cube(a.leafKey[l], a.leafLev[l], a.rootLo, a.rootSide, cx, cy, cz, side);
  const double h = side / 2;
  BlockBounds b;
  b.x0 = (float)((cx - h - a.unitOff[0]) * a.perStep[0] - X);
  b.x1 = (float)((cx + h - a.unitOff[0]) * a.perStep[0] - X);
  b.y0 = (float)((cy - h - a.unitOff[1]) * a.perStep[1] - Y);
  b.y1 = (float)((cy + h - a.unitOff[1]) * a.perStep[1] - Y);
  b.top = (float)((cz + h - a.unitOff[2]) * a.perStep[2] - Z);
  b.bottom = (float)((cz - h - a.unitOff[2]) * a.perStep[2] - Z);
  return b;
}

/* STRAYS: some cloud of the launch has points beside or above the root cube (those
 * below it are members by themselves, when their block meets the hyperboloid). */
template <bool STRAYS>
__device__ __forceinline__ void classifyGroupArcs(const ClsArgs &a, uint64_t group, int lane, GroupShared &sm)
{
  constexpr unsigned kAll = 0xffffffffu;
  bool act = false;
  int4 me = make_int4(0, 0, 0, 0);
  PtSetup ps{};
  uint32_t j = 0;
  const int4 own = a.groups[2 * group + 1];
  if (lane < own.z)
  {
    const int2 p = a.bxy[(uint32_t)own.y + lane], q = a.bzw[(uint32_t)own.y + lane];
    me = make_int4(p.x, p.y, q.x, q.y);
    j = (uint32_t)me.w & 0x7fffffffu;
    if (a.owner[j] >= 0)
    {
      act = true;
      ps = a.setup[j];
    }
    else
      a.label[j] = 0;
  }
  if (!__any_sync(kAll, act))
    return;
  if (!a.exactInts)
  {
    // FP32 differences are not exact for this cloud: the exact pass decides
    if (act)
    {
      a.label[j] = 2;
      a.ambList[atomicAdd(a.ambCount, 1u)] = j;
    }
    return;
  }
  // the group's box in record integers; its low corner is the origin of the
  // FP32 frame, in which the group's own points are exact
  const int gx0 = __reduce_min_sync(kAll, act ? me.x : INT32_MAX), gx1 = __reduce_max_sync(kAll, act ? me.x : INT32_MIN);
  const int gy0 = __reduce_min_sync(kAll, act ? me.y : INT32_MAX), gy1 = __reduce_max_sync(kAll, act ? me.y : INT32_MIN);
  const int gz0 = __reduce_min_sync(kAll, act ? me.z : INT32_MAX), gz1 = __reduce_max_sync(kAll, act ? me.z : INT32_MIN);
  const float ky = a.gky, kz = a.gkz, inv = a.gInv;
  const bool wideBox = max(max(gx1 - gx0, gy1 - gy0), gz1 - gz0) >= (1 << 22) || !(fminf(ky, kz) > 1e-9f) || !(fmaxf(ky, kz) < 1e9f);
  const float czp = ps.czp * inv, por2 = ps.por2f * inv * inv;
  // relative error of zd^2 at the boundary: 1e-5 covers the FP32 arithmetic
  // while |czp| is of the order of por (a thickness of the order of the
  // hyperboloid size); it grows with |czp| / por
  const float ratio = fabsf(czp) * rsqrtf(por2);
  const float eps = 1e-5f + 4e-7f * ratio;
  bool deferred = act && (wideBox || !(ratio < 1e5f) || !(por2 > 0.f && por2 < 1e30f));
  if (deferred)
    a.deferList[atomicAdd(a.deferCount, 1u)] = j;
  bool done = !act || deferred;
  // zd^2 kOut - pOut < r2: surely outside; zd^2 > kOut (r2 + pIn): surely inside
  const float kOut = (1.f + eps) / (1.f - eps);
  const float pOut = por2 - a.gTiny;
  const float mx = (float)(me.x - gx0), my = (float)(me.y - gy0);
  const float mys = my * ky, bw = (float)(gx1 - gx0), bh = (float)(gy1 - gy0) * ky;
  float mz = (float)(me.z - gz0);   // -infinity once the lane is done: then nothing is inside
  const int ci0 = min(max((__reduce_min_sync(kAll, act ? ps.ci : INT32_MAX) + __reduce_max_sync(kAll, act ? ps.ci : INT32_MIN)) / 2, 0), a.nx - 1);
  const int cj0 = min(max((__reduce_min_sync(kAll, act ? ps.cj : INT32_MAX) + __reduce_max_sync(kAll, act ? ps.cj : INT32_MIN)) / 2, 0), a.ny - 1);
  const int offG = max(abs(ps.ci - ci0), abs(ps.cj - cj0));
  const int smaxL = ps.smax + (offG + WB_SUPER - 1) / WB_SUPER + 1;

  // the lane's open arcs (LaneArcs); slow: addDirection decides whether a
  // candidate's direction falls into one (arcMin is -infinity then)
  int nDir = 0;
  bool slow = true, two = false;
  float side = 1.f, arcMin = -INFINITY, ax = 0.f, ay = 0.f, bx = 0.f, by = 0.f;
  if (done)
    mz = -INFINITY;

  // the envelope of the lanes still undecided.  The apex, and a box's height below
  // it, are rounded eight times in all by 6e-8 of |czp| (the centre, the two
  // factors, their products and sums) and four times by 6e-8 of the lane's height in
  // the group: the apex is raised by 6e-7 of both, so that the envelope holds every
  // lane's hyperboloid however far its centre lies from it (|czp| / por below 1e5)
  float apex, pK;
  int smaxG;
  auto envelope = [&]() {
    apex = orderedFloat(__reduce_max_sync(kAll, orderedInt(done ? -INFINITY : __fmaf_rn(mz, kz, czp) + 6e-7f * __fmaf_rn(mz, kz, fabsf(czp)))));
    // members have zd^2 - r2 >= por^2; 1.0004 zd^2 - r2 >= pK allows for rounding
    pK = __int_as_float(__reduce_min_sync(kAll, done ? 0x7f800000 : __float_as_int(por2))) * 0.9998f - a.gTiny;
    smaxG = __reduce_max_sync(kAll, done ? 0 : smaxL);
  };
  envelope();
  // can a box {x0, y0, x1, y1} with lowest point zmin hold a member of any lane?
  auto envReached = [&](const int4 &b, int32_t zmin) -> bool {
    if (b.x == INT32_MAX)
      return false;
    const float dx = (float)max(0, max(b.x - gx1, gx0 - b.z)), dy = (float)max(0, max(b.y - gy1, gy0 - b.w)) * ky;
    const float zd = apex - (float)(zmin - gz0) * kz;
    const float r2 = __fmaf_rn(dx, dx, dy * dy);
    return __fmaf_rn(zd * fabsf(zd), 1.0004f, -pK) >= r2;
  };
  // the same of a super-cell or group (bounds, record), also by the blocks of its
  // points beside or above the root cube (flags, sr): one whose block lies in a
  // lane's hyperboloid as a whole is a member wherever it is itself
  auto envMeets = [&](const int4 &b, const int4 &r, const int4 *sr) -> bool {
    return envReached(b, r.x) || (STRAYS && r.w && envReached(sr[0], sr[1].x));
  };
#ifdef WB_CLASSIFY_STATS
  unsigned long long gst[16] = {0};
  const long long tG = clock64();
#endif

  // adds the direction of lanes with `add`, any state
  auto addAny = [&](bool add, float ex, float ey, float rr) {
    if (add)
    {
      const float il = rsqrtf(rr);
      const LaneArcs r = addDirection(LaneArcs{ax, ay, bx, by, side, nDir, two, true}, ex * il, ey * il,
                                      &sm.arc2a[lane], &sm.arc2b[lane]);
      ax = r.ax;
      ay = r.ay;
      bx = r.bx;
      by = r.by;
      side = r.side;
      nDir = r.nDir;
      two = r.two;
      slow = two || nDir < 2;
      arcMin = slow ? -INFINITY : 0.f;
      if (!r.open)
      {
        done = true;   // surrounded
        mz = -INFINITY;
      }
    }
  };
  // Tests the octet of the staged group from entry k0.  Four candidates a
  // step, so that their latencies overlap; then the lanes that found some
  // inside an open arc add them, each lane its own, and those FP32 cannot
  // decide wait for the exact test at the end (pend, by entry).
  unsigned pend = 0;
  auto testOctet = [&](int k) {
    {
      unsigned hits = 0;
      const f32x2 mx2 = pair(-mx, -mx), my2 = pair(-my, -my), ky2 = pair(ky, ky), mz2 = pair(mz, mz), kz2 = pair(kz, kz), czp2 = pair(czp, czp);
      const f32x2 ax2 = pair(ax, ax), nay2 = pair(-ay, -ay), by2 = pair(by, by), nbx2 = pair(-bx, -bx), side2 = pair(side, side);
      const f32x2 kOut2 = pair(kOut, kOut), pOut2 = pair(-pOut, -pOut);
#pragma unroll
      for (int q = 0; q < 8; q += 4)
      {
        const ulonglong2 vx = *(const ulonglong2 *)&sm.cx[k + q], vy = *(const ulonglong2 *)&sm.cy[k + q], vz = *(const ulonglong2 *)&sm.cz[k + q];
#pragma unroll
        for (int p = 0; p < 2; p++)
        {
          const f32x2 ex = add2(p ? vx.y : vx.x, mx2), ey = mul2(add2(p ? vy.y : vy.x, my2), ky2);
          const f32x2 zd = fma2(add2(p ? vz.y : vz.x, mz2), kz2, czp2);   // cz holds -z
          const f32x2 rr = fma2(ex, ex, mul2(ey, ey));
          const f32x2 t0 = fma2(ax2, ey, mul2(nay2, ex)), t1 = fma2(by2, ex, mul2(nbx2, ey));
          float z0, z1, r0, r1, u0, u1, v0, v1;
          split(zd, z0, z1);
          split(rr, r0, r1);
          split(t0, u0, u1);
          split(t1, v0, v1);
          const f32x2 w = fma2(pair(z0 * fabsf(z0), z1 * fabsf(z1)), kOut2, pOut2);
          const f32x2 v = mul2(pair(fminf(u0, v0), fminf(u1, v1)), side2);
          float w0, w1, m0, m1;
          split(w, w0, w1);
          split(v, m0, m1);
          hits |= (unsigned)((w0 >= r0) & (m0 > arcMin)) << (q + 2 * p);
          hits |= (unsigned)((w1 >= r1) & (m1 > arcMin)) << (q + 2 * p + 1);
        }
      }
#pragma unroll 1
      while (__any_sync(kAll, hits != 0))
      {
        WB_STAT(gst[10], 1);
        const int kk = max(k + __ffs(hits) - 1, 0);
        const float ex = sm.cx[kk] - mx, ey = (sm.cy[kk] - my) * ky;
        // the arc may have shrunk since the candidate was found in it, and a lane
        // with two arcs found all candidates inside
        bool in = side * fminf(__fmaf_rn(ax, ey, -(ay * ex)), __fmaf_rn(ex, by, -(ey * bx))) > (two ? 0.f : arcMin);
        if (two & !in)
        {
          const float2 p2 = sm.arc2a[lane], q2 = sm.arc2b[lane];
          const float c0 = p2.x * ey - p2.y * ex, c1 = ex * q2.y - ey * q2.x;
          in = p2.x * q2.y - p2.y * q2.x < 0.f ? (c0 > 0.f) | (c1 > 0.f) : (c0 > 0.f) & (c1 > 0.f);
        }
        in = in & (hits != 0) & !done;
        hits &= hits - 1;
        if (!__any_sync(kAll, in))
          continue;
        const float zd = __fmaf_rn(mz + sm.cz[kk], kz, czp);
        const float rr = __fmaf_rn(ex, ex, ey * ey);
        in = in & (rr > 0.f);
        const bool sure = zd * zd > kOut * (rr + por2 + a.gTiny);
        if (in & !sure)
          pend |= 1u << kk;
        in = in & sure;
        const bool any = in & slow;
        if (__any_sync(kAll, any))
          addAny(any, ex, ey, rr);
        in = in & !any;
        if (__any_sync(kAll, in))
        {
          const float il = rsqrtf(rr), ux = ex * il, uy = ey * il;
          if (in)
          {
            float2 l, q;
            const int open = splitArc(ux, uy, ax, ay, bx, by, side, l, q);
            if (open == 2)
            {
              sm.arc2a[lane] = l;
              sm.arc2b[lane] = q;
              two = slow = true;
              arcMin = -INFINITY;
            }
            if (open == 0)
            {
              done = true;   // surrounded
              mz = -INFINITY;
            }
          }
        }
      }
    }
  };
  // the candidates of the staged group (first: its first point) that FP32
  // could not decide, and members outside the root cube
  auto testExact = [&](uint32_t first, unsigned members) {
#pragma unroll 1
    while (__any_sync(kAll, pend != 0))
    {
      bool in = false;
      float ex = 0.f, ey = 0.f, rr = 0.f;
      if (pend && !done)
      {
        const uint32_t at = first + __ffs(pend) - 1;
        const int2 q = a.bxy[at], r = a.bzw[at];
        const int dxi = q.x - me.x, dyi = q.y - me.y;
        // dist(p,q) == 0 gives no direction (classify.cpp:142,153)
        if (dxi != 0 || dyi != 0)
        {
          if (STRAYS && (members & pend & (0u - pend)))
            in = true;
          else if (a.fp32Only && r.y >= 0)
          {
            const float dx = (float)dxi * a.fsx, dy = (float)dyi * a.fsy;
            const float zd = (float)(me.z - r.x) * a.fsz + a.setup[j].czp;
            const float r2 = a.fs2 * __fmaf_rn(dx, dx, dy * dy);
            in = zd > 0 && __fmaf_rn(zd, zd, -r2) - a.setup[j].por2f > 0;
          }
          else
            in = memberExact(a, exactHyp(a, j), (uint32_t)r.y, q.x, q.y, r.x);
        }
        ex = (float)dxi;
        ey = (float)dyi * ky;
        rr = __fmaf_rn(ex, ex, ey * ey);
      }
      pend &= pend - 1;
      addAny(in, ex, ey, rr);
    }
  };

  // Boxes as {centre x, centre y, half width, half height} from the origin in x
  // record units, the halves widened by more than the rounding here and below.
  auto boxOf = [&](float x0, float x1, float y0, float y1) -> float4 {
    const float cx = 0.5f * (x0 + x1), cy = 0.5f * (y0 + y1), hx = 0.5f * (x1 - x0), hy = 0.5f * (y1 - y0);
    const float pad = 4e-6f * (fabsf(cx) + fabsf(cy) + hx + hy + bw + bh);
    return make_float4(cx, cy, hx + pad, hy + pad);
  };
  auto boxOfInts = [&](const int4 &b) -> float4 {
    return boxOf((float)(b.x - gx0), (float)(b.z - gx0), (float)(b.y - gy0) * ky, (float)(b.w - gy0) * ky);
  };
  // whether a box whose lowest point is zmin may hold a member of some
  // undecided lane in a direction of the lane's open arc: the nearest point of
  // the box against the hyperboloid, and the largest value of a cross product
  // over a box, its value at the centre plus the halves' shares.  Boxes holding
  // points beside or above the root cube (flags, their record's number plus one)
  // are also reached by those points' blocks.
  auto blocksReached = [&](const int4 &c, int z) -> bool {
    const float4 b = boxOfInts(c);
    const float dx = fmaxf(0.f, fabsf(b.x - mx) - b.z), dy = fmaxf(0.f, fabsf(b.y - mys) - b.w);
    const float zd = __fmaf_rn(mz - (float)(z - gz0), kz, czp);
    return __fmaf_rn(zd * fabsf(zd), kOut, -pOut) >= __fmaf_rn(dx, dx, dy * dy);
  };
  auto blockWanted = [&](int flags, const int4 *strays) -> bool {
    return STRAYS && flags && blocksReached(strays[2 * (flags - 1)], strays[2 * (flags - 1) + 1].x);
  };
  auto boxWanted = [&](const float4 &b, float zmin, bool block) -> bool {
    const float ex = b.x - mx, ey = b.y - mys;
    const float dx = fmaxf(0.f, fabsf(ex) - b.z), dy = fmaxf(0.f, fabsf(ey) - b.w);
    const float zd = __fmaf_rn(mz - zmin, kz, czp);
    const bool reach = __fmaf_rn(zd * fabsf(zd), kOut, -pOut) >= __fmaf_rn(dx, dx, dy * dy);
    const float A = __fmaf_rn(side, __fmaf_rn(ax, ey, -(ay * ex)), __fmaf_rn(fabsf(ay), b.z, fabsf(ax) * b.w));
    const float B = __fmaf_rn(side, __fmaf_rn(ex, by, -(ey * bx)), __fmaf_rn(fabsf(by), b.z, fabsf(bx) * b.w));
    const float v = side < 0.f ? fmaxf(A, B) : fminf(A, B);
    return __any_sync(kAll, (block | reach) & !done & (v >= arcMin));
  };

  // The walk, as one loop so that each part is there once: the next group of
  // the list; else put the next super-cell's groups in the list, 32 at a time;
  // else find the next 32 super-cells of the ring or the next ring.
  constexpr int S = WB_SUPER;
  const int si = ci0 / S, sj = cj0 / S;
  unsigned list = 0, supers = 0;             // left in the two lists
  uint32_t gNext = 0, gEnd = 0;              // groups of the current super-cell not listed yet
  int sr = -1, m0 = 0, nsc = 0;
  int reads = 0;
#pragma unroll 1
  for (;;)
  {
    if (list)
    {
      const int src = __ffs(list) - 1;
      list &= list - 1;
      WB_STAT(gst[3], 1);
      const int4 r = sm.nrec[src];
      if (!boxWanted(sm.nbox[src], __int_as_float(r.x), blockWanted(r.w, a.strayGrp)))
        continue;
      if (reads >= kGroupReads)
      {
        // a group whose neighbourhood is very large would hold one warp while
        // the rest of the GPU idles: its undecided points go to the one-point
        // kernel
        if (!done)
        {
          deferred = true;
          a.deferList[atomicAdd(a.deferCount, 1u)] = j;
        }
        break;
      }
      reads++;
      // stage the group, with its octets' boxes
      float x = 0.f, y = 0.f, z = INFINITY;
      int where = 0;   // store position and stray bit
      if (lane < r.z)
      {
        const int2 p = a.bxy[(uint32_t)r.y + lane], q = a.bzw[(uint32_t)r.y + lane];
        x = (float)(p.x - gx0);
        y = (float)(p.y - gy0);
        z = (float)(q.x - gz0);
        where = q.y;
      }
      const unsigned strays = __ballot_sync(kAll, where < 0);
      float x0 = z < INFINITY ? x : INFINITY, x1 = z < INFINITY ? x : -INFINITY;
      float y0 = z < INFINITY ? y : INFINITY, y1 = z < INFINITY ? y : -INFINITY, z0 = z;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1)
      {
        x0 = fminf(x0, __shfl_xor_sync(kAll, x0, o));
        x1 = fmaxf(x1, __shfl_xor_sync(kAll, x1, o));
        y0 = fminf(y0, __shfl_xor_sync(kAll, y0, o));
        y1 = fmaxf(y1, __shfl_xor_sync(kAll, y1, o));
        z0 = fminf(z0, __shfl_xor_sync(kAll, z0, o));
      }
      __syncwarp();
      sm.cx[lane] = x;
      sm.cy[lane] = y;
      sm.cz[lane] = where < 0 ? -INFINITY : -z;   // not in the octets' test
      if ((lane & 7) == 0)
      {
        sm.obox[lane >> 3] = boxOf(x0, x1, y0 * ky, y1 * ky);
        sm.oz[lane >> 3] = z0;
      }
      __syncwarp();
      const bool wasDone = done;
      pend = STRAYS || done ? 0u : strays;   // for the exact test
      unsigned members = 0;   // of pend: members for certain
      if (STRAYS && strays)
      {
        BlockBounds block{};
        if (where < 0)
          block = blockBounds(a, (uint32_t)where & 0x7fffffffu, gx0, gy0, gz0);
        __syncwarp();
        // The points outside the root cube, one after another: a member's block
        // meets the lane's hyperboloid (its cube's nearest point at the bottom),
        // and either the point is inside or the block as a whole is (its farthest
        // corner at the top).  Decided in FP32 with the rounding of the bounds
        // (half a record unit and 1e-6) and of the heights allowed for either way;
        // what that leaves in doubt waits for the exact test.
#pragma unroll 1
        for (unsigned left = strays; left; left &= left - 1)
        {
          const int k = __ffs(left) - 1;
          const float x0 = __shfl_sync(kAll, block.x0, k), x1 = __shfl_sync(kAll, block.x1, k);
          const float y0 = __shfl_sync(kAll, block.y0, k) * ky, y1 = __shfl_sync(kAll, block.y1, k) * ky;
          const float zt = __shfl_sync(kAll, block.top, k), zb = __shfl_sync(kAll, block.bottom, k);
          const float ex = sm.cx[k] - mx, ey = (sm.cy[k] - my) * ky, rr = __fmaf_rn(ex, ex, ey * ey);
          const float zd = __fmaf_rn(mz - __shfl_sync(kAll, z, k), kz, czp);
          const float px = 0.5f + 1e-6f * (fabsf(x0) + fabsf(x1) + bw), py = 0.5f * ky + 1e-6f * (fabsf(y0) + fabsf(y1) + bh);
          const float nx = fmaxf(x0 - mx, mx - x1), ny = fmaxf(y0 - mys, mys - y1);
          const float fx = fmaxf(mx - x0, x1 - mx), fy = fmaxf(mys - y0, y1 - mys), pz = 0.5f * kz;
          auto may = [&](float h, float dx, float dy) -> bool {
            const float d = fmaxf(0.f, dx), e = fmaxf(0.f, dy);
            return __fmaf_rn(h * fabsf(h), kOut, -pOut) >= __fmaf_rn(d, d, e * e);
          };
          auto sure = [&](float h, float dx, float dy) -> bool {
            const float d = fmaxf(0.f, dx), e = fmaxf(0.f, dy);
            return h > 0.f && h * h > kOut * (__fmaf_rn(d, d, e * e) + por2 + a.gTiny);
          };
          const float hb = __fmaf_rn(mz - zb, kz, czp), ht = __fmaf_rn(mz - zt, kz, czp);
          const bool arc = side * fminf(__fmaf_rn(ax, ey, -(ay * ex)), __fmaf_rn(ex, by, -(ey * bx))) > arcMin;
          const bool wanted = !done & arc & (rr > 0.f);
          const bool out = !may(hb + pz, nx - px, ny - py) || !(may(zd, fabsf(ex), fabsf(ey)) || may(ht + pz, fx - px, fy - py));
          const bool in = sure(hb - pz, nx + px, ny + py) && (sure(zd, fabsf(ex), fabsf(ey)) || sure(ht - pz, fx + px, fy + py));
          if (wanted & (in | !out))
            pend |= 1u << k;
          if (wanted & in)
            members |= 1u << k;
        }
      }
#pragma unroll 1
      for (int o = 0; 8 * o < r.z; o++)
      {
        WB_STAT(gst[2], 1);
        if (boxWanted(sm.obox[o], sm.oz[o], false))
        {
          WB_STAT(gst[6], 8);
          WB_STAT(gst[7], 8 * __popc(__ballot_sync(kAll, !done)));
#ifdef WB_CLASSIFY_STATS
          const long long tB = clock64();
#endif
          testOctet(8 * o);
          WB_STAT(gst[8], clock64() - tB);
        }
      }
      testExact((uint32_t)r.y, members);
      if (__any_sync(kAll, done != wasDone))
      {
        if (__all_sync(kAll, done))
          break;
        envelope();
      }
      continue;
    }
    int4 b = make_int4(INT32_MAX, 0, 0, 0), r = make_int4(0, 0, 0, 0);
    if (gNext < gEnd)
    {
      // the super-cell's next 32 groups
      if (gNext + lane < gEnd)
      {
        b = a.groups[2 * (uint64_t)(gNext + lane)];
        r = a.groups[2 * (uint64_t)(gNext + lane) + 1];
      }
      gNext += 32;
      if constexpr (STRAYS)
        list = __ballot_sync(kAll, envMeets(b, r, a.strayGrp + 2 * (uint64_t)(gNext - 32 + lane)));
      else
        list = __ballot_sync(kAll, envReached(b, r.x));
      __syncwarp();
      sm.nbox[lane] = boxOfInts(b);
      sm.nrec[lane] = make_int4(__float_as_int((float)(r.x - gz0)), r.y, r.z, STRAYS ? (r.w ? (int)(gNext - 32 + lane) + 1 : 0) : r.w);
      __syncwarp();
      continue;
    }
    if (supers)
    {
      const int src = __ffs(supers) - 1;
      supers &= supers - 1;
      WB_STAT(gst[4], 1);
      const int4 s1 = sm.srec[src];
      if (sr < 2 || boxWanted(sm.sbox[src], __int_as_float(s1.x), blockWanted(s1.w, a.straySuper)))
      {
        gNext = (uint32_t)s1.y;
        gEnd = gNext + (uint32_t)s1.z;
      }
      continue;
    }
    m0 += 32;
    if (m0 >= nsc)
    {
      sr++;
      // rings up to the undecided lanes' reach, while they touch the grid
      if (sr > smaxG || (si - sr < 0 && si + sr >= a.snx && sj - sr < 0 && sj + sr >= a.sny))
        break;
      nsc = sr == 0 ? 1 : 8 * sr;
      m0 = 0;
    }
    WB_STAT(gst[5], 1);
    uint32_t cell = 0;
    if (m0 + lane < nsc)
    {
      int di, dj;
      ringCell(sr, m0 + lane, di, dj);
      const int SI = si + di, SJ = sj + dj;
      if (SI >= 0 && SI < a.snx && SJ >= 0 && SJ < a.sny)
      {
        const uint64_t sc = (uint64_t)SJ * a.snx + SI;
        cell = (uint32_t)sc;
        b = a.super[2 * sc];
        r = a.super[2 * sc + 1];
      }
    }
    if constexpr (STRAYS)
      supers = __ballot_sync(kAll, envMeets(b, r, a.straySuper + 2 * (uint64_t)cell));
    else
      supers = __ballot_sync(kAll, envReached(b, r.x));
    __syncwarp();
    sm.sbox[lane] = boxOfInts(b);
    sm.srec[lane] = make_int4(__float_as_int((float)(r.x - gz0)), r.y, r.z, STRAYS ? (r.w ? (int)cell + 1 : 0) : r.w);
    __syncwarp();
  }
#ifdef WB_CLASSIFY_STATS
  {
    gst[0] = 1;
    gst[1] = reads;
    gst[11] = clock64() - tG;
    gst[12] = __popc(__ballot_sync(kAll, deferred));
    gst[15] = __popc(__ballot_sync(kAll, act && !deferred && !done));
    if (lane == 0)
      for (int q = 0; q < 16; q++)
        atomicAdd(&gClassifyStats[0][q], gst[q]);
  }
#endif
  if (act && !deferred)
  {
    bool amb = false;
    if (!done && nDir == 2)
    {
      // the widest open arc against 144 degrees + kArcBand
      auto sureOpen = [&](float px, float py, float qx, float qy) {
        return px * qy - py * qx < 0.f || px * qx + py * qy <= kCosSure;
      };
      amb = !sureOpen(ax * side, ay * side, bx * side, by * side);
      if (amb && two)
        amb = !sureOpen(sm.arc2a[lane].x, sm.arc2a[lane].y, sm.arc2b[lane].x, sm.arc2b[lane].y);
    }
    a.label[j] = done ? 1 : 2;
    if (amb)
      a.ambList[atomicAdd(a.ambCount, 1u)] = j;
  }
}

/* ---- One point per warp: the points of groups whose neighbourhood is large ----
 *
 * The same walk, arcs and tests as classifyGroupArcs, with the lanes over the
 * boxes and candidates instead of the points: a super-cell's groups are tested
 * 32 at a time and a group's points all at once against the one point's own
 * hyperboloid and open arc, so a point whose neighbours (those of a group
 * under trees, whose hyperboloids are several metres wide) need many groups
 * reads only its own, and no group holds one warp while the rest of the GPU
 * idles.  FP32 differences are taken from the point itself. */
struct PointShared
{
  float2 arc2a, arc2b;   /* the point's second open arc, while it has one */
};

template <bool STRAYS>
__device__ __forceinline__ void classifyPointArcs(const ClsArgs &a, uint64_t j, int lane, PointShared &sm)
{
  constexpr unsigned kAll = 0xffffffffu;
  if (a.owner[j] < 0)
  {
    if (lane == 0)
      a.label[j] = 0;
    return;
  }
  const int mex = a.sx[j], mey = a.sy[j], mez = a.sz[j];
  const PtSetup ps = a.setup[j];
  const float ky = a.gky, kz = a.gkz, inv = a.gInv;
  const float czp = ps.czp * inv, por2 = ps.por2f * inv * inv;
  const float ratio = fabsf(czp) * rsqrtf(por2);
  const float eps = 1e-5f + 4e-7f * ratio;
  if (!a.exactInts || !(fminf(ky, kz) > 1e-9f) || !(fmaxf(ky, kz) < 1e9f) || !(ratio < 1e5f) || !(por2 > 0.f && por2 < 1e30f))
  {
    // not for FP32 arcs: the last pass decides
    if (lane == 0)
    {
      a.label[j] = 2;
      a.ambList[atomicAdd(a.ambCount, 1u)] = (uint32_t)j;
    }
    return;
  }
  const float kOut = (1.f + eps) / (1.f - eps), pOut = por2 - a.gTiny;
  const int ci0 = min(max(ps.ci, 0), a.nx - 1), cj0 = min(max(ps.cj, 0), a.ny - 1);
  const int off = max(abs(ps.ci - ci0), abs(ps.cj - cj0));
  const int smax = ps.smax + (off + WB_SUPER - 1) / WB_SUPER + 1;
  // every lane holds the same arcs (LaneArcs)
  int nDir = 0;
  bool slow = true, two = false, done = false;
  float side = 1.f, arcMin = -INFINITY, ax = 0.f, ay = 0.f, bx = 0.f, by = 0.f;

  // whether the point's hyperboloid reaches a box (record integers) at height z
  auto reached = [&](const int4 &b, int32_t z) -> bool {
    const float x0 = (float)(b.x - mex), x1 = (float)(b.z - mex), y0 = (float)(b.y - mey) * ky, y1 = (float)(b.w - mey) * ky;
    const float pad = 2e-6f * (fabsf(x0) + fabsf(x1) + fabsf(y0) + fabsf(y1));
    const float dx = fmaxf(0.f, fmaxf(x0, -x1) - pad), dy = fmaxf(0.f, fmaxf(y0, -y1) - pad);
    const float zd = __fmaf_rn((float)(mez - z), kz, czp);
    return __fmaf_rn(zd * fabsf(zd), kOut, -pOut) >= __fmaf_rn(dx, dx, dy * dy);
  };
  // whether the lane's box may hold a member in a direction that matters (flags,
  // strays: as in classifyGroupArcs)
  auto meets = [&](const int4 &b, int32_t zmin, int flags, const int4 *strays) -> bool {
    const float x0 = (float)(b.x - mex), x1 = (float)(b.z - mex), y0 = (float)(b.y - mey) * ky, y1 = (float)(b.w - mey) * ky;
    const float ex = 0.5f * (x0 + x1), ey = 0.5f * (y0 + y1);
    const float pad = 2e-6f * (fabsf(x0) + fabsf(x1) + fabsf(y0) + fabsf(y1));
    const float hx = 0.5f * (x1 - x0) + pad, hy = 0.5f * (y1 - y0) + pad;
    const float dx = fmaxf(0.f, fabsf(ex) - hx), dy = fmaxf(0.f, fabsf(ey) - hy);
    const float zd = __fmaf_rn((float)(mez - zmin), kz, czp);
    bool reach = __fmaf_rn(zd * fabsf(zd), kOut, -pOut) >= __fmaf_rn(dx, dx, dy * dy);
    if (STRAYS && flags && !reach)
      reach = reached(strays[0], strays[1].x);
    const float A = __fmaf_rn(side, __fmaf_rn(ax, ey, -(ay * ex)), __fmaf_rn(fabsf(ay), hx, fabsf(ax) * hy));
    const float B = __fmaf_rn(side, __fmaf_rn(ex, by, -(ey * bx)), __fmaf_rn(fabsf(by), hx, fabsf(bx) * hy));
    const float v = side < 0.f ? fmaxf(A, B) : fminf(A, B);
    return (b.x != INT32_MAX) & reach & (v >= arcMin);
  };
  // adds the directions (ex, ey) of the lanes in hits; after each, those the
  // open arc no longer holds drop out
  auto add = [&](unsigned hits, float ex, float ey, float rr) {
    const float il = rsqrtf(rr), ux = ex * il, uy = ey * il;
    while (hits && !done)
    {
      const int src = __ffs(hits) - 1;
      hits &= hits - 1;
      const float vx = __shfl_sync(kAll, ux, src), vy = __shfl_sync(kAll, uy, src);
      if (slow)
      {
        __syncwarp();
        const LaneArcs r = addDirection(LaneArcs{ax, ay, bx, by, side, nDir, two, true}, vx, vy, &sm.arc2a, &sm.arc2b);
        __syncwarp();
        ax = r.ax;
        ay = r.ay;
        bx = r.bx;
        by = r.by;
        side = r.side;
        nDir = r.nDir;
        two = r.two;
        slow = two || nDir < 2;
        done = !r.open;
      }
      else
      {
        float2 l, q;
        const int open = splitArc(vx, vy, ax, ay, bx, by, side, l, q);
        done = open == 0;
        if (open == 2)
        {
          __syncwarp();
          sm.arc2a = l;
          sm.arc2b = q;
          __syncwarp();
          two = slow = true;
        }
      }
      arcMin = slow ? -INFINITY : 0.f;
      hits &= __ballot_sync(kAll, side * fminf(__fmaf_rn(ax, uy, -(ay * ux)), __fmaf_rn(ux, by, -(uy * bx))) > arcMin);
    }
  };

  const int si = ci0 / WB_SUPER, sj = cj0 / WB_SUPER;
  for (int sr = 0; sr <= smax && !done; sr++)
  {
    if (si - sr < 0 && si + sr >= a.snx && sj - sr < 0 && sj + sr >= a.sny)
      break;
    const int nsc = sr == 0 ? 1 : 8 * sr;
    for (int m0 = 0; m0 < nsc && !done; m0 += 32)
    {
      int4 b = make_int4(INT32_MAX, 0, 0, 0), r = make_int4(0, 0, 0, 0);
      uint64_t sc = 0;
      if (m0 + lane < nsc)
      {
        int di, dj;
        ringCell(sr, m0 + lane, di, dj);
        const int SI = si + di, SJ = sj + dj;
        if (SI >= 0 && SI < a.snx && SJ >= 0 && SJ < a.sny)
        {
          sc = (uint64_t)SJ * a.snx + SI;
          b = a.super[2 * sc];
          r = a.super[2 * sc + 1];
        }
      }
      unsigned supers = __ballot_sync(kAll, meets(b, r.x, r.w, a.straySuper + 2 * sc));
      while (supers && !done)
      {
        const int src = __ffs(supers) - 1;
        supers &= supers - 1;
        const uint32_t g0 = (uint32_t)__shfl_sync(kAll, r.y, src), g1 = g0 + (uint32_t)__shfl_sync(kAll, r.z, src);
        for (uint32_t g = g0; g < g1 && !done; g += 32)
        {
          int4 gb = make_int4(INT32_MAX, 0, 0, 0), gr = make_int4(0, 0, 0, 0);
          if (g + lane < g1)
          {
            gb = a.groups[2 * (uint64_t)(g + lane)];
            gr = a.groups[2 * (uint64_t)(g + lane) + 1];
          }
          unsigned list = __ballot_sync(kAll, meets(gb, gr.x, gr.w, a.strayGrp + 2 * (uint64_t)(g + lane)));
          while (list && !done)
          {
            const int gs = __ffs(list) - 1;
            list &= list - 1;
            const uint32_t first = (uint32_t)__shfl_sync(kAll, gr.y, gs);
            const int n = __shfl_sync(kAll, gr.z, gs);
            int2 p = make_int2(0, 0), q = make_int2(0, 0);
            if (lane < n)
            {
              p = a.bxy[first + lane];
              q = a.bzw[first + lane];
            }
            const int dxi = p.x - mex, dyi = p.y - mey;
            const float ex = (float)dxi, ey = (float)dyi * ky, zd = __fmaf_rn((float)(mez - q.x), kz, czp);
            const float rr = __fmaf_rn(ex, ex, ey * ey), w = zd * fabsf(zd);
            const bool arc = side * fminf(__fmaf_rn(ax, ey, -(ay * ex)), __fmaf_rn(ex, by, -(ey * bx))) > arcMin;
            // dist(p,q) == 0 gives no direction (classify.cpp:142,153)
            const bool cand = (lane < n) & ((dxi != 0) | (dyi != 0)), stray = q.y < 0;
            // points outside the root cube: in or not by their blocks too
            bool blockMeets = true, blockHolds = false;
            if (STRAYS && __shfl_sync(kAll, gr.w, gs))
            {
              const int4 *s = a.strayGrp + 2 * (uint64_t)(g + gs);
              blockMeets = reached(s[0], s[1].y);
              blockHolds = reached(s[0], s[1].x);
            }
            const bool may = (__fmaf_rn(w, kOut, -pOut) >= rr) & arc, sure = w > kOut * (rr + por2 + a.gTiny);
            const unsigned hits = __ballot_sync(kAll, cand & !stray & may & sure);
            const bool unsure = cand & (stray ? (may & blockMeets) | (arc & blockHolds) : may & !sure);
            if (hits)
              add(hits, ex, ey, rr);
            if (__any_sync(kAll, unsure) && !done)
            {
              bool in = false;
              if (unsure)
              {
                if (a.fp32Only && !stray)
                {
                  const float dx = (float)dxi * a.fsx, dy = (float)dyi * a.fsy;
                  const float z = (float)(mez - q.x) * a.fsz + ps.czp;
                  const float r2 = a.fs2 * __fmaf_rn(dx, dx, dy * dy);
                  in = z > 0 && __fmaf_rn(z, z, -r2) - ps.por2f > 0;
                }
                else
                  in = memberExact(a, exactHyp(a, (uint32_t)j), (uint32_t)q.y, p.x, p.y, q.x);
              }
              const bool still = side * fminf(__fmaf_rn(ax, ey, -(ay * ex)), __fmaf_rn(ex, by, -(ey * bx))) > arcMin;
              const unsigned more = __ballot_sync(kAll, in & still);
              if (more)
                add(more, ex, ey, rr);
            }
          }
        }
      }
    }
  }
  bool amb = false;
  if (!done && nDir == 2)
  {
    auto sureOpen = [&](float px, float py, float qx, float qy) {
      return px * qy - py * qx < 0.f || px * qx + py * qy <= kCosSure;
    };
    amb = !sureOpen(ax * side, ay * side, bx * side, by * side);
    if (amb && two)
      amb = !sureOpen(sm.arc2a.x, sm.arc2a.y, sm.arc2b.x, sm.arc2b.y);
  }
  if (lane == 0)
  {
    a.label[j] = done ? 1 : 2;
    if (amb)
      a.ambList[atomicAdd(a.ambCount, 1u)] = (uint32_t)j;
  }
}
