// Bounds of one group of a lot from the few features that attain them.
//
// The bounds mode of the grammar (kernels/sink.cu:15-20 of the reference) takes
// the union of up to 56 feature boxes a group, 1,859 a lot.  Most of them cannot
// touch the union: they repeat along a facade (only the first and the last of a
// row reach its ends, since every operation that places them is monotone in
// the row's counter), or lie inside a neighbour by constants that differ by
// more than any rounding (0.005 m and more against 1e-5 m).  fastBounds() visits
// only the features that can attain one of the six bounds (2-9 a group, 300 a
// lot) and places them with the grammar's own operations in the grammar's
// order, so the bounds are the same bits (checked against the whole grammar on
// the CPU for every lot family, floor count and group).
//
// The dominated features are dominated for the dimensions that describe()
// (kernels/world.cu:37-56) gives a lot; a row with any other dimensions is
// not `regular` and goes through the whole grammar.
#pragma once
#include "grammar_ra.cuh"

namespace st {

// The ranges of describe(): floors 2..6, storey 3.2..4.35, h = 4.2 + floors *
// storey, w 9.4..13.7, d 9..13.7, roof scale 0.85..1.25 (with a little room).
HD bool regularLot(const LotDesc& l) {
  return l.type >= 0 && l.type <= 5 && l.floors >= 2 && l.floors <= 6 && l.storey >= 3.199f && l.storey <= 4.351f &&
         l.h == 4.2f + float(l.floors) * l.storey && l.w >= 9.399f && l.w <= 13.701f && l.d >= 8.999f &&
         l.d <= 13.701f && l.roofScale >= 0.849f && l.roofScale <= 1.251f;
}

struct BoxUnion {
  f3 lo{1000000.0f, 1000000.0f, 1000000.0f}, hi{-1000000.0f, -1000000.0f, -1000000.0f};
};
// One feature (kernels/sink.cu:10-20): the roof rescale, then the padded box;
// prisms and arches (`base`) stand on p.y.
struct BoundsOf {
  const LotDesc& l;
  BoxUnion u;
  HD void box(float px, float py, float pz, float hx, float hy, float hz, bool base = false) {
    if (py >= l.h) { py = l.h + (py - l.h) * l.roofScale; hy *= l.roofScale; }
    const f3 p = mk(px, py, pz), h = mk(hx, hy, hz), pad = mk(0.025f, 0.025f, 0.025f);
    f3 a = p - h;
    if (base) a.y = p.y;
    u.lo = vmin(u.lo, a - pad);
    u.hi = vmax(u.hi, (p + h) + pad);
  }
  // A box on facade `face`, in the facade's own axes (x along it, z out of it,
  // `base` = the facade's distance); facing() turns the union into the lot's.
  HD void wall(float reach, float along, float y, float out, float hw, float hy, float hd) {
    box(along, y, reach + out, hw, hy, hd);
  }
  HD void facing(int face) {
    const BoxUnion f = u;
    if (face == 1) {
      u.lo = mk(f.lo.z, f.lo.y, f.lo.x);
      u.hi = mk(f.hi.z, f.hi.y, f.hi.x);
    } else if (face == 2) {
      u.lo.z = -f.hi.z;
      u.hi.z = -f.lo.z;
    } else if (face == 3) {
      u.lo = mk(-f.hi.z, f.lo.y, f.lo.x);
      u.hi = mk(-f.lo.z, f.hi.y, f.hi.x);
    }
  }
};

// A park's tree (group 1..8): its height, trunk, and crown envelope j (0..27).
HD bool isTree(const LotDesc& l, int group) { return l.type == 3 && group >= 1 && group <= 8; }
HD float treeHeight(const LotDesc& l, int group) { return 5.0f + hash1(int(l.seed) + group - 1) * 3.0f; }
HD float treeX(int group) { return 0.0f + (group - 1 < 4 ? -10.0f : 10.0f); }
HD float treeZ(int group) { return 0.0f + (float((group - 1) % 4) - 1.5f) * 6.7f; }
HD void treeTrunk(BoundsOf& b, int group, float th) {
  b.box(treeX(group), th * 0.4f, treeZ(group), 0.19f, th * 0.4f, 0.19f);
}
HD void treeCrown(BoundsOf& b, int group, float th, int j) {
  const int seed = int(b.l.seed);
  const float yy = hash1(seed + j + 991) * 3.3f - 0.5f;
  const float rr = sqrtf(hash1(seed + j + 330)) * 2.1f * (1.0f - yy * 0.12f);
  const float size = 0.48f + hash1(seed + j + 62) * 0.30f;
  b.box(treeX(group) + TreeCos(j) * rr, th + yy, treeZ(group) + TreeSin(j) * rr, size, size * 1.25f, size);
}

// Bounds of a non-empty group of a regular lot.
HD void fastBounds(const LotDesc& l, int group, BoxUnion& u) {
  BoundsOf b{l, BoxUnion{}};
  const float w = l.w, d = l.d, h = l.h, storey = l.storey;
  const int type = l.type, floors = l.floors;
  if (type == 4) {  // bridge: deck and parapets (the posts end below and inside them)
    b.box(0.0f, 0.25f, 0.0f, 18.0f, 0.5f, 5.0f);
    b.box(0.0f, 1.25f, 0.0f - 5.0f, 18.0f, 0.2f, 0.23f);
    b.box(0.0f, 1.25f, 0.0f + 5.0f, 18.0f, 0.2f, 0.23f);
  } else if (type == 3) {
    if (group == 0) {
      b.box(0.0f, -0.12f, 0.0f, 15.5f, 0.22f, 15.5f);
    } else if (group == 9) {  // fountain: the basin, and the ball on top
      b.box(0.0f, 0.8f, 0.0f, 3.6f, 0.45f, 3.6f);
      b.box(0.0f, 3.15f, 0.0f, 0.5f, 0.5f, 0.5f);
    } else {  // a tree: the trunk and every envelope of its crown
      const float th = treeHeight(l, group);
      treeTrunk(b, group, th);
#pragma unroll 1
      for (int j = 0; j < 28; j++) treeCrown(b, group, th, j);
    }
  } else if (group == 0) {  // the plinth around and below, the mass above
    b.box(0.0f, 0.15f, 0.0f, w + 1.1f, 0.25f, d + 1.1f);
    b.box(0.0f, (h + 4.0f) * 0.5f, 0.0f, w, (h - 4.0f) * 0.5f, d);
  } else if (group == 1) {  // eaves; ridge and chimney pot, dome and ball, or tower and finial
    b.box(0.0f, h + 0.25f, 0.0f, w + 0.6f, 0.24f, d + 0.6f);
    if (type == 0) {
      b.box(0.0f, h + 4.8f, 0.0f, 0.12f, 0.14f, d + 0.7f);
      b.box(0.0f - w * 0.52f, h + 6.32f, 0.0f, 0.2f, 0.25f, 0.2f);
    } else if (type == 1) {
      b.box(0.0f, h + 3.1f, 0.0f, w * 0.79f, 8.4f, w * 0.79f);
      b.box(0.0f, h + 13.8f, 0.0f, 0.6f, 0.6f, 0.6f);
    } else {
      const float xx = 0.0f - w * 0.75f, zz = 0.0f + d * 0.60f;
      b.box(xx, h + 3.5f, zz, 2.3f, 7.2f, 2.3f);
      b.box(xx, h + 16.0f, zz, 0.17f, 1.2f, 0.17f);
    }
  } else if (group < 30 || (group >= 32 && group < 60)) {  // facade groups
    const int face = group < 6 ? group - 2 : (group < 30 ? (group - 6) / 6 : (group < 56 ? (group - 32) / 6 : group - 56));
    const float ext = face % 2 == 0 ? w : d, reach = 0.0f + (face % 2 == 0 ? d : w);
    if (group < 6) {  // lowest string, top string, a pilaster, a dentil
      const float top = 4.2f + float(floors) * storey;
      b.wall(reach, 0.0f, 4.2f + 0.0f * storey, 0.17f, ext + 0.15f, 0.11f, 0.22f);
      b.wall(reach, 0.0f, top + 0.21f, 0.1f, ext + 0.10f, 0.052f, 0.16f);
      b.wall(reach, (0.0f / 4.0f * 2.0f - 1.0f) * (ext - 0.3f), (h + 4.0f) * 0.5f, 0.16f, 0.19f, (h - 4.0f) * 0.5f, 0.22f);
      b.wall(reach, (0.0f - 3.5f) * (ext / 4.0f), h - 0.24f, 0.4f, 0.15f, 0.12f, 0.19f);
    } else if (group < 56) {
      const bool windows = group < 30;
      const int row = windows ? (group - 6) % 6 : (group - 32) % 6;
      const float y = 4.2f + storey * 0.5f + float(row) * storey;
      const float u0 = (0.0f - 1.5f) * (ext * 0.48f), u3 = (3.0f - 1.5f) * (ext * 0.48f);
      if (windows) {  // outer sills, then one window's sill, head and flower rail
        const float wy = 1.2f;
        b.wall(reach, u0, y - 1.31f, 0.30f, 1.18f, 0.045f, 0.07f);
        b.wall(reach, u3, y - 1.31f, 0.30f, 1.18f, 0.045f, 0.07f);
        b.wall(reach, u0, y - wy - 0.13f, 0.22f, 1.13f, 0.14f, 0.29f);
        b.wall(reach, u0, y + wy + 0.12f, 0.18f, 1.11f, 0.14f, 0.23f);
        b.wall(reach, u0, y - wy + 0.46f, 0.56f, 1.10f, 0.035f, 0.035f);
      } else {  // outer hand rails, then one balcony's slab and bracket
        b.wall(reach, u0, y - 0.22f, 1.17f, 1.20f, 0.028f, 0.035f);
        b.wall(reach, u3, y - 0.22f, 1.17f, 1.20f, 0.028f, 0.035f);
        b.wall(reach, u0, y - 1.18f, 0.56f, 1.16f, 0.085f, 0.65f);
        b.wall(reach, u0 - 0.72f, y - 1.42f, 0.46f, 0.075f, 0.22f, 0.42f);
      }
    } else {  // lowest (wide) and highest (narrow) quoins; a tower's rose window
      const float y0 = 4.45f + 0.0f * (h - 4.0f) / 14.0f, y13 = 4.45f + 13.0f * (h - 4.0f) / 14.0f;
      b.wall(reach, -ext + 0.52f, y0, 0.12f, 0.52f, 0.16f, 0.16f);
      b.wall(reach, ext - 0.52f, y0, 0.12f, 0.52f, 0.16f, 0.16f);
      b.wall(reach, -ext + 0.30f, y13, 0.12f, 0.30f, 0.16f, 0.16f);
      b.wall(reach, ext - 0.30f, y13, 0.12f, 0.30f, 0.16f, 0.16f);
      if (type == 2) b.wall(reach, 0.0f, h - 2.3f, 0.21f, 2.35f, 2.35f, 0.26f);
    }
    b.facing(face);
  } else if (group == 30) {  // lamp heads and a lamp foot, strip and bollard behind, a drainpipe
    const float pz = 0.0f + 15.9f;
    b.box(0.0f - 16.0f, 4.44f, pz, 0.37f, 0.1f, 0.37f, true);
    b.box(0.0f + 16.0f, 4.44f, pz, 0.37f, 0.1f, 0.37f, true);
    b.box(0.0f - 16.0f, 0.15f, pz, 0.27f, 0.18f, 0.27f);
    b.box(0.0f - 14.0f + 0.0f * 4.0f, 0.055f, 0.0f - d - 2.2f, 1.75f, 0.035f, 0.045f);
    b.box(0.0f - 14.9f, 0.43f, 0.0f - 12.0f + 0.0f * 3.3f, 0.10f, 0.43f, 0.10f);
    b.box(0.0f + -1.0f * (w + 0.34f), h * 0.38f, 0.0f + -0.58f * d, 0.075f, h * 0.38f, 0.075f);
  } else if (group == 31) {  // dormers, outer planters, the awnings' sides, roof services
    if (type == 0) {
      const float x0 = 0.0f - w * 0.68f, x1 = 0.0f + w * 0.68f, z0 = 0.0f + (0.0f - 0.5f) * d * 0.96f;
      b.box(x0, h + 3.55f, z0, 1.2f, 1.0f, 1.45f, true);  // turned
      b.box(x0 + -1.36f, h + 2.5f, z0, 0.035f, 0.70f, 0.65f);
      b.box(x1 + 1.36f, h + 2.5f, z0, 0.035f, 0.70f, 0.65f);
    }
    const float pz = 0.0f + d + 1.5f;
    b.box(0.0f + (0.0f - 1.0f) * 7.0f, 0.48f, pz, 0.52f, 0.42f, 0.52f);
    b.box(0.0f + (0.0f - 1.0f) * 7.0f, 1.13f, pz, 0.7f, 0.8f, 0.7f);
    b.box(0.0f + (2.0f - 1.0f) * 7.0f, 1.13f, pz, 0.7f, 0.8f, 0.7f);
    b.box(0.0f + (w - 3.5f) + 0.6f, 3.1f, 0.0f, 0.7f, 0.10f, 1.38f);
    b.box(0.0f - (w - 3.5f) - 0.6f, 3.1f, 0.0f, 0.7f, 0.10f, 1.38f);
    b.box(0.0f, 3.1f, 0.0f - (d - 3.5f) - 0.6f, 1.38f, 0.10f, 0.7f);
    b.box(0.0f + (0.0f - 0.5f) * w, h + 1.18f, 0.0f + (0.0f - 0.5f) * d, 0.46f, 0.055f, 0.46f);
  } else if (group < 62) {  // roof slats: the first and the last of a side
    const int side = group - 60;
    b.box(0.0f, h + 0.395f, 0.0f - d + (float(0 + side * 32) + 0.5f) * d / 32.0f, w + 0.46f, 4.42f, 0.023f, true);
    b.box(0.0f, h + 0.395f, 0.0f - d + (float(31 + side * 32) + 0.5f) * d / 32.0f, w + 0.46f, 4.42f, 0.023f, true);
  } else if (group == 62) {  // curbs: two opposite corners
    b.box(0.0f + (-15.5f + 0.0f * 2.0f), 0.16f, 0.0f - 16.3f, 0.98f, 0.19f, 0.19f);
    b.box(0.0f + (-15.5f + 15.0f * 2.0f), 0.16f, 0.0f + 16.3f, 0.98f, 0.19f, 0.19f);
  } else {  // roofline brackets: one of each side
    const float uw = (0.0f - 3.5f) * w * 0.25f, ud = (0.0f - 3.5f) * d * 0.25f;
    b.box(0.0f + uw, h - 0.36f, 0.0f + d + 0.48f, 0.12f, 0.24f, 0.24f);
    b.box(0.0f + w + 0.48f, h - 0.36f, 0.0f + ud, 0.24f, 0.24f, 0.12f);
    b.box(0.0f + uw, h - 0.36f, 0.0f - d - 0.48f, 0.12f, 0.24f, 0.24f);
    b.box(0.0f - w - 0.48f, h - 0.36f, 0.0f + ud, 0.24f, 0.24f, 0.12f);
  }
  u = b.u;
}

// Bounds and feature count of one group as seven words [lo.xyz, count, hi.xyz].
// The whole grammar, out of line: rows whose dimensions describe() never gives.
static __host__ __device__ __noinline__ void anyBounds(LotDesc l, int group, float* o) {
  BoundsSink s;
  const int count = runGroup(l, group, s);
  o[0] = s.lo.x; o[1] = s.lo.y; o[2] = s.lo.z; o[3] = float(count);
  o[4] = s.hi.x; o[5] = s.hi.y; o[6] = s.hi.z;
}
HD void groupBounds(const LotDesc& l, bool regular, int group, float* o) {
  if (!regular) {
    anyBounds(l, group, o);
    return;
  }
  const int count = groupCount(l, group);
  BoxUnion u;
  if (count > 0) fastBounds(l, group, u);
  o[0] = u.lo.x; o[1] = u.lo.y; o[2] = u.lo.z; o[3] = float(count);
  o[4] = u.hi.x; o[5] = u.hi.y; o[6] = u.hi.z;
}

}  // namespace st
