// The ring of tensor memory's slots that the tiles of moe_tcgen05.cu take in turn: where a tile's slots lie, what they are
// multiplied as, and which slots have to be waited for.  Plain functions of whole numbers, so that a check on the host can follow
// every sequence of tiles.
//
// Who uses a slot: the issuer of products writes it for a tile; the epilogue's warps, in two teams, read a tile's even slots (team
// 0) and odd ones (team 1), in order, tile after tile.  Every slot counts sixteen signals a use, one from each warp: from those
// that read it when they have, from the others when they begin with the tile.
//
// What a tile waits for is that all its slots have been read.  A wait for each of ten would take longer than the products of a
// short tile leave, and two say it: as long as uses follow the ring's order, where a slot and the one before it have been read, so has
// all that was used earlier.  A tile that passes over slots to begin at slot 0 breaks that order: those slots, from `top` on, keep
// a use of an earlier turn until a tile takes them, and to wait for them says nothing (tiles of 8, 6, 6, 10 slots: the last one
// takes 6 to 15, of which nobody has ever used 14 and 15).  So a tile waits for its last two slots BELOW top; what lies from there on was
// read earlier than slot top - 1, which the tile that takes it waits for.  (To have the warps signal the slots passed over keeps the
// order too, but the next tile to take these would wait for the products of the one that passed over them.)
#pragma once

#ifdef __CUDACC__
#define CCB_RING __host__ __device__ __forceinline__
#else
#define CCB_RING inline
#endif

namespace ccb {

constexpr int kSlots = 16;       // of 32 columns of tensor memory
constexpr int kMostSlots = 8;    // of a product (256 columns)

struct SlotRing {
  int at = 0, top = kSlots;   // where the next tile may begin; slots from top on were passed over this turn
  // To a tile of `slots` slots: it begins at `at`, but one that fits a product is not cut by the ring's end.
  CCB_RING void enter(int slots) {
    if (slots <= kMostSlots && at + slots > kSlots) top = at, at = 0;
  }
  // Its slots first_waited() .. end_waited() - 1, counted from its first one, are waited for.
  CCB_RING int end_waited(int slots) const { return at + slots > kSlots || at + slots <= top ? slots : top - at; }
  CCB_RING int first_waited(int slots) const {
    const int end = end_waited(slots);
    return end > 2 ? end - 2 : 0;
  }
  CCB_RING void leave(int slots) {
    at += slots;
    if (at >= kSlots) at -= kSlots, top = kSlots;
  }
};

// A bit for each of `n` slots from slot `at` on.
CCB_RING unsigned slot_bits(int at, int n) {
  const unsigned bits = ((1u << n) - 1) << at;
  return (bits | bits >> kSlots) & ((1u << kSlots) - 1);
}

// The products of a tile of `slots` slots from slot `at` on: runs that neither pass the ring's end nor have more than kMostSlots
// slots, of about the same size where a run is cut; at most three (slots of the first, second, third).
struct TileParts {
  int len[3];
  CCB_RING TileParts(int at, int slots) {
    const int head = slots < kSlots - at ? slots : kSlots - at, tail = slots - head;
    const int h = head > kMostSlots ? (head + 1) / 2 : head, t = tail > kMostSlots ? (tail + 1) / 2 : tail;
    len[0] = h;
    len[1] = head > h ? head - h : t;
    len[2] = head > h ? t : tail - t;
  }
  CCB_RING int count() const { return 1 + (len[1] > 0) + (len[2] > 0); }
};

}  // namespace ccb
