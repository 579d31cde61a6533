// wg_layout.h -- how many sheets and slots the buckets of a pool member get (plain
// host code).
#pragma once
#include <cstdint>

namespace wg {

constexpr int kBucketCap = 2048;      // sheets a bucket's shared-memory pass can hold
constexpr int kMaxTarget = kBucketCap * 3 / 4;  // largest bucket target
constexpr int kSmallestTarget = 64;  // smallest target a tuning row may ask for
constexpr int kMinTarget = 384;  // smallest target that launches with few buckets are cut to

// Buckets of `target` sheets at a re-sort, `capg` slots each.
struct MemberLayout {
  int target = 0;
  int64_t nb = 0;
  int capg = kBucketCap;
};

// Buckets of `target` sheets in the slots of nb_tuned buckets of kBucketCap.
inline MemberLayout layout_for(int64_t n, int64_t nb_tuned, int target) {
  MemberLayout l;
  l.target = target;
  l.nb = (n + target - 1) / target;
  const int64_t slots = nb_tuned * kBucketCap / l.nb & ~(int64_t)3;
  l.capg = slots < kBucketCap ? (int)slots : kBucketCap;
  return l;
}

// Whether as large a share of the slots is spare as in the tuned layouts, which
// hold at most kMaxTarget of kBucketCap sheets: a quarter.  Sheets come and go
// between re-sorts; a layout without spare slots overflows at once, and one with
// fewer slots than sheets cannot hold them.
inline bool has_spare_slots(const MemberLayout& l) {
  return (int64_t)l.capg * kMaxTarget >= (int64_t)l.target * kBucketCap;
}

// Layout of a member whose step would like buckets of t sheets: that, or as many
// buckets all of one size (1200 sheets and t = 1056: two of 600, not 1056 + 144 in
// slots for 1024 each), or the tuned one.
inline MemberLayout member_layout(int64_t n, int tuned, int64_t nb_tuned, int64_t nb_room,
                                  int64_t t) {
  if (t < tuned && (n + t - 1) / t <= nb_room) {
    MemberLayout l = layout_for(n, nb_tuned, (int)t);
    if (!has_spare_slots(l)) l = layout_for(n, nb_tuned, (int)((n + l.nb - 1) / l.nb));
    if (has_spare_slots(l)) return l;
  }
  return layout_for(n, nb_tuned, tuned);
}

}  // namespace wg
