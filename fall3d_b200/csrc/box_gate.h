// box_gate.h -- host side: whether a step's sweeps look for their non-zero
// boxes first (active.cuh) or march whole pencils.
//
// Finding the boxes costs two launches and a pass over the state, and pays
// when it shortens the march.  How long a march is depends on the state, which
// the host does not read; so a step with ranges leaves their lengths in
// page-locked memory, and the host looks there, without waiting, when it puts
// the next step together.  Either way the step has the same result, so a value
// that is some steps old costs time at most.
//
// Looking for the boxes in every step, whatever they gained, made a step of
// 48 x 40 x 24 x 4 cells 71 to 86 us, one of 157 x 93 x 37 x 8 full of ash 181
// to 211, and the operators called one by one up to half as slow again
// (compensated form).  With the gate these are 68, 179 and unchanged, and the
// plume in 400 x 300 x 60 x 8 cells keeps its gain (x alone 514 to 199 us).
#pragma once
#include <algorithm>
#include <atomic>

namespace f3d {

// What such a step leaves: a count of them, written last; the longest range
// and the sum of all ranges per direction; the directions it ran for.
constexpr int kGateWords = 8;

class BoxGate {
 public:
  // pub: kGateWords page-locked words, zeroed.  Before any result the boxes
  // are taken to pay: a run starts with an empty domain.
  void attach(const unsigned int* pub, bool compensated) {
    pub_ = pub;
    slower_ = compensated ? 1.12 : 1.05;
    step_cost_ = compensated ? 22.0 : 30.0;
    operator_cost_ = compensated ? 55.0 : 100.0;
  }
  // The state was replaced (nothing in flight): start over.
  void reset() {
    for (Way& w : way_) w = Way();
    if (pub_) seen_ = pub_[0];
  }
  // Once per launch sequence over dirs (a bit mask): blocks march `longest`
  // cells at most and `total` in all per direction.
  bool use(int dirs, const int longest[3], const long long total[3]) {
    if (!pub_) return false;
    const unsigned int run = pub_[0];
    std::atomic_thread_fence(std::memory_order_acquire);
    if (run != seen_) {
      seen_ = run;
      const int d = (int)(pub_[7] & 7u);
      int most[3];
      long long sum[3];
      for (int q = 0; q < 3; ++q) {
        most[q] = (int)pub_[1 + q];
        sum[q] = pub_[4 + q];
      }
      way_[d].pays = cost(d) + slower_ * length(d, most, sum) < length(d, longest, total);
    }
    Way& w = way_[dirs & 7];
    if (length(dirs, longest, total) <= cost(dirs)) return false;
    if (w.pays) return true;
    if (++w.idle < kLook) return false;
    w.idle = 0;
    return true;
  }

 private:
  // How long a march is, in cells of a full device: 592 blocks are resident
  // (four on each of 148 SMs), and where that is a round or less, the longest
  // block's cells take 0.64 of a full device's time each, and the others' work
  // the rest (a compensated step marches a cell in 0.42 us with few blocks, in
  // 0.66 with all).
  static double length(int dirs, const int longest[3], const long long total[3]) {
    double s = 0.0;
    for (int d = 0; d < 3; ++d) {
      const double all = (double)total[d] / 592.0;
      if (dirs >> d & 1) s += std::max(0.64 * longest[d] + 0.36 * all, all);
    }
    return s;
  }
  // The two launches in such cells: a step has them behind other work (14 us;
  // a cell takes 0.66 us compensated, 0.47 in FP32), a lone operator waits for
  // them (20 us and more: y of 200 x 150 x 40 x 8 in FP32, a plume, 83 us
  // without and 98 with).  A march over a range takes longer per cell than one
  // over the pencil, whose ends the compiler knows to be the domain's (400 x
  // 300 x 60 x 4 full of ash, compensated: 0.88 ms a step with ranges, 0.78
  // without; FP32 0.56 and 0.55).
  double cost(int dirs) const { return (dirs & (dirs - 1)) ? step_cost_ : operator_cost_; }
  double slower_ = 1.12, step_cost_ = 22.0, operator_cost_ = 55.0;
  static constexpr int kLook = 32;  // steps between two looks at a state that boxes do not help
  struct Way {
    bool pays = true;
    int idle = 0;
  };
  Way way_[8];
  const volatile unsigned int* pub_ = nullptr;
  unsigned int seen_ = 0;
};

}  // namespace f3d
