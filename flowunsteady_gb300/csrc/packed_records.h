// packed_records.h — which pair pass finds its packed source records written already.
#pragma once

namespace vpm {

// The update between two pair passes may write the packed records of the second.  What
// they hold is good for that pass of the same call alone: the next pass takes them or
// drops them, and a Scope around the call drops what an error left behind.
class PackedRecords {
 public:
  // The records of `pass` at cores σ·scale are written (pass < 0: none).
  void hold(int pass, double scale) {
    pass_ = pass;
    scale_ = scale;
  }
  // Whether they are those of `pass` at `scale`; none are held after this.
  bool take(int pass, double scale) {
    const bool same = pass_ >= 0 && pass_ == pass && scale_ == scale;
    pass_ = -1;
    return same;
  }
  class Scope {
   public:
    explicit Scope(PackedRecords& r) : r_(r) { r_.pass_ = -1; }
    ~Scope() { r_.pass_ = -1; }
    Scope(const Scope&) = delete;
    Scope& operator=(const Scope&) = delete;

   private:
    PackedRecords& r_;
  };

 private:
  int pass_ = -1;
  double scale_ = 1.0;
};

}  // namespace vpm
