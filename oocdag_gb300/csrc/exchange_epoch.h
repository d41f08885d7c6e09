// The tags of successive launches on one exchange buffer of the triangular solves (trsolve.cuh): a tag counts only if
// nothing in the buffer can carry it, and the buffer's error word has to be 0 before a launch.
#pragma once

class ExchangeEpoch {
 public:
  explicit ExchangeEpoch(unsigned last = 0) : last_(last) {}
  // The next launch's tag; *clear: the buffer is to be zeroed before it.
  unsigned next(bool* clear) {
    if (++last_ == 0) last_ = 1;  // (every tag used: start again on a zeroed buffer)
    *clear = last_ == 1;
    return last_;
  }
  // The buffer is new, or a launch on it ended with its error word raised: its contents are void.
  void restart() { last_ = 0; }

 private:
  unsigned last_;
};
