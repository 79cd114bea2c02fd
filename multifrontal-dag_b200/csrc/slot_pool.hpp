// Page-locked slots that the handles' last kernels write their status to.
#pragma once
#include <cstddef>
#include <mutex>
#include <vector>

namespace mfd {

// Slots cut from page-locked blocks, shared by the handles of a process (page-locking memory for
// every handle takes 0.15-0.5 ms, a fifth of a small handle's set-up).  A block belongs to the
// context that was current when it was locked and goes with it (a device reset), so slots are only
// handed out from blocks of the current one.  Api::context() is that context's id (never used
// again by another; 0: none), Api::lock / unlock allocate and free a block.  When all slots are
// back one block per device stays.
template <class Api>
class SlotPool {
 public:
  static constexpr int kSlots = 256;
  static constexpr size_t kSlotBytes = 256;
  struct Slot {
    void* p = nullptr;
    unsigned long long ctx = 0;
  };

  // A slot for a handle on `device`, whose context is current; p is null if there is no memory.
  Slot take(int device) {
    std::lock_guard<std::mutex> lk(mu_);
    Slot s;
    s.ctx = Api::context();
    if (s.ctx == 0) return s;
    Block* b = nullptr;
    for (size_t k = 0; k < blocks_.size();) {
      if (blocks_[k].device == device && blocks_[k].ctx != s.ctx) {   // gone with the device's last context
        blocks_.erase(blocks_.begin() + k);
        continue;
      }
      if (blocks_[k].ctx == s.ctx && !blocks_[k].free.empty() && !b) b = &blocks_[k];
      ++k;
    }
    if (!b) {
      char* base = static_cast<char*>(Api::lock(kSlots * kSlotBytes));
      if (!base) return s;
      blocks_.push_back({device, s.ctx, base, {}});
      b = &blocks_.back();
      for (int i = kSlots; i-- > 0;) b->free.push_back(i);
    }
    s.p = b->base + b->free.back() * kSlotBytes;
    b->free.pop_back();
    return s;
  }
  void give(const Slot& s) {
    if (!s.p) return;
    std::lock_guard<std::mutex> lk(mu_);
    char* p = static_cast<char*>(s.p);
    size_t at = blocks_.size(), of_ctx = 0;
    for (size_t k = 0; k < blocks_.size(); ++k) {
      if (blocks_[k].ctx != s.ctx) continue;
      ++of_ctx;
      if (p >= blocks_[k].base && p < blocks_[k].base + kSlots * kSlotBytes) at = k;
    }
    if (at == blocks_.size()) return;                    // its block is gone
    Block& b = blocks_[at];
    b.free.push_back((int)((p - b.base) / kSlotBytes));
    if ((int)b.free.size() == kSlots && of_ctx > 1) {
      Api::unlock(b.base);
      blocks_.erase(blocks_.begin() + at);
    }
  }

 private:
  struct Block {
    int device;
    unsigned long long ctx;
    char* base;
    std::vector<int> free;
  };
  std::mutex mu_;
  std::vector<Block> blocks_;
};

}  // namespace mfd
