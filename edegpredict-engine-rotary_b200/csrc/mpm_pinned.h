// Small pieces of pinned host memory, shared by the handles of a process.
//
// A pinned allocation of a few hundred bytes and its release cost 2.1 and
// 0.5 ms on a B200 host, more than all the rest of creating and closing the
// handle of a small workpiece (1.15 and 1.5 ms); a copy into pageable memory
// instead costs every metrics and status call 5.7 us of 30 and 16.  So handles
// take slots of a block that stays.
//
// A block belongs to the CUDA context that allocated it and is only handed
// out, and only freed, while that context is the current one: a reset of the
// device ends the context and with it the block, and the next context, which
// has another id, gets a new one.  A block whose last slot comes back is freed
// while another of its context has a slot to spare; the last one stays for the
// next handle and ends with its context.
#pragma once

#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

namespace mpmb {

// Ops: context(uint64_t*) (the current context's id, unique in the process;
// false: not known), alloc(size_t) (nullptr on failure) and release(void*).
template <typename Ops> class PinnedSlots {
  public:
    static constexpr size_t kSlotBytes = 512;
    static constexpr int kSlots = 32;

    explicit PinnedSlots(Ops ops = Ops()) : ops_(ops) {}

    // A slot of kSlotBytes, or nullptr.  Any thread.
    void* take() {
        std::lock_guard<std::mutex> lock(m_);
        uint64_t ctx = 0;
        const bool known = ops_.context(&ctx);
        if (known)
            for (Block& b : blocks_)
                if (b.known && b.ctx == ctx && b.used != ~0u) return slot(b);
        char* p = static_cast<char*>(ops_.alloc(kSlotBytes * kSlots));
        if (!p) return nullptr;
        // a block that is still listed at these addresses ended with its context
        for (size_t k = blocks_.size(); k-- > 0;)
            if (p < blocks_[k].base + kSlotBytes * kSlots && blocks_[k].base < p + kSlotBytes * kSlots)
                blocks_.erase(blocks_.begin() + k);
        blocks_.push_back(Block{p, ctx, 0u, known});
        return slot(blocks_.back());
    }

    // Gives a slot back; nothing on the device may still write it.
    void give(void* s) {
        std::lock_guard<std::mutex> lock(m_);
        const char* at = static_cast<const char*>(s);
        for (size_t k = 0; k < blocks_.size(); ++k) {
            Block& b = blocks_[k];
            if (!(b.base <= at && at < b.base + kSlotBytes * kSlots)) continue;
            b.used &= ~(1u << ((at - b.base) / kSlotBytes));
            uint64_t ctx = 0;
            if (b.used == 0u && (!b.known || (ops_.context(&ctx) && ctx == b.ctx && spare(k)))) {
                ops_.release(b.base);
                blocks_.erase(blocks_.begin() + k);
            }
            return;
        }
    }

    size_t blocks() {
        std::lock_guard<std::mutex> lock(m_);
        return blocks_.size();
    }

  private:
    struct Block {
        char* base;
        uint64_t ctx;
        uint32_t used;   // a bit per slot
        bool known;      // its context's id is known (else it is freed when empty)
    };

    static void* slot(Block& b) {
        int k = 0;
        while ((b.used >> k) & 1u) ++k;
        b.used |= 1u << k;
        return b.base + kSlotBytes * k;
    }
    // another block of the same context has a free slot
    bool spare(size_t k) const {
        for (size_t q = 0; q < blocks_.size(); ++q)
            if (q != k && blocks_[q].known && blocks_[q].ctx == blocks_[k].ctx && blocks_[q].used != ~0u) return true;
        return false;
    }

    Ops ops_;
    std::mutex m_;
    std::vector<Block> blocks_;
};

// Slots of page-locked memory (csrc/mpm_engine.cu).
void* pinned_take();
void pinned_give(void* slot);

}  // namespace mpmb
