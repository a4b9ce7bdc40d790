// call_lock.hpp -- one call at a time per context, and what a callback of that call may do.
//
// A fit holds the lock while it asks the host for row indices (vqb_draw_fn, vqb_init_fn, vqb_restart_fn).  What runs there may come
// back into the library on the same thread without anybody having written so: a garbage collector that starts inside a Python
// callback destroys quantizers that nobody refers to any more.  With a plain mutex that thread waits for itself, for good and
// with an idle GPU.  So the lock knows its holder, and the caller decides: destroying an object goes on (its memory is freed
// in the stream's order and is none of the fit's), anything else is refused.
#pragma once
#include <atomic>
#include <mutex>
#include <thread>

namespace vqb {

class CallLock {
  public:
    // Waits for another thread's call to end; empty when the calling thread is inside a call of this lock itself.
    class Hold {
      public:
        explicit Hold(CallLock &l) : lock_(l.owner_.load(std::memory_order_relaxed) == std::this_thread::get_id() ? nullptr : &l)
        {
            if (!lock_) return;
            lock_->mu_.lock();
            lock_->owner_.store(std::this_thread::get_id(), std::memory_order_relaxed);
        }
        ~Hold()
        {
            if (!lock_) return;
            lock_->owner_.store(std::thread::id(), std::memory_order_relaxed);
            lock_->mu_.unlock();
        }
        Hold(const Hold &) = delete;
        Hold &operator=(const Hold &) = delete;
        explicit operator bool() const { return lock_ != nullptr; }

      private:
        CallLock *lock_;
    };

  private:
    std::mutex mu_;
    std::atomic<std::thread::id> owner_{std::thread::id()}; // only its holder ever finds its own number here
};

} // namespace vqb
