// workspace_pool.h -- workspaces kept between calls.
//
// A workspace is in the pool only while no call uses it.  The pool holds at
// most kMost of them and a given number of bytes of each device's memory; the
// longest idle leave first.  A workspace belongs to the CUDA context that it
// was made in: once the program has reset that context, its addresses may
// belong to someone else and its handles to nobody, so it is forgotten, not
// freed, wherever it leaves the pool.
//
// Workspace: `int device`, `unsigned long long context`, `size_t bytes()`
// (device memory) and `drop_host_memory()` (what no context owns).
// Contexts::of(device): the id of the context that the device has now, 0 when
// it has none or that is unknown.
#pragma once

#include <cstddef>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

namespace necsim {

template <typename Workspace, typename Contexts>
class WorkspacePool {
  public:
    static constexpr size_t kMost = 4;

    // The idle workspace that `fits` likes best of the given device (a smaller
    // value is better, 0: does not fit), or null.
    template <typename Fits>
    std::unique_ptr<Workspace> take(int device, Fits &&fits) {
        const unsigned long long id = Contexts::of(device);
        std::lock_guard<std::mutex> lock(mu_);
        size_t best = idle_.size();
        unsigned long long best_fit = 0;
        for (size_t j = 0; j < idle_.size(); ++j) {
            const Workspace &w = *idle_[j];
            if (id == 0 || w.device != device || w.context != id) continue;
            const unsigned long long fit = fits(w);
            if (fit != 0 && (best == idle_.size() || fit < best_fit)) {
                best = j;
                best_fit = fit;
            }
        }
        if (best == idle_.size()) return nullptr;
        return remove(best);
    }

    // Keeps a workspace of a finished call, within `limit` bytes of its device.
    void put(std::unique_ptr<Workspace> w, size_t limit) {
        const unsigned long long id = Contexts::of(w->device);
        if (id == 0 || w->bytes() > limit) return;
        w->context = id;
        std::vector<std::unique_ptr<Workspace>> gone;
        {
            std::lock_guard<std::mutex> lock(mu_);
            for (size_t j = 0; j < idle_.size();) {
                if (idle_[j]->device == w->device && idle_[j]->context != id)
                    gone.push_back(remove(j));
                else
                    ++j;
            }
            size_t bytes = w->bytes();
            for (auto &o : idle_) bytes += o->device == w->device ? o->bytes() : 0;
            while (!idle_.empty() && (idle_.size() >= kMost || bytes > limit)) {
                if (idle_.front()->device == w->device) bytes -= idle_.front()->bytes();
                gone.push_back(remove(0));
            }
            idle_.push_back(std::move(w));
        }
        dispose(gone);
    }

    // Empties the pool; whether device memory was freed.
    bool empty_out() {
        std::vector<std::unique_ptr<Workspace>> gone;
        {
            std::lock_guard<std::mutex> lock(mu_);
            gone.swap(idle_);
        }
        return dispose(gone);
    }

  private:
    std::unique_ptr<Workspace> remove(size_t j) {
        std::unique_ptr<Workspace> w = std::move(idle_[j]);
        idle_.erase(idle_.begin() + (std::ptrdiff_t)j);
        return w;
    }

    // (outside the lock)
    static bool dispose(std::vector<std::unique_ptr<Workspace>> &gone) {
        bool freed = false;
        for (auto &w : gone) {
            if (Contexts::of(w->device) == w->context) {
                w.reset();
                freed = true;
            } else {
                w->drop_host_memory();
                (void)w.release();
            }
        }
        return freed;
    }

    std::mutex mu_;
    std::vector<std::unique_ptr<Workspace>> idle_;
};

}  // namespace necsim
