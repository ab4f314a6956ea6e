// A setup step done once on every device of the process: module-scope device arrays (the procedural
// textures' tables) exist once per device, so a flag for the whole process would leave the second device's
// at zero.
#pragma once

#include <mutex>
#include <set>
#include <string>

namespace lts {

class OncePerDevice {
   public:
    // Runs f ("" on success) unless it has succeeded for `device` before; callers of other threads wait.
    template <class F>
    std::string run(int device, F&& f) {
        std::lock_guard<std::mutex> lock(mu_);
        if (done_.count(device)) return "";
        std::string e = f();
        if (e.empty()) done_.insert(device);
        return e;
    }

   private:
    std::mutex mu_;
    std::set<int> done_;
};

}  // namespace lts
