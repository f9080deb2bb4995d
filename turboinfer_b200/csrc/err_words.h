// err_words.h -- error words that kernels set and the host reads behind a synchronisation: one for every model, so that of several models (driven by
// several threads, on the library's one stream) each hears of its own kernels only.  Word 0 belongs to calls that concern no model, and to
// the models beyond the first kWords - 1.
#pragma once
#include <mutex>

namespace tib {

struct ErrWords {
    static constexpr int kWords = 1024;
    int* host = nullptr;   // [kWords] mapped host memory
    int* dev = nullptr;    // ... as kernels see it
    int take() {
        std::lock_guard<std::mutex> lk(mu);
        for (int i = 1; i < kWords; ++i)
            if (!used[i]) {
                used[i] = true;
                if (host) host[i] = 0;
                return i;
            }
        return 0;
    }
    void give(int i) {
        std::lock_guard<std::mutex> lk(mu);
        used[i] = false;
    }
    // whether word i was set; clears it
    bool fetch(int i) {
        if (!host) return false;
        volatile int* w = host + i;
        if (!*w) return false;
        *w = 0;
        return true;
    }

private:
    std::mutex mu;
    bool used[kWords] = {};
};

}  // namespace tib
