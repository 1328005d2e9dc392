// restart_order.h -- restart files of the mixed state.
#pragma once
#include <cstddef>

namespace falcon {

// Restart files hold the state, eight variables, as [block][var][cell] and the correction
// as [block][var][interior cell]; the mixed device arrays hold G variables of a cell side
// by side (Layout). Whole blocks, in host memory, from the device's order to the file's: n
// values per variable and block. The type and G are constants, so that the loops become
// structure loads (64 MB of FP32 on 16 cores: 1.8 -> 0.4 ms). A load reorders on the GPU
// (launch_state_from_file), since the copies there read what other cores have just
// written: 21.2M cells 129 ms, 112 without.
template <class T, int G>
void blocks_to_file(const unsigned char* src, unsigned char* dst, size_t nblocks, size_t n) {
#pragma omp parallel for schedule(static)
    for (long g = 0; g < (long)(nblocks * (8 / G)); ++g) {
        const T* s = reinterpret_cast<const T*>(src) + (size_t)g * G * n;
        T* d = reinterpret_cast<T*>(dst) + (size_t)g * G * n;
        for (size_t c = 0; c < n; ++c)
            for (int v = 0; v < G; ++v) d[v * n + c] = s[c * G + v];
    }
}

}  // namespace falcon
