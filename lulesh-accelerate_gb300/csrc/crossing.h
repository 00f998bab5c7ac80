// crossing.h -- how a Domain record's eleven arrays cross between the host and
// the device, chosen from what is known about the host's arrays.  No CUDA
// calls: api.cu asks the driver about the arrays and passes on its answers.
#pragma once

#include <cstddef>
#include <cstdint>

namespace lulesh {

enum class HostMemory {
    kPageable,   // the C library's, nothing that CUDA knows
    kPinned,     // page-locked by CUDA, allocated or registered
    kOther       // the device's own or managed memory
};

// One array of the host, and for a pinned one the driver's description of the
// allocation or registered piece that its first value lies in.
struct HostArray {
    uintptr_t at;        // 0: left out
    size_t bytes;
    HostMemory memory;
    uintptr_t device;    // a kernel's address of the first value, 0: not mapped
    uintptr_t piece;     // where the piece begins
    size_t piece_bytes;
    bool writable;       // by a kernel
};

// Through the context's pinned buffer, by a kernel on the host's own arrays,
// or field by field through the copy engine.
enum class Crossing { kStaged, kDirect, kCopied };

inline bool overlap(const HostArray &a, const HostArray &b)
{
    return a.at && b.at && a.at < b.at + b.bytes && b.at < a.at + a.bytes;
}

// A kernel takes 8-byte words, so it needs arrays aligned to them, each mapped
// and within one pinned piece from its first value to its last (two pieces
// with a gap between them look the same from both ends), and for the way
// back writable and apart from one another: copies to arrays that share
// memory leave the last one's values there, a kernel whichever came last.  The
// copy engine asks for none of that, and answers memory that is not the
// host's with an error or its own rules.
inline Crossing crossing(const HostArray *arrays, int n, bool to_host, bool have_buffer)
{
    bool pageable = false, direct = true;
    for (int i = 0; i < n; ++i) {
        const HostArray &a = arrays[i];
        if (!a.at) continue;
        if (a.memory == HostMemory::kOther) return Crossing::kCopied;
        if (a.memory == HostMemory::kPageable) {
            pageable = true;
            continue;
        }
        if (a.at % sizeof(double) || a.device % sizeof(double) || !a.device) direct = false;
        if (a.at < a.piece || a.bytes > a.piece_bytes || a.at - a.piece > a.piece_bytes - a.bytes) direct = false;
        if (to_host && !a.writable) direct = false;
        for (int j = 0; to_host && j < i; ++j)
            if (overlap(a, arrays[j])) direct = false;
    }
    if (pageable) return have_buffer ? Crossing::kStaged : Crossing::kCopied;
    return direct ? Crossing::kDirect : Crossing::kCopied;
}

}  // namespace lulesh
