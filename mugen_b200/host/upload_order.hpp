// Which uploads of step metadata still lie last on their stream.
//
// The kernel that uploads lets the next launch on its stream start before it has stored anything, and the library's kernels read
// metadata ahead of their own wait.  So the first of them behind an upload, on the upload's stream, is launched without
// that overlap, or it is one that waits before it reads metadata and before it lets the next kernel start.  Uploads of one step can stand on several streams at once (mla_step_begin on one, the plan of a group of layers on
// another), so each region of the metadata buffer remembers its own; a region that is written anew forgets the
// upload before, which the caller has ordered ahead of this one.
#pragma once

#include <array>
#include <cstddef>
#include <cstdint>

namespace mugen::mla {

template <size_t Regions>
class UploadOrder {
public:
    // `stream`: names one stream, whatever handle it goes by
    void uploaded(size_t region, uint64_t stream) { at_[region] = {stream, true}; }
    // a kernel that waits for the upload has been launched on `stream`
    void followed(uint64_t stream) { for (auto& u : at_) if (u.stream == stream) u.open = false; }
    bool open(uint64_t stream) const
    {
        for (const auto& u : at_) if (u.open && u.stream == stream) return true;
        return false;
    }

private:
    struct Upload { uint64_t stream = 0; bool open = false; };
    std::array<Upload, Regions> at_{};
};

}  // namespace mugen::mla
