// Bookkeeping of a run's record buffer, apart from the run driver and free of CUDA so that it can be
// checked without a device.
#pragma once
#include <algorithm>
#include <array>
#include <cstddef>

namespace stb {

// Records that fit a run's buffer on the device (Buf: bytes, ensure(bytes), grow_keep(bytes, keep
// bytes, stream)), each `one` bytes.  The kernels store below `cap`, so cap follows this process's own
// buffer: over several ranks the buffers differ (a context keeps the room of its earlier runs), and
// the ranks exchange record counts only.
template <typename Buf>
struct RecordRoom {
    Buf &buf;
    size_t one;
    unsigned long long cap = 0;    // records the buffer holds
    unsigned long long asked = 0;  // records a re-run after an overflow is given

    RecordRoom(Buf &b, size_t record_bytes) : buf(b), one(record_bytes) {}
    // start of the run or of a re-run: room for at least `least` records
    auto begin(unsigned long long least) {
        const auto e = buf.ensure(size_t(std::max(asked, least)) * one);
        cap = buf.bytes / one;
        return e;
    }
    // room for `need` records, keeping the first `keep`
    template <typename Stream>
    auto room(unsigned long long need, unsigned long long keep, Stream st) {
        decltype(buf.ensure(size_t(0))) e{};
        if (need <= cap) return e;
        e = buf.grow_keep(size_t(std::max(need, cap + cap / 2)) * one, size_t(keep) * one, st);
        cap = buf.bytes / one;
        return e;
    }
    // what a rank tells the others after a batch that has brought the run to n records
    std::array<unsigned long long, 2> report(unsigned long long n) const { return {n > cap ? 1ull : 0ull, n}; }
    // whether the run starts again: any rank's records did not fit (all ranks see the same reports)
    bool overflowed(const unsigned long long *reports, int ranks) {
        bool over = false;
        unsigned long long most = 0;
        for (int k = 0; k < ranks; ++k) {
            over = over || reports[2 * k] != 0;
            most = std::max(most, reports[2 * k + 1]);
        }
        if (over) asked = most + most / 4 + 4096;
        return over;
    }
};

}  // namespace stb
