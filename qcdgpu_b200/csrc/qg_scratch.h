// qg_scratch.h -- device scratch that its owner keeps between calls, and the
// pieces in which a link table passes through it.  Host code without CUDA:
// the calls come through Api (Error with kSuccess and kNoMemory; alloc, free
// and sync in the order of one stream), so that each of them can be made to
// fail without a GPU.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace qg {

struct Scratch {
    void *p = nullptr;
    size_t bytes = 0;
};

// `want` bytes, or where they are not free a half, a quarter, ... of them,
// `least` at least.  A buffer that came out smaller is asked for in full
// again by the next call.
template <class Api>
typename Api::Error scratch_reserve(Api &api, Scratch &st, size_t want, size_t least)
{
    if (st.bytes >= want) return Api::kSuccess;
    api.free(st.p);
    st = Scratch{};
    for (size_t n = want;;) {
        void *p = nullptr;
        const typename Api::Error e = api.alloc(&p, n);
        if (e == Api::kSuccess) {
            st.p = p;
            st.bytes = n;
            return e;
        }
        if (e != Api::kNoMemory || n <= least) return e;
        n = n / 2 < least ? least : n / 2;
    }
}

// A table of `planes` rows of `rowsize` elements of `es` bytes through a stage of
// `bytes`: whole rows, or pieces of one row, each converted and copied
// (to_host; else copied and converted) in stream order.  convert(row, rows,
// s0, s1) handles elements [s0, s1) of the rows, copy(offset, n) the n table
// bytes there.  After an error nothing is in flight any more: the caller may
// give back its table, and the owner the stage.
template <class Api, class Convert, class Copy>
typename Api::Error table_pieces(Api &api, size_t bytes, int planes, uint32_t rowsize, size_t es, bool to_host,
                                 Convert convert, Copy copy)
{
    const size_t row = (size_t)rowsize * es;
    const int step = (int)(bytes / row);                 // whole rows at a time; 0: pieces of one row
    const uint32_t piece = step ? rowsize : (uint32_t)(bytes / es);
    for (int p = 0; p < planes; p += step ? step : 1) {
        const int np = step ? (planes - p < step ? planes - p : step) : 1;
        for (uint32_t s0 = 0; s0 < rowsize;) {
            const uint32_t s1 = rowsize - s0 > piece ? s0 + piece : rowsize;
            const size_t at = (size_t)p * row + (size_t)s0 * es, n = (size_t)np * (s1 - s0) * es;
            typename Api::Error e = to_host ? convert(p, np, s0, s1) : copy(at, n);
            if (e == Api::kSuccess) e = to_host ? copy(at, n) : convert(p, np, s0, s1);
            if (e != Api::kSuccess) {
                api.sync();
                return e;
            }
            s0 = s1;
        }
    }
    return Api::kSuccess;
}

}  // namespace qg
