// Tags of the messages of the path in windows of steps (resident_window.cuh): how a reader knows the words of a head.
//
// A head is two 64-bit words, stored and loaded together; but that both arrive together is not promised, so each says of itself whose it
// is.  The first has room for the launch (20 bits) and the message (24), the second for 8 bits of each.  What a launch leaves in a
// buffer lies there until another writes it, and launches of few messages write the first buffers only: the heads are therefore
// cleared before the lower 8 bits of a launch's number come round, and the number of buffers, after which a launch writes a
// buffer again, is not a multiple of 256.
#pragma once

#ifdef __CUDACC__
#define B200_TAG __host__ __device__ __forceinline__
#else
#define B200_TAG inline
#endif

namespace b200
{
constexpr unsigned int WINDOW_EPOCH_BITS = 20, WINDOW_MESSAGE_BITS = 24;

// (no tag of a launch is 0, which is what a cleared word says)
B200_TAG unsigned long long windowTag(unsigned int epoch, unsigned int message)
{
    return ((unsigned long long)epoch << WINDOW_MESSAGE_BITS) | (message & ((1u << WINDOW_MESSAGE_BITS) - 1u));
}

B200_TAG unsigned int windowShortTag(unsigned int epoch, unsigned int message) { return ((epoch & 0xFFu) << 8) | (message & 0xFFu); }

// The number of the launch behind one with number `epoch`; `clear`: once all heads are cleared.
inline unsigned int windowNextEpoch(unsigned int epoch, bool *clear)
{
    const unsigned int next = (epoch + 1u) & ((1u << WINDOW_EPOCH_BITS) - 1u);
    *clear = (next & 0xFFu) == 0u;
    return *clear ? next + 1u : next;
}

inline unsigned int windowBuffers(unsigned int least) { return least % 256u ? least : least + 1u; }
}   // namespace b200
