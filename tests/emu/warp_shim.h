// shim.h with warp collectives that order no memory, as the hardware's: a ballot or shuffle hands over values only, and
// between lanes just __syncwarp and the block barrier order loads and stores. ThreadSanitizer then reports any shared or
// global access that a kernel leaves unordered. Full-warp masks only; a block's threads are whole warps. Blocks of more
// than 256 threads keep shim.h's collectives on barriers: a thousand spinning threads take seconds.
#pragma once
#define __shfl_sync shim_shfl_sync
#define __shfl_up_sync shim_shfl_up_sync
#define __shfl_down_sync shim_shfl_down_sync
#define __shfl_xor_sync shim_shfl_xor_sync
#define __ballot_sync shim_ballot_sync
#define __match_any_sync shim_match_any_sync
#define __any_sync shim_any_sync
#define __all_sync shim_all_sync
#include "shim.h"
#undef __shfl_sync
#undef __shfl_up_sync
#undef __shfl_down_sync
#undef __shfl_xor_sync
#undef __ballot_sync
#undef __match_any_sync
#undef __any_sync
#undef __all_sync

#include <atomic>

namespace emu {
// A lane's contribution to its warp's collective number n lies in slot n % 2 as two words, each half of the value
// tagged with n: readers look until both tags are n, with relaxed accesses only. A slot is written again two collectives
// later, when every lane has read it.
struct Slot {
	std::atomic<uint64_t> half[2];
};
extern Slot slots[2][1024];
extern thread_local uint32_t collectives;

inline void Put(uint64_t v)
{
	const uint64_t tag = static_cast<uint64_t>(++collectives) << 32;
	Slot& s = slots[collectives & 1][threadIdx.x];
	s.half[0].store(tag | (v & 0xffffffffu), std::memory_order_relaxed);
	s.half[1].store(tag | (v >> 32), std::memory_order_relaxed);
}

inline uint64_t Get(int src)
{
	Slot& s = slots[collectives & 1][wid() * 32 + src];
	uint64_t v[2];
	for (int h = 0; h < 2; ++h) {
		for (;;) {
			v[h] = s.half[h].load(std::memory_order_relaxed);
			if (static_cast<uint32_t>(v[h] >> 32) == collectives) { break; }
			std::this_thread::yield();
		}
	}
	return (v[1] << 32) | (v[0] & 0xffffffffu);
}

template <class T> inline T Exchange(T v, int src, bool valid)
{
	Put(bits(v));
	T r = v;
	for (int l = 0; l < 32; ++l) {  // every lane's value, so that no lane runs two collectives ahead
		const uint64_t b = Get(l);
		if (valid && l == src) { r = unbits<T>(b); }
	}
	return r;
}

template <class Pred> inline unsigned Lanes(uint64_t v, Pred pred)
{
	Put(v);
	unsigned b = 0;
	for (int l = 0; l < 32; ++l) {
		if (pred(Get(l))) { b |= 1u << l; }
	}
	return b;
}
}  // namespace emu

namespace emu {
inline bool Large() { return blockDim.x > 256; }
}  // namespace emu

template <class T> inline T __shfl_sync(unsigned m, T v, int src)
{
	return emu::Large() ? shim_shfl_sync(m, v, src) : emu::Exchange(v, src & 31, true);
}
template <class T> inline T __shfl_up_sync(unsigned m, T v, unsigned d)
{
	const int s = emu::lane() - static_cast<int>(d);
	return emu::Large() ? shim_shfl_up_sync(m, v, d) : emu::Exchange(v, s, s >= 0);
}
template <class T> inline T __shfl_down_sync(unsigned m, T v, unsigned d)
{
	const int s = emu::lane() + static_cast<int>(d);
	return emu::Large() ? shim_shfl_down_sync(m, v, d) : emu::Exchange(v, s, s <= 31);
}
template <class T> inline T __shfl_xor_sync(unsigned m, T v, int x)
{
	return emu::Large() ? shim_shfl_xor_sync(m, v, x) : emu::Exchange(v, emu::lane() ^ x, true);
}
inline unsigned __ballot_sync(unsigned m, int pred)
{
	return emu::Large() ? shim_ballot_sync(m, pred) : emu::Lanes(pred ? 1u : 0u, [](uint64_t v) { return v != 0; });
}
template <class T> inline unsigned __match_any_sync(unsigned m, T v)
{
	if (emu::Large()) { return shim_match_any_sync(m, v); }
	const uint64_t mine = emu::bits(v);
	return emu::Lanes(mine, [mine](uint64_t x) { return x == mine; });
}
inline int __any_sync(unsigned m, int pred) { return __ballot_sync(m, pred) != 0; }
inline int __all_sync(unsigned m, int pred) { return __ballot_sync(m, !pred) == 0; }
