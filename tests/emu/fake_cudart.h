// State of the stand-in CUDA runtime (fake_cudart.cpp).
#pragma once
#include <cstddef>
#include <map>
#include <utility>

namespace fake {
constexpr int kDevices = 2;
struct Block {
	size_t bytes;
	int device;
	bool host;
	void* pool;
};
struct Pool {
	int device;
	size_t kept, threshold;  // freed bytes still held; most of them that a synchronisation leaves
};
extern size_t limit;
extern size_t used[kDevices];
extern size_t launches[kDevices];
}  // namespace fake
