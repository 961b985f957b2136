// The word through which the threads of a query row hand its reference maximum from tile to tile in suffix attention: the value's bits below, the number of
// tiles it stands for above (tests/test_reference_word_cpu.py runs it).
#pragma once

#include <cstdint>

#ifndef B200KV_HD
#ifdef __CUDACC__
#define B200KV_HD __host__ __device__ __forceinline__
#else
#define B200KV_HD inline
#endif
#endif

namespace b200kv {

B200KV_HD unsigned long long reference_word(uint32_t value, uint32_t seq) { return (static_cast<unsigned long long>(seq) << 32) | value; }

// The value a thread has published, by way of the number above it as the thread finds it afterwards (any thread's: the next tile's may have put its own word there
// from the store on).  Numbers stay below 2^31, so their top bit adds nothing; the compiler, which cannot know, has to wait for it.
B200KV_HD uint32_t own_reference(uint32_t seq_found, uint32_t own) { return own | (seq_found & 0x80000000u); }

}  // namespace b200kv
