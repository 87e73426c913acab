// The hash by which rtgb_prepare_scene tells a changed scene from the prepared
// one (what the geometry and scene signatures of
// gpu_scene_acceleration.cpp:116-135 do).
//
// A step takes one 64-bit word: exclusive or, then the running hash's upper bits
// folded 29 places down, then an odd multiplier (2^64 over the golden ratio,
// Knuth's multiplicative hashing). Each step is a bijection of the running hash
// for a given word and of the word for a given hash, so inputs that differ in one
// word always hash differently. The fold is there for inputs that differ in
// several: a multiplication carries bits upwards only, so without it a flipped
// bit 63 (the sign of the float in a word's upper half) stays exactly bit 63, and
// flipping it in any two words gives the hash of the unchanged input. Folded, the
// sign bits of a word's two floats (63 and 31, alone or together) reach the
// multiplier as lower bits whose carries depend on the hash so far. (Folded 32
// places, flipping both signs of a word would again leave bit 63 alone.)
//
// Words go to kHashLanes interleaved lanes folded in order at the end, the tail
// byte by byte. One running hash is a chain of dependent multiplies, 8 bytes per
// five or so clocks: 13.5 ms of a million triangles' 108 MB, more than half of
// preparing them; the lanes' multiplies overlap.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <thread>

namespace rtgb {

constexpr uint64_t kHashSeed = 14695981039346656037ull;
constexpr int kHashLanes = 8;

inline uint64_t hash_step(uint64_t h, uint64_t word) {
    h ^= word;
    h ^= h >> 29;
    return h * 0x9e3779b97f4a7c15ull;
}

inline uint64_t hash_words(uint64_t h, const void* data, size_t bytes) {
    const unsigned char* p = static_cast<const unsigned char*>(data);
    size_t i = 0;
    if (bytes >= 8 * kHashLanes) {
        uint64_t lane[kHashLanes];
        for (int k = 0; k < kHashLanes; ++k) lane[k] = h + static_cast<uint64_t>(k);
        for (; i + 8 * kHashLanes <= bytes; i += 8 * kHashLanes) {
            uint64_t w[kHashLanes];
            std::memcpy(w, p + i, sizeof w);
            for (int k = 0; k < kHashLanes; ++k) lane[k] = hash_step(lane[k], w[k]);
        }
        for (int k = 0; k < kHashLanes; ++k) h = hash_step(h, lane[k]);
    }
    for (; i + 8 <= bytes; i += 8) {
        uint64_t w;
        std::memcpy(&w, p + i, 8);
        h = hash_step(h, w);
    }
    for (; i < bytes; ++i) h = hash_step(h, p[i]);
    return h;
}

// Arrays of kHashSplit bytes or more are hashed in kHashParts slices on as many
// threads and the slices' hashes folded, so the value does not depend on whether
// the threads could be started. Below it starting them (some 20 us each) costs
// what they save.
constexpr size_t kHashSplit = 4u << 20;
constexpr int kHashParts = 4;

inline uint64_t hash_bytes(uint64_t h, const void* data, size_t bytes) {
    if (bytes < kHashSplit) return hash_words(h, data, bytes);
    const unsigned char* p = static_cast<const unsigned char*>(data);
    const size_t part = (bytes / kHashParts) & ~size_t(63);
    uint64_t hash[kHashParts];
    auto slice = [&](int k) {
        const size_t from = part * static_cast<size_t>(k);
        hash[k] = hash_words(h + static_cast<uint64_t>(k), p + from, k + 1 < kHashParts ? part : bytes - from);
    };
    std::thread workers[kHashParts];
    for (int k = 1; k < kHashParts; ++k) {
        try {
            workers[k] = std::thread(slice, k);
        } catch (...) {  // no thread to be had, or no memory for its state: this one does the slice
            slice(k);
        }
    }
    slice(0);
    for (int k = 1; k < kHashParts; ++k) {
        if (workers[k].joinable()) workers[k].join();
    }
    return hash_words(h, hash, sizeof hash);
}

// An array of `count` elements with its length; a missing array is an empty one.
template <typename T>
uint64_t hash_array(uint64_t h, const T* data, long long count) {
    const long long n = count > 0 && data ? count : 0;
    h = hash_words(h, &n, sizeof n);
    return n > 0 ? hash_bytes(h, data, static_cast<size_t>(n) * sizeof(T)) : h;
}

}  // namespace rtgb
