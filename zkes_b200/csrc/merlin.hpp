// Host-side Fiat-Shamir transcript: Merlin (STROBE-128 over Keccak-f[1600]) as wrapped by
// src/util/transcript.rs:13-46 of the reference.  Written from the STROBE v1.0.2 and Merlin
// v1.0 specifications; only the three STROBE operations Merlin uses are present.
#pragma once
#include <cstdint>
#include <cstring>
#include <cstddef>

namespace zk {

template <int N>
inline uint64_t turn(uint64_t x) {
  return N ? (x << (N & 63)) | (x >> ((64 - N) & 63)) : x;
}
inline void chi(uint64_t* row, uint64_t x0, uint64_t x1, uint64_t x2, uint64_t x3, uint64_t x4) {
  row[0] = x0 ^ (~x1 & x2);
  row[1] = x1 ^ (~x2 & x3);
  row[2] = x2 ^ (~x3 & x4);
  row[3] = x3 ^ (~x4 & x0);
  row[4] = x4 ^ (~x0 & x1);
}

// One round from a to b, every lane and rotation by name: lane (x, y) of the rho step, turned by its offset, is lane (y, 2x + 3y) of
// the chi step.  A permutation takes a CPU core 0.35 us; with the lanes found by index arithmetic it was 3.3 us, most of a host-stepped
// round's 7 us and 10 us of the start of a transcript.
inline void keccak_round(const uint64_t* a, uint64_t* b, uint64_t constant) {
  const uint64_t c0 = a[0] ^ a[5] ^ a[10] ^ a[15] ^ a[20], c1 = a[1] ^ a[6] ^ a[11] ^ a[16] ^ a[21];
  const uint64_t c2 = a[2] ^ a[7] ^ a[12] ^ a[17] ^ a[22], c3 = a[3] ^ a[8] ^ a[13] ^ a[18] ^ a[23];
  const uint64_t c4 = a[4] ^ a[9] ^ a[14] ^ a[19] ^ a[24];
  const uint64_t d0 = c4 ^ turn<1>(c1), d1 = c0 ^ turn<1>(c2), d2 = c1 ^ turn<1>(c3), d3 = c2 ^ turn<1>(c4), d4 = c3 ^ turn<1>(c0);
  chi(b + 0, turn<0>(a[0] ^ d0), turn<44>(a[6] ^ d1), turn<43>(a[12] ^ d2), turn<21>(a[18] ^ d3), turn<14>(a[24] ^ d4));
  chi(b + 5, turn<28>(a[3] ^ d3), turn<20>(a[9] ^ d4), turn<3>(a[10] ^ d0), turn<45>(a[16] ^ d1), turn<61>(a[22] ^ d2));
  chi(b + 10, turn<1>(a[1] ^ d1), turn<6>(a[7] ^ d2), turn<25>(a[13] ^ d3), turn<8>(a[19] ^ d4), turn<18>(a[20] ^ d0));
  chi(b + 15, turn<27>(a[4] ^ d4), turn<36>(a[5] ^ d0), turn<10>(a[11] ^ d1), turn<15>(a[17] ^ d2), turn<56>(a[23] ^ d3));
  chi(b + 20, turn<62>(a[2] ^ d2), turn<55>(a[8] ^ d3), turn<39>(a[14] ^ d4), turn<41>(a[15] ^ d0), turn<2>(a[21] ^ d1));
  b[0] ^= constant;
}

inline void keccak_f1600(uint64_t a[25]) {
  static const uint64_t RC[24] = {
      0x0000000000000001ull, 0x0000000000008082ull, 0x800000000000808Aull, 0x8000000080008000ull,
      0x000000000000808Bull, 0x0000000080000001ull, 0x8000000080008081ull, 0x8000000000008009ull,
      0x000000000000008Aull, 0x0000000000000088ull, 0x0000000080008009ull, 0x000000008000000Aull,
      0x000000008000808Bull, 0x800000000000008Bull, 0x8000000000008089ull, 0x8000000000008003ull,
      0x8000000000008002ull, 0x8000000000000080ull, 0x000000000000800Aull, 0x800000008000000Aull,
      0x8000000080008081ull, 0x8000000000008080ull, 0x0000000080000001ull, 0x8000000080008008ull};
  uint64_t b[25];
  for (int round = 0; round < 24; round += 2) {
    keccak_round(a, b, RC[round]);
    keccak_round(b, a, RC[round + 1]);
  }
}

class Strobe128 {
 public:
  static constexpr int kRate = 166;
  explicit Strobe128(const uint8_t* label, size_t n) {
    memset(st_, 0, sizeof st_);
    const uint8_t head[6] = {1, kRate + 2, 1, 0, 1, 96};
    memcpy(st_, head, 6);
    memcpy(st_ + 6, "STROBEv1.0.2", 12);
    permute();
    pos_ = pos_begin_ = cur_flags_ = 0;
    meta_ad(label, n, false);
  }
  void meta_ad(const uint8_t* d, size_t n, bool more) { begin_op(kM | kA, more); absorb(d, n); }
  void ad(const uint8_t* d, size_t n, bool more) { begin_op(kA, more); absorb(d, n); }
  void prf(uint8_t* out, size_t n, bool more) { begin_op(kI | kA | kC, more); squeeze(out, n); }

  // raw state access (the device-resident transcript is seeded from / written back to it)
  uint8_t* state() { return st_; }
  uint8_t& pos() { return pos_; }
  uint8_t& pos_begin() { return pos_begin_; }
  uint8_t& cur_flags() { return cur_flags_; }

 private:
  enum : uint8_t { kI = 1, kA = 2, kC = 4, kT = 8, kM = 16, kK = 32 };
  void permute() {
    uint64_t lanes[25];
    memcpy(lanes, st_, 200);  // little-endian host
    keccak_f1600(lanes);
    memcpy(st_, lanes, 200);
  }
  void run_f() {
    st_[pos_] ^= pos_begin_;
    st_[pos_ + 1] ^= 0x04;
    st_[kRate + 1] ^= 0x80;
    permute();
    pos_ = 0;
    pos_begin_ = 0;
  }
  void absorb(const uint8_t* d, size_t n) {
    for (size_t i = 0; i < n; i++) {
      st_[pos_++] ^= d[i];
      if (pos_ == kRate) run_f();
    }
  }
  void squeeze(uint8_t* out, size_t n) {
    for (size_t i = 0; i < n; i++) {
      out[i] = st_[pos_];
      st_[pos_++] = 0;
      if (pos_ == kRate) run_f();
    }
  }
  void begin_op(uint8_t flags, bool more) {
    if (more) return;  // continuation of the current operation
    const uint8_t old_begin = pos_begin_;
    pos_begin_ = pos_ + 1;
    cur_flags_ = flags;
    const uint8_t hdr[2] = {old_begin, flags};
    absorb(hdr, 2);
    if ((flags & (kC | kK)) && pos_ != 0) run_f();
  }
  uint8_t st_[200];
  uint8_t pos_, pos_begin_, cur_flags_;
};

class MerlinTranscript {
 public:
  MerlinTranscript(const uint8_t* label, size_t n) : strobe_(reinterpret_cast<const uint8_t*>("Merlin v1.0"), 11) {
    append_message(reinterpret_cast<const uint8_t*>("dom-sep"), 7, label, n);
  }
  void append_message(const uint8_t* label, size_t ln, const uint8_t* msg, size_t n) {
    const uint32_t len = (uint32_t)n;
    uint8_t le[4] = {(uint8_t)len, (uint8_t)(len >> 8), (uint8_t)(len >> 16), (uint8_t)(len >> 24)};
    strobe_.meta_ad(label, ln, false);
    strobe_.meta_ad(le, 4, true);
    strobe_.ad(msg, n, false);
  }
  void append_u64(const uint8_t* label, size_t ln, uint64_t v) {
    uint8_t le[8];
    for (int i = 0; i < 8; i++) le[i] = (uint8_t)(v >> (8 * i));
    append_message(label, ln, le, 8);
  }
  void challenge_bytes(const uint8_t* label, size_t ln, uint8_t* out, size_t n) {
    const uint32_t len = (uint32_t)n;
    uint8_t le[4] = {(uint8_t)len, (uint8_t)(len >> 8), (uint8_t)(len >> 16), (uint8_t)(len >> 24)};
    strobe_.meta_ad(label, ln, false);
    strobe_.meta_ad(le, 4, true);
    strobe_.prf(out, n, false);
  }
  Strobe128& strobe() { return strobe_; }

 private:
  Strobe128 strobe_;
};

}  // namespace zk
