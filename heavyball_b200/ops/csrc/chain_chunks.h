// How many elements a block of a specialised fused-chain launch covers (plain C++: the launcher, and a CPU test of the rule).
//
// A block walks its chunk in steps of 1024 elements times the vectors that a thread has in flight.  Few elements: as many blocks as
// possible, since the dependent steps of one block are what the launch takes.  Many: long chunks, which pay for finding the tensor
// once; and a chunk shorter than one step leaves vectors without work, which the kinds with four vectors feel first.  Measured on
// one B200 over eight tensors, us at chunks of 2048 / 4096 / 8192:
//                                  0.6 M           2.4 M            4.8 M            7.0 M           9.6 M elements
//   Adam fp32 (2 vectors)      4.1/4.9/7.2     9.6/10.4/8.9    16.4/15.7/18.0   31.0/30.2/29.8  43.6/44.0/44.6
//   Adam bf16 + 8 bits (1)     6.6/9.5/14.1   17.6/16.9/18.5   32.4/31.9/31.8   47.3/46.3/47.1  63.6/61.7/61.5
//   momentum fp32 (4)          4.2/4.9/6.7     9.6/8.0/7.4     16.3/12.2/13.7   23.6/17.1/16.1  36.5/28.4/28.3
//   parameter update (4)       3.0/3.0/3.8     5.9/4.2/4.7      9.6/6.8/6.1     12.8/8.8/8.5    17.6/12.3/11.4
#pragma once

namespace hb {

constexpr int kChunk = 8192;  // the general kernel's, and the largest
constexpr int kMediumChunk = 4096, kSmallChunk = 2048;

// `vectors`: four-element vectors a thread of the kind has in flight; `elems`: of the whole launch.
constexpr int chain_chunk(int vectors, long long elems) {
  const bool wide = vectors > 2;
  if (elems <= (wide ? 900'000 : 2'400'000)) return kSmallChunk;
  return elems <= (wide ? 4'800'000 : 9'700'000) ? kMediumChunk : kChunk;
}

}  // namespace hb
