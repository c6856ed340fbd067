// Which CUDA-core kernel takes a call: tiles in shared memory (na2d_tile*.cuh) or one warp per pixel (na2d_simt.cuh).
//
// A tile works through its channel chunks one after the other (copies, barrier, arithmetic), so on a GPU that is
// not filled a tiled kernel takes the same time however small the problem is.  One warp per pixel needs
// many pixels to fill a wave and re-reads every row, but a wave of it is short.  Both times are estimated, in
// microseconds:
//   tiles      fixed + chunks * (chunk + chunk_ks * ks) * (1 + unaligned, where rows are not multiples of four channels)
//   per pixel  (wave + groups * (group + group_lane * lanes) + taps * tap_lane * lanes) * max(1, 0.6 + pixels / 4300)
// with chunks of 32 channels, taps window members in groups of 32, and `lanes` channels to a lane (1, 2, 4, 8).  Up to
// 1700 pixels are in flight at once, one to a warp; beyond that the time grows with their number.
// The constants are fitted to times of both kernels on one B200: 128 to 65536 pixels, 16 to 256 channels, windows 3 to
// 13 (240 to 700 points each).  There the kernel chosen takes 1.00 (unfused pair 1.01) times the better one's time on
// average, 1.2 times (pair 1.6) at worst; tiles alone took up to 3.0 (pair 6.3) times in fp32 and 7.5 times in 16 bits.
//
// The constants are those of the tiled kernels also for the 1D rows that na2d_line.cuh takes, where "tiles" means a kernel twice as fast,
// and for the fp32 2D calls that na2d_box.cuh takes: such calls cross over later than they could.  One sequence of 64 channels, window 7,
// bf16, per pixel / na2d_line, us: forward 2048 tokens 6.2 / 8.2, 4096 10.9 / 8.3, 8192 16.5 / 8.1; backward 1024 tokens 19.1 / 17.8,
// 4096 38.5 / 18.0.
#pragma once

namespace na2d_tile {

enum class Work { kForward, kQueryHalf, kBackward, kDot, kApply, kKeySum };

struct Cost {
    float fixed, chunk, chunk_ks, unaligned, wave, group, group_lane, tap_lane;
};

inline const Cost& cost_of(Work work, bool one_d, bool half) {
    static constexpr Cost kOneD[3][2] = {                                                              // fp32, 16 bits
        {{6.97f, 2.89f, 0.54f, 1.14f, 5.88f, 2.42f, 0.27f, 0.25f}, {7.38f, 9.55f, 0.20f, 0.08f, 6.69f, 1.65f, 0.07f, 0.10f}},
        {{11.22f, 3.68f, 0.05f, 1.29f, 7.58f, 2.44f, 0.69f, 0.16f}, {6.72f, 14.10f, 0.34f, 0.02f, 9.62f, 3.83f, 0.03f, 0.48f}},
        {{16.88f, 5.21f, 1.27f, 0.39f, 13.45f, 7.95f, 1.44f, 0.95f}, {17.31f, 9.77f, 0.11f, 0.02f, 11.62f, 6.92f, 0.00f, 0.46f}},
    };
    static constexpr Cost kTwoD[6][2] = {
        {{3.48f, 2.63f, 1.56f, 0.43f, 2.69f, 2.98f, 0.28f, 0.19f}, {3.58f, 8.85f, 1.88f, 0.00f, 0.10f, 9.58f, 0.16f, 0.13f}},
        {{7.74f, 5.33f, 0.75f, 0.63f, 6.19f, 3.73f, 0.69f, 0.19f}, {2.82f, 9.31f, 1.11f, 0.08f, 0.28f, 7.81f, 0.25f, 0.20f}},
        {{9.82f, 8.13f, 4.87f, 0.64f, 1.40f, 18.81f, 0.08f, 1.09f}, {11.55f, 15.96f, 2.44f, 0.00f, 0.07f, 23.71f, 0.08f, 0.56f}},
        {{5.97f, 1.64f, 1.08f, 0.37f, 1.39f, 2.45f, 0.44f, 0.17f}, {5.26f, 8.12f, 0.07f, 0.37f, 0.34f, 5.67f, 0.08f, 0.05f}},
        {{4.82f, 3.47f, 0.03f, 0.64f, 0.76f, 2.28f, 0.00f, 0.01f}, {4.77f, 4.21f, 0.58f, 0.64f, 0.83f, 1.78f, 0.05f, 0.04f}},
        {{3.15f, 0.52f, 2.77f, 0.24f, 0.04f, 9.44f, 0.04f, 0.02f}, {2.68f, 0.58f, 3.23f, 0.24f, 0.03f, 7.55f, 0.01f, 0.04f}},
    };
    return one_d ? kOneD[(int)work][half] : kTwoD[(int)work][half];
}

// `pixels`: (batch, head, row, column) positions; half: 16-bit tensors.
inline bool faster_in_tiles(Work work, bool one_d, bool half, long long pixels, int C, int ks) {
    const Cost& c = cost_of(work, one_d, half);
    const int chunks = (C + 31) / 32, taps = one_d ? ks : ks * ks, groups = (taps + 31) / 32;
    const int lanes = C <= 32 ? 1 : C <= 64 ? 2 : C <= 128 ? 4 : 8;
    const float waves = 0.6f + (float)pixels / 4300.f;
    const float tiles = c.fixed + chunks * (c.chunk + c.chunk_ks * ks) * (C % 4 ? 1.f + c.unaligned : 1.f);
    const float per_pixel = c.wave + groups * (c.group + c.group_lane * lanes) + taps * c.tap_lane * lanes;
    return tiles <= per_pixel * (waves < 1.f ? 1.f : waves);
}

}  // namespace na2d_tile
