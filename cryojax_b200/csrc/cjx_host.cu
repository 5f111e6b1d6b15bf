// Host-side steps of a batched call in native code: the per-image parameter
// records, the processing order of a batch and the quaternion's share of the
// pose gradient.  Each was a few dozen NumPy or autograd operations on arrays
// of one to a few thousand images, whose fixed cost per operation was most of
// a small call: one 64^2 image spent 240 us on the host around 20 us of
// kernels.  No device work, no state: safe from any thread.
#include <cmath>
#include <cstdint>
#include <new>
#include <utility>
#include <vector>

#include "cjx_common.cuh"

namespace cjx {
namespace {

constexpr double kRadPerDeg = 3.14159265358979323846 / 180.0;

enum Source { kQuat, kOffset, kPixel, kKilovolts, kScale, kDefocus, kAstig, kAngle, kCsMm, kContrast, kPhase, kEnvAmp, kEnvB, kSources };

// Rotation matrix of q / |q|: q scaled by sqrt(2 / |q|^2), products of its entries.
void quat_to_matrix(const double* quat, bool normalise, double* R) {
  double q[4] = {quat[0], quat[1], quat[2], quat[3]};
  if (normalise) {
    const double len = std::sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
    for (double& v : q) v /= len;
  }
  const double s = std::sqrt(2.0 / (q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]));
  const double w = q[0] * s, x = q[1] * s, y = q[2] * s, z = q[3] * s;
  R[0] = 1.0 - y * y - z * z;
  R[1] = x * y - z * w;
  R[2] = x * z + y * w;
  R[3] = x * y + z * w;
  R[4] = 1.0 - x * x - z * z;
  R[5] = y * z - x * w;
  R[6] = x * z - y * w;
  R[7] = y * z + x * w;
  R[8] = 1.0 - x * x - y * y;
}

// Hilbert-curve index of (x, y) in [0, 2^bits)^2 (two's complement throughout, as NumPy's int64).
int64_t hilbert_index(uint64_t x, uint64_t y, int bits) {
  uint64_t d = 0;
  for (uint64_t s = 1ull << (bits - 1); s > 0; s >>= 1) {
    const bool rx = (x & s) != 0, ry = (y & s) != 0;
    d += s * s * ((3u * rx) ^ (unsigned)ry);
    if (!ry) {
      if (rx) {
        x = s - 1 - x;
        y = s - 1 - y;
      }
      const uint64_t t = x;
      x = y;
      y = t;
    }
  }
  return (int64_t)d;
}

double clip(double v, double lo, double hi) { return v < lo ? lo : (v > hi ? hi : v); }  // NaN stays NaN

}  // namespace
}  // namespace cjx

extern "C" int cjx_pack_image_params(int64_t n_images, uint32_t flags, int offset_dim, const void* const* sources,
                                     const int64_t* strides, cjx_image_params* out) {
  using namespace cjx;
  if (n_images < 0) return fail(CJX_ERR_INVALID_ARGUMENT, "n_images < 0");
  if (n_images == 0) return CJX_OK;
  if (!sources || !strides || !out) return fail(CJX_ERR_INVALID_ARGUMENT, "sources, strides and out must be non-NULL");
  if (offset_dim != 2 && offset_dim != 3) return fail(CJX_ERR_INVALID_ARGUMENT, "offset_dim must be 2 or 3");
  const bool theory = (flags & CJX_PACK_THEORY) != 0, envelope = (flags & CJX_PACK_ENVELOPE) != 0;
  if (envelope && !theory) return fail(CJX_ERR_INVALID_ARGUMENT, "an envelope belongs to a transfer theory");
  const double* src[kSources];
  for (int s = 0; s < kSources; ++s) {
    src[s] = static_cast<const double*>(sources[s]);
    const bool needed = s <= kScale || (theory && s <= kPhase) || envelope;
    if (needed && !src[s]) return fail(CJX_ERR_INVALID_ARGUMENT, "a needed source is NULL");
  }
  for (int64_t i = 0; i < n_images; ++i) {
    cjx_image_params p{};
    auto at = [&](Source s) { return src[s][i * strides[s]]; };
    quat_to_matrix(src[kQuat] + i * strides[kQuat], (flags & CJX_PACK_NORMALISE) != 0, p.rot);
    const double* off = src[kOffset] + i * strides[kOffset];
    p.shift_x = off[0];
    p.shift_y = off[1];
    p.pixel_size = at(kPixel);
    const double v = 1000.0 * at(kKilovolts);
    p.wavelength = 12.2639 / std::sqrt(v + 0.97845e-6 * (v * v));  // relativistic electron wavelength, Angstrom
    p.scale = at(kScale);
    p.envelope_amplitude = 1.0;
    if (theory) {
      p.defocus = at(kDefocus) + (offset_dim == 3 ? off[2] : 0.0);
      p.astigmatism = at(kAstig);
      p.astigmatism_angle = at(kAngle) * kRadPerDeg;
      p.spherical_aberration = at(kCsMm) * 1e7;
      const double ac = at(kContrast);
      p.phase_shift = at(kPhase) * kRadPerDeg;
      p.phase_total = p.phase_shift + std::atan(ac / std::sqrt(1.0 - ac * ac));
      p.amplitude_contrast_ratio = ac;
    }
    if (envelope) {
      p.envelope_amplitude = at(kEnvAmp);
      p.envelope_b_factor = at(kEnvB);
    }
    out[i] = p;
  }
  return CJX_OK;
}

extern "C" int cjx_orientation_order(int64_t n_images, const double* rotations, int64_t stride, int bits,
                                     int32_t* order) {
  using namespace cjx;
  if (n_images < 0 || n_images > INT32_MAX) return fail(CJX_ERR_INVALID_ARGUMENT, "n_images out of range");
  // beyond 32 bits an index needs more than 64
  if (bits < 1 || bits > 32) return fail(CJX_ERR_INVALID_ARGUMENT, "bits must be in [1, 32]");
  if (n_images == 0) return CJX_OK;
  if (!rotations || !order) return fail(CJX_ERR_INVALID_ARGUMENT, "rotations and order must be non-NULL");
  try {
    std::vector<int64_t> key(n_images);
    std::vector<int32_t> other(n_images);
    const double scale = (double)((1ll << bits) - 1), root2 = std::sqrt(2.0);
    for (int64_t i = 0; i < n_images; ++i) {
      const double* R = rotations + i * stride;
      double nx = R[2], ny = R[5], nz = R[8];  // the plane's normal, sign-free
      if (nz < 0 || (nz == 0 && ny < 0)) {
        nx = -nx;
        ny = -ny;
        nz = -nz;
      }
      const double k = std::sqrt(2.0 / (1.0 + clip(nz, 0.0, 1.0)));  // Lambert's equal-area disk of radius sqrt(2)
      const double gx = clip(std::nearbyint((k * nx / root2 + 1.0) * 0.5 * scale), 0.0, scale);
      const double gy = clip(std::nearbyint((k * ny / root2 + 1.0) * 0.5 * scale), 0.0, scale);
      const uint64_t none = 1ull << 63;  // a NaN's place: no index bit set
      // sorted as unsigned bytes below: at 32 bits, where an index fills the signed type, its sign bit is turned
      // over so that the order stays that of signed 64-bit integers
      key[i] = hilbert_index(gx == gx ? (uint64_t)gx : none, gy == gy ? (uint64_t)gy : none, bits) ^
               (bits == 32 ? INT64_MIN : 0);
    }
    for (int64_t i = 0; i < n_images; ++i) order[i] = (int32_t)i;
    int32_t *from = order, *to = other.data();
    for (int shift = 0; shift < 2 * bits; shift += 8) {  // stable counting sort, a byte of the key at a time
      int64_t count[257] = {0};
      for (int64_t i = 0; i < n_images; ++i) ++count[((key[i] >> shift) & 255) + 1];
      for (int b = 0; b < 256; ++b) count[b + 1] += count[b];
      for (int64_t i = 0; i < n_images; ++i) to[count[(key[from[i]] >> shift) & 255]++] = from[i];
      std::swap(from, to);
    }
    if (from != order)
      for (int64_t i = 0; i < n_images; ++i) order[i] = from[i];
  } catch (const std::bad_alloc&) {
    return fail(CJX_ERR_INVALID_ARGUMENT, "out of host memory");
  }
  return CJX_OK;
}

extern "C" int cjx_quaternion_grad(int64_t n_images, const double* wxyz, int64_t quat_stride, const double* d_rot,
                                   int columns, double* d_wxyz) {
  using namespace cjx;
  if (n_images < 0) return fail(CJX_ERR_INVALID_ARGUMENT, "n_images < 0");
  if (columns != 2 && columns != 3) return fail(CJX_ERR_INVALID_ARGUMENT, "columns must be 2 or 3");
  if (n_images == 0) return CJX_OK;
  if (!wxyz || !d_rot || !d_wxyz) return fail(CJX_ERR_INVALID_ARGUMENT, "wxyz, d_rot and d_wxyz must be non-NULL");
  for (int64_t i = 0; i < n_images; ++i) {
    const double* q = wxyz + i * quat_stride;
    const double w = q[0], x = q[1], y = q[2], z = q[3];
    double G[3][3] = {};
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < columns; ++b) G[a][b] = d_rot[(i * 3 + a) * columns + b];
    // R = 1 + s P(q), s = 2 / |q|^2, P quadratic: dL/dq = s G.dP/dq - s^2 (G.P) q
    const double s = 2.0 / (w * w + x * x + y * y + z * z);
    const double m01 = G[0][1] - G[1][0], m02 = G[0][2] - G[2][0], m12 = G[1][2] - G[2][1];
    const double p01 = G[0][1] + G[1][0], p02 = G[0][2] + G[2][0], p12 = G[1][2] + G[2][1];
    const double gp = -G[0][0] * (y * y + z * z) - G[1][1] * (x * x + z * z) - G[2][2] * (x * x + y * y) +
                      p01 * x * y + p02 * x * z + p12 * y * z - m01 * z * w + m02 * y * w - m12 * x * w;
    const double dw = -m01 * z + m02 * y - m12 * x;
    const double dx = -2.0 * x * (G[1][1] + G[2][2]) + p01 * y + p02 * z - m12 * w;
    const double dy = -2.0 * y * (G[0][0] + G[2][2]) + p01 * x + p12 * z + m02 * w;
    const double dz = -2.0 * z * (G[0][0] + G[1][1]) + p02 * x + p12 * y - m01 * w;
    const double c = s * s * gp;
    d_wxyz[4 * i] = s * dw - c * w;
    d_wxyz[4 * i + 1] = s * dx - c * x;
    d_wxyz[4 * i + 2] = s * dy - c * y;
    d_wxyz[4 * i + 3] = s * dz - c * z;
  }
  return CJX_OK;
}
