// Fourier-space work around the gravity step: the reference's initial-condition generator
// (Zel'dovich and 2LPT displacements of a lattice, src/initialize.cpp:261-355,436-898) and its
// matter power spectrum (src/power.cpp:33-77, src/power.cu:32-85, src/fft.cpp:172-330).
//
// Both follow the reference's conventions: grids of Nfour^3 points in x-major order, the
// half-complex layout N x N x (N/2 + 1) of a real-to-complex transform along z, the 6-point
// quintic-spline cloud kernel (CLOUD_MIN -2 .. CLOUD_MAX 3, fft.hpp:113-134) for mass
// assignment and interpolation with its window deconvolved in k-space, and the random field
// drawn row by row (one generator per (x, y) row of k-space) from GSL's "taus" generator
// (L'Ecuyer 1996), so that a seed gives the reference's field.  The transforms are cuFFT's
// (single precision, out of place); the reference's normalisations are applied around them.
#include "ct_internal.cuh"

#include <cub/cub.cuh>
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace ct {
namespace {

constexpr int FT_TPB = 256;
constexpr int CLOUD_MIN = -2;
constexpr int CLOUD_MAX = 3;

// ---------------------------------------------------------------- the cloud kernel
// Quintic spline of support 3 (fft.hpp:116-131), with the reference's mixed float / double
// arithmetic.
__host__ __device__ inline float cloud_weight(float x) {
	x = fabsf(x);
	const float x2 = x * x;
	const float x3 = x * x2;
	const float x4 = x2 * x2;
	const float x5 = x3 * x2;
	if (x > 3.0f) {
		return 0.0f;
	} else if (x < 1.0f) {
		return (33.0f - 30.0 * x2 + 15.0f * x4 - 5.0f * x5) / 60.0f;
	} else if (x < 2.0f) {
		return (51.0 + 75.0 * x - 210 * x2 + 150 * x3 - 45 * x4 + 5 * x5) / 120.0;
	} else {
		return (243.0 - 405.0 * x + 270 * x2 - 90 * x3 + 15 * x4 - x5) / 120.0;
	}
}

__host__ __device__ inline double sinc(double x) {
	return x == 0.0 ? 1.0 : sin(x) / x;
}

// Inverse of the kernel's window at wavenumber kh (grid units): 1 / sinc(kh / 2)^6.
__host__ __device__ inline double cloud_filter(double kh) {
	const double s = sinc(0.5 * kh);
	const double s3 = s * (s * s);
	return 1.0 / (s3 * s3);
}

__device__ __forceinline__ int wrap(int i, int n) {
	i %= n;
	return i < 0 ? i + n : i;
}

// ---------------------------------------------------------------- GSL "taus"
// The maximally equidistributed combined Tausworthe generator of L'Ecuyer (Math. Comp. 65,
// 1996, 203-213): three 32-bit components, output their XOR.  Seeding as GSL's gsl_rng_taus
// does: seed 0 is taken as 1, the components are successive values of the LCG
// x -> 69069 x mod 2^32 from the seed, and six outputs are discarded.  uniform_pos divides an
// output by 2^32 and skips zero.
struct Taus {
	uint32_t s1, s2, s3;

	__host__ __device__ uint32_t next() {
		s1 = ((s1 & 4294967294u) << 12) ^ (((s1 << 13) ^ s1) >> 19);
		s2 = ((s2 & 4294967288u) << 4) ^ (((s2 << 2) ^ s2) >> 25);
		s3 = ((s3 & 4294967280u) << 17) ^ (((s3 << 3) ^ s3) >> 11);
		return s1 ^ s2 ^ s3;
	}
	__host__ __device__ void seed(uint32_t s) {
		if (s == 0) {
			s = 1;
		}
		s1 = 69069u * s;
		s2 = 69069u * s1;
		s3 = 69069u * s2;
		for (int i = 0; i < 6; i++) {
			next();
		}
	}
	__host__ __device__ double uniform_pos() {
		uint32_t v;
		do {
			v = next();
		} while (v == 0);
		return v / 4294967296.0;
	}
};

// ---------------------------------------------------------------- power table
// P(k) in Mpc^3 at k_i = exp(logkmin + i dlogk): cubic interpolation of log P in log k over
// four table points (power_spectrum_function::operator(), initialize.cpp:110-139).  Indices
// are clamped to the table (the reference reads past it when k is out of range; the host
// checks the range before generating).
struct PowerTable {
	const float* P;
	int n;
	float logkmin, dlogk;

	__host__ __device__ float operator()(float k) const {
		const float logk = logf(k);
		const float k0 = (logk - logkmin) / dlogk;
		int i0 = int(k0) - 1;
		i0 = i0 < 0 ? 0 : (i0 > n - 4 ? n - 4 : i0);
		const int i1 = i0 + 1, i2 = i0 + 2, i3 = i0 + 3;
		const float x = k0 - i1;
		const float y0 = logf(P[i0]);
		const float y1 = logf(P[i1]);
		const float y2 = logf(P[i2]);
		const float y3 = logf(P[i3]);
		const float k1 = (y2 - y0) * 0.5;
		const float k2 = (y3 - y1) * 0.5;
		const float a = y1;
		const float b = k1;
		const float c = -2 * k1 - k2 - 3 * y1 + 3 * y2;
		const float d = k1 + k2 + 2 * y1 - 2 * y2;
		return expf(a + b * x + c * x * x + d * x * x * x);
	}
};

// ---------------------------------------------------------------- k-space fields
// The Gaussian field for the displacement derivatives dim1, dim2 (3: none):
// Y(k) = n(k) sqrt(P(|k|)) box^-1.5 N^3 (-i k_dim1)(-i k_dim2) / k^2, n a unit complex normal,
// times the cloud kernel's inverse window (twolpt_generate, initialize.cpp:436-540).  Every
// (x, y) row of k-space has its own generator (seed (I0 N + I1) 1234 + 42, eight draws
// discarded) for kz > 0; the kz = 0 element takes the generator of the mirrored row and its
// conjugate on the lower half, which makes the kz = 0 plane Hermitian.  The seeds do not depend
// on dim1, dim2, so every field of one call draws the same numbers: the amplitude
// n(k) sqrt(P) box^-1.5 N^3 is made once (row generators, then one thread per mode) and each
// field is an elementwise pass over it.

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
	return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ float wavenumber(int I, int N, float box_size) {
	const int i = I < N / 2 ? I : I - N;
	return 2.f * (float) M_PI / box_size * float(i);
}

// sigma8 normalisation of the table (power_spectrum_function::normalize and
// sigma8_integrand, initialize.cpp:141-172): Simpson's rule over 8192 log-k intervals of the
// top-hat variance at R = 8 / h Mpc, the integrand in float as the reference takes it, the sum in
// double; the table is scaled in place and the factor kept in norm.  One block: the host took 0.8 ms
// for the same 8193 values.
constexpr int SIGMA_TPB = 1024;
constexpr int SIGMA_N = 8 * 1024;
__global__ void __launch_bounds__(SIGMA_TPB) k_sigma8(PowerTable t, float* P, float logkmax_table, float hubble, double sigma8, float* norm) {
	__shared__ double s_sum[SIGMA_TPB / 32];
	const float logkmax = logkmax_table - 2.5 * t.dlogk;
	const float logkmin = t.logkmin + 1.5 * t.dlogk;
	const float dlogk = (logkmax - logkmin) / SIGMA_N;
	const float R = 8 / hubble;
	const float c0 = float(9) / (2. * float(M_PI) * float(M_PI)) / powf(R, 6);
	double sum = 0.0;
	for (int i = threadIdx.x; i <= SIGMA_N; i += SIGMA_TPB) {
		const float x = i == SIGMA_N ? logkmax : logkmin + i * dlogk;
		const float k = expf(x);
		const float p = t(k);
		const float tmp = (sinf(k * R) - k * R * cosf(k * R));
		const float f = c0 * p * tmp * tmp * powf(k, -3.f);
		const double w = i == 0 || i == SIGMA_N ? 1.0 / 3.0 : (i & 1) ? 4.0 / 3.0 : 2.0 / 3.0;
		sum += w * f * dlogk;
	}
	for (int o = 16; o; o >>= 1) {
		sum += __shfl_xor_sync(0xffffffffu, sum, o);
	}
	if ((threadIdx.x & 31) == 0) {
		s_sum[threadIdx.x >> 5] = sum;
	}
	__syncthreads();
	sum = 0.0;
	for (int i = 0; i < SIGMA_TPB / 32; i++) {
		sum += s_sum[i];
	}
	const float f = (float) ((sigma8 * sigma8) / sum);
	for (int i = threadIdx.x; i < t.n; i += SIGMA_TPB) {
		P[i] *= f;
	}
	if (threadIdx.x == 0) {
		*norm = f;
	}
}

// Per-axis values of one call, by grid index: the inverse window at the axis' wavenumber and the
// lattice point's stencil (first cell and six weights).  Evaluated once an axis; every mode and
// every point used to evaluate its own in double, which bounded the field and interpolation passes
// (256^3: 161 us a field against 25 us of memory traffic, 1,260 us an interpolation against 70).
struct AxisTables {
	float* filter;  // [N]
	int* cell;      // [N]
	double* weight; // [6][N]
};

__global__ void k_ic_axis(int N, float box_size, AxisTables t) {
	const int I = blockIdx.x * blockDim.x + threadIdx.x;
	if (I >= N) {
		return;
	}
	t.filter[I] = (float) cloud_filter(wavenumber(I, N, box_size) * box_size / N);
	const double x0 = fixed_to_double(fixed_from_double(I * (1.0 / N)));
	const int i1 = (int) (x0 * N);
	const double f = x0 * N - i1;
	t.cell[I] = i1;
	for (int j = 0; j < 6; j++) {
		t.weight[j * N + I] = cloud_weight((float) (-(j + CLOUD_MIN) + f));
	}
}

// A mode times the inverse window, axis by axis.
__device__ __forceinline__ float2 filtered(float2 v, float fx, float fy, float fz) {
	v = make_float2(v.x * fx, v.y * fx);
	v = make_float2(v.x * fy, v.y * fy);
	return make_float2(v.x * fz, v.y * fz);
}

// The uniforms (x, y) of every mode, as floats, row by row (the generators are sequential).
__global__ void __launch_bounds__(FT_TPB) k_ic_uniforms(int N, float2* __restrict__ U) {
	const int NZ = N / 2 + 1;
	const int64_t rows = (int64_t) N * N;
	for (int64_t row = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; row < rows; row += (int64_t) gridDim.x * blockDim.x) {
		const int I0 = (int) (row / N), I1 = (int) (row % N);
		float2* out = U + row * NZ;
		Taus g;
		g.seed((uint32_t) (((int64_t) I0 * N + I1) * 1234 + 42));
		for (int l = 0; l < 8; l++) {
			g.uniform_pos();
		}
		for (int I2 = 1; I2 < NZ; I2++) {
			const double x = g.uniform_pos();
			const double y = g.uniform_pos();
			out[I2] = make_float2((float) x, (float) y);
		}
		// kz = 0: the mirrored row's generator (no draw for the k = 0 mode)
		const int J0 = I0 > N / 2 ? N - I0 : I0;
		const int J1 = I1 > N / 2 ? N - I1 : I1;
		g.seed((uint32_t) (((int64_t) J0 * N + J1) * 1234 + 42));
		for (int l = 0; l < 8; l++) {
			g.uniform_pos();
		}
		float2 u = make_float2(1.f, 0.f);
		if (I0 != 0 || I1 != 0) {
			const double x = g.uniform_pos();
			const double y = g.uniform_pos();
			u = make_float2((float) x, (float) y);
		}
		out[0] = u;
	}
}

// In place: uniforms -> amplitude n(k) sqrt(P(|k|)) factor (0 at k = 0).
__global__ void __launch_bounds__(FT_TPB) k_ic_amplitude(int N, float box_size, float factor, PowerTable power, float2* __restrict__ U) {
	const int NZ = N / 2 + 1;
	const int64_t total = (int64_t) N * N * NZ;
	for (int64_t e = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; e < total; e += (int64_t) gridDim.x * blockDim.x) {
		const int I2 = (int) (e % NZ);
		const int64_t row = e / NZ;
		const int I0 = (int) (row / N), I1 = (int) (row % N);
		if (I0 == 0 && I1 == 0 && I2 == 0) {
			U[e] = make_float2(0.f, 0.f);
			continue;
		}
		const float kx = wavenumber(I0, N, box_size), ky = wavenumber(I1, N, box_size), kz = wavenumber(I2, N, box_size);
		const float K0 = sqrtf(kx * kx + ky * ky + kz * kz);
		const float2 u = U[e];
		const float ang = 2.f * float(M_PI) * u.y;
		const float mag = sqrtf(-logf(fabsf(u.x)));
		float2 r = make_float2(cosf(ang) * mag, sinf(ang) * mag);
		const float sp = sqrtf(power(K0));
		r = make_float2(r.x * sp, r.y * sp);
		U[e] = make_float2(r.x * factor, r.y * factor);
	}
}

// One field: Y = A (-i k_dim1)(-i k_dim2) / k^2, conjugated (times the parity sign) on the lower
// half of the kz = 0 plane, times the inverse window.
__global__ void __launch_bounds__(FT_TPB) k_ic_field(int N, float box_size, int dim1, int dim2, const float* __restrict__ filter, const float2* __restrict__ A,
		cufftComplex* __restrict__ Y) {
	const int NZ = N / 2 + 1;
	float sgn = 1.f;
	sgn *= dim1 != 3 ? -1.f : 1.f;
	sgn *= dim2 != 3 ? -1.f : 1.f;
	const int64_t stride = (int64_t) gridDim.x * blockDim.x, total = (int64_t) N * N * NZ;
	// the mode's indices advance with e: no division inside the loop
	const int64_t e0 = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	int I2 = (int) (e0 % NZ), row = (int) (e0 / NZ);
	const int d2 = (int) (stride % NZ), drow = (int) (stride / NZ);
	for (int64_t e = e0; e < total; e += stride) {
		const int I0 = (unsigned) row / (unsigned) N, I1 = row - I0 * N;
		const float kx = wavenumber(I0, N, box_size), ky = wavenumber(I1, N, box_size), kz = wavenumber(I2, N, box_size);
		float2 v = make_float2(0.f, 0.f);
		if (I2 > 0 || I0 != 0 || I1 != 0) {
			const float k2 = kx * kx + ky * ky + kz * kz;
			const float2 K[4] = { make_float2(0.f, -kx), make_float2(0.f, -ky), make_float2(0.f, -kz), make_float2(1.f, 0.f) };
			v = cmul(A[e], K[dim1]);
			v = cmul(v, K[dim2]);
			v = make_float2(v.x / k2, v.y / k2);
			if (I2 == 0 && (I0 > N / 2 || (I0 == 0 && I1 > N / 2))) {
				v = make_float2(v.x * sgn, -v.y * sgn);
			}
		}
		v = filtered(v, __ldg(filter + I0), __ldg(filter + I1), __ldg(filter + I2));
		Y[e] = make_cuComplex(v.x, v.y);
		I2 += d2;
		row += drow;
		if (I2 >= NZ) {
			I2 -= NZ;
			row++;
		}
	}
}

// Second-order displacement field of axis dim from the transformed 2LPT source:
// Y = -i k_dim delta2(k) / k^2 times the inverse window, 0 at k = 0 (twolpt_correction2,
// initialize.cpp:384-434).
__global__ void __launch_bounds__(FT_TPB) k_ic_correction(const cufftComplex* __restrict__ src, cufftComplex* __restrict__ Y, int N, float box_size, int dim,
		const float* __restrict__ filter) {
	const int NZ = N / 2 + 1;
	const int64_t total = (int64_t) N * N * NZ;
	for (int64_t e = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; e < total; e += (int64_t) gridDim.x * blockDim.x) {
		const unsigned row = (unsigned) (e / NZ);  // (at most 2^20 rows)
		const int I2 = (int) (e - (int64_t) row * NZ);
		const int I0 = (int) (row / (unsigned) N), I1 = (int) (row - (unsigned) I0 * (unsigned) N);
		const int i = I0 < N / 2 ? I0 : I0 - N;
		const int j = I1 < N / 2 ? I1 : I1 - N;
		const int k = I2 < N / 2 ? I2 : I2 - N;
		float2 v = make_float2(0.f, 0.f);
		if (i * i + j * j + k * k > 0) {
			const float kx = 2.f * (float) M_PI / box_size * float(i);
			const float ky = 2.f * (float) M_PI / box_size * float(j);
			const float kz = 2.f * (float) M_PI / box_size * float(k);
			const float k2 = kx * kx + ky * ky + kz * kz;
			const float K[3] = { kx, ky, kz };
			const cufftComplex s = src[e];
			// -i K y / k^2
			v = make_float2(K[dim] * s.y, -K[dim] * s.x);
			v = make_float2(v.x / k2, v.y / k2);
			v = filtered(v, __ldg(filter + I0), __ldg(filter + I1), __ldg(filter + I2));
		}
		Y[e] = make_cuComplex(v.x, v.y);
	}
}

// ---------------------------------------------------------------- real space
// The lattice (init_X0, initialize.cpp:650-798): particle (I0 N + I1) N + I2 at I / N, at rest,
// rung 0.
__global__ void __launch_bounds__(FT_TPB) k_ic_lattice(int N, uint32_t* __restrict__ x, uint32_t* __restrict__ y, uint32_t* __restrict__ z,
		float* __restrict__ v0, float* __restrict__ v1, float* __restrict__ v2, int8_t* __restrict__ rung) {
	const int64_t n = (int64_t) N * N * N;
	const double Ninv = 1.0 / N;
	for (int64_t p = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; p < n; p += (int64_t) gridDim.x * blockDim.x) {
		const int I2 = (int) (p % N);
		const int I1 = (int) ((p / N) % N);
		const int I0 = (int) (p / ((int64_t) N * N));
		x[p] = fixed_from_double(I0 * Ninv);
		y[p] = fixed_from_double(I1 * Ninv);
		z[p] = fixed_from_double(I2 * Ninv);
		v0[p] = v1[p] = v2[p] = 0.f;
		rung[p] = 0;
	}
}

// Displacement of axis dim (zeldovich_end, initialize.cpp:800-868): the field interpolated
// with the cloud kernel at each particle's lattice point, dx = -D field / box; the position
// moves by dx (periodic) and the velocity by prefac dx.  Particle (I0 N + I1) N + I2 sits at
// lattice point I, and the kernel's 6^3 weights there are products of per-axis weights that
// depend only on I0, I1, I2, so the 216-term sum is taken as 6-term sums along x, y and z (double
// precision, as the reference accumulates), in two passes: along x into a double grid, each thread
// eight points of a line (a field value is read and converted to double 13 / 8 times; in one pass over
// tiles 10 times); then y and z with the update, the y sums of DISP_ROWS rows of one x in shared memory,
// where a thread keeps to one z and its columns.  256^3, an axis: 276 us in one pass, now 46 + 140,
// against 90 for the bytes of both; four blocks an SM (2lpt 3.72 ms; two 3.88, three 3.80).  The largest
// dx in units of the mean spacing goes to dxmax (float bits: a positive float orders like its bits).
constexpr int DISP_ROWS = 8;
constexpr int DISP_X = 8;
constexpr int IC_MAX_N = 1024;  // points of a grid's axis, at most

// An index at most one grid length outside 0 .. n - 1.
__device__ __forceinline__ int wrap1(int i, int n) {
	return i < 0 ? i + n : (i >= n ? i - n : i);
}

// Sums along x: points x0 .. x0 + 7 (x0 = 8 blockIdx.y) of the line (y, z).
__global__ void __launch_bounds__(FT_TPB) k_ic_sum_x(int N, const float* __restrict__ R, AxisTables t, double* __restrict__ G) {
	const int line = blockIdx.x * FT_TPB + threadIdx.x, plane = N * N;  // (a grid has at most 2^30 points)
	if (line >= plane) {
		return;
	}
	const int x0 = blockIdx.y * DISP_X, nx = min(DISP_X, N - x0);
	const int c0 = __ldg(t.cell + x0);
	// a lattice point's cell is its index or, where I / N rounds below itself, one less
	bool regular = nx == DISP_X;
	for (int i = 1; i < nx; i++) {
		regular = regular && __ldg(t.cell + x0 + i) == c0 + i;
	}
	if (regular) {
		double v[DISP_X + 5];
#pragma unroll
		for (int j = 0; j < DISP_X + 5; j++) {
			v[j] = (double) R[wrap1(c0 + CLOUD_MIN + j, N) * plane + line];
		}
#pragma unroll
		for (int i = 0; i < DISP_X; i++) {
			double acc = 0.0;
#pragma unroll
			for (int j = 0; j < 6; j++) {
				acc += __ldg(t.weight + j * N + x0 + i) * v[i + j];
			}
			G[(x0 + i) * plane + line] = acc;
		}
	} else {
		for (int i = 0; i < nx; i++) {
			const int c = __ldg(t.cell + x0 + i) + CLOUD_MIN;
			double acc = 0.0;
#pragma unroll
			for (int j = 0; j < 6; j++) {
				acc += __ldg(t.weight + j * N + x0 + i) * (double) R[wrap1(c + j, N) * plane + line];
			}
			G[(x0 + i) * plane + line] = acc;
		}
	}
}

// Sums along y and z, scaled by the inverse transform's normalisation, and the update of rows
// (x, 8 blockIdx.x ..) of x = blockIdx.y.
__global__ void __launch_bounds__(FT_TPB, 4) k_ic_displace(int N, const double* __restrict__ G, AxisTables t, double scale, float D, float prefac,
		double box_size_inv, uint32_t* __restrict__ X, float* __restrict__ V, unsigned int* dxmax) {
	extern __shared__ double s_y[];  // [DISP_ROWS][N]
	const int x = blockIdx.y, y0 = blockIdx.x * DISP_ROWS;
	const int ny = min(DISP_ROWS, N - y0);
	const int c0 = __ldg(t.cell + y0);
	bool regular = ny == DISP_ROWS;
	for (int i = 1; i < ny; i++) {
		regular = regular && __ldg(t.cell + y0 + i) == c0 + i;
	}
	for (int z = threadIdx.x; z < N; z += FT_TPB) {
		const double* col = G + (size_t) x * N * N + z;
		if (regular) {
			double v[DISP_ROWS + 5];
#pragma unroll
			for (int j = 0; j < DISP_ROWS + 5; j++) {
				v[j] = col[wrap1(c0 + CLOUD_MIN + j, N) * N];
			}
#pragma unroll
			for (int i = 0; i < DISP_ROWS; i++) {
				double acc = 0.0;
#pragma unroll
				for (int j = 0; j < 6; j++) {
					acc += __ldg(t.weight + j * N + y0 + i) * v[i + j];
				}
				s_y[i * N + z] = acc;
			}
		} else {
			for (int i = 0; i < ny; i++) {
				const int c = __ldg(t.cell + y0 + i) + CLOUD_MIN;
				double acc = 0.0;
#pragma unroll
				for (int j = 0; j < 6; j++) {
					acc += __ldg(t.weight + j * N + y0 + i) * col[wrap1(c + j, N) * N];
				}
				s_y[i * N + z] = acc;
			}
		}
	}
	__syncthreads();
	float mymax = 0.f;
	for (int z = threadIdx.x; z < N; z += FT_TPB) {
		const int p0 = (x * N + y0) * N + z;
		// the rows' positions and velocities are read before any is written: a read behind a write that
		// might be to the same place waits for it, eight trips to memory one after another
		uint32_t xr[DISP_ROWS];
		float vr[DISP_ROWS];
#pragma unroll
		for (int y = 0; y < DISP_ROWS; y++) {
			xr[y] = y < ny ? X[p0 + y * N] : 0u;
			vr[y] = y < ny ? V[p0 + y * N] : 0.f;
		}
		const int c = __ldg(t.cell + z) + CLOUD_MIN;
		int at[6];
		double wz[6];
#pragma unroll
		for (int j = 0; j < 6; j++) {
			at[j] = wrap1(c + j, N);
			wz[j] = __ldg(t.weight + j * N + z);
		}
#pragma unroll
		for (int y = 0; y < DISP_ROWS; y++) {
			if (y < ny) {
				double dx = 0.0;
#pragma unroll
				for (int j = 0; j < 6; j++) {
					dx += wz[j] * s_y[y * N + at[j]];
				}
				dx *= scale;
				dx *= -D * box_size_inv;
				double q = fixed_to_double(xr[y]) + dx;
				if (q >= 1.0) {
					q -= 1.0;
				} else if (q < 0.0) {
					q += 1.0;
				}
				X[p0 + y * N] = fixed_from_double(q);
				V[p0 + y * N] = (float) (vr[y] + prefac * dx);
				mymax = fmaxf(mymax, (float) (dx * N));
			}
		}
	}
	for (int o = 16; o; o >>= 1) {
		mymax = fmaxf(mymax, __shfl_xor_sync(0xffffffffu, mymax, o));
	}
	if ((threadIdx.x & 31) == 0 && mymax > 0.f) {
		atomicMax(dxmax, __float_as_uint(mymax));
	}
}

// The 2LPT source (twolpt_phase, initialize.cpp:565-589).  The reference brings the second
// derivatives in nine phases (yy, zz, xx, zz, xx, yy, xy, xz, yz): an even phase up to 6 keeps its
// field, an odd one adds the product with the kept field, and phases 7 and 8 subtract their squares:
// delta2 = p_yy p_zz + p_xx p_zz + p_xx p_yy - p_xz^2 - p_yz^2 (it keeps p_xy at phase 6 without
// using it, so -p_xy^2 is not part of its source; reproduced as is).  Here each of the five fields
// that count is transformed once; the products and squares are added in the same order.
__global__ void __launch_bounds__(FT_TPB) k_twolpt_products(int64_t n, const float* __restrict__ xx, const float* __restrict__ yy, float* __restrict__ zz,
		float scale) {
	for (int64_t p = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; p < n; p += (int64_t) gridDim.x * blockDim.x) {
		const float a = xx[p] * scale, b = yy[p] * scale, c = zz[p] * scale;
		float d = b * c;
		d += a * c;
		d += a * b;
		zz[p] = d;
	}
}
__global__ void __launch_bounds__(FT_TPB) k_twolpt_squares(int64_t n, const float* __restrict__ xz, const float* __restrict__ yz, float* __restrict__ delta2,
		float scale) {
	for (int64_t p = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; p < n; p += (int64_t) gridDim.x * blockDim.x) {
		const float a = xz[p] * scale, b = yz[p] * scale;
		float d = delta2[p];
		d -= a * a;
		d -= b * b;
		delta2[p] = d;
	}
}

__global__ void k_fill(int64_t n, float* __restrict__ a, float v) {
	for (int64_t p = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; p < n; p += (int64_t) gridDim.x * blockDim.x) {
		a[p] = v;
	}
}

// ---------------------------------------------------------------- power spectrum
// Mass assignment with the cloud kernel on the N^3 grid after folding the box M times
// (accumulate_density_kernel, power.cu:32-61): x -> frac(M x), 216 weights per particle.
__global__ void __launch_bounds__(FT_TPB) k_density(int64_t n, const uint32_t* __restrict__ X, const uint32_t* __restrict__ Yp, const uint32_t* __restrict__ Z,
		int M, int N, float* __restrict__ rho) {
	for (int64_t p = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; p < n; p += (int64_t) gridDim.x * blockDim.x) {
		const float x = fmodf(M * (float(X[p]) * (1.f / 4294967296.f)), 1.0f);
		const float y = fmodf(M * (float(Yp[p]) * (1.f / 4294967296.f)), 1.0f);
		const float z = fmodf(M * (float(Z[p]) * (1.f / 4294967296.f)), 1.0f);
		const int j = (int) (x * N), k = (int) (y * N), l = (int) (z * N);
		const float x0 = x * N - j, y0 = y * N - k, z0 = z * N - l;
		float wy[6], wz[6];
		int cy[6], cz[6];
#pragma unroll
		for (int q = 0; q < 6; q++) {
			wy[q] = cloud_weight(y0 - (q + CLOUD_MIN));
			wz[q] = cloud_weight(z0 - (q + CLOUD_MIN));
			cy[q] = wrap(k + q + CLOUD_MIN, N);
			cz[q] = wrap(l + q + CLOUD_MIN, N);
		}
		for (int a = 0; a < 6; a++) {
			const float wx = cloud_weight(x0 - (a + CLOUD_MIN));
			const int64_t ox = (int64_t) wrap(j + a + CLOUD_MIN, N) * N;
#pragma unroll
			for (int b = 0; b < 6; b++) {
				const int64_t oy = (ox + cy[b]) * N;
				const float wxy = wx * wy[b];
#pragma unroll
				for (int c = 0; c < 6; c++) {
					atomicAdd(rho + oy + cz[c], wxy * wz[c]);
				}
			}
		}
	}
}

// The same deposit through shared memory.  216 float atomics a particle go to the L2 at about 390 G/s
// whatever the particles' order (256^3 particles on 256^3 cells: 9.4 ms); here the particles are first
// listed by tile of 8^3 cells, and a warp adds a tile's particles one after the other to its own copy
// of the tile (13^3 cells with the kernel's reach), each lane one (x, y) row of the 6^3 cells, so that
// no two lanes meet; the block's copies are summed and go to the grid with one atomic a cell and unit
// of at most DEP_UNIT particles.  The row strides put the 32 rows of a warp on distinct banks.  256^3
// on 256^3: 1.93 ms, shared memory 81% busy (14 trips a particle for the cells, 8 for the weights).
constexpr int DEP_TILE = 8;                // cells of a tile per axis
constexpr int DEP_SPAN = DEP_TILE + 5;     // cells its particles reach
constexpr int DEP_SY = 13, DEP_SX = 174;   // strides of y and x in the copy
constexpr int DEP_CELLS = 12 * DEP_SX + 12 * DEP_SY + 13;
constexpr int DEP_WARPS = 4;
constexpr int DEP_UNIT = 1024;             // particles of a work unit
constexpr int DEP_W = 20;                  // floats of a particle's weights: z, the last of x, -, x, y

// cloud_weight at distance f - k of a cell k = CLOUD_MIN + q (a constant) from a particle at fraction f of
// its cell, in double throughout: the cell says which piece of the spline it is (the pieces join with four
// derivatives, so a fraction that rounds to either end may take either).  Its error is the final rounding
// alone; the mixed form takes six conversions and a division a weight.
__device__ __forceinline__ float deposit_weight(double f, int q) {
	const double x = fabs(f - (double) (q + CLOUD_MIN));
	const double x2 = x * x;
	if (q == 2 || q == 3) {
		return (float) (fma(x2, fma(x2, fma(x, -5.0, 15.0), -30.0), 33.0) * (1.0 / 60.0));
	}
	if (q == 1 || q == 4) {
		return (float) (fma(x, fma(x, fma(x, fma(x, fma(x, 5.0, -45.0), 150.0), -210.0), 75.0), 51.0) * (1.0 / 120.0));
	}
	return (float) (fma(x, fma(x, fma(x, fma(x, fma(x, -1.0, 15.0), -90.0), 270.0), -405.0), 243.0) * (1.0 / 120.0));
}

// Cell and fraction of a coordinate (the grid of accumulate_density_kernel, power.cu:32-61).
__device__ __forceinline__ int deposit_cell(uint32_t X, int M, int N, float& frac) {
	const float x = fmodf(M * (float(X) * (1.f / 4294967296.f)), 1.0f);
	const int j = (int) (x * N);
	frac = x * N - j;
	return j < N ? j : j - N;  // (a product rounded up to N is cell 0's)
}

// Tile of every particle: counted, with the particle's rank among its tile's (in no order).
__global__ void __launch_bounds__(FT_TPB) k_dep_count(int64_t n, const uint32_t* __restrict__ X, const uint32_t* __restrict__ Y, const uint32_t* __restrict__ Z,
		int M, int N, int nt, uint32_t* __restrict__ count, uint32_t* __restrict__ rank) {
	for (int64_t p0 = blockIdx.x * (int64_t) blockDim.x; p0 < n; p0 += (int64_t) gridDim.x * blockDim.x) {
		const int64_t p = p0 + threadIdx.x;
		uint32_t tile = 0xffffffffu;
		if (p < n) {
			float f;
			const int j = deposit_cell(X[p], M, N, f) / DEP_TILE, k = deposit_cell(Y[p], M, N, f) / DEP_TILE, l = deposit_cell(Z[p], M, N, f) / DEP_TILE;
			tile = (uint32_t) ((j * nt + k) * nt + l);
		}
		// one atomic for the lanes that share a tile (particles near in memory usually are near)
		const unsigned same = __match_any_sync(0xffffffffu, tile);
		const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
		uint32_t base = 0;
		if (lane == leader && p < n) {
			base = atomicAdd(count + tile, (uint32_t) __popc(same));
		}
		base = __shfl_sync(0xffffffffu, base, leader);
		if (p < n) {
			rank[p] = base + (uint32_t) __popc(same & ((1u << lane) - 1u));
		}
	}
}

// The particles' indices by tile.
__global__ void __launch_bounds__(FT_TPB) k_dep_order(int64_t n, const uint32_t* __restrict__ X, const uint32_t* __restrict__ Y, const uint32_t* __restrict__ Z,
		int M, int N, int nt, const uint32_t* __restrict__ offset, const uint32_t* __restrict__ rank, uint32_t* __restrict__ order) {
	for (int64_t p = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; p < n; p += (int64_t) gridDim.x * blockDim.x) {
		float f;
		const int j = deposit_cell(X[p], M, N, f) / DEP_TILE, k = deposit_cell(Y[p], M, N, f) / DEP_TILE, l = deposit_cell(Z[p], M, N, f) / DEP_TILE;
		order[offset[(j * nt + k) * nt + l] + rank[p]] = (uint32_t) p;
	}
}

// Work units (tile, first particle, particles) of the tiles that hold any.
__global__ void __launch_bounds__(FT_TPB) k_dep_units(int ntile, const uint32_t* __restrict__ count, const uint32_t* __restrict__ offset, uint4* __restrict__ units,
		unsigned int* __restrict__ nunits) {
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= ntile || count[t] == 0) {
		return;
	}
	const uint32_t c = count[t], nu = (c + DEP_UNIT - 1) / DEP_UNIT;
	const unsigned int u = atomicAdd(nunits, nu);
	for (uint32_t q = 0; q < nu; q++) {
		units[u + q] = make_uint4((uint32_t) t, offset[t] + q * DEP_UNIT, min((uint32_t) DEP_UNIT, c - q * DEP_UNIT), 0u);
	}
}

__global__ void __launch_bounds__(32 * DEP_WARPS) k_density_tiles(const uint32_t* __restrict__ X, const uint32_t* __restrict__ Y, const uint32_t* __restrict__ Z,
		int M, int N, int nt, const uint32_t* __restrict__ order, const uint4* __restrict__ units, const unsigned int* __restrict__ nunits,
		unsigned int* __restrict__ next, float* __restrict__ rho) {
	__shared__ float s_rho[DEP_WARPS][DEP_CELLS];
	__shared__ __align__(16) float s_w[DEP_WARPS][32][DEP_W];
	__shared__ unsigned int s_unit;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const unsigned int total = *nunits;
	// this lane's rows of the 6 x 6 (x, y) rows: one of the first 32, and a quarter of one of the last
	// four (24 lanes, one cell each)
	const int a1 = lane / 6, b1 = lane % 6, o1 = a1 * DEP_SX + b1 * DEP_SY;
	const int b2 = 2 + min(lane, 23) / 6, c2 = min(lane, 23) % 6, o2 = 5 * DEP_SX + b2 * DEP_SY + c2;
	float* T = s_rho[w];
	for (;;) {
		if (threadIdx.x == 0) {
			s_unit = atomicAdd(next, 1u);
		}
		__syncthreads();
		const unsigned int u = s_unit;
		if (u >= total) {
			break;
		}
		const uint4 un = units[u];
		const int tx = (int) (un.x / (uint32_t) (nt * nt)), ty = (int) (un.x / (uint32_t) nt % (uint32_t) nt), tz = (int) (un.x % (uint32_t) nt);
		for (int i = lane; i < DEP_CELLS; i += 32) {
			T[i] = 0.f;
		}
		__syncwarp();
		// (the next particles' positions are on their way while these are added)
		uint32_t px = 0, py = 0, pz = 0;
		if (32u * w + lane < un.z) {
			const uint32_t p = order[un.y + 32 * w + lane];
			px = X[p];
			py = Y[p];
			pz = Z[p];
		}
		for (uint32_t q0 = 32 * w; q0 < un.z; q0 += 32 * DEP_WARPS) {
			// a particle a lane: its first cell in the tile and its 18 weights
			const int cnt = min(32, (int) (un.z - q0));
			int base = 0;
			if (lane < cnt) {
				float fx, fy, fz;
				const int j = deposit_cell(px, M, N, fx), k = deposit_cell(py, M, N, fy), l = deposit_cell(pz, M, N, fz);
				base = (j - tx * DEP_TILE) * DEP_SX + (k - ty * DEP_TILE) * DEP_SY + (l - tz * DEP_TILE);
				float* sw = s_w[w][lane];
				const double dx = fx, dy = fy, dz = fz;
#pragma unroll
				for (int q = 0; q < 6; q++) {
					sw[q] = deposit_weight(dz, q);
					sw[8 + q] = deposit_weight(dx, q);
					sw[14 + q] = deposit_weight(dy, q);
				}
				sw[6] = sw[13];
			}
			if (q0 + 32 * DEP_WARPS + lane < un.z) {
				const uint32_t p = order[un.y + q0 + 32 * DEP_WARPS + lane];
				px = X[p];
				py = Y[p];
				pz = Z[p];
			}
			__syncwarp();
			// (a particle's weights are read while the one before it is added: the pass is a chain of
			// trips to shared memory, 16 warps an SM)
			float4 z0, z1;
			float wxy, w2;
			int bs;
			auto fetch = [&](int i) {
				bs = __shfl_sync(0xffffffffu, base, i);
				const float* sw = s_w[w][i];
				z0 = *reinterpret_cast<const float4*>(sw);
				z1 = *reinterpret_cast<const float4*>(sw + 4);  // (z, z, last x, -)
				wxy = sw[8 + a1] * sw[14 + b1];
				w2 = z1.z * sw[14 + b2] * sw[c2];
			};
			fetch(0);
			for (int i = 0; i < cnt; i++) {
				const float4 y0 = z0, y1 = z1;
				const float u1 = wxy, u2 = w2;
				float* r = T + bs + o1;
				float* r2 = T + bs + o2;
				if (i + 1 < cnt) {
					fetch(i + 1);
				}
				r[0] += u1 * y0.x;
				r[1] += u1 * y0.y;
				r[2] += u1 * y0.z;
				r[3] += u1 * y0.w;
				r[4] += u1 * y1.x;
				r[5] += u1 * y1.y;
				if (lane < 24) {
					*r2 += u2;
				}
				__syncwarp();  // the next particle's rows may be these
			}
		}
		__syncthreads();
		// the copies' sum to the grid (the reach wraps around the box)
		for (int i = threadIdx.x; i < DEP_SPAN * DEP_SPAN * DEP_SPAN; i += 32 * DEP_WARPS) {
			const int cz = i % DEP_SPAN, cy = i / DEP_SPAN % DEP_SPAN, cx = i / (DEP_SPAN * DEP_SPAN);
			float v = 0.f;
#pragma unroll
			for (int q = 0; q < DEP_WARPS; q++) {
				v += s_rho[q][cx * DEP_SX + cy * DEP_SY + cz];
			}
			if (v != 0.f) {
				auto cell = [&](int t, int c) {
					int g = t * DEP_TILE + c + CLOUD_MIN;
					g = g < 0 ? g + N : g;
					while (g >= N) {
						g -= N;
					}
					return (int64_t) g;
				};
				atomicAdd(rho + (cell(tx, cx) * N + cell(ty, cy)) * N + cell(tz, cz), v);
			}
		}
		__syncthreads();
	}
}

// Bin of |k| (grid units) among the log-spaced edges (search_kbins, fft.cpp:219-237): -1 below
// 0 or at / above the last edge.
__device__ __forceinline__ int k_bin(const float* kb, int nb, double k) {
	if (k < 0.0 || k >= kb[nb]) {
		return -1;
	}
	int lo = 0, hi = nb;
	while (hi - lo > 1) {
		const int mid = (lo + hi) / 2;
		if (k >= kb[mid]) {
			lo = mid;
		} else {
			hi = mid;
		}
	}
	return lo;
}

constexpr int MAX_BINS = 1024;

// Per-axis factors of the two passes by grid index: the inverse window, and sinc(pi i / N).
__global__ void k_power_axis(int N, double* __restrict__ axis) {
	const int I = blockIdx.x * blockDim.x + threadIdx.x;
	if (I < N) {
		const int64_t i = I < N / 2 ? I : I - N;
		axis[I] = cloud_filter(2.0 * M_PI * i / N);
		axis[N + I] = sinc(M_PI * i / N);
	}
}

// Pass 1 (power_spectrum_compute, fft.cpp:240-304): each mode of the half-complex box,
// deconvolved by the kernel's window (in place), adds |Y|^2, 1 and |k| to its bin.
// Pass 2 (power_spectrum_compute2, :306-360): the mode is multiplied further by
// (sinc(pi i/N) sinc(pi j/N) sinc(pi k/N))^-3 and adds (|Y|^2 - P_bin)^2 to its bin.
__global__ void __launch_bounds__(FT_TPB) k_power_bins(cufftComplex* __restrict__ Y, int N, const float* __restrict__ kb, int nb, int pass,
		const double* __restrict__ axis, const double* __restrict__ pmean, double* __restrict__ out) {
	__shared__ double s_p[MAX_BINS], s_c[MAX_BINS], s_k[MAX_BINS];
	for (int b = threadIdx.x; b < nb; b += blockDim.x) {
		s_p[b] = s_c[b] = s_k[b] = 0.0;
	}
	__syncthreads();
	const int NZ = N / 2 + 1;
	const int64_t total = (int64_t) N * N * NZ;
	const double* f = axis + (pass == 1 ? 0 : N);
	const int lane = threadIdx.x & 31;
	// whole warps step together: the lanes' sums of a bin are added before they go to shared memory
	// (the modes of a warp lie along a row and share few bins; an atomic each met in the same word)
	for (int64_t e0 = blockIdx.x * (int64_t) blockDim.x; e0 < total; e0 += (int64_t) gridDim.x * blockDim.x) {
		const int64_t e = e0 + threadIdx.x;
		int bin = -1;
		double vp = 0.0, vk = 0.0;
		if (e < total) {
			const unsigned row = (unsigned) (e / NZ);  // (at most 2^20 rows)
			const int I2 = (int) (e - (int64_t) row * NZ);
			const int I0 = (int) (row / (unsigned) N), I1 = (int) (row - (unsigned) I0 * (unsigned) N);
			const int64_t i = I0 < N / 2 ? I0 : I0 - N;
			const int64_t j = I1 < N / 2 ? I1 : I1 - N;
			const int64_t k = I2 < N / 2 ? I2 : I2 - N;
			double c0 = f[I0] * f[I1] * f[I2];
			if (pass == 2) {
				c0 = 1.0 / c0;
				c0 = c0 * c0 * c0;
			}
			cufftComplex y = Y[e];
			y.x *= c0;
			y.y *= c0;
			Y[e] = y;
			const double kk = sqrt((double) (i * i + j * j + k * k));
			if (kk > 0) {
				bin = k_bin(kb, nb, kk);
				const float pwr = y.x * y.x + y.y * y.y;
				if (pass == 1) {
					vp = (double) pwr;
					vk = kk;
				} else if (bin >= 0) {
					const double d = (double) (pwr - (float) pmean[bin]);
					vp = d * d;
				}
			}
		}
		unsigned todo = __ballot_sync(0xffffffffu, bin >= 0);
		while (todo) {
			const int b = __shfl_sync(0xffffffffu, bin, __ffs(todo) - 1);
			const unsigned mine = __ballot_sync(0xffffffffu, bin == b);
			double p = bin == b ? vp : 0.0, q = bin == b ? vk : 0.0;
			for (int o = 16; o; o >>= 1) {
				p += __shfl_xor_sync(0xffffffffu, p, o);
				q += __shfl_xor_sync(0xffffffffu, q, o);
			}
			if (lane == 0) {
				atomicAdd(&s_p[b], p);
				if (pass == 1) {
					atomicAdd(&s_c[b], (double) __popc(mine));
					atomicAdd(&s_k[b], q);
				}
			}
			todo &= ~mine;
		}
	}
	__syncthreads();
	for (int b = threadIdx.x; b < nb; b += blockDim.x) {
		if (s_p[b] != 0.0) {
			atomicAdd(&out[b], s_p[b]);
		}
		if (pass == 1 && s_c[b] != 0.0) {
			atomicAdd(&out[nb + b], s_c[b]);
			atomicAdd(&out[2 * nb + b], s_k[b]);
		}
	}
}

}  // namespace
}  // namespace ct

namespace ct {
namespace {

int ft_grid(const Ctx* c, int64_t n) {
	return (int) std::max<int64_t>(1, std::min<int64_t>((n + FT_TPB - 1) / FT_TPB, (int64_t) c->nsm * 8));
}

ct_status fft_check(Ctx* c, cufftResult r, const char* what) {
	if (r != CUFFT_SUCCESS) {
		return fail(c, r == CUFFT_ALLOC_FAILED ? CT_ERR_MEMORY : CT_ERR_CUDA, std::string(what) + ": cuFFT error " + std::to_string((int) r));
	}
	return CT_OK;
}

}  // namespace

// The context's cuFFT plans, one of each kind: kept from one call to the next of the same grid (a
// plan's making took 0.3 to 0.8 ms, several times the transforms of a 64^3 grid), replaced for
// another grid, freed with the context.  They hold no work area: each call lends one from the
// context's pool.
struct FtPlans {
	cufftHandle plan[2] = { 0, 0 };
	size_t work[2] = { 0, 0 };
	int n[2] = { 0, 0 };
};

namespace {

// Device buffers of one call, released on every return path.
struct FtScope {
	Ctx* c;
	std::vector<std::pair<void*, size_t>> bufs;
	std::vector<void*> work;
	cufftHandle plans[2] = { 0, 0 };

	explicit FtScope(Ctx* c_) : c(c_) {
	}
	~FtScope() {
		for (auto& b : bufs) {
			dfree(c, b.first, b.second);
		}
		for (auto p : work) {
			cudaFreeAsync(p, c->stream);
		}
	}
	template<class T>
	ct_status alloc(T** p, size_t count, const char* what) {
		CT_TRY(dalloc(c, (void**) p, sizeof(T) * count, what));
		bufs.push_back({ (void*) *p, sizeof(T) * count });
		return CT_OK;
	}
	ct_status plan(int which, int N, cufftType type) {
		if (!c->ft) {
			c->ft = new FtPlans();
		}
		FtPlans& F = *c->ft;
		if (F.n[which] != N) {
			if (F.n[which]) {
				cufftDestroy(F.plan[which]);
				F.n[which] = 0;
			}
			CT_TRY(fft_check(c, cufftCreate(&F.plan[which]), "cufftCreate"));
			cufftResult r = cufftSetAutoAllocation(F.plan[which], 0);
			if (r == CUFFT_SUCCESS) {
				r = cufftMakePlan3d(F.plan[which], N, N, N, type, &F.work[which]);
			}
			if (r != CUFFT_SUCCESS) {
				cufftDestroy(F.plan[which]);
				return fft_check(c, r, "cufftMakePlan3d");
			}
			F.n[which] = N;
		}
		plans[which] = F.plan[which];
		// the work area is cuFFT's own business and outside the budget, as when plans allocated it
		void* w = nullptr;
		if (F.work[which]) {
			const cudaError_t e = cudaMallocFromPoolAsync(&w, F.work[which], c->pool, c->stream);
			if (e != cudaSuccess) {
				cudaGetLastError();
				return fail(c, CT_ERR_MEMORY, std::string("device allocation failed for a transform's work area: ") + cudaGetErrorString(e));
			}
			work.push_back(w);
			CT_TRY(fft_check(c, cufftSetWorkArea(plans[which], w), "cufftSetWorkArea"));
		}
		return fft_check(c, cufftSetStream(plans[which], c->stream), "cufftSetStream");
	}
};

// The particles' mass on the grid.  By tiles where the tiles hold enough particles for their copies
// to pay (DEP_MIN a tile on average) and the index arrays fit the budget, else particle by particle.
constexpr int64_t DEP_MIN = 16;

ct_status deposit(Ctx* c, FtScope& S, Box* b, int fold, int N, float* rho) {
	cudaStream_t st = c->stream;
	const int64_t np = b->n;
	const int nt = (N + DEP_TILE - 1) / DEP_TILE;
	const int64_t ntile = (int64_t) nt * nt * nt, max_units = np / DEP_UNIT + std::min(ntile, np) + 1;
	size_t tmp_bytes = 0;
	uint32_t *count = nullptr, *offset = nullptr, *rank = nullptr, *order = nullptr;
	uint4* units = nullptr;
	char* tmp = nullptr;
	bool tiles = np >= DEP_MIN * ntile;
	if (tiles) {
		CT_CUDA(c, cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, count, offset, (int) ntile, st));
		tiles = S.alloc(&count, ntile + 2, "tile counts") == CT_OK && S.alloc(&offset, ntile, "tile offsets") == CT_OK && S.alloc(&rank, np, "tile ranks") == CT_OK
				&& S.alloc(&order, np, "tile order") == CT_OK && S.alloc(&units, max_units, "deposit units") == CT_OK && S.alloc(&tmp, tmp_bytes, "scan") == CT_OK;
	}
	if (!tiles) {
		c->launches++;
		k_density<<<ft_grid(c, np), FT_TPB, 0, st>>>(np, b->x[0], b->x[1], b->x[2], fold, N, rho);
		return CT_OK;
	}
	unsigned int* ctr = (unsigned int*) (count + ntile);  // units made, units taken
	CT_CUDA(c, cudaMemsetAsync(count, 0, sizeof(uint32_t) * (ntile + 2), st));
	c->launches += 4;
	k_dep_count<<<ft_grid(c, np), FT_TPB, 0, st>>>(np, b->x[0], b->x[1], b->x[2], fold, N, nt, count, rank);
	CT_CUDA(c, cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, count, offset, (int) ntile, st));
	k_dep_order<<<ft_grid(c, np), FT_TPB, 0, st>>>(np, b->x[0], b->x[1], b->x[2], fold, N, nt, offset, rank, order);
	k_dep_units<<<(int) ((ntile + FT_TPB - 1) / FT_TPB), FT_TPB, 0, st>>>((int) ntile, count, offset, units, ctr);
	const int nblk = (int) std::min<int64_t>(max_units, (int64_t) c->nsm * 4);
	k_density_tiles<<<nblk, 32 * DEP_WARPS, 0, st>>>(b->x[0], b->x[1], b->x[2], fold, N, nt, order, units, ctr, ctr + 1, rho);
	return CT_OK;
}

// cosmos_growth_factor (src/cosmology.cpp:80-87): the linear growth factor's fitting formula.
double growth_factor(double omega_m, float a) {
	const double omega_l = 1.f - omega_m;
	const double a3 = a * (a * a);
	const double deninv = 1.f / (omega_m + a3 * omega_l);
	const double Om = omega_m * deninv;
	const double Ol = a3 * omega_l * deninv;
	return a * 2.5 * Om / (pow(Om, 4.f / 7.f) - Ol + (1.f + 0.5f * Om) * (1.f + 0.014285714f * Ol));
}

}  // namespace

void fourier_release(Ctx* c) {
	if (c->ft) {
		for (int i = 0; i < 2; i++) {
			if (c->ft->n[i]) {
				cufftDestroy(c->ft->plan[i]);
			}
		}
		delete c->ft;
		c->ft = nullptr;
	}
}

}  // namespace ct

using namespace ct;

extern "C" ct_status ct_initialize(ct_ctx* ctx, int box_id, const ct_ic_params* p, ct_ic_return* ret) {
	Ctx* c = (Ctx*) ctx;
	if (!c || box_id < 0 || box_id >= (int) c->boxes.size() || !c->boxes[box_id] || !p) {
		return fail(c, CT_ERR_ARG, "ct_initialize: bad arguments");
	}
	Box* b = c->boxes[box_id];
	const int N = p->nfour;
	if (N < 4 || N > IC_MAX_N || N % 2 != 0) {
		// (cuFFT's 3-D plans take 32-bit sizes)
		return fail(c, CT_ERR_ARG, "ct_initialize: nfour must be even, 4 .. 1024");
	}
	const int64_t n = (int64_t) N * N * N;
	if (b->nsub != 1 || b->n != n) {
		return fail(c, CT_ERR_ARG, "ct_initialize: the box must be a single box of nfour^3 particles");
	}
	if (!p->table_k || !p->table_p || p->ntable < 8 || !(p->box_size > 0.0) || !(p->hubble > 0.0) || !(p->sigma8 > 0.0) || !(p->omega_m > 0.0) ||
			!(p->z0 > -1.0)) {
		return fail(c, CT_ERR_ARG, "ct_initialize: bad parameters or power table");
	}
	// the table as read_power_spectrum takes it (initialize.cpp:870-898): k h / Mpc -> 1 / Mpc,
	// P (Mpc / h)^3 -> Mpc^3, log-uniform in k
	const float h = (float) p->hubble;
	std::vector<float> P(p->ntable);
	float kmax = 0.0, kmin = 3.4e38f;
	for (int i = 0; i < p->ntable; i++) {
		const float k = p->table_k[i] * h;
		P[i] = p->table_p[i] / (h * h * h);
		if (!(k > 0.f) || !(P[i] > 0.f)) {
			return fail(c, CT_ERR_ARG, "ct_initialize: power table entries must be positive");
		}
		kmax = std::max(kmax, k);
		kmin = std::min(kmin, k);
	}
	PowerTable tab;
	tab.P = P.data();
	tab.n = p->ntable;
	tab.logkmin = std::log(kmin);
	const float logkmax = std::log(kmax);
	tab.dlogk = (logkmax - tab.logkmin) / (p->ntable - 1);
	const float box = (float) p->box_size;
	// the interpolation needs two table points below and three above each |k| of the grid
	const double kf = 2.0 * M_PI / box, kN = kf * std::sqrt(3.0) * (N / 2);
	if (std::log(kf) < tab.logkmin + 1.0 * tab.dlogk || std::log(kN) > logkmax - 2.0 * tab.dlogk) {
		return fail(c, CT_ERR_ARG, "ct_initialize: the power table does not cover the grid's wavenumbers " + std::to_string(kf) + " .. " +
				std::to_string(kN) + " / Mpc");
	}
	// growth and velocity factors (initialize(), initialize.cpp:262-275)
	const float omega_m = (float) p->omega_m;
	const float a0 = 1.0 / (p->z0 + 1.0);
	const float D1 = growth_factor(omega_m, a0) / growth_factor(omega_m, 1.0);
	const float Om = omega_m / (omega_m + (a0 * a0 * a0) * (1.0 - omega_m));
	const float f1 = std::pow(Om, 5.f / 9.f);
	const float H0 = (float) p->H0;
	const float H = H0 * std::sqrt(omega_m / (a0 * a0 * a0) + 1.0 - omega_m);
	const float prefac1 = f1 * H * a0 * a0;
	const float D2 = -3.f * (D1 * D1) / 7.f;
	const float f2 = 2.f * std::pow(Om, 6.f / 11.f);
	const float prefac2 = f2 * H * a0 * a0;
	cudaSetDevice(c->device);
	cudaStream_t st = c->stream;
	FtScope S(c);
	const int NZ = N / 2 + 1;
	const int64_t ncx = (int64_t) N * N * NZ;
	float* dP = nullptr;
	float2* A = nullptr;
	cufftComplex* Y = nullptr;
	float* R = nullptr;
	AxisTables ax = {};
	double* G = nullptr;
	unsigned int* dmax = nullptr;  // six displacement maxima, then the table's factor
	CT_TRY(S.alloc(&dP, P.size(), "power table"));
	CT_TRY(S.alloc(&A, ncx, "mode amplitudes"));
	CT_TRY(S.alloc(&Y, ncx, "k-space field"));
	CT_TRY(S.alloc(&R, n, "real-space field"));
	CT_TRY(S.alloc(&G, n, "interpolation pass"));
	CT_TRY(S.alloc(&ax.filter, N, "axis tables"));
	CT_TRY(S.alloc(&ax.cell, N, "axis tables"));
	CT_TRY(S.alloc(&ax.weight, 6 * (size_t) N, "axis tables"));
	CT_TRY(S.alloc(&dmax, 7, "displacement maxima"));
	CT_TRY(S.plan(0, N, CUFFT_C2R));
	CT_CUDA(c, cudaMemcpyAsync(dP, P.data(), sizeof(float) * P.size(), cudaMemcpyHostToDevice, st));
	CT_CUDA(c, cudaMemsetAsync(dmax, 0, 6 * sizeof(unsigned int), st));
	PowerTable dtab = tab;
	dtab.P = dP;
	const float factor = std::pow(box, -1.5) * N * N * N;
	const double scale = 1.0 / ((double) N * N * N);  // cuFFT's inverse is unnormalised
	const float fscale = (float) scale;
	const double box_inv = 1.0 / box;
	const int gn = ft_grid(c, n), gx = ft_grid(c, ncx);
	c->launches += 5;
	k_sigma8<<<1, SIGMA_TPB, 0, st>>>(dtab, dP, logkmax, (float) p->hubble, p->sigma8, (float*) (dmax + 6));
	k_ic_axis<<<(N + 127) / 128, 128, 0, st>>>(N, box, ax);
	k_ic_lattice<<<gn, FT_TPB, 0, st>>>(N, b->x[0], b->x[1], b->x[2], b->v[0], b->v[1], b->v[2], b->rung);
	k_ic_uniforms<<<ft_grid(c, (int64_t) N * N), FT_TPB, 0, st>>>(N, A);
	k_ic_amplitude<<<gx, FT_TPB, 0, st>>>(N, box, factor, dtab, A);
	// interpolation at the lattice points and update of axis dim
	const size_t disp_smem = sizeof(double) * DISP_ROWS * N;
	// (the limit belongs to the kernel, whatever context launches it: always the largest grid's 64 KB, so
	// that calls on other grids from other threads never lower it)
	CT_CUDA(c, cudaFuncSetAttribute(k_ic_displace, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(double) * DISP_ROWS * IC_MAX_N));
	auto displace = [&](int dim, float D, float prefac, unsigned int* mx) {
		c->launches += 2;
		k_ic_sum_x<<<dim3((N * N + FT_TPB - 1) / FT_TPB, (N + DISP_X - 1) / DISP_X), FT_TPB, 0, st>>>(N, R, ax, G);
		k_ic_displace<<<dim3((N + DISP_ROWS - 1) / DISP_ROWS, N), FT_TPB, disp_smem, st>>>(N, G, ax, scale, D, prefac, box_inv, b->x[dim], b->v[dim], mx);
		const cudaError_t e = cudaGetLastError();
		return e == cudaSuccess ? CT_OK : cuda_check(c, e, "interpolation");
	};
	// the field of dim1, dim2 in real space
	auto field = [&](int dim1, int dim2, float* out) {
		c->launches++;
		k_ic_field<<<gx, FT_TPB, 0, st>>>(N, box, dim1, dim2, ax.filter, A, Y);
		return fft_check(c, cufftExecC2R(S.plans[0], Y, out), "cufftExecC2R");
	};
	for (int dim = 0; dim < 3; dim++) {
		CT_TRY(field(dim, 3, R));
		CT_TRY(displace(dim, D1, prefac1, dmax + dim));
	}
	if (p->twolpt) {
		float* R1 = nullptr;
		float* R2 = nullptr;
		cufftComplex* d2k = nullptr;
		CT_TRY(S.alloc(&R1, n, "2LPT field"));
		CT_TRY(S.alloc(&R2, n, "2LPT field"));
		CT_TRY(S.alloc(&d2k, ncx, "2LPT source transform"));
		CT_TRY(S.plan(1, N, CUFFT_R2C));
		CT_TRY(field(1, 1, R1));
		CT_TRY(field(2, 2, R2));
		CT_TRY(field(0, 0, R));
		c->launches += 2;
		k_twolpt_products<<<gn, FT_TPB, 0, st>>>(n, R, R1, R2, fscale);
		CT_TRY(field(0, 2, R));
		CT_TRY(field(1, 2, R1));
		k_twolpt_squares<<<gn, FT_TPB, 0, st>>>(n, R, R1, R2, fscale);
		CT_TRY(fft_check(c, cufftExecR2C(S.plans[1], R2, d2k), "cufftExecR2C"));
		for (int dim = 0; dim < 3; dim++) {
			c->launches++;
			k_ic_correction<<<gx, FT_TPB, 0, st>>>(d2k, Y, N, box, dim, ax.filter);
			CT_TRY(fft_check(c, cufftExecC2R(S.plans[0], Y, R), "cufftExecC2R"));
			CT_TRY(displace(dim, -D2, prefac2, dmax + 3 + dim));
		}
	}
	CT_CUDA(c, cudaGetLastError());
	unsigned int hm[7];
	CT_CUDA(c, cudaMemcpyAsync(hm, dmax, sizeof(hm), cudaMemcpyDeviceToHost, st));
	CT_CUDA(c, cudaStreamSynchronize(st));
	b->rung_begin = 0;
	b->rung_stack.clear();
	b->tree_valid = false;
	if (ret) {
		ret->D1 = D1;
		ret->D2 = D2;
		ret->prefac1 = prefac1;
		ret->prefac2 = prefac2;
		float norm;
		memcpy(&norm, hm + 6, 4);
		ret->norm = norm;
		for (int d = 0; d < 3; d++) {
			float a, q;
			memcpy(&a, hm + d, 4);
			memcpy(&q, hm + 3 + d, 4);
			ret->dxmax[d] = a;
			ret->dxmax2[d] = q;
		}
	}
	return CT_OK;
}

extern "C" ct_status ct_power_spectrum(ct_ctx* ctx, int box_id, int nfour, int fold, double box_size, int max_bins, float* k, float* P, float* Perr,
		int* nbins) {
	Ctx* c = (Ctx*) ctx;
	if (!c || box_id < 0 || box_id >= (int) c->boxes.size() || !c->boxes[box_id] || !nbins) {
		return fail(c, CT_ERR_ARG, "ct_power_spectrum: bad arguments");
	}
	Box* b = c->boxes[box_id];
	if (b->nsub != 1) {
		return fail(c, CT_ERR_ARG, "ct_power_spectrum: the spectrum is of a single box, not an ensemble");
	}
	const int N = nfour;
	if (N < 4 || N > 1024 || N % 2 != 0 || fold < 1 || !(box_size > 0.0)) {
		return fail(c, CT_ERR_ARG, "ct_power_spectrum: nfour must be even, 4 .. 1024; fold >= 1; box_size > 0");
	}
	// log-spaced bin edges in grid units from 1 to N / 2 (fft3d_power_spectrum, fft.cpp:172-214)
	std::vector<float> kb;
	const double Ns = std::max(N / 8.0, 64.0);
	const double lkmin = std::log(0.999999), lkmax = std::log(N / 2.0);
	const double dl = (lkmax - lkmin) / Ns;
	for (int i = 0; i <= Ns; i++) {
		kb.push_back(std::exp(lkmin + dl * i));
	}
	const int nb = (int) kb.size() - 1;
	*nbins = nb;
	if (!k || !P || max_bins < nb) {
		return k || P ? fail(c, CT_ERR_ARG, "ct_power_spectrum: room for " + std::to_string(nb) + " bins needed") : CT_OK;
	}
	cudaSetDevice(c->device);
	cudaStream_t st = c->stream;
	FtScope S(c);
	const int64_t ng = (int64_t) N * N * N, ncx = (int64_t) N * N * (N / 2 + 1);
	float* rho = nullptr;
	cufftComplex* Y = nullptr;
	float* dkb = nullptr;
	double* acc = nullptr;
	double* pmean = nullptr;
	CT_TRY(S.alloc(&rho, ng, "density grid"));
	CT_TRY(S.alloc(&Y, ncx, "density transform"));
	CT_TRY(S.alloc(&dkb, kb.size(), "k bins"));
	CT_TRY(S.alloc(&acc, 3 * nb, "bin sums"));
	CT_TRY(S.alloc(&pmean, nb, "bin means"));
	double* axis = nullptr;
	CT_TRY(S.alloc(&axis, 2 * (size_t) N, "axis factors"));
	CT_TRY(S.plan(1, N, CUFFT_R2C));
	CT_CUDA(c, cudaMemcpyAsync(dkb, kb.data(), sizeof(float) * kb.size(), cudaMemcpyHostToDevice, st));
	CT_CUDA(c, cudaMemsetAsync(acc, 0, sizeof(double) * 3 * nb, st));
	// the grid starts at -1 (fft3d_init(N, -1), power.cpp:35) and gains the particles' weights
	c->launches += 3;
	k_power_axis<<<(N + 127) / 128, 128, 0, st>>>(N, axis);
	k_fill<<<ft_grid(c, ng), FT_TPB, 0, st>>>(ng, rho, -1.0f);
	const int64_t np = b->n;
	if (np > 0) {
		CT_TRY(deposit(c, S, b, fold, N, rho));
	}
	CT_TRY(fft_check(c, cufftExecR2C(S.plans[1], rho, Y), "cufftExecR2C"));
	k_power_bins<<<ft_grid(c, ncx), FT_TPB, 0, st>>>(Y, N, dkb, nb, 1, axis, nullptr, acc);
	std::vector<double> h(3 * nb);
	CT_CUDA(c, cudaMemcpyAsync(h.data(), acc, sizeof(double) * 3 * nb, cudaMemcpyDeviceToHost, st));
	CT_CUDA(c, cudaStreamSynchronize(st));
	std::vector<double> mean(nb, 0.0);
	for (int i = 0; i < nb; i++) {
		const double cnt = h[nb + i];
		mean[i] = cnt > 0 ? h[i] / cnt : 0.0;
		P[i] = (float) mean[i];
		k[i] = (float) (std::sqrt((double) kb[i] * kb[i + 1]) * (2.0 * M_PI / box_size) * fold);
	}
	CT_CUDA(c, cudaMemcpyAsync(pmean, mean.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, st));
	CT_CUDA(c, cudaMemsetAsync(acc, 0, sizeof(double) * nb, st));
	c->launches++;
	k_power_bins<<<ft_grid(c, ncx), FT_TPB, 0, st>>>(Y, N, dkb, nb, 2, axis, pmean, acc);
	std::vector<double> dev(nb);
	CT_CUDA(c, cudaMemcpyAsync(dev.data(), acc, sizeof(double) * nb, cudaMemcpyDeviceToHost, st));
	CT_CUDA(c, cudaStreamSynchronize(st));
	for (int i = 0; i < nb; i++) {
		const double cnt = h[nb + i];
		float e = 0.f;
		if (cnt > 0) {
			if (cnt > 1) {
				e = (float) (std::sqrt(dev[i]) / std::sqrt(cnt - 1) / std::sqrt(cnt));
			} else {
				P[i] = 0.f;
			}
		}
		if (Perr) {
			Perr[i] = e;
		}
	}
	CT_CUDA(c, cudaGetLastError());
	return CT_OK;
}
