// The library's host code on the stand-in runtime (fake_cudart.cpp), one check per name on the command line. A check
// prints what it saw and the driver returns 0 when all hold. Test harness only.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <signal.h>
#include <sys/wait.h>
#include <time.h>
#include <unistd.h>

#include <cuda_runtime_api.h>

#include "../../include/palmtracer_b200.h"
#include "fake_cudart.h"

namespace ptb {
void ParallelCopy(void* dst, const void* src, size_t bytes);
}

namespace {

int failures = 0;

void Expect(bool ok, const char* what)
{
	std::printf("%s %s (%s)\n", ok ? "ok  " : "FAIL", what, PTB_LastError());
	failures += ok ? 0 : 1;
}

const double kParams[4] = {7, 1, 2, 0};

// A call that was refused (here: no device memory) is over: the next one does not fail for it.
void AfterAnError()
{
	const uint64_t H = 64, W = 80, Z = 3, n = 5;
	std::vector<uint16_t> stack(2 * H * W * Z, 100);
	std::vector<double> pos(n * 6, 1.0), rows(n * 18);
	auto fit = [&](uint64_t planes) { return Fitting(stack.data(), pos.data(), n, rows.data(), rows.size(), H, W, planes, 2, kParams); };
	Expect(fit(Z) == n * 18, "Fitting");
	const size_t had = fake::limit;
	fake::limit = 0;
	Expect(fit(2 * Z) == 0 && *PTB_LastError(), "Fitting without device memory");
	fake::limit = had;
	Expect(fit(Z) == n * 18, "Fitting afterwards");
}

// Null buffers are refused with the runtime's error by every entry point that hands host memory to a copy.
void NullBuffers()
{
	const uint64_t H = 64, W = 80, Z = 3, n = 5;
	std::vector<uint16_t> stack(H * W * Z, 100);
	std::vector<double> pos(n * 6, 1.0), rows(n * 18), plane(H * W * Z), points(n * 4, 1.0);
	std::vector<uint64_t> tracks(n * 2);
	Expect(Fitting(nullptr, pos.data(), n, rows.data(), rows.size(), H, W, Z, 2, kParams) == 0 && *PTB_LastError(), "Fitting of a null stack");
	Expect(Fitting(stack.data(), pos.data(), n, nullptr, rows.size(), H, W, Z, 2, kParams) == 0 && *PTB_LastError(), "Fitting into a null buffer");
	Wavelett(nullptr, plane.data(), H, W, Z, 2);
	Expect(*PTB_LastError(), "Wavelett of a null stack");
	Wavelett(stack.data(), nullptr, H, W, Z, 2);
	Expect(*PTB_LastError(), "Wavelett into a null buffer");
	Tracking(nullptr, tracks.data(), n, 5.0);
	Expect(*PTB_LastError(), "Tracking of a null table");
	Expect(Localization(nullptr, rows.data(), rows.size(), H, W, Z, 10.0, 0.0, 0, kParams) == 0 && *PTB_LastError(), "Localization of a null stack");
	Expect(Fitting(stack.data(), pos.data(), n, rows.data(), rows.size(), H, W, Z, 2, kParams) == n * 18, "Fitting afterwards");
}

// A child forked from a process whose copies have helper threads exits with its own code: it has none of the threads.
void ForkedChild()
{
	std::vector<char> from(8 << 20, 7), to(from.size());
	ptb::ParallelCopy(to.data(), from.data(), from.size());
	const timespec pause{0, 20000000};
	nanosleep(&pause, nullptr);  // the helpers have gone to sleep
	std::fflush(stdout);
	const pid_t child = fork();
	if (child == 0) { std::exit(7); }
	int status = 0, seen = 0;
	for (int i = 0; i < 500 && (seen = waitpid(child, &status, WNOHANG)) == 0; ++i) { nanosleep(&pause, nullptr); }
	if (seen == 0) { kill(child, SIGKILL); }
	Expect(to == from, "the copy");
	Expect(seen == child && WIFEXITED(status) && WEXITSTATUS(status) == 7, "exit of a forked child");
}

// Every entry point on a second device after the first: kernels are allowed their shared memory on each.
void SecondDevice()
{
	const uint64_t H = 64, W = 80, Z = 3, n = 5;
	std::vector<uint16_t> stack(H * W * Z, 100);
	std::vector<double> pos(n * 6, 1.0), rows(n * 18 * Z), plane(H * W * Z);
	for (int device = 0; device < fake::kDevices; ++device) {
		cudaSetDevice(device);
		const size_t before = fake::launches[device];
		Localization(stack.data(), rows.data(), rows.size(), H, W, Z, 10.0, 10.0, 2, kParams);
		Expect(!*PTB_LastError() && fake::launches[device] > before, device ? "Localization on device 1" : "Localization on device 0");
		const int mode = PTB_SetSegmentationMode(1);
		Localization(stack.data(), rows.data(), rows.size(), H, W, Z, 10.0, 10.0, 0, kParams);
		Expect(!*PTB_LastError(), device ? "strict segmentation on device 1" : "strict segmentation on device 0");
		PTB_SetSegmentationMode(mode);
		Wavelett(stack.data(), plane.data(), H, W, Z, 2);
		Expect(!*PTB_LastError(), device ? "Wavelett on device 1" : "Wavelett on device 0");
	}
	cudaSetDevice(0);
}

// Scratch that the library keeps between calls is given back when another of its allocations needs the memory.
void KeptScratch()
{
	const uint64_t H = 1000, W = 1000, n = 250000;
	const uint64_t small = 1, large = 30;  // planes: 2 and 60 MB
	std::vector<uint16_t> stack(H * W * large, 100);
	std::vector<double> pos(n * 6, 1.0), rows(n * 18);
	fake::limit = 100 << 20;
	auto fit = [&](uint64_t points, uint64_t planes) {
		return Fitting(stack.data(), pos.data(), points, rows.data(), rows.size(), H, W, planes, 2, kParams);
	};
	Expect(fit(n, small) == n * 18, "Fitting of many points");
	const size_t kept = fake::used[0];
	Expect(kept > (40u << 20), "scratch is kept");
	Expect(fit(5, large) == 5 * 18, "Fitting on a large stack");
	Expect(fake::used[0] < kept + (30u << 20), "scratch was given back for it");
	Expect(fit(5, large) == 5 * 18, "Fitting afterwards");
}

// Chunks of a nine-frame host stack under the budget and chunk slots of the environment.
void Chunks(uint64_t want)
{
	const uint64_t H = 256, W = 256, Z = 9;
	std::vector<uint16_t> stack(H * W * Z, 100);
	std::vector<double> rows((H * W / 5 + 1) * Z * 18);
	uint64_t counts[3] = {};
	Localization(stack.data(), rows.data(), rows.size(), H, W, Z, 10.0, 0.0, 0, kParams);
	PTB_GraphStats(counts, 3);
	Expect(!*PTB_LastError() && counts[0] + counts[1] + counts[2] == want, "chunks");
	std::printf("     %llu\n", static_cast<unsigned long long>(counts[0] + counts[1] + counts[2]));
}

}  // namespace

int main(int argc, char** argv)
{
	for (int i = 1; i < argc; ++i) {
		if (!std::strcmp(argv[i], "after")) { AfterAnError(); }
		else if (!std::strcmp(argv[i], "null")) { NullBuffers(); }
		else if (!std::strcmp(argv[i], "fork")) { ForkedChild(); }
		else if (!std::strcmp(argv[i], "devices")) { SecondDevice(); }
		else if (!std::strcmp(argv[i], "scratch")) { KeptScratch(); }
		else if (!std::strcmp(argv[i], "chunks") && i + 1 < argc) { Chunks(static_cast<uint64_t>(std::atoi(argv[++i]))); }
		else { return 2; }
	}
	return failures ? 1 : 0;
}
