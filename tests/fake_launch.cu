// The launches of fake_cudart.cpp: they run nothing.  A chosen launch fails, as one without resources does; the others do to
// the words and counters that live from call to call what their kernels do, and note where they do not find them at zero.
#include <stdlib.h>
#include <string.h>
#include <map>
#include <string>
#include "pbg_common.cuh"

static std::map<const void *, std::string> names;
static std::string launched;                        // the kernels since fake_arm, one after the other
static int launches, fail_at, behind_failure, unclean;
static bool failed, bad_ids;
extern "C" cudaError_t fake_refuse(cudaError_t);
extern "C" void fake_arm(int at, int ids) { fail_at = at; bad_ids = ids != 0; launches = behind_failure = unclean = 0; failed = false; launched.clear(); }
extern "C" const char *fake_launched() { return launched.c_str(); }
extern "C" int fake_launches() { return launches; }
extern "C" int fake_behind_failure() { return behind_failure; }
extern "C" int fake_unclean() { return unclean; }

template <class T> static T &arg(void **args, int i) { return *(T *)args[i]; }
template <class T> static void expect_zero(T &word) { if (word) ++unclean; }

static void run(const std::string &name, void **args) {
  auto is = [&](const char *part) { return name.find(part) != std::string::npos; };
  if (is("allnegs_rows_kernel")) {
    if (bad_ids) *arg<WaveBufs>(args, 1).errflag |= 1;
    unsigned *seam = arg<AllNegs>(args, 2).seam;
    if (seam) { expect_zero(*seam); *seam = 1; }
  } else if (is("allnegs_slab_kernel")) {
    if (arg<AllNegs>(args, 2).seam) *arg<AllNegs>(args, 2).seam = 0;
  } else if (is("narrow_tile_kernel") || is("tile_update_kernel") || is("hub_kernel")) {
    const WaveDims &d = arg<WaveDims>(args, 0);
    int *cnt = arg<int *>(args, 8), seam = is("hub_kernel") ? HUB_SEAM_HUB : HUB_SEAM_TILE;
    const bool operators = !is("narrow_tile_kernel") && is("ELi1EE");            // <VEC, RULE_REL>
    if (is("hub_kernel")) arg<int *>(args, 9)[0] = 0;
    else { expect_zero(cnt[0]); cnt[0] = 1; }
    if (operators) cnt[seam - HUB_REL] = 0;
    else if (d.dynamic && d.op != PBG_OP_NONE) { expect_zero(cnt[seam]); cnt[seam] = 1; }
  } else if (is("randperm_deal_kernel")) {
    unsigned *count = arg<unsigned *>(args, 5);
    expect_zero(count[0]);
    count[0] = 1;
    arg<unsigned *>(args, 6)[0] = 0;
  } else if (is("gather") && bad_ids) *arg<WaveBufs>(args, 2).errflag |= 1;
}

static cudaError_t launch(const void *func, void **args) {
  if (failed) ++behind_failure;
  if (++launches == fail_at) { failed = true; return fake_refuse(cudaErrorLaunchOutOfResources); }
  launched += names[func] + " ";
  run(names[func], args);
  return cudaSuccess;
}

extern "C" {
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t) { return launch(f, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *f, void **args) { return launch(f, args); }
const char *fake_kernel_name(const void *f) { return names[f].c_str(); }
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) { names[f] = name; }
}
