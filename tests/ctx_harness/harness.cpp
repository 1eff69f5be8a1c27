// CPU harness of the context (test infrastructure only): the real host code of
// luthe_b200/csrc/api.cu -- budget, key upload, the choice of launch forms,
// capture -- over a fake CUDA runtime.  Kernels do nothing; a launch notes its
// form and batch size, and which of the context's buffers it uses.
#include <stdio.h>
#include "../../luthe_b200/csrc/api.cu"

static std::string g_log;  // "form count;" per launch
static int g_fail_map, g_fail_ks_attr, g_fail_brx;

static void note(const char *form, size_t count) { g_log += std::string(form) + " " + std::to_string(count) + ";"; }

namespace luthe {
void build_twiddles(uint64_t *tw) { memset(tw, 0, 4096 * 8); }
bool ks_supported(uint32_t, uint32_t) { return true; }
bool pbs_supported(uint32_t) { return true; }
cudaError_t set_slab_wait_polls(unsigned long long) { return cudaSuccess; }
cudaError_t slab_wait_polls_address(const unsigned long long **a)
{
    static unsigned long long polls;
    *a = &polls;
    return cudaSuccess;
}
size_t br_smem_bytes(const BrConfig &, uint32_t) { return 100000; }
cudaError_t br_set_attributes(const BrConfig &, uint32_t) { return cudaSuccess; }
void br_cluster_limits(BrConfig *cfg)
{
    cfg->oct_max = 15;
    cfg->quad_max = 33;
}
cudaError_t launch_bsk_prepare(const uint64_t *d_std, uint64_t *d_slab, const uint64_t *, uint32_t n, cudaStream_t)
{
    memcpy(d_slab, d_std, n * SLAB_BYTES);
    return cudaSuccess;
}
cudaError_t launch_ntt_fwd(const uint64_t *, uint64_t *, const uint64_t *, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ntt_inv(const uint64_t *, uint64_t *, const uint64_t *, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ntt_mul(const uint64_t *, const uint64_t *, uint64_t *, const uint64_t *, size_t, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_lwe_op(int, const uint64_t *, const uint64_t *, uint64_t *, uint64_t, size_t, uint32_t, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_keyswitch(const uint64_t *, const uint32_t *, uint32_t *, uint32_t *, size_t B, uint32_t, uint32_t,
                             cudaStream_t, const uint32_t *, uint32_t, uint32_t, uint32_t, uint32_t *)
{
    note("ks_dp4a", B);
    return cudaSuccess;
}
size_t kstc_ksk_bytes(uint32_t n, uint32_t L) { return (size_t)(n / kstc::XT + 1) * 64 * L * 8192; }
size_t kstc_digit_bytes(size_t rows, uint32_t L) { return (rows + 127) / 128 * 64 * (size_t)L * 4096; }
cudaError_t launch_ks_layout(const uint32_t *, uint32_t *, uint32_t, uint32_t, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_kstc_layout(const uint32_t *, uint8_t *, uint32_t, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t kstc_set_attributes() { return g_fail_ks_attr; }
cudaError_t launch_keyswitch_tc(const KsTc &t, int, const uint64_t *, uint32_t *, uint32_t *, size_t B, uint32_t, uint32_t,
                                uint32_t, uint32_t, uint32_t, uint32_t *, cudaStream_t s)
{
    note("ks_tc", B);
    fake_use(t.dig, s);
    fake_use(t.part, s);
    return cudaSuccess;
}
cudaError_t launch_blind_rotate(const BrConfig &cfg, int, const uint32_t *, const uint64_t *, const uint32_t *, uint32_t,
                                const uint64_t *, const uint64_t *, uint64_t *, size_t B, uint32_t, uint32_t *, cudaStream_t,
                                const uint32_t *, uint32_t, uint32_t, uint32_t, cudaEvent_t, size_t *main_count)
{
    if (main_count) *main_count = B;
    note(B <= (size_t)cfg.oct_max ? "br_oct" : B <= (size_t)cfg.quad_max ? "br_quad" : "br", B);
    return cudaSuccess;
}
namespace brx {
void build_weights(uint8_t *w) { memset(w, 0, WEIGHT_BYTES); }
cudaError_t set_attributes() { return cudaSuccess; }
cudaError_t make_prod_map(Workspace &) { return g_fail_map; }
bool limited_stream(cudaStream_t s) { return fake_of(s)->limited; }
// the expanded key's first word: that of the key it was made from
cudaError_t launch_expand(const uint64_t *d_std, const Workspace &ws, uint32_t, cudaStream_t)
{
    memcpy(ws.bsk, d_std, 8);
    return cudaSuccess;
}
cudaError_t launch(const Workspace &ws, int, const uint32_t *, const uint64_t *, const uint32_t *, uint32_t, uint64_t *,
                   size_t B, uint32_t, uint32_t *, cudaStream_t s, uint32_t, uint32_t, uint32_t)
{
    if (g_fail_brx) return g_fail_brx;
    note(fake_of(s)->limited ? "brx_limited" : "brx", B);
    fake_use(ws.sync, s);
    return cudaSuccess;
}
}  // namespace brx
}  // namespace luthe

extern "C" {
fake_stream *harness_stream() { return new fake_stream; }
void harness_limit(fake_stream *s) { s->limited = true; }
void harness_fail_brx(int error) { g_fail_brx = error; }
void harness_begin_capture(fake_stream *s)  // the caller's
{
    s->capture = new fake_graph;
    s->caller = true;
}
void harness_fork(fake_stream *from, fake_stream *to)  // `to` joins the capture of `from`
{
    to->capture = from->capture;
    to->caller = from->caller;
    to->before = from->before;
}
fake_graph *harness_end_capture(fake_stream *s)
{
    fake_graph *g = s->capture;
    s->capture = nullptr;
    s->caller = false;
    return g;
}
void harness_replay(fake_graph *g, fake_stream *s) { cudaGraphLaunch(g, s); }
int harness_races() { return g_fake.races; }
void harness_reset()
{
    g_fake.ops = g_fake.races = 0;
    g_fake.uses.clear();
    g_fake.fail_malloc.clear();
    g_log.clear();
    g_fail_map = g_fail_ks_attr = g_fail_brx = 0;
}
int harness_log(char *buf, int cap)
{
    const int n = (int)g_log.size();
    snprintf(buf, cap, "%s", g_log.c_str());
    g_log.clear();
    return n;
}
void harness_fail_malloc(int nth, int error) { g_fake.fail_malloc[nth] = error; }
void harness_fail_optional(int map_error, int ks_error)
{
    g_fail_map = map_error;
    g_fail_ks_attr = ks_error;
}
// first words of the two device forms of the BSK (0: form not there)
void harness_bsk_words(luthe_ctx *c, uint64_t *slab, uint64_t *expanded)
{
    *slab = c->d_bsk ? c->d_bsk[0] : 0;
    *expanded = 0;
    if (c->ws.bsk) memcpy(expanded, c->ws.bsk, 8);
}
}
