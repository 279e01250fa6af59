// Which steps run as the one fused kernel of step_fused.cuh, and its launch from a plan.
#include "step_fused.cuh"

namespace b200dec_detail {

namespace {

bool all_kinds(const b200dec_plan* pl, int attn, int ffn) {
  for (int i = 0; i < pl->layers; ++i) {
    const b200dec_layer& l = pl->layer[i];
    const b200dec_weight* a[4] = {&l.qkv, &l.o, &l.cq, &l.co};
    for (const b200dec_weight* w : a)
      if (w->kind != attn || w->k != D_MODEL) return false;
    if (l.qkv.n != 3 * D_MODEL || l.o.n != D_MODEL || l.cq.n != D_MODEL || l.co.n != D_MODEL) return false;
    if (l.fc1.kind != ffn || l.fc2.kind != ffn || l.fc1.n != 4 * D_MODEL || l.fc1.k != D_MODEL || l.fc2.n != D_MODEL ||
        l.fc2.k != 4 * D_MODEL)
      return false;
    if (!l.qkv.ln_g || !l.qkv.ln_bias || !l.cq.ln_g || !l.cq.ln_bias || !l.fc1.ln_g || !l.fc1.ln_bias) return false;
  }
  return true;
}

// the kernel's weight mode for this plan and row count, or -1
int fused_mode(const b200dec_plan* pl, int rows) {
  if (rows < 1 || rows > F_MAX_ROWS || pl->layers > F_MAX_LAYERS || pl->attn_ring) return -1;
  if (!((pl->heads == 16 && pl->head_dim == 64) || (pl->heads == 8 && pl->head_dim == 128))) return -1;
  const b200dec_weight& h = pl->head;
  if (!h.ln_g || !h.ln_bias || h.k != D_MODEL || h.n != pl->vocab || pl->vocab % 16) return -1;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < FC)
    return -1;
  // 16-bit weights at 9 to 16 rows: twice the weight pieces, a quarter of fc2 waiting in the ring, and every CTA polls the
  // operand of all the rows (bf16 weights: as fp32). The sequence of kernels is ahead where its attention shares a row's
  // keys, from 128 (row, head) items on (step.cu), and for bf16 weights a little earlier. Sequence / fused, us a step, ragged
  // rows: 16 heads, fp16 248 / 261 at 9 rows, 268 / 292 at 16, bf16 284 / 292 and 309 / 350; 8 heads, fp16 309 / 290 at 15 rows,
  // 280 / 298 at 16, bf16 355 / 343 at 14, 323 / 352 at 16; with all rows at 350 positions bf16 387 / 384 at 14, 385 / 394 at 15,
  // over int8 caches 366 / 362 at 12, 365 / 376 at 13.
  const int kind = pl->layer[0].qkv.kind, items = rows * pl->heads;
  if (rows > 8 && ((kind == B200DEC_W_F16 && items >= 128) || (kind == B200DEC_W_BF16 && items >= (pl->kv_int8 ? 104 : 120))))
    return -1;
  const bool a16 = pl->a_kind == B200DEC_A_F16;
  // a vocabulary projection in the fragment layout is taken with the operand precision its mode has here
  const bool head8 = h.kind == B200DEC_W_INT8_UMMA || (h.kind == B200DEC_W_INT8 && pl->head_a_kind == B200DEC_A_F16);
  const bool head16 = h.kind == B200DEC_W_F16_UMMA || (h.kind == B200DEC_W_F16 && pl->head_a_kind == B200DEC_A_F16);
  if (a16 && head8 && all_kinds(pl, B200DEC_W_INT8, B200DEC_W_INT8)) return FM_INT8;
  if (a16 && head8 && all_kinds(pl, B200DEC_W_INT8, B200DEC_W_INT8_24)) return FM_INT8_24;
  if (a16 && head16 && all_kinds(pl, B200DEC_W_F16, B200DEC_W_F16)) return FM_F16;
  if (pl->a_kind == B200DEC_A_F32_SPLIT && h.kind == B200DEC_W_BF16 && pl->head_a_kind == B200DEC_A_F32_SPLIT &&
      all_kinds(pl, B200DEC_W_BF16, B200DEC_W_BF16))
    return FM_BF16;
  return -1;
}

FProj proj(const b200dec_weight& w) {
  return FProj{(const uint8_t*)w.w, (const uint32_t*)w.meta, w.scale, w.bias, w.ln_g, w.ln_bias};
}

}  // namespace

// Does this step run fused? The caller gave it a workspace, asks for the whole step, and no test switch of the other
// kernels is on.
bool fused_step_applies(const b200dec_plan* pl, int row0, int rows) {
  return row0 == 0 && rows >= 1 && rows <= F_MAX_ROWS && pl->fused_ws[rows - 1] && !pl->classes && !(pl->withhold & 3) &&
         fused_mode(pl, rows) >= 0;
}

int fused_step(const b200dec_plan* pl, int rows, void* stream) {
  const int mode = fused_mode(pl, rows);
  FArgs a{};
  a.layers = pl->layers, a.rows = rows, a.heads = pl->heads, a.act = pl->act, a.slots = pl->slots, a.seq = pl->seq;
  a.frames = pl->frames, a.vocab = pl->vocab, a.max_prompt = pl->max_prompt, a.out_cols = pl->out_cols, a.eos = pl->eos;
  a.max_pos = pl->max_pos, a.head_umma = is_umma_kind(pl->head.kind);
  a.wait_limit = pl->wait_limit > 0 ? (uint32_t)pl->wait_limit : 1u << 20, a.withhold = (pl->withhold >> 2) & 1;
  a.embed = (const __nv_bfloat16*)pl->embed, a.ptab = (const __nv_bfloat16*)pl->pos_table, a.ln0 = pl->emb_ln;
  a.head = proj(pl->head), a.gamma_f = pl->final_ln.w, a.eps_f = pl->final_ln.eps;
  a.scale_log2 = (1.0f / sqrtf((float)pl->head_dim)) * 1.4426950408889634f;
  a.active = pl->active, a.tok = pl->tok, a.pos = pl->pos, a.plen = pl->plen, a.limit = pl->limit, a.cross_len = pl->cross_len;
  a.finished = pl->finished, a.forced = pl->forced, a.out = pl->out, a.flags_host = pl->flags_host, a.status = pl->status;
  a.logits = pl->logits, a.argmax = pl->argmax, a.ws = (uint32_t*)pl->fused_ws[rows - 1];
  a.set_words = fused_set_words(pl->layers, rows, mode == FM_BF16);
  B200_REQUIRE(((uintptr_t)a.ws & 15) == 0, "fused step: the workspace must be 16-byte aligned");
  for (int i = 0; i < pl->layers; ++i) {
    const b200dec_layer& s = pl->layer[i];
    FLayer& d = a.layer[i];
    d.qkv = proj(s.qkv), d.o = proj(s.o), d.cq = proj(s.cq), d.co = proj(s.co), d.fc1 = proj(s.fc1), d.fc2 = proj(s.fc2);
    d.gamma[0] = s.ln1.w, d.gamma[1] = s.ln2.w, d.gamma[2] = s.ln3.w;
    d.eps[0] = s.ln1.eps, d.eps[1] = s.ln2.eps, d.eps[2] = s.ln3.eps;
    d.sk = s.self_k, d.sv = s.self_v, d.ck = (void*)s.cross_k, d.cv = (void*)s.cross_v;
    d.sks = s.self_ks, d.svs = s.self_vs, d.cks = s.cross_ks, d.cvs = s.cross_vs;
  }
  const bool q8 = pl->kv_int8 != 0;
  cudaStream_t st = (cudaStream_t)stream;
  switch (mode) {
    case FM_INT8: return launch_fused_int8(a, pl->head_dim, q8, st);
    case FM_INT8_24: return launch_fused_24(a, pl->head_dim, q8, st);
    case FM_F16: return launch_fused_f16(a, pl->head_dim, q8, st);
    case FM_BF16: return launch_fused_bf16(a, pl->head_dim, q8, st);
  }
  return fail(B200DEC_EINVAL, "fused step: no kernel for this plan");
}

}  // namespace b200dec_detail

using namespace b200dec_detail;

extern "C" int64_t b200dec_fused_words(const b200dec_plan* pl, int rows) {
  if (!pl || !pl->layer || pl->layers < 1) return 0;
  const int mode = fused_mode(pl, rows);
  if (mode < 0) return 0;
  return 16 + 2 * (int64_t)fused_set_words(pl->layers, rows, mode == FM_BF16);
}
