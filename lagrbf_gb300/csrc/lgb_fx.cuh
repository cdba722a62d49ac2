/*
 * lgb_fx.cuh -- 64-bit fixed-point arithmetic on the integer pipe in place of FP64.
 *
 * GB300 issues 2 FP64 multiply-adds per clock and SM, but 25-55 32 x 32 + 64-bit integer ones
 * (mad.wide; the operands' register banks decide), so three integer multiply-adds for a 56-bit product
 * are four to eight times an FP64 one.  Values are integers in units of 2^-56, multiplied as
 *     t = hi 2^28 + lo,  |lo| <= 2^27:   t t' 2^-56 = hi hi' + (hi lo' + lo hi') 2^-28  (+ lo lo' 2^-56)
 * where the last product, at most a quarter unit, is left out.  Every operation below is exact up to
 * about one unit, 2^-56, which is an eighth of the rounding unit 2^-53 of FP64 at one.
 * The functions compile for the host too, where the unit tests compare them with extended precision.
 */
#pragma once
#include <math.h>
#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD static inline
struct int2 { int x, y; };
static inline int2 make_int2(int x, int y) { int2 v = {x, y}; return v; }
#endif

#define FX_ONE 72057594037927936.0 /* 2^56 */
#define FX_ONE_I (1LL << 56)

/* a += x y */
FX_HD void fx_mad(long long &a, int x, int y)
{
#ifdef __CUDA_ARCH__
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a) : "r"(x), "r"(y));
#else
  a += (long long)x * y;
#endif
}
/* The value of the two sums of products. */
FX_HD long long fx_sum(long long hh, long long hl) { return hh + ((hl + (1LL << 27)) >> 28); }
FX_HD int2 fx_split(long long t)
{
  const int hi = (int)((t + (1LL << 27)) >> 28);
  return make_int2(hi, (int)(t - ((long long)hi << 28)));
}
FX_HD long long fx_mul(long long a, long long b)
{
  const int2 p = fx_split(a), q = fx_split(b);
  long long hh = 0, hl = 0;
  fx_mad(hh, p.x, q.x);
  fx_mad(hl, p.x, q.y);
  fx_mad(hl, p.y, q.x);
  return fx_sum(hh, hl);
}
FX_HD long long fx_sq(long long a)
{
  const int2 p = fx_split(a);
  long long hh = 0, hl = 0;
  fx_mad(hh, p.x, p.x);
  fx_mad(hl, p.x, p.y);
  return fx_sum(hh, hl + hl);
}
/* eps d rounded to the grid with the product's rounding error, |eps d| < 64. */
FX_HD long long fx_coord(double eps, double d)
{
  const double p = eps * d, e = fma(eps, d, -p);
#ifdef __CUDA_ARCH__
  return __double2ll_rn(p * FX_ONE) + __double2ll_rn(e * FX_ONE);
#else
  return llrint(p * FX_ONE) + llrint(e * FX_ONE);
#endif
}
FX_HD float fx_rsqrtf(float f)
{
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
  return y;
#else
  return 1.0f / sqrtf(f);
#endif
}
FX_HD int fx_f2i(float f)
{
#ifdef __CUDA_ARCH__
  return __float2int_rn(f);
#else
  return (int)lrintf(f);
#endif
}

/* -lim 2^32 <= d < lim 2^32 */
FX_HD bool fx_below(long long d, unsigned lim) { return (unsigned)((int)(d >> 32) + (int)lim) < 2 * lim; }

/* Squared distance of two points, or FX_ONE_I where it is 1 or more (|differences| < 2^62). */
template <int DIM> FX_HD long long fx_dist2(long long dx, long long dy, long long dz)
{
  /* |d| < 1 for every component, by the high words */
  bool in = fx_below(dx, 1u << 24) && fx_below(dy, 1u << 24);
  if (DIM == 3) in = in && fx_below(dz, 1u << 24);
  if (!in) return FX_ONE_I;
  const int2 x = fx_split(dx), y = fx_split(dy);
  long long hh = 0, hl = 0;
  fx_mad(hh, x.x, x.x);
  fx_mad(hl, x.x, x.y);
  fx_mad(hh, y.x, y.x);
  fx_mad(hl, y.x, y.y);
  if (DIM == 3) {
    const int2 z = fx_split(dz);
    fx_mad(hh, z.x, z.x);
    fx_mad(hl, z.x, z.y);
  }
  return fx_sum(hh, hl + hl);
}

/* Wendland C2 (1 - r)^4 (4 r + 1) of s = r^2 < 1.  The root: R0 = round(2^28 r) from the
   single-precision reciprocal root y of s, then two Newton corrections (s - r^2) / (2 r) with the
   residuals formed exactly in integers; the second residual is a few thousand units at most. */
FX_HD long long fx_phi_c2(long long s)
{
  const int sh = (int)(s >> 28), sl = (int)(s & 0xfffffff);
  const float f = fmaf((float)sh, 268435456.0f, (float)sl);
  const float y = fx_rsqrtf(fmaxf(f, 1.0f)); /* 2^-28 / r */
  const int R0 = fx_f2i(f * y);
  long long e = s;
  fx_mad(e, R0, -R0);
  const float yc = y * 134217728.0f; /* 2^27 */
  const int D0 = fx_f2i((float)(int)((e + 32) >> 6) * yc);
  const long long r1 = ((long long)R0 << 28) + ((long long)D0 << 6);
  const int2 q = fx_split(r1);
  long long e1 = s, hl = 0, ll = 0;
  fx_mad(e1, q.x, -q.x);
  fx_mad(hl, q.x, q.y);
  fx_mad(ll, q.y, q.y);
  e1 -= (hl + hl + (ll >> 28) + (1LL << 27)) >> 28;
  const int D1 = fx_f2i((float)(int)e1 * yc);
  long long u = FX_ONE_I - (r1 + D1);
  if (u < 0) u = 0;
  const long long u2 = fx_sq(u), u4 = fx_sq(u2);
  return fx_mul(u4, 5 * FX_ONE_I - 4 * u);
}

/* exp(-a) and exp(-b / 256) rounded to 2^-56 (computed in decimal arithmetic of 60 digits). */
#ifdef __CUDACC__
#define FX_TAB __device__ const
#else
#define FX_TAB const
#endif
static FX_TAB long long fx_exp1[41] = {
  72057594037927936LL, 26508507426831583LL, 9751934898471831LL, 3587536360790103LL, 1319780871589693LL,
  485520249509175LL, 178612918066855LL, 65708020484435LL, 24172629856296LL, 8892613563178LL,
  3271409708176LL, 1203484375286LL, 442737159439LL, 162873898800LL, 59917958872LL,
  22042585226LL, 8109013935LL, 2983139515LL, 1097435698LL, 403724031LL,
  148521771LL, 54638106LL, 20100236LL, 7394464LL, 2720271LL,
  1000732LL, 368149LL, 135434LL, 49824LL, 18329LL,
  6743LL, 2481LL, 913LL, 336LL, 124LL,
  45LL, 17LL, 6LL, 2LL, 1LL,
  0LL,
};
static FX_TAB long long fx_exp256[256] = {
  72057594037927936LL, 71776668101901790LL, 71496837392306472LL, 71218097639258780LL, 70940444589522213LL,
  70663874006442063LL, 70388381669880777LL, 70113963376153557LL, 69840614937964221LL, 69568332184341305LL,
  69297110960574424LL, 69026947128150872LL, 68757836564692478LL, 68489775163892696LL, 68222758835453955LL,
  67956783505025242LL, 67691845114139934LL, 67427939620153870LL, 67165062996183664LL, 66903211231045260LL,
  66642380329192729LL, 66382566310657296LL, 66123765210986618LL, 65865973081184282LL, 65609185987649558LL,
  65353400012117367LL, 65098611251598503LL, 64844815818320068LL, 64592009839666157LL, 64340189458118763LL,
  64089350831198916LL, 63839490131408053LL, 63590603546169612LL, 63342687277770860LL, 63095737543304942LL,
  62849750574613160LL, 62604722618227472LL, 62360649935313224LL, 62117528801612096LL, 61875355507385275LL,
  61634126357356849LL, 61393837670657422LL, 61154485780767946LL, 60916067035463778LL, 60678577796758949LL,
  60442014440850654LL, 60206373358063954LL, 59971650952796701LL, 59737843643464670LL, 59504947862446911LL,
  59272960056031308LL, 59041876684360358LL, 58811694221377152LL, 58582409154771577LL, 58354017985926716LL,
  58126517229865469LL, 57899903415197373LL, 57674173084065636LL, 57449322792094370LL, 57225349108336036LL,
  57002248615219092LL, 56780017908495846LL, 56558653597190508LL, 56338152303547452LL, 56118510662979671LL,
  55899725324017442LL, 55681792948257181LL, 55464710210310509LL, 55248473797753506LL, 55033080411076170LL,
  54818526763632069LL, 54604809581588192LL, 54391925603874991LL, 54179871582136626LL, 53968644280681394LL,
  53758240476432361LL, 53548656958878176LL, 53339890530024088LL, 53131938004343145LL, 52924796208727588LL,
  52718461982440433LL, 52512932177067240LL, 52308203656468076LL, 52104273296729658LL, 51901137986117685LL,
  51698794625029362LL, 51497240125946097LL, 51296471413386393LL, 51096485423858919LL, 50897279105815766LL,
  50698849419605882LL, 50501193337428690LL, 50304307843287891LL, 50108189932945441LL, 49912836613875708LL,
  49718244905219815LL, 49524411837740149LL, 49331334453775061LL, 49139009807193728LL, 48947434963351207LL,
  48756606999043647LL, 48566523002463692LL, 48377180073156046LL, 48188575321973216LL, 48000705871031429LL,
  47813568853666715LL, 47627161414391170LL, 47441480708849383LL, 47256523903775030LL, 47072288176947650LL,
  46888770717149575LL, 46705968724123034LL, 46523879408527431LL, 46342499991896773LL, 46161827706597285LL,
  45981859795785168LL, 45802593513364543LL, 45624026123945541LL, 45446154902802570LL, 45268977135832734LL,
  45092490119514423LL, 44916691160866059LL, 44741577577405003LL, 44567146697106625LL, 44393395858363533LL,
  44220322409944957LL, 44047923710956298LL, 43876197130798828LL, 43705140049129552LL, 43534749855821225LL,
  43365023950922522LL, 43195959744618369LL, 43027554657190424LL, 42859806118977713LL, 42692711570337421LL,
  42526268461605836LL, 42360474253059439LL, 42195326414876160LL, 42030822427096766LL, 41866959779586416LL,
  41703735971996357LL, 41541148513725773LL, 41379194923883778LL, 41217872731251565LL, 41057179474244696LL,
  40897112700875540LL, 40737669968715861LL, 40578848844859547LL, 40420646905885490LL, 40263061737820604LL,
  40106090936102992LL, 39949732105545257LL, 39793982860297951LL, 39638840823813172LL, 39484303628808301LL,
  39330368917229878LL, 39177034340217623LL, 39024297558068595LL, 38872156240201490LL, 38720608065121077LL,
  38569650720382781LL, 38419281902557392LL, 38269499317195919LL, 38120300678794581LL, 37971683710759932LL,
  37823646145374121LL, 37676185723760292LL, 37529300195848117LL, 37382987320339458LL, 37237244864674172LL,
  37092070604996042LL, 36947462326118847LL, 36803417821492556LL, 36659934893169663LL, 36517011351771647LL,
  36374645016455564LL, 36232833714880771LL, 36091575283175781LL, 35950867565905239LL, 35810708416037038LL,
  35671095694909555LL, 35532027272199020LL, 35393501025887007LL, 35255514842228056LL, 35118066615717420LL,
  34981154249058936LL, 34844775653133026LL, 34708928746964815LL, 34573611457692381LL, 34438821720535126LL,
  34304557478762266LL, 34170816683661454LL, 34037597294507513LL, 33904897278531300LL, 33772714610888687LL,
  33641047274629668LL, 33509893260667576LL, 33379250567748433LL, 33249117202420411LL, 33119491179003413LL,
  32990370519558776LL, 32861753253859088LL, 32733637419358127LL, 32606021061160913LL, 32478902231993879LL,
  32352278992175158LL, 32226149409584988LL, 32100511559636224LL, 31975363525244980LL, 31850703396801368LL,
  31726529272140366LL, 31602839256512788LL, 31479631462556378LL, 31356904010267006LL, 31234655026969984LL,
  31112882647291490LL, 30991585013130108LL, 30870760273628470LL, 30750406585145017LL, 30630522111225871LL,
  30511105022576804LL, 30392153497035335LL, 30273665719542918LL, 30155639882117250LL, 30038074183824685LL,
  29920966830752750LL, 29804316035982776LL, 29688120019562627LL, 29572377008479544LL, 29457085236633090LL,
  29342242944808200LL, 29227848380648342LL, 29113899798628769LL, 29000395460029894LL, 28887333632910756LL,
  28774712592082588LL, 28662530619082500LL, 28550786002147253LL, 28439477036187139LL, 28328602022759968LL,
  28218159270045144LL, 28108147092817859LL, 27998563812423371LL, 27889407756751394LL, 27780677260210581LL,
  27672370663703111LL, 27564486314599373LL, 27457022566712747LL, 27349977780274488LL, 27243350321908701LL,
  27137138564607423LL, 27031340887705793LL, 26925955676857322LL, 26820981324009262LL, 26716416227378071LL,
  26612258791424967LL,
};

#define FX_EXP_END (40LL << 56) /* exp(-40) < 2^-57 */

/* Squared distance of two points, or FX_EXP_END where a component is 6.5 or more (|differences| < 2^62). */
template <int DIM> FX_HD long long fx_dist2_wide(long long dx, long long dy, long long dz)
{
  bool in = fx_below(dx, 13u << 23) && fx_below(dy, 13u << 23);
  if (DIM == 3) in = in && fx_below(dz, 13u << 23);
  if (!in) return FX_EXP_END;
  const int2 x = fx_split(dx), y = fx_split(dy);
  long long hh = 0, hl = 0;
  fx_mad(hh, x.x, x.x);
  fx_mad(hl, x.x, x.y);
  fx_mad(hh, y.x, y.x);
  fx_mad(hl, y.x, y.y);
  if (DIM == 3) {
    const int2 z = fx_split(dz);
    fx_mad(hh, z.x, z.x);
    fx_mad(hl, z.x, z.y);
  }
  return fx_sum(hh, hl + hl);
}

/* exp(-s) for 0 <= s < 40: s = a + b / 256 + g; two table values and the Taylor polynomial of exp(-g) to
   fifth order (g < 2^-8: the sixth is below 2^-57), its terms from the fourth on in single precision. */
FX_HD long long fx_exp_neg(long long s)
{
  const int m = (int)(s >> 48);
  const long long g = s & ((1LL << 48) - 1), g2 = fx_sq(g);
  const long long p = fx_mul(g2, FX_ONE_I / 2 - fx_mul(g, FX_ONE_I / 6));
  const float gf = (float)(int)(g >> 24) * 2.3283064365386963e-10f, q = gf * gf; /* 2^-32 */
  const int t = fx_f2i(q * q * fmaf(gf, -600479950316066.0f, 3002399751580331.0f)); /* 2^56 (1/24 - g/120) */
  const long long e = FX_ONE_I - g + p + t;
#ifdef __CUDA_ARCH__
  return fx_mul(fx_mul(__ldg(&fx_exp1[m >> 8]), __ldg(&fx_exp256[m & 255])), e);
#else
  return fx_mul(fx_mul(fx_exp1[m >> 8], fx_exp256[m & 255]), e);
#endif
}
