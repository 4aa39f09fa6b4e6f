// imc_math64.cuh -- the double precision functions of a transport segment,
// with few FP64 operations: GB300 issues FP64 at 1/64 of the FP32 rate (an FP64
// instruction takes as long as 64 in FP32), so an FP64 history costs its FP64
// instructions and little else, and a function in 64-bit integers -- about a
// hundred instructions of the FP32 kind -- is a tenth of the same function in
// sixteen FP64 instructions.
//
//   neglog_k53   -log(k 2^-53) of a 53-bit uniform integer k: table-driven
//                reduction after Tang (ACM TOMS 16, 1990) in fixed point: the
//                mantissa m times a short table reciprocal c leaves r = m c - 1,
//                |r| <= 2^-8, exactly; -log v = e ln 2 + log c - log1p(r)
//   expm1_neg    exp(-y) - 1 for y >= 0.  Below 1, in fixed point, y = j/64 + r:
//                1 - exp(-y) = D_j + (1 - D_j) q with D_j = 1 - exp(-j/64) and
//                q = r g(r), g(r) = 1 - r/2 + r^2/6 - ...; for j = 0 y g(y), so
//                that small results keep their relative accuracy.  From 1 on in
//                FP64 (Tang, ACM TOMS 15, 1989)
//   attenuate    E exp(-y), a history's weight after a segment
//   div_r        a / b with r = 1/b at hand: one residual correction
//                (Markstein, IBM J. Res. Dev. 34, 1990)
//   pow_law      x^p of the opacity laws
//   rcp64, Sum128   a reciprocal and the sum of a cell's deposits, in integers
//   u53, one_minus_2u53   uniforms from their integers without a conversion
//
// Largest errors seen (tests/test_math64.py, against extended precision):
// 0.60 units in the last place for neglog_k53, 0.99 for expm1_neg; 1.94 units
// of 2^-53 for attenuate (tests/test_attenuate64.py); div_r
// equals the IEEE quotient wherever it was compared.  CUDA's log, exp and expm1 are good to 1 unit each.
// Table entries are the nearest integers to the stated expressions, computed
// with 400-bit arithmetic; the polynomials are the Taylor series.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef IMC_HD
#define IMC_HD __host__ __device__ __forceinline__
#endif

namespace imc {
namespace m64 {

// one row per 1/256 of the mantissa [1, 2): log(c) 2^62 and 512 c.  Mantissas
// from 1.5 up are halved, so the rows next to 1 on both sides have c = 1.
struct LogRow { long long l, c; };
#define IMC_LOG_ROWS \
    {0ll, 512ll}, \
    {-27101073204424016ll, 509ll}, \
    {-45257340823377788ll, 507ll}, \
    {-63485372532455475ll, 505ll}, \
    {-81785737890161276ll, 503ll}, \
    {-100159013262507360ll, 501ll}, \
    {-118605781931934706ll, 499ll}, \
    {-137126634208421142ll, 497ll}, \
    {-146415028120619150ll, 496ll}, \
    {-165048128291145683ll, 494ll}, \
    {-183756819338657074ll, 492ll}, \
    {-202541717077322504ll, 490ll}, \
    {-221403444877355111ll, 488ll}, \
    {-240342633789136771ll, 486ll}, \
    {-249841475496346632ll, 485ll}, \
    {-268898056407992778ll, 483ll}, \
    {-288033710495916050ll, 481ll}, \
    {-307249096706100262ll, 479ll}, \
    {-326544882255865699ll, 477ll}, \
    {-336223135584348451ll, 476ll}, \
    {-355640789612337420ll, 474ll}, \
    {-375140548129827607ll, 472ll}, \
    {-384921434125820140ll, 471ll}, \
    {-404545659561483878ll, 469ll}, \
    {-424253749463135451ll, 467ll}, \
    {-434139468186319879ll, 466ll}, \
    {-453974707445850668ll, 464ll}, \
    {-473895628350361066ll, 462ll}, \
    {-483888451368428307ll, 461ll}, \
    {-503939291730314290ll, 459ll}, \
    {-524077690624727309ll, 457ll}, \
    {-534179964146264212ll, 456ll}, \
    {-554451144118913011ll, 454ll}, \
    {-564620246405707431ll, 453ll}, \
    {-585025970045847207ll, 451ll}, \
    {-595262791160234820ll, 450ll}, \
    {-615804856387649007ll, 448ll}, \
    {-626110304292690010ll, 447ll}, \
    {-646790545308295307ll, 445ll}, \
    {-657165546351034578ll, 444ll}, \
    {-677985834619673835ll, 442ll}, \
    {-688431334030819940ll, 441ll}, \
    {-709393579297559686ll, 439ll}, \
    {-719910541708256709ll, 438ll}, \
    {-741016693049569391ll, 436ll}, \
    {-751606103025968078ll, 435ll}, \
    {-772858149937245866ll, 433ll}, \
    {-783521012533614846ll, 432ll}, \
    {-804920986054532345ll, 430ll}, \
    {-815658327385686451ll, 429ll}, \
    {-826420726712327630ll, 428ll}, \
    {-848021169098865055ll, 426ll}, \
    {-858859449101412339ll, 425ll}, \
    {-880612725371488827ll, 423ll}, \
    {-891527963646838293ll, 422ll}, \
    {-902469098122669217ll, 421ll}, \
    {-924429549231742015ll, 419ll}, \
    {-935449114853454346ll, 418ll}, \
    {-946495074669527710ll, 417ll}, \
    {-968666684771920437ll, 415ll}, \
    {-979792591298436692ll, 414ll}, \
    {-990945404517476615ll, 413ll}, \
    {-1002125254885922439ll, 412ll}, \
    {-1024566593663252558ll, 410ll}, \
    {-1035828347778509098ll, 409ll}, \
    {-1047117670474792364ll, 408ll}, \
    {-1069779563833499675ll, 406ll}, \
    {-1081152408113732256ll, 405ll}, \
    {-1092553368230430985ll, 404ll}, \
    {-1103982583543593542ll, 403ll}, \
    {-1126926342403200110ll, 401ll}, \
    {-1138441169904712895ll, 400ll}, \
    {-1149984820533913219ll, 399ll}, \
    {-1161557438949134583ll, 398ll}, \
    {-1173159170900473790ll, 397ll}, \
    {-1196450563936932904ll, 395ll}, \
    {-1208140522080887569ll, 394ll}, \
    {-1219860187901362382ll, 393ll}, \
    {-1231609712775298014ll, 392ll}, \
    {-1243389249239614210ll, 391ll}, \
    {-1255198951003091802ll, 390ll}, \
    {-1278909471194322142ll, 388ll}, \
    {-1290810603008029780ll, 387ll}, \
    {-1302742526917661759ll, 386ll}, \
    {-1314705402674956551ll, 385ll}, \
    {-1326699391278092920ll, 384ll}, \
    {-1338724654984690639ll, 383ll}, \
    {-1350781357324981151ll, 382ll}, \
    {-1374989738470859697ll, 380ll}, \
    {-1387141750820937955ll, 379ll}, \
    {-1399325868921263853ll, 378ll}, \
    {-1411542262868825059ll, 377ll}, \
    {-1423791104115966901ll, 376ll}, \
    {-1436072565484830305ll, 375ll}, \
    {-1448386821181982498ll, 374ll}, \
    {-1460734046813243573ll, 373ll}, \
    {-1473114419398712070ll, 372ll}, \
    {-1485528117387992781ll, 371ll}, \
    {-1497975320675630063ll, 370ll}, \
    {-1510456210616749994ll, 369ll}, \
    {-1522970970042914766ll, 368ll}, \
    {-1535519783278192789ll, 367ll}, \
    {-1548102836155448031ll, 366ll}, \
    {-1560720316032852194ll, 365ll}, \
    {-1573372411810623399ll, 364ll}, \
    {-1586059313947995113ll, 363ll}, \
    {-1598781214480419132ll, 362ll}, \
    {-1611538307037006498ll, 361ll}, \
    {-1624330786858210330ll, 360ll}, \
    {-1637158850813754575ll, 359ll}, \
    {-1650022697420812822ll, 358ll}, \
    {-1662922526862441371ll, 357ll}, \
    {-1675858541006270817ll, 356ll}, \
    {-1688830943423460540ll, 355ll}, \
    {-1701839939407920528ll, 354ll}, \
    {-1714885735995805087ll, 353ll}, \
    {-1727968541985283054ll, 352ll}, \
    {-1741088567956589237ll, 351ll}, \
    {-1754246026292361902ll, 350ll}, \
    {-1767441131198271204ll, 349ll}, \
    {-1780674098723943588ll, 348ll}, \
    {-1793945146784187257ll, 347ll}, \
    {-1807254495180523925ll, 346ll}, \
    {-1820602365623032176ll, 345ll}, \
    {-1833988981752507855ll, 344ll}, \
    {-1833988981752507855ll, 344ll}, \
    {-1847414569162947021ll, 343ll}, \
    {-1860879355424357132ll, 342ll}, \
    {1322193591194761711ll, 682ll}, \
    {1308649716501276066ll, 680ll}, \
    {1295065948157571726ll, 678ll}, \
    {1288259030289399357ll, 677ll}, \
    {1274614978862336174ll, 675ll}, \
    {1260930440576458077ll, 673ll}, \
    {1247205174438025750ll, 671ll}, \
    {1240327192524140639ll, 670ll}, \
    {1226540378015585561ll, 668ll}, \
    {1212712223671536416ll, 666ll}, \
    {1198842480830767967ll, 664ll}, \
    {1191891935402897159ll, 663ll}, \
    {1177959338647209446ll, 661ll}, \
    {1163984521836834621ll, 659ll}, \
    {1156981200797048007ll, 658ll}, \
    {1142942571939435847ll, 656ll}, \
    {1135907199074706049ll, 655ll}, \
    {1121804172736868012ll, 653ll}, \
    {1107657885514302838ll, 651ll}, \
    {1100568435972976629ll, 650ll}, \
    {1086356757488956149ll, 648ll}, \
    {1072101147935129264ll, 646ll}, \
    {1064956783968038650ll, 645ll}, \
    {1050634766188671844ll, 643ll}, \
    {1043457043310243364ll, 642ll}, \
    {1029067995697975510ll, 640ll}, \
    {1021856600923705940ll, 639ll}, \
    {1007399893102391509ll, 637ll}, \
    {1000154509022227221ll, 636ll}, \
    {985629501681226295ll, 634ll}, \
    {971058601665755500ll, 632ll}, \
    {963755851100267971ll, 631ll}, \
    {949115565730358898ll, 629ll}, \
    {941777957152272781ll, 628ll}, \
    {927067622451560875ll, 626ll}, \
    {919694821491238125ll, 625ll}, \
    {904913763906744091ll, 623ll}, \
    {897505431360282709ll, 622ll}, \
    {882652967577356360ll, 620ll}, \
    {875208759312948373ll, 619ll}, \
    {867752515136648555ll, 618ll}, \
    {852803762927731854ll, 616ll}, \
    {845311176359318437ll, 615ll}, \
    {830289384515648153ll, 613ll}, \
    {822760099547778631ll, 612ll}, \
    {807664550820620399ll, 610ll}, \
    {800098206189071320ll, 609ll}, \
    {792519427131828708ll, 608ll}, \
    {777324401792140010ll, 606ll}, \
    {769708073028073317ll, 605ll}, \
    {754437575570643203ll, 603ll}, \
    {746783323160507053ll, 602ll}, \
    {739116345470348965ll, 601ll}, \
    {723744044508635127ll, 599ll}, \
    {716038635834774757ll, 598ll}, \
    {700589086985402910ll, 596ll}, \
    {692844860113627059ll, 595ll}, \
    {685087606781766015ll, 594ll}, \
    {669533844927058342ll, 592ll}, \
    {661737247941683425ll, 591ll}, \
    {653927447568147903ll, 590ll}, \
    {638268057247272981ll, 588ll}, \
    {630418377022834815ll, 587ll}, \
    {622555312852915764ll, 586ll}, \
    {606788849569836211ll, 584ll}, \
    {598885358315037087ll, 583ll}, \
    {590968298828248853ll, 582ll}, \
    {583037624443118960ll, 581ll}, \
    {567135243104909236ll, 579ll}, \
    {559163441606601112ll, 578ll}, \
    {551177836116122077ll, 577ll}, \
    {543178378744478074ll, 576ll}, \
    {527137715551786840ll, 574ll}, \
    {519096412697589843ll, 573ll}, \
    {511041063892406469ll, 572ll}, \
    {494888031551711298ll, 570ll}, \
    {486790248929492881ll, 569ll}, \
    {478678222179227865ll, 568ll}, \
    {470551901101307142ll, 567ll}, \
    {462411235230280503ll, 566ll}, \
    {446086665906604093ll, 564ll}, \
    {437902660176841357ll, 563ll}, \
    {429704105095901985ll, 562ll}, \
    {421490948840588497ll, 561ll}, \
    {413263139310326503ll, 560ll}, \
    {396763350623858924ll, 558ll}, \
    {388491265861683732ll, 557ll}, \
    {380204316608565210ll, 556ll}, \
    {371902449346940932ll, 555ll}, \
    {363585610269703183ll, 554ll}, \
    {346906799979656229ll, 552ll}, \
    {338544719685978041ll, 551ll}, \
    {330167449410667966ll, 550ll}, \
    {321774933867122964ll, 549ll}, \
    {313367117466351674ll, 548ll}, \
    {304943944314765187ll, 547ll}, \
    {296505358211947596ll, 546ll}, \
    {279581720803300556ll, 544ll}, \
    {271096555542151863ll, 543ll}, \
    {262595749414529602ll, 542ll}, \
    {254079244651718042ll, 541ll}, \
    {245546983164360664ll, 540ll}, \
    {236998906540082847ll, 539ll}, \
    {228434956041092464ll, 538ll}, \
    {219855072601758172ll, 537ll}, \
    {211259196826165129ll, 536ll}, \
    {194019229016300178ll, 534ll}, \
    {185375016516461455ll, 533ll}, \
    {176714570744179701ll, 532ll}, \
    {168037830614650467ll, 531ll}, \
    {159344734697631736ll, 530ll}, \
    {150635221214834383ll, 529ll}, \
    {141909228037287941ll, 528ll}, \
    {133166692682681406ll, 527ll}, \
    {124407552312678784ll, 526ll}, \
    {115631743730209093ll, 525ll}, \
    {106839203376730539ll, 524ll}, \
    {98029867329468553ll, 523ll}, \
    {89203671298627407ll, 522ll}, \
    {80360550624575084ll, 521ll}, \
    {71500440275001118ll, 520ll}, \
    {62623274842047070ll, 519ll}, \
    {53728988539409335ll, 518ll}, \
    {44817515199413960ll, 517ll}, \
    {35888788270063140ll, 516ll}, \
    {26942740812053071ll, 515ll}, \
    {17979305495762817ll, 514ll}, \
    {0ll, 512ll}
// D_j = 1 - exp(-j/64), times 2^64
#define IMC_EXPM_ROWS \
    0ull, 285990258791865196ull, 567546649590711158ull, 844737913148277362ull, \
    1117631724489728397ull, 1386294709436213052ull, 1650792460871264869ull, 1911189554755015531ull, \
    2167549565890130884ull, 2419935083443318773ull, 2668407726226198211ull, 2913028157739260623ull, \
    3153856100982596093ull, 3390950353037000583ull, 3624368799419024035ull, 3854168428213464087ull, \
    4080405343986755773ull, 4303134781484654118ull, 4522411119117553846ull, 4738287892236738577ull, \
    4950817806204800870ull, 5160052749263424177ull, 5366043805201668333ull, 5568841265827851480ull, \
    5768494643248073388ull, 5965052681954377915ull, 6158563370725505876ull, 6349073954343143847ull, \
    6536630945126529359ull, 6721280134288228618ull, 6903066603113859213ull, 7082034733968487284ull, \
    7258228221132386316ull, 7431690081468803075ull, 7602462664926335147ull, 7770587664878484220ull, \
    7936106128302909442ull, 8099058465802866082ull, 8259484461473276195ull, 8417423282613840026ull, \
    8572913489291559591ull, 8725993043755009064ull, 8876699319702650433ull, 9025069111407457241ull, \
    9171138642700074143ull, 9314943575812705491ull, 9456519020085892127ull, 9595899540540302124ull, \
    9733119166315628212ull, 9868211398978652248ull, 10001209220702505067ull, 10132145102319118672ull, \
    10261051011246836720ull, 10387958419295118804ull, 10512898310348244006ull, 10635901187929889672ull, \
    10756997082650432255ull, 10876215559538788475ull, 10993585725260586803ull, 11109136235224431575ull, \
    11222895300577994696ull, 11334890695095642989ull, 11445149761959282784ull, 11553699420434077252ull
struct ExpRow { double hi, lo; };  // 2^(-j/64)
#define IMC_EXP2_ROWS \
    {0x1.0000000000000p+0, 0x0.0p+0}, \
    {0x1.fa7c1819e90d8p-1, 0x1.74853f3a5931ep-56}, \
    {0x1.f50765b6e4540p-1, 0x1.9d3e12dd8a18bp-55}, \
    {0x1.efa1bee615a27p-1, 0x1.dc7f486a4b6b0p-55}, \
    {0x1.ea4afa2a490dap-1, -0x1.e9c23179c2893p-55}, \
    {0x1.e502ee78b3ff6p-1, 0x1.39e8980a9cc8fp-56}, \
    {0x1.dfc97337b9b5fp-1, -0x1.1a5cd4f184b5cp-55}, \
    {0x1.da9e603db3285p-1, 0x1.c2300696db532p-55}, \
    {0x1.d5818dcfba487p-1, 0x1.2ed02d75b3707p-56}, \
    {0x1.d072d4a07897cp-1, -0x1.cbc3743797a9cp-55}, \
    {0x1.cb720dcef9069p-1, 0x1.503cbd1e949dbp-57}, \
    {0x1.c67f12e57d14bp-1, 0x1.2884dff483cadp-55}, \
    {0x1.c199bdd85529cp-1, 0x1.11065895048ddp-56}, \
    {0x1.bcc1e904bc1d2p-1, 0x1.23dd07a2d9e84p-56}, \
    {0x1.b7f76f2fb5e47p-1, -0x1.5584f7e54ac3bp-57}, \
    {0x1.b33a2b84f15fbp-1, -0x1.2805e3084d708p-58}, \
    {0x1.ae89f995ad3adp-1, 0x1.7a1cd345dcc81p-55}, \
    {0x1.a9e6b5579fdbfp-1, 0x1.0fac90ef7fd31p-55}, \
    {0x1.a5503b23e255dp-1, -0x1.d2f6edb8d41e1p-55}, \
    {0x1.a0c667b5de565p-1, -0x1.359495d1cd533p-55}, \
    {0x1.9c49182a3f090p-1, 0x1.c7c46b071f2bep-57}, \
    {0x1.97d829fde4e50p-1, -0x1.d185b7c1b85d1p-55}, \
    {0x1.93737b0cdc5e5p-1, -0x1.75fc781b57ebcp-58}, \
    {0x1.8f1ae99157736p-1, 0x1.5cc13a2e3976cp-56}, \
    {0x1.8ace5422aa0dbp-1, 0x1.6e9f156864b27p-55}, \
    {0x1.868d99b4492edp-1, -0x1.fc6f89bd4f6bap-55}, \
    {0x1.82589994cce13p-1, -0x1.d4c1dd41532d8p-55}, \
    {0x1.7e2f336cf4e62p-1, 0x1.05d02ba15797ep-57}, \
    {0x1.7a11473eb0187p-1, -0x1.41577ee04992fp-56}, \
    {0x1.75feb564267c9p-1, -0x1.0245957316dd3p-55}, \
    {0x1.71f75e8ec5f74p-1, -0x1.16e4786887a99p-56}, \
    {0x1.6dfb23c651a2fp-1, -0x1.bbe3a683c88abp-58}, \
    {0x1.6a09e667f3bcdp-1, -0x1.bdd3413b26456p-55}, \
    {0x1.6623882552225p-1, -0x1.bb60987591c34p-55}, \
    {0x1.6247eb03a5585p-1, -0x1.383c17e40b497p-55}, \
    {0x1.5e76f15ad2148p-1, 0x1.ba6f93080e65ep-55}, \
    {0x1.5ab07dd485429p-1, 0x1.6324c054647adp-55}, \
    {0x1.56f4736b527dap-1, 0x1.9bb2c011d93adp-55}, \
    {0x1.5342b569d4f82p-1, -0x1.07abe1db13cadp-56}, \
    {0x1.4f9b2769d2ca7p-1, -0x1.4b309d25957e3p-55}, \
    {0x1.4bfdad5362a27p-1, 0x1.d4397afec42e2p-57}, \
    {0x1.486a2b5c13cd0p-1, 0x1.3c1a3b69062f0p-57}, \
    {0x1.44e086061892dp-1, 0x1.89b7a04ef80d0p-60}, \
    {0x1.4160a21f72e2ap-1, -0x1.ef3691c309278p-59}, \
    {0x1.3dea64c123422p-1, 0x1.ada0911f09ebcp-56}, \
    {0x1.3a7db34e59ff7p-1, -0x1.5e436d661f5e3p-57}, \
    {0x1.371a7373aa9cbp-1, -0x1.63aeabf42eae2p-55}, \
    {0x1.33c08b26416ffp-1, 0x1.32721843659a6p-55}, \
    {0x1.306fe0a31b715p-1, 0x1.6f46ad23182e4p-56}, \
    {0x1.2d285a6e4030bp-1, 0x1.0024754db41d5p-55}, \
    {0x1.29e9df51fdee1p-1, 0x1.612e8afad1255p-56}, \
    {0x1.26b4565e27cddp-1, 0x1.2bd339940e9d9p-56}, \
    {0x1.2387a6e756238p-1, 0x1.9b07eb6c70573p-55}, \
    {0x1.2063b88628cd6p-1, 0x1.dc775814a8495p-56}, \
    {0x1.1d4873168b9aap-1, 0x1.e016e00a2643cp-55}, \
    {0x1.1a35beb6fcb75p-1, 0x1.e5b4c7b4968e4p-56}, \
    {0x1.172b83c7d517bp-1, -0x1.19041b9d78a76p-56}, \
    {0x1.1429aaea92de0p-1, -0x1.32fbf9af1369ep-55}, \
    {0x1.11301d0125b51p-1, -0x1.6c51039449b3ap-55}, \
    {0x1.0e3ec32d3d1a2p-1, 0x1.03a1727c57b53p-60}, \
    {0x1.0b5586cf9890fp-1, 0x1.8a62e4adc610bp-55}, \
    {0x1.0874518759bc8p-1, 0x1.186be4bb284ffp-58}, \
    {0x1.059b0d3158574p-1, 0x1.d73e2a475b465p-56}, \
    {0x1.02c9a3e778061p-1, -0x1.19083535b085dp-57}


static const LogRow h_log_rows[256] = {IMC_LOG_ROWS};
static const uint64_t h_expm_rows[64] = {IMC_EXPM_ROWS};
static const ExpRow h_exp2_rows[64] = {IMC_EXP2_ROWS};
#ifdef __CUDACC__
static __device__ const LogRow d_log_rows[256] = {IMC_LOG_ROWS};
static __device__ const uint64_t d_expm_rows[64] = {IMC_EXPM_ROWS};
static __device__ const ExpRow d_exp2_rows[64] = {IMC_EXP2_ROWS};
#endif
#undef IMC_LOG_ROWS
#undef IMC_EXPM_ROWS
#undef IMC_EXP2_ROWS

constexpr double kStepInv = 0x1.71547652b82fep+6;  // 64 / ln 2
constexpr double kStepHi = 0x1.62e42fefa3800p-7, kStepLo = 0x1.ef35793c76730p-51;  // ln 2 / 64: grid 2^-48, rest
IMC_HD uint64_t bits(double v) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u; memcpy(&u, &v, 8); return u;
#endif
}
IMC_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v; memcpy(&v, &u, 8); return v;
#endif
}
IMC_HD uint32_t hi32(double v) { return (uint32_t)(bits(v) >> 32); }

// k 2^-53 (k < 2^53) without an integer conversion: the low 52 bits as the
// fraction of a number in [1/2, 1), whose 1/2 goes unless bit 52 is set
IMC_HD double u53(uint64_t k) {
    const double w = from_bits(0x3FE0000000000000ull | (k & 0xFFFFFFFFFFFFFull));
    return w - ((k >> 52) ? 0.0 : 0.5);
}
// 1 - 2 u53(k): exact, one subtraction
IMC_HD double one_minus_2u53(uint64_t k) {
    const double w = from_bits(0x3FF0000000000000ull | (k & 0xFFFFFFFFFFFFFull));
    return ((k >> 52) ? 1.0 : 2.0) - w;
}

IMC_HD uint64_t mulhi_u(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
IMC_HD long long mulhi_s(long long a, long long b) {
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return (long long)(((__int128)a * b) >> 64);
#endif
}
IMC_HD int mulhi_s32(int a, int b) {
#ifdef __CUDA_ARCH__
    return __mulhi(a, b);
#else
    return (int)(((long long)a * b) >> 32);
#endif
}
IMC_HD uint32_t mulhi_u32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
IMC_HD int clz64(uint64_t v) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return __builtin_clzll(v);
#endif
}
// v 2^-scale rounded to the nearest double, v > 0
IMC_HD double fixed_to_double(uint64_t v, int scale) {
    const int z = clz64(v);
    const uint64_t n = v << z;  // the leading bit at 63
    const uint64_t m = (n >> 11) + ((n >> 10) & 1u);  // 53 bits, or 2^53
    // the leading bit and a carry add to the exponent
    return from_bits(((uint64_t)(1023 + 63 - scale - z - 1) << 52) + m);
}

// -log(k 2^-53), 0 < k < 2^53
IMC_HD double neglog_k53(uint64_t k) {
    const int z = clz64(k);  // 11..63
    const uint64_t f = k << (z - 11);  // mantissa in [1, 2), times 2^52
    const int row = (int)(f >> 44) & 255;
    const int up = row >> 7;  // mantissa at or above 1.5: halved
    const int e = z - 10 - up;  // k 2^-53 = m 2^-e
    if (e == 0 && row >= 254) {
        // within 2^-8 of 1, where the result is small and wants its relative
        // accuracy: the series in FP64
        const double r = -u53((1ull << 53) - k);
        const double r2 = r * r;
        double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
        p = fma(r, p, 1.0 / 5.0);
        p = fma(r, p, -1.0 / 4.0);
        p = fma(r, p, 1.0 / 3.0);
        p = fma(r, p, -1.0 / 2.0);
        return fma(-r2, p, -r);
    }
#ifdef __CUDA_ARCH__
    const longlong2 t = __ldg(reinterpret_cast<const longlong2 *>(&d_log_rows[row]));
    const long long tl = t.x, tc = t.y;
#else
    const long long tl = h_log_rows[row].l, tc = h_log_rows[row].c;
#endif
    // r 2^62, exact
    const long long R = (long long)(f * (uint64_t)tc - (1ull << (61 + up))) << (1 - up);
    // log1p(r) = r - r^2 P, P = 1/2 - r Q, Q = 1/3 - r (1/4 - r/5 + r^2/6 - r^3/7)
    const int rh = (int)(R >> 24);  // r 2^38
    int w = 715827883 - (mulhi_s32(rh, 613566757) >> 6);  // times 2^32 from here
    w = 858993459 - (mulhi_s32(rh, w) >> 6);
    w = 1073741824 - (mulhi_s32(rh, w) >> 6);
    const long long Q = 1537228672809129301ll - (((long long)rh * w) >> 8);  // times 2^62
    const long long P = (1ll << 61) - mulhi_s(R << 1, Q << 1);
    const uint64_t a = (uint64_t)(R < 0 ? -R : R);
    const uint64_t S = mulhi_u(a << 5, a << 5);  // r^2 2^70
    const long long l = R - (long long)(mulhi_u(S << 1, (uint64_t)P << 1) >> 8);
    const long long B = tl - l;  // log c - log1p(r), times 2^62
    const uint64_t v = e ? (uint64_t)(e * 199786072581291495ll + ((B + 8) >> 4)) : (uint64_t)B;  // ln 2 times 2^58
    return fixed_to_double(v, e ? 58 : 62);
}

// exp(-y) - 1 and *ex = exp(-y), 1 <= y <= 760, in FP64
IMC_HD double expm1_neg_fp64(double y, double *ex) {
    // n = floor(64 y / ln 2): the remainder r >= 0 keeps 2^(-n/64) - 1 and
    // exp(-r) - 1 of one sign, so their sum cancels nothing
#ifdef __CUDA_ARCH__
    const double big = __fma_rd(y, kStepInv, 0x1.8p52);
#else
    const double big = std::floor(y * kStepInv) + 0x1.8p52;
#endif
    const double n = big - 0x1.8p52;
    const uint32_t ni = (uint32_t)bits(big);
    double r = fma(-n, kStepHi, y);  // exact: y >= 1 and kStepHi are multiples of 2^-52, r is below 2^-6
    r = fma(-n, kStepLo, r);
    const double r2 = r * r;
    double q = fma(r, -1.0 / 5040.0, 1.0 / 720.0);
    q = fma(r, q, -1.0 / 120.0);
    q = fma(r, q, 1.0 / 24.0);
    q = fma(r, q, -1.0 / 6.0);
    q = fma(r, q, 1.0 / 2.0);
    const double p = fma(r2, q, -r);  // exp(-r) - 1
    const uint32_t j = ni & 63u;
#ifdef __CUDA_ARCH__
    const double2 t = __ldg(reinterpret_cast<const double2 *>(&d_exp2_rows[j]));
    const double th0 = t.x, tl0 = t.y;
#else
    const double th0 = h_exp2_rows[j].hi, tl0 = h_exp2_rows[j].lo;
#endif
    // times 2^-(n / 64), by the exponents, what is beyond 2^-512 at the end; the
    // low part of row 0 is 0
    const uint32_t k = ni >> 6, k1 = k < 512u ? k : 512u;
    const uint64_t sh = (uint64_t)k1 << 52;
    const double th = from_bits(bits(th0) - sh), tl = j ? from_bits(bits(tl0) - sh) : 0.0;
    double e = th + fma(th, p, tl);
    if (k > 512u) e *= from_bits((uint64_t)(1023u - (k - 512u)) << 52);
    *ex = e;
    return e - 1.0;
}

// exp(-y) - 1, 0 <= y < 1, in fixed point; where it is -1/2 or below, *ex is
// left with exp(-y), to 0.51 units in its last place
IMC_HD double expm1_neg_fixed(double y, double *ex) {
    const uint64_t yb = bits(y);
    const int e = (int)(yb >> 52);
    const int s = 1022 - e;
    uint64_t Y = ((yb & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11;  // y 2^64 once shifted
    Y = s < 64 ? Y >> s : 0ull;
    const int j = (int)(Y >> 58);
    const uint64_t r = Y & 0x3FFFFFFFFFFFFFFull;  // (y - j/64) 2^64
    // g = 1 - r (1/2 - r (1/6 - r (1/24 - r K))), K = 1/120 - r (1/720 - r (1/5040 - r/40320))
    const uint32_t rh = (uint32_t)(r >> 26);  // r 2^38
    uint32_t K = 54539267u - (mulhi_u32(rh, 6817408u) >> 6);  // times 2^38
    K = 381774871u - (mulhi_u32(rh, K) >> 6);
    K = 2290649225u - (mulhi_u32(rh, K) >> 6);
    const uint64_t J = 192153584101141163ull - (((uint64_t)rh * K) >> 14);  // times 2^62 from here
    const uint64_t I = 768614336404564651ull - mulhi_u(r, J);
    const uint64_t H = (1ull << 61) - mulhi_u(r, I);
    const uint64_t g = (1ull << 62) - mulhi_u(r, H);
    if (j == 0) return -(y * fixed_to_double(g, 62));
#ifdef __CUDA_ARCH__
    const uint64_t D = __ldg(reinterpret_cast<const unsigned long long *>(&d_expm_rows[j]));
#else
    const uint64_t D = h_expm_rows[j];
#endif
    const uint64_t q = mulhi_u(r, g << 2);  // (r g) 2^64; g = 1 only where r < 2^-60
    const uint64_t v = D + q - mulhi_u(D, q);
    if (v >> 63) *ex = fixed_to_double(0ull - v, 64);  // 1 - v 2^-64
    return -fixed_to_double(v, 64);
}

// exp(-y) - 1, y >= 0 (NaN gives NaN); from 760 on exp(-y) rounds to 0
IMC_HD double expm1_neg(double y) {
    double ex;
    if (hi32(y) < 0x3FF00000u) return expm1_neg_fixed(y, &ex);
    return y == y ? expm1_neg_fp64(y > 760.0 ? 760.0 : y, &ex) : y;
}

// E exp(-y), the weight E after a path of y mean free paths of absorption, and
// *em1 = exp(-y) - 1.  Up to ln 2 the weight is E + E em1.  Beyond, that sum
// would cancel, an error of em1 growing e^y times in the weight (50 units in
// the last place at the 1 % cut-off), and the weight is E exp(-y): one
// fused multiply-add either way.  A negative y (a path past the census time by a
// rounding, a negative opacity) and NaN take CUDA's expm1, whose sum with 1
// cancels nothing.  (FP64 heat waves of 60,000 and 200,000 histories 45.0 and 46.7
// ms, the 98 x 28 channel 10.36 ms; with E + E em1 throughout 46.1, 45.3 and
// 10.26; with CUDA's exp in the kernel for what lies beyond the table's range
// 48.4, 46.2 and 10.45.)
IMC_HD double attenuate(double E, double y, double *em1) {
    const uint32_t yh = hi32(y);
    double ex = 0.0, m;
    if (yh < 0x3FF00000u) m = expm1_neg_fixed(y, &ex);
    else if (yh <= 0x7FF00000u) m = expm1_neg_fp64(yh < 0x4087C000u ? y : 760.0, &ex);
    else m = expm1(-y);
    *em1 = m;
    const bool thick = (yh >= 0x3FF00000u && yh <= 0x7FF00000u) || bits(ex) != 0;
    return fma(E, thick ? ex : m, thick ? 0.0 : E);
}

// 1 / b: binary32's reciprocal and two Newton steps in 64-bit integers, then
// rounded (off by at most 0.52 units in the last place).  Beyond 2^+-1020, and
// for zeros, infinities and NaN, the division.
IMC_HD double rcp64(double b) {
    const uint64_t u = bits(b);
    const int ex = (int)(u >> 52) & 0x7FF;
    if ((unsigned)(ex - 3) > 2040u) return 1.0 / b;
    const uint64_t M = ((u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11;  // |b| 2^(1022 - ex), times 2^64
    const float f = (float)(uint32_t)(M >> 40);  // 24 bits of it
    float r0;
#ifdef __CUDA_ARCH__
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(f));
#else
    r0 = 1.0f / f;
#endif
    // the reciprocal, in (1, 2], times 2^61
    long long R = (long long)(uint64_t)(uint32_t)(r0 * 0x1p53f) << 32;
    for (int i = 0; i < 2; ++i) {
        const long long e = (1ll << 61) - (long long)mulhi_u(M, (uint64_t)R);
        R += mulhi_s(R, e << 3);
    }
    const double r = fixed_to_double((uint64_t)R, 61);
    return from_bits((bits(r) + ((uint64_t)(int64_t)(1022 - ex) << 52)) | (u & 0x8000000000000000ull));
}

// The deposits of one cell of a history as an exact 128-bit sum in units of the
// tally's 2^b, in place of a compensated pair: an addition in integers costs
// less than the pair's four in FP64, and the flush has nothing left to convert.
struct Sum128 {
    uint64_t lo;
    long long hi;
    IMC_HD void clear() { lo = 0; hi = 0; }
    IMC_HD void add128(uint64_t l, uint64_t h, bool neg) {
        if (neg) {
            h = ~h + (l == 0 ? 1u : 0u);
            l = ~l + 1u;
        }
        const uint64_t t = lo + l;
        hi += (long long)(h + (t < lo ? 1u : 0u));
        lo = t;
    }
    // man 2^sh, rounded half up; false where it does not fit below 2^94
    IMC_HD bool add(uint64_t man, int sh, bool neg) {
        if (man == 0) return true;
        if (sh >= 0) {
            if (64 - clz64(man) + sh > 94) return false;
            const uint64_t l = sh < 64 ? man << sh : 0ull;
            const uint64_t h = sh == 0 ? 0ull : sh < 64 ? man >> (64 - sh) : man << (sh - 64);
            add128(l, h, neg);
        } else if (sh >= -64) {
            const uint64_t half = (man >> (-sh - 1)) & 1u;
            add128((sh == -64 ? 0ull : man >> -sh) + half, 0ull, neg);
        }
        return true;
    }
    // v in units of 2^b; false for infinities, NaN and values out of range
    IMC_HD bool add(double v, int b) {
        const uint64_t u = bits(v);
        const int ex = (int)(u >> 52) & 0x7FF;
        if (ex == 0x7FF) return false;
        uint64_t man = u & 0xFFFFFFFFFFFFFull;
        if (ex) man |= 0x10000000000000ull;
        return add(man, (ex ? ex : 1) - 1075 - b, (u >> 63) != 0);
    }
    // the sum's sign and magnitude; false from 2^94 on, beyond a tally's words
    IMC_HD bool magnitude(bool &neg, uint64_t &l, uint64_t &h) const {
        neg = hi < 0;
        l = neg ? ~lo + 1u : lo;
        h = neg ? ~(uint64_t)hi + (lo == 0 ? 1u : 0u) : (uint64_t)hi;
        return (h >> 30) == 0;
    }
    // x y to 64 bits (both finite), negated
    IMC_HD bool add_minus_product(double x, double y, int b) {
        const uint64_t u = bits(x), v = bits(y);
        const int ex = (int)(u >> 52) & 0x7FF, ey = (int)(v >> 52) & 0x7FF;
        if (ex == 0 || ey == 0 || ex == 0x7FF || ey == 0x7FF) return add(-(x * y), b);
        const uint64_t m = (u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull, n = (v & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
        // (m 2^11)(n 2^11) = p 2^64
        return add(mulhi_u(m << 11, n << 11), ex - 1075 + ey - 1075 + 42 - b, ((u ^ v) >> 63) == 0);
    }
};

// x^p; the small whole powers of opacity laws by products, without pow's
// hundred instructions, each with the products' rounding errors carried along:
// 0.51 units in the last place (the products alone 1.3 and, for 1 / x^3, 2.4
// where CUDA's pow has 1.3).  Beyond 2^+-300, and for zeros, infinities and NaN,
// where errors would be lost or x^3 leaves the range, pow.  pow(x, 0) is 1
// for every x, NaN included.
IMC_HD double pow_law(double x, double p) {
    if (p == 0.0) return 1.0;
    if (p == 1.0) return x;
    const uint32_t e = hi32(x) >> 20 & 0x7FFu;
    if (e - (1023u - 300u) <= 600u) {
        if (p == -1.0) return 1.0 / x;
        const bool two = p == 2.0 || p == -2.0;
        if (two || p == 3.0 || p == -3.0) {
            // x^2 or x^3 as h + l
            double h = x * x, l = fma(x, x, -h);
            if (!two) {
                const double q = h * x;
                l = fma(l, x, fma(h, x, -q));
                h = q;
            }
            if (p > 0.0) return h + l;
            // 1 / (h + l): the quotient's residual, one Newton step
            const double r = 1.0 / h;
            return fma(fma(-l, r, fma(-h, r, 1.0)), r, r);
        }
    }
    return pow(x, p);
}

// a / b while nothing under- or overflows.  For rb = RN(1 / b) it is correctly
// rounded (Markstein).  rcp64's rb may be RN(1 / b)'s neighbour where 1 / b lies
// within 1/32 of a unit of a tie; the sum that is rounded here is then off by
// less than 2^-52 units in the last place, and the quotient its neighbour only
// where a / b is that close to a tie itself (none found in 4e6 draws, most of them
// next to one: tests/test_div64.py).
IMC_HD double div_r(double a, double b, double rb) {
    const double q = a * rb;
    return fma(fma(-q, b, a), rb, q);
}

}  // namespace m64
}  // namespace imc
